"""Performance cases: what a program asks of this library, through its public entry points.

Every case is one of these kinds of use:

  query      tgpu_see_noalloc on agents already in device memory: a neighbour count and
             displacement sum per agent, at the density of the 100,000-agent test workload
  frames     a viewer's loop: tay_run(state, 1), then the host reads the agents
  agents     the test model resident on the device for a run of steps, then read by id
  boxes      the same with box (non-point) agents
  groups     two groups that see each other, on a plane (dims 2), four see passes and two acts
  flock      boids: the host hands over its records, some steps run, the host reads them;
             one state of Gaussian flocks, or many uneven states in one batch
  dam        SPH dam break, all four passes, handed over and read like the flocks
  calibrate  the differentiable SPH rollout: forward, and the gradients of a loss on the
             final positions

Flocks tighten and dams collapse while they run, so these start every pass from the
records the program holds; the bouncing test and box agents are stationary and stay
resident.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

F32 = torch.float32


# ------------------------------------------------------------------ the cases


def listed():
    return [
        # one scene object's neighbour query from a program that may not allocate: latency
        {"name": "query_1k", "kind": "query", "n": 1000},
        # the most agents that entry point takes
        {"name": "query_65k", "kind": "query", "n": 65536},
        # a small simulation drawn on screen: one step and a read per frame
        {"name": "frames_2k", "kind": "frames", "n": 2048},
        # the reference's own test workload: 100,000 agents, r = 50 in a cube of side 1000
        {"name": "agents_100k", "kind": "agents", "n": 100000, "steps": 20},
        # the reference's non-point test agents (edges 1..50, r = 50), a ragged count
        {"name": "boxes_12k", "kind": "boxes", "n": 12345, "steps": 10},
        # the reference's combination test on a plane: two groups, see passes between them
        {"name": "groups_50k", "kind": "groups", "n": 30000, "m": 20001, "steps": 10},
        # boids on the host's side every step: push, one step, read back
        {"name": "flock_250k_edit", "kind": "flock", "n": 250007, "steps": 1, "states": 1},
        # the 1M-boid workload, ten steps on the device
        {"name": "flock_1m", "kind": "flock", "n": 1 << 20, "steps": 10, "states": 1},
        # an ensemble of uneven flocks (1,000 to 65,536 agents, radius 5 to 20) in one batch
        {"name": "flocks_32", "kind": "flock", "n": 32, "steps": 4, "states": 32},
        # a small fluid, as an interactive program has it
        {"name": "dam_2k", "kind": "dam", "nx": 16, "ny": 16, "nz": 8, "steps": 20},
        # the 524,288-particle dam break
        {"name": "dam_524k", "kind": "dam", "nx": 64, "ny": 128, "nz": 64, "steps": 5},
        # fitting viscosity and sound speed: rollout and gradients of several instances
        {"name": "calibrate_4x5k", "kind": "calibrate", "nx": 16, "ny": 20, "nz": 16, "instances": 4, "steps": 20,
         "every": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "frames", "agents", "boxes", "groups", "flock", "flock", "flocks", "dam", "dam",
                       "calibrate"])
    if kind == "query":
        return {"kind": kind, "n": _log(rng, 500, 65536)}
    if kind == "frames":
        return {"kind": kind, "n": _log(rng, 500, 20000)}
    if kind == "agents":
        return {"kind": kind, "n": _log(rng, 5000, 400000), "steps": rng.choice([10, 20])}
    if kind == "boxes":
        return {"kind": kind, "n": _log(rng, 2000, 20000), "steps": 10}
    if kind == "groups":
        return {"kind": kind, "n": _log(rng, 4000, 100000), "m": _log(rng, 4000, 100000), "steps": 10}
    if kind == "flock":
        return {"kind": kind, "n": _log(rng, 4000, 900000), "steps": rng.choice([1, 5, 10]), "states": 1}
    if kind == "flocks":
        s = _log(rng, 4, 32)
        return {"kind": "flock", "n": s, "steps": rng.choice([2, 4]), "states": s}
    if kind == "dam":
        return {"kind": kind, "nx": _log(rng, 10, 64), "ny": _log(rng, 10, 100), "nz": _log(rng, 8, 60),
                "steps": rng.choice([3, 5])}
    return {"kind": kind, "nx": _log(rng, 8, 16), "ny": _log(rng, 8, 20), "nz": _log(rng, 8, 16),
            "instances": rng.choice([1, 2, 3, 4]), "steps": rng.choice([12, 20]), "every": rng.choice([5, 10])}


# ------------------------------------------------------------------ inputs

SIDE, RADIUS = 1000.0, 50.0  # of the 100,000-agent test workload


def _side(n):
    """The cube side that gives n test agents the density of the 100,000-agent workload."""
    return SIDE * (n / 100000.0) ** (1.0 / 3.0)


def _plane_side(n):
    """The square side at which an agent has about 50 neighbours within RADIUS on a plane."""
    return math.sqrt(n * (2 * RADIUS) ** 2 / 50.0)


def _flocks(case, seed):
    """(points, radius) of every state of a flock case."""
    if case["states"] == 1:
        return [(W.boids_points(case["n"], seed=seed), 10.0)]
    # the batched workload's sizes and radii (agent counts log-uniform in [1000, 65536], radius
    # U[5, 20], 125 unit^3 per agent); positions and headings from the seed
    shape, out = W.Stream(4), []
    counts = np.exp(shape.uniform(case["states"], math.log(1000), math.log(65536))).round().astype(int)
    radii = shape.uniform(case["states"], 5.0, 20.0).astype(np.float32)
    for k, (n, r) in enumerate(zip(counts, radii)):
        rng = np.random.default_rng([seed, k])
        p, v = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
        p[:, :3] = rng.uniform(0.0, (125.0 * n) ** (1.0 / 3.0), (n, 3))
        d = rng.standard_normal((n, 3))
        v[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(1.0, 2.0, (n, 1))
        out.append((W.PointSet(p, v), float(r)))
    return out


TANK = ((0.0, 0.0, 0.0), (2.0, 1.5, 0.8))
DX, H = 0.01, 0.02


def _fluid(case, seed):
    """A block of fluid in motion: the dam's lattice with positions off it by up to 2% of its
    spacing and velocities of standard deviation 0.02 m/s."""
    s = W.sph_dam(case["nx"], case["ny"], case["nz"], DX, TANK[1])
    rng = np.random.default_rng(seed)
    p, v = s.points.p.copy(), s.points.v.copy()
    p[:, :3] += rng.uniform(-0.02 * DX, 0.02 * DX, (p.shape[0], 3)).astype(np.float32)
    v[:, :3] = (0.02 * rng.standard_normal((p.shape[0], 3))).astype(np.float32)
    return W.PointSet(p, v)


def _instances(case, seed):
    pars = [(0.05, 20.0), (0.08, 22.0), (0.12, 18.0), (0.06, 21.0)]
    return [(_fluid(case, 16 * seed + k), *pars[k], *TANK) for k in range(case["instances"])]


# ------------------------------------------------------------------ what the program keeps


class Pinned:
    """Page-locked records of the program's own (tgpu_host_alloc)."""

    def __init__(self, dtype, n):
        self.L = api.lib()
        self.bytes = n * dtype.itemsize
        self.ptr = self.L.tgpu_host_alloc(self.bytes)
        raw = (ctypes.c_char * self.bytes).from_address(self.ptr)
        self.rec = np.frombuffer(raw, dtype=dtype)
        self.words = torch.from_numpy(np.frombuffer(raw, dtype=np.float32).reshape(n, dtype.itemsize // 4))

    def __del__(self):
        self.L.tgpu_host_free(self.ptr)


def _by_id(words, id_word, spans, offset=None):
    """Fields of the records (word ranges `spans`), handed to torch on the GPU in id order."""
    g = words.cuda()
    ids = g[:, id_word].contiguous().view(torch.int32).long()
    if offset is not None:
        ids += offset
    out = []
    for a, b in spans:
        x = torch.empty((g.shape[0], b - a), dtype=F32, device=g.device)
        x[ids] = g[:, a:b]
        out.append(x)
    return out


class Resident:
    """A Tay state whose agents stay on the device between runs (the C API)."""

    def __init__(self, groups, passes, funcs, dtype, see, act, part, dims=3, is_point=True):
        self.st, self.dtype = api.State(), dtype
        self.gs, self.words, self.recs = [], [], []
        for rec in groups:
            g = self.st.add_group(dtype.itemsize, rec.shape[0], is_point)
            self.st.configure_space(g, api.TAY_GPU_Z_GRID, dims, part, 250)
            self.gs.append(g)
        for p in passes:
            if p[0] == "see":
                self.st.add_see(self.gs[p[1]], self.gs[p[2]], funcs[0], RADIUS, False, see)
            else:
                self.st.add_act(self.gs[p[1]], funcs[1], act)
        for g, rec in zip(self.gs, groups):
            self.st.commit(g, rec)
            raw = (ctypes.c_char * rec.nbytes).from_address(self.st.agent_ptr(g))
            self.words.append(torch.from_numpy(np.frombuffer(raw, np.float32).reshape(rec.shape[0], -1)))
            self.recs.append(np.frombuffer(raw, dtype))
        self.st.start()

    def fetch(self):
        for g in self.gs:
            self.st.agent_ptr(g)


COMBO = [("see", 0, 0), ("see", 0, 1), ("see", 1, 1), ("see", 1, 0), ("act", 0), ("act", 1)]
ALONE = [("see", 0, 0), ("act", 0)]


def _test_records(n, seed, side, flat=False):
    ps = W.basic_points(n, seed=seed, side=side)
    if flat:
        ps.p[:, 2] = 0.0
        ps.v[:, 2] = 0.0
    return M.records(M.TEST_RECORD, ps.p, ps.v)


class Episode:
    """Records the program keeps, a batch they are pushed to, and where results come back."""

    def __init__(self, setups, recs, dtype):
        n = [r.shape[0] for r in recs]
        total = sum(n)
        self.start, self.result = Pinned(dtype, total), Pinned(dtype, total)
        at = np.concatenate([[0], np.cumsum(n)])
        for k, r in enumerate(recs):
            self.start.rec[at[k]:at[k + 1]] = r
        self.batch = api.Batch([(s, self.start.rec[at[k]:at[k + 1]]) for k, s in enumerate(setups)])
        self.to = [self.result.ptr + int(at[k]) * dtype.itemsize for k in range(len(n))]
        for k, p in enumerate(self.to):
            self.batch.write_through(k, p)
        self.offset = torch.repeat_interleave(torch.from_numpy(at[:-1]), torch.tensor(n)).cuda() if len(n) > 1 else None

    def __del__(self):
        self.batch.close()

    def run(self, steps):
        B = self.batch
        B.push()
        _, pairs = B.run(steps)
        for k, p in enumerate(self.to):
            B._check(B.L.tgpu_batch_fetch(B.ptr, k, p), "tgpu_batch_fetch")
        return pairs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "query":
        n = case["n"]
        pos = torch.from_numpy(W.basic_points(n, seed=seed, side=_side(n)).p).cuda()
        r = (ctypes.c_float * 4)(RADIUS, RADIUS, RADIUS, 0.0)
        return {"case": case, "pos": pos, "r": r, "L": api.lib()}
    if kind in ("frames", "agents"):
        n = case["n"]
        see, act = M.test_contexts(RADIUS, 0.0, _side(n))
        return {"case": case, "R": Resident([_test_records(n, seed, _side(n))], ALONE, ("agent_see", "agent_act"),
                                            M.TEST_RECORD, see, act, RADIUS)}
    if kind == "boxes":
        b = W.box_agents(case["n"], seed=seed)
        see, act = M.test_contexts(RADIUS)
        return {"case": case, "R": Resident([M.box_records(b.lo, b.hi, b.v)], ALONE,
                                            ("box_agent_see", "box_agent_act"), M.BOX_RECORD, see, act, RADIUS,
                                            is_point=False)}
    if kind == "groups":
        side = _plane_side(case["n"] + case["m"])
        see, act = M.test_contexts(RADIUS, 0.0, side)
        recs = [_test_records(case["n"], 2 * seed, side, True), _test_records(case["m"], 2 * seed + 1, side, True)]
        return {"case": case, "R": Resident(recs, COMBO, ("agent_see", "agent_act"), M.TEST_RECORD, see, act, RADIUS,
                                            dims=2)}
    if kind == "flock":
        fl = _flocks(case, seed)
        return {"case": case, "E": Episode([M.boids_setup(r=r, part=r) for _, r in fl],
                                           [M.records(M.BOIDS_RECORD, ps.p, ps.v) for ps, _ in fl], M.BOIDS_RECORD)}
    if kind == "dam":
        ps = _fluid(case, seed)
        return {"case": case, "E": Episode([M.sph_setup(h=H, dx=DX, tank_min=TANK[0], tank_max=TANK[1])],
                                           [M.records(M.SPH_RECORD, ps.p, ps.v)], M.SPH_RECORD)}
    from tay_gb300.adjoint import SphRollout

    roll = SphRollout(_instances(case, seed), case["steps"], checkpoint_every=case["every"], h=H, dx=DX)
    rng = np.random.default_rng(seed + 99)
    x0 = np.concatenate([ps.p[:, :3] for ps, *_ in roll.instances]).astype(np.float64)
    return {"case": case, "roll": roll, "target": x0 + 1e-3 * rng.standard_normal(x0.shape)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "query":
        n = case["n"]
        out = torch.empty((n, 4), dtype=F32, device="cuda")
        rc = state["L"].tgpu_see_noalloc(state["pos"].data_ptr(), n, state["r"], state["r"], out.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise api.TayError(state["L"].tgpu_noalloc_last_error().decode())
        return {"sum": out[:, :3], "count": out[:, 3].view(torch.int32)}
    if kind == "frames":
        R = state["R"]
        R.st.run(1)
        R.fetch()
        rec = R.recs[0]
        p, f = np.empty((case["n"], 4), np.float32), np.empty((case["n"], 4), np.float32)
        p[rec["id"]] = rec["p"]
        f[rec["id"]] = rec["f_buffer"]
        return {"p": p, "f": f, "pairs": R.st.pairs()}
    if kind in ("agents", "groups"):
        R = state["R"]
        R.st.run(case["steps"])
        R.fetch()
        out = [_by_id(w, 19, [(2, 5), (6, 9), (15, 18)]) for w in R.words]
        return {"p": [o[0] for o in out], "v": [o[1] for o in out], "f": [o[2] for o in out], "pairs": R.st.pairs()}
    if kind == "boxes":
        R = state["R"]
        R.st.run(case["steps"])
        R.fetch()
        lo, hi, v, f = _by_id(R.words[0], 23, [(2, 5), (6, 9), (10, 13), (19, 22)])
        return {"min": lo, "max": hi, "v": v, "f": f, "pairs": R.st.pairs()}
    if kind == "flock":
        E = state["E"]
        pairs = E.run(case["steps"])
        p, v = _by_id(E.result.words, 24, [(2, 5), (6, 9)], E.offset)
        return {"p": p, "v": v, "pairs": pairs}
    if kind == "dam":
        E = state["E"]
        E.run(case["steps"])
        p, v, P = _by_id(E.result.words, 16, [(2, 5), (6, 9), (15, 16)])
        return {"p": p, "v": v, "P": P}
    roll = state["roll"]
    x, v = roll.forward()
    per = case["nx"] * case["ny"] * case["nz"]
    dx0, dv0, dp = roll.backward(2.0 * (x.astype(np.float64) - state["target"]) / per)
    return {"x": x, "v": v, "dx0": dx0, "dv0": dv0, "dparams": dp}


# ------------------------------------------------------------------ the work of a pass


def work(case):
    """Bytes and operations that a pass cannot do without: per step every agent's state read
    once and written once, and the pair terms of the neighbours that count (box-test passes,
    or those inside the radius); per pass the records over the host link and back."""
    kind = case["kind"]
    if kind == "query":
        n = case["n"]
        return {"bytes": 32 * n, "flops": n * 100.0 * 6}
    if kind in ("frames", "agents"):
        n, k = case["n"], case.get("steps", 1)
        return {"bytes": (2 * 64 * k + 80) * n, "flops": n * 100.0 * 6 * k}
    if kind == "boxes":
        n, k = case["n"], case["steps"]
        mates = n * (2 * RADIUS + 51.0) ** 3 / SIDE ** 3
        return {"bytes": (2 * 80 * k + 96) * n, "flops": n * mates * 6 * k}
    if kind == "groups":
        n, k = case["n"] + case["m"], case["steps"]
        return {"bytes": (2 * 64 * k + 80) * n, "flops": n * 50.0 * 6 * k}
    if kind == "flock":
        k = case["steps"]
        if case["states"] == 1:
            n = case["n"]
            # pairs within r = 10 of each other inside Gaussian clusters of sigma 40
            mates = n / 64.0 * (4.0 / 3.0 * math.pi * 1000.0) / (4.0 * math.pi * 1600.0) ** 1.5
        else:
            n = int(case["states"] * 64536.0 / math.log(65.536))
            mates = 4.0 / 3.0 * math.pi * (20.0 ** 4 - 5.0 ** 4) / 60.0 / 125.0
        return {"bytes": (2 * 36 * k + 2 * 104) * n, "flops": n * mates * 14 * k}
    per = case["nx"] * case["ny"] * case["nz"]
    if kind == "dam":
        return {"bytes": (2 * 36 * case["steps"] + 2 * 72) * per, "flops": per * 240.0 * 45 * case["steps"]}
    n = per * case["instances"]
    return {"bytes": (4 * 36 * case["steps"] + 6 * 16) * n, "flops": n * 240.0 * 150 * case["steps"]}


# ------------------------------------------------------------------ the same in 64 bits


def _candidates(seer_lo, seer_hi, seen, reach, most=1 << 25):
    """Index pairs (i, j) in chunks: every j whose point may lie in seer i's interval, from a
    sort of the seen points into cells of edge `reach` (no smaller than any interval's part
    on either side of its lower corner's cell)."""
    dev, dims = seen.device, seen.shape[1]
    mn = torch.minimum(seen.min(0).values, seer_lo.min(0).values)
    cell = torch.floor((seen - mn) / reach).long()
    lo = torch.floor((seer_lo - mn) / reach).long()
    hi = torch.floor((seer_hi - mn) / reach).long()
    nx = int(max(cell[:, 0].max(), hi[:, 0].max())) + 2
    ny = int(max(cell[:, 1].max(), hi[:, 1].max())) + 2 if dims > 1 else 1
    row = torch.zeros_like(cell[:, 0])
    if dims > 1:
        row = row + cell[:, 1]
    if dims > 2:
        row = row + cell[:, 2] * ny
    key, order = torch.sort(row * nx + cell[:, 0])
    span = [int((hi[:, a] - lo[:, a]).max()) + 1 for a in range(dims)]
    for dz in range(span[2] if dims > 2 else 1):
        for dy in range(span[1] if dims > 1 else 1):
            y = lo[:, 1] + dy if dims > 1 else torch.zeros_like(lo[:, 0])
            z = lo[:, 2] + dz if dims > 2 else torch.zeros_like(y)
            r = y + z * ny
            ok = (y <= hi[:, 1] if dims > 1 else True) & (z <= hi[:, 2] if dims > 2 else y == y)
            a = torch.searchsorted(key, r * nx + lo[:, 0])
            b = torch.searchsorted(key, r * nx + hi[:, 0], right=True)
            cnt = torch.where(ok, b - a, torch.zeros_like(a))
            ends = torch.cumsum(cnt, 0)
            total, first = int(ends[-1]), 0
            while first < cnt.shape[0]:
                base = int(ends[first - 1]) if first else 0
                last = int(torch.searchsorted(ends, torch.tensor(base + most, device=dev)))
                last = max(first + 1, min(last, cnt.shape[0]))
                c = cnt[first:last]
                if int(c.sum()):
                    i = torch.repeat_interleave(torch.arange(first, last, device=dev), c)
                    j = torch.arange(i.shape[0], device=dev) - (ends[i] - cnt[i] - base) + a[i]
                    yield i, order[j]
                first = last
                if base >= total:
                    break


def _near(p, q, r, same):
    """(i, j) with every |p_i - q_j| <= r on each axis, i != j when the sets are the same."""
    for i, j in _candidates(p - r, p + r, q, r):
        ok = ((p[i] - q[j]).abs() <= r).all(1)
        if same:
            ok &= i != j
        yield i[ok], j[ok]


def _t64(x, cols=3):
    return torch.from_numpy(np.ascontiguousarray(x[:, :cols])).cuda().double()


def _displacements(p, q, r, same):
    s = torch.zeros_like(p)
    n = torch.zeros(p.shape[0], dtype=torch.float64, device=p.device)
    for i, j in _near(p, q, r, same):
        s.index_add_(0, i, q[j] - p[i])
        n += torch.bincount(i, minlength=p.shape[0])
    return s, n


def _bounce(p, v, side, dims):
    p = p + v
    for a in range(dims):
        low, high = p[:, a] < 0, p[:, a] > side
        v[:, a] = torch.where(low | high, -v[:, a], v[:, a])
        p[:, a] = p[:, a].clamp(0, side)
    return p, v


def _agents64(recs, side, steps, dims):
    """The test model's steps in 64 bits over one group, or two that also see each other."""
    p, v = [_t64(r["p"], dims) for r in recs], [_t64(r["v"], dims) for r in recs]
    f = [torch.zeros_like(x) for x in p]
    for _ in range(steps):
        for a in range(len(p)):
            s, n = 0, 0
            for b in range(len(p)):
                ds, dn = _displacements(p[a], p[b], RADIUS, a == b)
                s, n = s + ds, n + dn
            f[a] += s / n.clamp(min=1)[:, None]
        for a in range(len(p)):
            p[a], v[a] = _bounce(p[a], v[a], side, dims)
    pad = lambda x: torch.cat([x, x.new_zeros((x.shape[0], 3 - dims))], 1) if dims < 3 else x  # noqa: E731
    return [pad(x) for x in p], [pad(x) for x in v], [pad(x) for x in f]


def _boxes64(b, steps):
    lo, hi, v = _t64(b.lo), _t64(b.hi), _t64(b.v)
    f = torch.zeros_like(lo)
    for _ in range(steps):
        big = float((hi - lo).max())
        s = torch.zeros_like(lo)
        n = torch.zeros(lo.shape[0], dtype=torch.float64, device=lo.device)
        for i, j in _candidates(lo - RADIUS - big, hi + RADIUS, lo, RADIUS + big):
            ok = ((lo[i] - hi[j] <= RADIUS) & (lo[j] - hi[i] <= RADIUS)).all(1) & (i != j)
            i, j = i[ok], j[ok]
            s.index_add_(0, i, lo[j] - lo[i])
            n += torch.bincount(i, minlength=lo.shape[0])
        f += s / n.clamp(min=1)[:, None]
        size = hi - lo
        lo, hi = lo + v, hi + v
        low, high = lo < 0, hi > SIDE
        lo = torch.where(low, torch.zeros_like(lo), lo)
        hi = torch.where(low, size, hi)
        hi = torch.where(high, torch.full_like(hi, SIDE), hi)
        lo = torch.where(high, SIDE - size, lo)
        v = torch.where(low ^ high, -v, v)
    return lo, hi, v, f


def _boids64(p, v, r, steps):
    rr, sep2 = float(np.float32(r)), float(np.float32(r / 2)) ** 2
    top, force = 2.0, float(np.float32(0.03))

    def limit(x, most):
        n = x.norm(dim=1, keepdim=True)
        return torch.where(n > most, x * (most / n.clamp(min=1e-300)), x)

    def steer(x, w):
        n = x.norm(dim=1, keepdim=True)
        s = limit(x * (top / n.clamp(min=1e-300)) - v, force)
        return torch.where(n > 0, w * s, torch.zeros_like(s))

    for _ in range(steps):
        coh, ali, sep = torch.zeros_like(p), torch.zeros_like(p), torch.zeros_like(p)
        for i, j in _near(p, p, rr, True):
            d = p[j] - p[i]
            d2 = (d * d).sum(1)
            ok = (d2 < rr * rr) & (d2 > 0)
            i, j, d, d2 = i[ok], j[ok], d[ok], d2[ok]
            coh.index_add_(0, i, d)
            ali.index_add_(0, i, v[j])
            close = d2 < sep2
            sep.index_add_(0, i[close], -d[close] / d2[close, None])
        v = limit(v + steer(sep, 1.5) + steer(ali, 1.0) + steer(coh, 1.0), top)
        p = p + v
    return p, v


def _sph_ctx(alpha=0.05, c0=20.0):
    c = [float(x) for x in M.sph_context(h=H, dx=DX, alpha=alpha, c0=c0, tank_min=TANK[0], tank_max=TANK[1])]
    names = ["h", "inv_h", "support2", "sigma", "m", "rho0", "B", "c0", "alpha", "eta2", "dt", "gx", "gy", "gz"]
    return dict(zip(names, c))


def _sph_step64(x, v, c, alpha, c0):
    """One SPH step in 64 bits (differentiable: x, v, alpha, c0 may carry gradients); the
    neighbours are found on the values alone.  Returns x, v, P."""
    h, m, rho0 = c["h"], c["m"], c["rho0"]
    at = x.detach()
    ii, jj = [], []
    for i, j in _near(at, at, math.sqrt(c["support2"]), True):
        ok = ((at[i] - at[j]) ** 2).sum(1) < c["support2"]
        ii.append(i[ok])
        jj.append(j[ok])
    I, J = torch.cat(ii), torch.cat(jj)
    d = x[I] - x[J]
    r2 = (d * d).sum(1)
    r = r2.sqrt()
    q = r / h
    near = q < 1
    Wq = c["sigma"] * torch.where(near, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2 - q) ** 3)
    rho = (m * c["sigma"] + torch.zeros_like(x[:, 0])).index_add(0, I, m * Wq)
    B = c0 * c0 * rho0 / 7.0
    P = B * ((rho / rho0) ** 7 - 1)
    dW = c["sigma"] / h * torch.where(near, -3 * q + 2.25 * q ** 2, -0.75 * (2 - q) ** 2)
    vr = ((v[I] - v[J]) * d).sum(1)
    bar = 0.5 * (rho[I] + rho[J])
    visc = torch.where(vr < 0, -alpha * c0 * h * vr / ((r2 + c["eta2"]) * bar), torch.zeros_like(vr))
    A = P / rho ** 2
    a = torch.zeros_like(x).index_add(0, I, (-m * (A[I] + A[J] + visc) * dW / r)[:, None] * d)
    g = torch.tensor([c["gx"], c["gy"], c["gz"]], dtype=torch.float64, device=x.device)
    v = v + c["dt"] * (a + g)
    x = x + c["dt"] * v
    lo = torch.tensor([float(np.float32(t)) for t in TANK[0]], dtype=torch.float64, device=x.device)
    hi = torch.tensor([float(np.float32(t)) for t in TANK[1]], dtype=torch.float64, device=x.device)
    out = (x < lo) | (x > hi)
    v = torch.where(out, -0.5 * v, v)
    x = torch.where(x < lo, lo.expand_as(x), torch.where(x > hi, hi.expand_as(x), x))
    return x, v, P


def _calibrate64(case, seed):
    rng = np.random.default_rng(seed + 99)
    inst = _instances(case, seed)
    x0 = np.concatenate([ps.p[:, :3] for ps, *_ in inst]).astype(np.float64)
    target = x0 + 1e-3 * rng.standard_normal(x0.shape)
    got = {"x": [], "v": [], "dx0": [], "dv0": [], "dparams": []}
    at = 0
    for ps, alpha, c0, *_ in inst:
        c = _sph_ctx(alpha, c0)
        x, v = _t64(ps.p).requires_grad_(), _t64(ps.v).requires_grad_()
        par = torch.tensor([c["alpha"], c["c0"]], dtype=torch.float64, device="cuda", requires_grad=True)
        xs, vs = x, v
        for _ in range(case["steps"]):
            xs, vs, _P = _sph_step64(xs, vs, c, par[0], par[1])
        t = torch.from_numpy(target[at:at + ps.n]).cuda()
        at += ps.n
        ((xs - t) ** 2).sum(1).mean().backward()
        for name, val in (("x", xs.detach()), ("v", vs.detach()), ("dx0", x.grad), ("dv0", v.grad),
                          ("dparams", par.grad[None])):
            got[name].append(val)
    return {k: torch.cat(w) for k, w in got.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "query":
        n = case["n"]
        p = _t64(W.basic_points(n, seed=seed, side=_side(n)).p)
        return {"sum": _displacements(p, p, RADIUS, True)[0], "count": None}
    if kind in ("frames", "agents"):
        n = case["n"]
        p, v, f = _agents64([_test_records(n, seed, _side(n))], _side(n), case.get("steps", 1), 3)
        if kind == "frames":
            z = torch.zeros((n, 1), dtype=torch.float64, device="cuda")
            return {"p": torch.cat([p[0], z], 1), "f": torch.cat([f[0], z], 1), "pairs": None}
        return {"p": p, "v": v, "f": f, "pairs": None}
    if kind == "boxes":
        lo, hi, v, f = _boxes64(W.box_agents(case["n"], seed=seed), case["steps"])
        return {"min": lo, "max": hi, "v": v, "f": f, "pairs": None}
    if kind == "groups":
        side = _plane_side(case["n"] + case["m"])
        recs = [_test_records(case["n"], 2 * seed, side, True), _test_records(case["m"], 2 * seed + 1, side, True)]
        p, v, f = _agents64(recs, side, case["steps"], 2)
        return {"p": p, "v": v, "f": f, "pairs": None}
    if kind == "flock":
        got = [_boids64(_t64(ps.p), _t64(ps.v), r, case["steps"]) for ps, r in _flocks(case, seed)]
        return {"p": torch.cat([g[0] for g in got]), "v": torch.cat([g[1] for g in got]), "pairs": None}
    if kind == "dam":
        ps, c = _fluid(case, seed), _sph_ctx()
        x, v = _t64(ps.p), _t64(ps.v)
        for _ in range(case["steps"]):
            x, v, P = _sph_step64(x, v, c, c["alpha"], c["c0"])
        return {"p": x, "v": v, "P": P[:, None]}
    return _calibrate64(case, seed)
