"""GPU: see passes whose seers share several lanes (small and middle launches) give the bits
of the row walk with one lane per seer.  The terms of a seer's neighbours are the same
floats, folded in the same order, so records and pair counts must be equal byte for byte
(no tolerance).  The hit-mask tuning keeps one lane per seer, walks in the same order and
keeps no pair lists, so it is the comparison for every model."""
import numpy as np
import pytest

from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _records(model, n):
    if model == "test":
        ps = W.basic_points(n, seed=91, side=1000.0 * (n / 1e5) ** (1 / 3) + 1.0)
        return M.test_setup(), M.records(M.TEST_RECORD, ps.p, ps.v)
    if model == "box":
        b = W.box_agents(n, seed=92)
        return M.box_setup(), M.box_records(b.lo, b.hi, b.v)
    if model == "boids":  # 64 neighbours inside the box, both halves of the separation test
        ps = W.basic_points(n, seed=93, side=(125.0 * n) ** (1 / 3))
        return M.boids_setup(r=10.0, part=10.0), M.records(M.BOIDS_RECORD, ps.p, ps.v)
    if model == "flock":  # scattered: a few neighbours, or none
        ps = W.boids_points(n, seed=97)
        return M.boids_setup(r=10.0, part=10.0), M.records(M.BOIDS_RECORD, ps.p, ps.v)
    if model == "heap":  # every particle inside every other's support: the pair lists overflow
        p = np.full((n, 4), 0.05, np.float32)
        p[:, :3] += np.random.default_rng(94).uniform(0, 0.01, (n, 3)).astype(np.float32)
        p[:, 3] = 0.0
        return M.sph_setup(mb=64), M.records(M.SPH_RECORD, p, np.zeros((n, 4), np.float32))
    side = int(np.ceil(n ** (1 / 3)))
    sph = W.sph_dam(side, side, side)
    return M.sph_setup(mb=64), M.records(M.SPH_RECORD, sph.points.p[:n], sph.points.v[:n])


def _run(setup, recs, steps, **tuning):
    api.set_tuning(**tuning)
    try:
        b = api.Batch([(setup, recs)])
        try:
            b.push()
            pairs = [b.run(1)[1] for _ in range(steps)]
            return M.by_id(b.fetch(0)).tobytes(), pairs
        finally:
            b.close()
    finally:
        api.set_tuning()


# a single agent, part of a CTA, a CTA and one more, and sizes at 32, 16, 8 and 1 lanes per
# seer for each model's density
@pytest.mark.parametrize("model,n", [
    ("test", 1), ("test", 2), ("test", 127), ("test", 129), ("test", 2500), ("test", 4097), ("test", 12289),
    ("test", 40000), ("test", 60001), ("box", 3), ("box", 3001), ("box", 12289), ("boids", 33), ("boids", 2049),
    ("boids", 8193), ("boids", 30001), ("flock", 600), ("flock", 5000), ("sph", 5), ("sph", 4097), ("sph", 20001), ("sph", 40001), ("sph", 130000),
    ("heap", 700)])
def test_shared_lanes_equal_one_lane(gpu, model, n):
    setup, recs = _records(model, n)
    assert _run(setup, recs, 3) == _run(setup, recs, 3, hit_masks=1)


def test_two_groups_read_every_step(gpu):
    """Groups of a state that see each other, each launch over one group's seers, and the
    records written through after every run."""
    a, b = W.basic_points(3001, seed=95, side=310.0), W.basic_points(1999, seed=96, side=310.0)
    recs = [M.records(M.TEST_RECORD, x.p, x.v) for x in (a, b)]
    passes = [("see", 0, 0, False), ("see", 0, 1, False), ("see", 1, 0, False), ("act", 0), ("act", 1)]
    see, act = M.test_contexts()
    out = []
    for tuning in ({}, {"hit_masks": 1}):
        api.set_tuning(**tuning)
        try:
            out.append(M.run_groups(M.TEST_RECORD, ("agent_see", "agent_act"), recs, passes, see, act, 50.0, 50.0, 4,
                                    host_loop="read" if not tuning else None))
        finally:
            api.set_tuning()
    for x, y in zip(*out):
        assert x.tobytes() == y.tobytes()


@pytest.mark.parametrize("shape,dx,box,dims", [
    ((32, 40, 16), 0.01, None, 3),                             # 64 particles per cubed part: a third
    ((32, 40, 16), 0.014, None, 3),                            # 23: a half
    ((32, 40, 16), 0.007, None, 3),                            # 187 (the lists overflow): a quarter
    ((32, 40, 64), 0.01, None, 3),                             # 64, and above 80,000 particles: a quarter
    ((44, 44, 44), 0.0126, None, 3),                           # 32: a third
    ((40, 40, 11), 0.01, ((0, 0, 0), (2.0, 1.5, 0.8)), 3),     # a fixed box, sparse by the mean: no change
    ((150, 150, 1), 0.01, None, 2),                            # a plane
    ((20000, 1, 1), 0.01, None, 3),                            # a line: one cell across
])
def test_cells_below_the_part_size(gpu, shape, dx, box, dims):
    """Dense SPH groups (above 16,384 particles) get cells below the part size.  The neighbour
    sets do not depend on the cells: the pair counts equal those of cells given by a tuning,
    and the densities agree to the rounding of a sum of positive float32 terms (2^-24 for each
    addition at worst; (0.04 / dx)^3 * 4/3 pi terms, and one in two sums each)."""
    import dataclasses

    sph = W.sph_dam(*shape, dx=dx, tank=(300.0, 3.0, 3.0))
    recs = M.records(M.SPH_RECORD, sph.points.p, sph.points.v)
    setup = dataclasses.replace(M.sph_setup(passes=("sph_density", "sph_pressure"), mb=64), dims=dims, fixed_box=box)
    got = []
    for tuning in ({}, {"x_cell_factor": 1.0}):
        api.set_tuning(**tuning)
        try:
            b = api.Batch([(setup, recs)])
            try:
                b.push()
                pairs = b.run(1)[1]
                got.append((pairs, M.by_id(b.fetch(0))))
            finally:
                b.close()
        finally:
            api.set_tuning()
    assert got[0][0] == got[1][0] > 0
    a, b = got[0][1]["rho"], got[1][1]["rho"]
    terms = (0.04 / dx) ** 3 * 4 / 3 * np.pi
    assert np.max(np.abs(a - b) / b) < 2 * terms * 2.0 ** -24


@pytest.mark.parametrize("most", [2, 9])
def test_replay_of_short_lists(gpu, most):
    """Clumps of 1 to `most` particles, further apart than the support: the force pass's lists
    end at every place of a group of four entries, and the next group's entries are loaded
    ahead.  One lane per seer (above 16,384 particles), the walk's bits."""
    k = 1 + np.arange(16384 * 2 // (most + 1) + most) % most
    site = np.repeat(np.arange(len(k)), k)
    p = np.zeros((len(site), 4), np.float32)
    p[:, :3] = 0.1 * np.stack([site % 32, site // 32 % 32, site // 1024], 1) + 0.05
    p[:, :3] += np.random.default_rng(most).uniform(-0.005, 0.005, (len(site), 3)).astype(np.float32)
    recs = M.records(M.SPH_RECORD, p, np.zeros_like(p))
    assert len(recs) > 16384
    got = []
    for tuning in ({}, {"pair_list_cap": 0}):
        api.set_tuning(**tuning)
        try:
            b = api.Batch([(M.sph_setup(tank_max=(4.0, 4.0, 4.0), mb=64), recs)])
            try:
                b.push()
                got.append((b.run(1)[1], b.run(1)[1], b.fetch(0).tobytes(), b.telemetry()["replay_warps"]))
            finally:
                b.close()
        finally:
            api.set_tuning()
    assert got[0][:3] == got[1][:3]
    assert got[0][3] == (len(recs) + 127) // 128 * 4 and got[1][3] == 0  # every warp of every block


def test_rollout_cells_depend_on_the_instance(gpu):
    """Rollouts give instances above 16,384 particles cells below the part size, by their own
    count: a large and a small instance have the same trajectories and gradients alone and
    together, bit for bit."""
    from tay_gb300.adjoint import SphRollout

    def rollout(shapes):
        inst = []
        for shape in shapes:
            s = W.sph_dam(*shape)
            s.points.v[:, :3] = 0.02 * np.random.default_rng(shape[0]).standard_normal((s.points.n, 3))
            inst.append((s.points, 0.05, 20.0, (0.0, 0.0, 0.0), (2.0, 1.5, 0.8)))
        roll = SphRollout(inst, 4, checkpoint_every=2)
        x, v = roll.forward()
        dx, dv, dp = roll.backward(2.0 * x)
        roll.close()
        return x, dx, dv, dp

    large, small = (32, 40, 16), (16, 16, 8)
    both, a, b = rollout([large, small]), rollout([large]), rollout([small])
    n = len(a[0])
    for k in range(3):
        assert both[k][:n].tobytes() == a[k].tobytes()
        assert both[k][n:].tobytes() == b[k].tobytes()
    assert both[3][0].tobytes() == a[3][0].tobytes() and both[3][1].tobytes() == b[3][0].tobytes()
