"""GPU: values that no workload has but that the entry points take: negative and zero see
radii, and box agents whose max corner lies below their min corner.  The reference's box test
decides (a pair is skipped when |seer - seen| > r on an axis), so a negative radius on any axis
of the space finds nothing, at every number of lanes per seer."""
import ctypes
import dataclasses

import numpy as np
import pytest

from oracle import pyoracle as O
from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# agents and neighbours per agent that give 32, 16, 8 and 1 lanes per seer
SPACE = [(2500, 100), (5000, 100), (6000, 25), (20000, 100)]
FLAT = [(2000, 100), (4000, 100), (2500, 10), (10000, 100)]


def _side(n, mates, dims, radius=50.0):
    return 2.0 * radius * (n / mates) ** (1.0 / dims)


def _set_radii(b, radii):
    for k in range(b._descs[0].pass_count):
        b._descs[0].passes[k].radii[:] = list(radii) + [0.0]
    b._check(b.L.tgpu_batch_set_contexts(b.ptr, 0, ctypes.byref(b._descs[0])), "tgpu_batch_set_contexts")


@pytest.mark.parametrize("dims,n,mates", [(3, *x) for x in SPACE] + [(2, *x) for x in FLAT] + [(1, *x) for x in FLAT])
def test_negative_radii_find_nothing(gpu, dims, n, mates):
    """Radii set to negative ones between runs (the batch keeps the lanes of its first run)."""
    ps = W.basic_points(n, seed=71, side=_side(n, mates, dims))
    recs = M.records(M.TEST_RECORD, ps.p, ps.v)
    setup = dataclasses.replace(M.test_setup(passes=("agent_see",), mb=16), dims=dims)
    b = api.Batch([(setup, recs)])
    try:
        b.push()
        pairs = b.run(1)[1]
        assert pairs > 0
        first = b.fetch(0).tobytes()
        for axis in range(dims):
            for r in (-1e-3, -1.0, -60.0, -1e6, -np.inf):
                radii = [50.0, 50.0, 50.0]
                radii[axis] = r
                _set_radii(b, radii)
                assert b.run(1)[1] == 0, radii
        for radii in ([-50.0] * 3, [-1.0, -60.0, -1e6]):
            _set_radii(b, radii)
            assert b.run(1)[1] == 0, radii
        assert M.by_id(b.fetch(0)).tobytes() == M.by_id(np.frombuffer(first, M.TEST_RECORD)).tobytes()
        _set_radii(b, [50.0] * 3)
        assert b.run(1)[1] == pairs
    finally:
        b.close()


@pytest.mark.parametrize("dims,n,mates", [(3, *SPACE[0])] + [(2, *x) for x in FLAT])
def test_states_of_negative_radius(gpu, dims, n, mates):
    ps = W.basic_points(n, seed=72, side=_side(n, mates, dims))
    recs = M.records(M.TEST_RECORD, ps.p, ps.v)
    setup = dataclasses.replace(M.test_setup(radius=-50.0, passes=("agent_see",), mb=16), dims=dims)
    b = api.Batch([(setup, recs)])
    try:
        b.push()
        assert b.run(1)[1] == 0
        assert not b.fetch(0)["b_buffer_count"].any()
    finally:
        b.close()


@pytest.mark.parametrize("n", [2000, 5000, 20000, 40000])
def test_recorded_lists_of_negative_radius(gpu, n):
    """SPH: the density pass records empty lists and the force pass replays them."""
    side = int(np.ceil(n ** (1 / 3)))
    sph = W.sph_dam(side, side, side)
    setup = M.sph_setup(passes=("sph_density", "sph_pressure", "sph_force"), mb=64)
    recs = M.records(M.SPH_RECORD, sph.points.p[:n], sph.points.v[:n])
    b = api.Batch([(setup, recs)])
    try:
        b.push()
        assert b.run(1)[1] > 0
        for axis in range(3):
            radii = [0.04, 0.04, 0.04]
            radii[axis] = -0.3
            _set_radii(b, radii)
            assert b.run(1)[1] == 0
            got = b.fetch(0)
            assert not got["rho"].any() and not got["a"].any()
    finally:
        b.close()


@pytest.mark.parametrize("n,mates", SPACE[:3] + [(31000, 100)])
def test_inverted_boxes(gpu, port, n, mates):
    """A box whose max corner lies far below its min corner, on one axis or on all: exact counts."""
    w = W.box_agents(n, seed=73, side=_side(n, mates, 3))
    for k in range(7):
        axes = [k] if k < 3 else [0, 1, 2]
        for a in axes:
            w.hi[k::28, a] = w.lo[k::28, a] - 400.0 * (k + 1)
    recs = M.box_records(w.lo, w.hi, w.v)
    setup = M.box_setup(passes=("box_agent_see",), mb=16)
    b = api.Batch([(setup, recs)])
    try:
        b.push()
        b.run(1)
        got = M.by_id(b.fetch(0))
    finally:
        b.close()
    want = port.run(O.MODEL_BOX, "simple", recs, setup.passes[0].ctx, setup.passes[0].ctx, 50.0, 50.0, 1,
                    O.PASS_SEE0).records
    assert got["b_buffer_count"].sum() > 0
    assert np.array_equal(got["b_buffer_count"], want["b_buffer_count"])


@pytest.mark.parametrize("n", [1, 1000, 5000, 20000, 65536])
def test_allocation_free_pass_of_negative_radius(gpu, n):
    torch = pytest.importorskip("torch")
    L = api.lib()
    pos = torch.from_numpy(W.basic_points(n, seed=74).p.copy()).cuda()
    parts = (ctypes.c_float * 4)(50.0, 50.0, 50.0, 50.0)
    for radii in ((50.0, 50.0, -1.0), (50.0, -300.0, 50.0), (-1e6, 50.0, 50.0), (-50.0, -50.0, -50.0)):
        out = torch.full((n, 4), -1.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        rc = L.tgpu_see_noalloc(ctypes.c_void_p(pos.data_ptr()), n, (ctypes.c_float * 4)(*radii, 0.0), parts,
                                ctypes.c_void_p(out.data_ptr()), None)
        assert rc == 0, L.tgpu_noalloc_last_error().decode()
        assert not out.cpu().numpy().any(), radii


def _far_seers(rng, n, radius, edge=0.0):
    """Seers whose search interval [p - radius, p + radius] ends inside [0, 5], half of them from
    each side; the other axes near 0."""
    u = rng.uniform(0.0, 5.0, n)
    p = np.zeros((n, 4), np.float32)
    p[:, 0] = np.where(np.arange(n) % 2, radius + edge + u, u - radius)
    p[:, 1:3] = rng.uniform(0.0, 0.004, (n, 2))
    return p


@pytest.mark.parametrize("radius", [1e4, 1e5])
@pytest.mark.parametrize("tuning", [{}, {"hit_masks": 1}, {"cell_order": 0, "cell_multiple": 0.5}])
def test_far_seers_of_another_group(gpu, radius, tuning):
    """Seers one radius away from a small group with fine cells: their coordinates, and the
    differences of the box test, round more coarsely than the group's cells.  Exact counts
    against the box test in float32 over all pairs."""
    rng = np.random.default_rng(75)
    seen = np.zeros((3000, 4), np.float32)
    seen[:, :3] = rng.uniform(0.0, 1.0, (3000, 3)) * [5.0, 0.004, 0.004]
    seers = _far_seers(rng, 4000, radius)
    r = np.float32(radius)
    want = np.ones((4000, 3000), bool)
    for a in range(3):
        want &= np.abs(seers[:, None, a] - seen[None, :, a]) <= r
    see, act = M.test_contexts(radius)
    zero = [np.zeros_like(x) for x in (seers, seen)]
    recs = [M.records(M.TEST_RECORD, x, v) for x, v in zip((seers, seen), zero)]
    api.set_tuning(**tuning)
    try:
        got = M.run_groups(M.TEST_RECORD, ("agent_see", "agent_act"), recs, [("see", 0, 1, False)], see, act, radius,
                           0.01, 1)
    finally:
        api.set_tuning()
    assert np.array_equal(got[0]["b_buffer_count"], want.sum(1))


@pytest.mark.parametrize("radius", [1e4, 1e5])
@pytest.mark.parametrize("tuning", [{}, {"cell_order": 0, "cell_multiple": 0.5}])
def test_far_boxes_of_another_group(gpu, radius, tuning):
    rng = np.random.default_rng(76)

    def box(lo, edge):
        hi = lo.copy()
        hi[:, :3] += np.float32(edge)
        return lo, hi

    lo = np.zeros((3000, 4), np.float32)
    lo[:, :3] = rng.uniform(0.0, 1.0, (3000, 3)) * [5.0, 0.004, 0.004]
    seen, seers = box(lo, 0.5), box(_far_seers(rng, 4000, radius, 0.5), 0.0)
    r = np.float32(radius)
    want = np.ones((4000, 3000), bool)
    for a in range(3):
        want &= ~(seers[0][:, None, a] - seen[1][None, :, a] > r) & ~(seen[0][None, :, a] - seers[1][:, None, a] > r)
    see, act = M.test_contexts(radius)
    recs = [M.box_records(x, y, np.zeros_like(x)) for x, y in (seers, seen)]
    api.set_tuning(**tuning)
    try:
        got = M.run_groups(M.BOX_RECORD, ("box_agent_see", "box_agent_act"), recs, [("see", 0, 1, False)], see, act,
                           radius, 0.01, 1, is_point=False)
    finally:
        api.set_tuning()
    assert np.array_equal(got[0]["b_buffer_count"], want.sum(1))


def _odd_records(model, n, kind, fixed):
    """A workload with positions (boxes: corners) that are NaN or infinite, on one axis or all."""
    if model == "box":
        w = W.box_agents(n, seed=81, side=_side(n, 100, 3))
        setup, corners, side = M.box_setup(mb=16), (w.lo, w.hi), _side(n, 100, 3)
    elif model == "sph":
        e = int(np.ceil(n ** (1 / 3)))
        w = W.sph_dam(e, e, e).points
        setup, corners, side = M.sph_setup(mb=16), (w.p[:n],), 0.01 * e
    elif model == "boids":
        side = (125.0 * n) ** (1 / 3)
        w = W.basic_points(n, seed=82, side=side)
        setup, corners = M.boids_setup(mb=16), (w.p,)
    else:
        side = _side(n, 100, 3)
        w = W.basic_points(n, seed=83, side=side)
        setup, corners = M.test_setup(mb=16), (w.p,)
    values = [np.nan] if kind == "nan" else [np.inf, -np.inf, np.nan]
    for k, axes in enumerate(([0], [1], [2], [0, 1, 2], [0, 2])):
        for c in corners:
            c[k::977, axes] = values[k % len(values)]
    if len(corners) == 2:
        corners[1][5::977, 1] = np.inf  # a box without an upper end
    if fixed:
        setup = dataclasses.replace(setup, fixed_box=((0.0, 0.0, 0.0), (side, side, side)))
    if model == "box":
        return setup, M.box_records(*corners, w.v)
    return setup, M.records(setup.dtype, corners[0], w.v[:n])


def _same(a, b):
    """Equal values in every field, NaNs of any payload equal."""
    for f in a.dtype.names:
        x, y = a[f], b[f]
        if x.dtype.kind == "f" or (x.dtype.subdtype and x.dtype.subdtype[0].kind == "f"):
            assert np.array_equal(x, y, equal_nan=True), f
        else:
            assert np.array_equal(x, y), f


def _run_odd(groups, steps):
    b = api.Batch(groups)
    try:
        b.push()
        pairs = b.run(steps)[1]
        return M.by_id(b.fetch(0)), pairs, b.launches_per_step()
    finally:
        b.close()


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("kind", ["nan", "inf"])
@pytest.mark.parametrize("model,n", [("test", 2500), ("test", 5001), ("test", 20000), ("box", 3001), ("box", 12289),
                                     ("boids", 2049), ("boids", 8193), ("sph", 4097), ("sph", 20001)])
def test_nan_and_infinite_positions(gpu, model, n, kind, fixed):
    """A state alone (shared lanes, cluster sort) and in a batch of so many agents and segments
    that every seer has one lane and the sort is the general one; the agents beside it are
    scattered over a large space.  The second step meets the NaNs that the first one computed."""
    setup, recs = _odd_records(model, n, kind, fixed)
    plain = dataclasses.replace(setup, fixed_box=None)
    x = W.basic_points(60000, seed=85, side=5000.0)
    if model == "box":
        other = M.box_records(x.p, x.p, x.v)
    else:
        other = M.records(setup.dtype, x.p, x.v)
    many = [(plain, other)] + [(plain, other[:5])] * 200
    for steps in (1, 2):
        got, pairs, launches = _run_odd([(setup, recs)], steps)
        want, _, general = _run_odd([(setup, recs)] + many, steps)
        assert pairs > 0 and launches < general
        _same(got, want)


@pytest.mark.parametrize("n,mates", SPACE)
def test_zero_radius(gpu, n, mates):
    """Neighbours are the agents in exactly the same place."""
    ps = W.basic_points(n, seed=84, side=_side(n, mates, 3))
    ps.p[n // 2:2 * (n // 2)] = ps.p[:n // 2]
    recs = M.records(M.TEST_RECORD, ps.p, ps.v)
    b = api.Batch([(M.test_setup(passes=("agent_see",), mb=16), recs)])
    try:
        b.push()
        assert b.run(1)[1] > 0
        _set_radii(b, [0.0] * 3)
        assert b.run(1)[1] == 2 * (n // 2)
    finally:
        b.close()
