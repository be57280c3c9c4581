"""GPU: the cells of an SPH state, and so the order of its float sums, depend on the state alone:
it steps through the same bits alone, among others in a batch, and as a recorded rollout."""
import ctypes

import numpy as np
import pytest

from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# below, between and above the agent counts at which the cells shrink
SHAPES = [(16, 16, 8), (32, 32, 16), (32, 40, 16), (44, 44, 44)]


def _state(shape):
    sph = W.sph_dam(*shape)
    v = sph.points.v
    v[:, :3] = 0.05 * np.random.default_rng(shape[0] + shape[1]).standard_normal((len(v), 3))
    return M.sph_setup(mb=16), M.records(M.SPH_RECORD, sph.points.p, v)


def _steps(b, steps):
    b.push()
    pairs = b.run(steps)[1]
    return pairs, [M.by_id(b.fetch(k)).tobytes() for k in range(len(b.groups))]


def test_alone_equals_in_a_batch(gpu):
    states = [_state(s) for s in SHAPES]
    batches = [api.Batch(states)] + [api.Batch([s]) for s in states]
    try:
        got = [_steps(b, 3) for b in batches]
    finally:
        for b in batches:
            b.close()
    assert got[0][0] == sum(g[0] for g in got[1:])
    for k, g in enumerate(got[1:]):
        assert got[0][1][k] == g[1][0], SHAPES[k]


def test_many_small_states_equal_one(gpu):
    """More agents than either threshold, in states below both."""
    state = _state(SHAPES[0])
    many, one = api.Batch([state] * 48), api.Batch([state])
    try:
        a, b = _steps(many, 3), _steps(one, 3)
    finally:
        many.close()
        one.close()
    assert a[0] == 48 * b[0] and set(a[1]) == set(b[1])


@pytest.mark.parametrize("shape", SHAPES)
def test_rollout_equals_plain_steps(gpu, shape):
    """The recorded forward steps, and plain steps of a batch that has recorded a rollout."""
    state = _state(shape)
    plain, b = api.Batch([state]), api.Batch([state])
    adj = ctypes.c_void_p()
    try:
        want = np.frombuffer(_steps(plain, 4)[1][0], M.SPH_RECORD)
        b.push()
        b._check(b.L.tgpu_adjoint_create(b.ptr, 4, 2, 1, ctypes.byref(adj)), "tgpu_adjoint_create")
        b._check(b.L.tgpu_adjoint_forward(adj), "tgpu_adjoint_forward")
        got = M.by_id(b.fetch(0))
        for f in ("p", "v", "rho"):
            assert got[f].tobytes() == want[f].tobytes(), f
        b.L.tgpu_adjoint_destroy(adj)
        adj = ctypes.c_void_p()
        assert _steps(b, 4)[1][0] == want.tobytes()
    finally:
        if adj:
            b.L.tgpu_adjoint_destroy(adj)
        plain.close()
        b.close()
