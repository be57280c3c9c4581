"""GPU: small segments are boxed, keyed and sorted by one launch (a thread-block cluster per
segment), middle ones by one such launch per radix pass.  The same keys and a stable sort give the same permutation as the general path,
which a batch of many segments takes, so the same states alone and in such a batch must end
with the same bytes."""
import numpy as np
import pytest

from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# one agent, edges of a warp, of a block's threads and of its chunk, of two, four and eight
# blocks, the largest segment of one launch, and on both sides of the sizes at which a block's
# chunk grows, up to the largest that a cluster sorts pass by pass
SIZES = [1, 2, 33, 1023, 1025, 2048, 2049, 4096, 4097, 8193, 16384, 16385, 32769, 65536, 65537, 131072]


def _state(model, n, k):
    if model == "boids":
        ps = W.boids_points(n, seed=60 + k, clusters=3, side=300.0)
        if k % 3 == 0:
            ps.p[:, 0] = 7.0                      # one cell across x: every key's low digit equal
        if k % 3 == 1:
            ps.p[n // 2:, :3] = ps.p[0, :3]       # half of the agents in one place
        return M.boids_setup(mb=4), M.records(M.BOIDS_RECORD, ps.p, ps.v)
    b = W.box_agents(n, seed=80 + k, side=1000.0 * max(1.0, n / 20000) ** (1 / 3))
    return M.box_setup(mb=4), M.box_records(b.lo, b.hi, b.v)


@pytest.mark.parametrize("model", ["boids", "box"])
@pytest.mark.parametrize("tuning", [{}, {"cell_order": 0}, {"cell_multiple": 0.3, "x_cell_factor": 0.25}])
def test_alone_equals_in_a_batch(gpu, model, tuning):
    states = [_state(model, n, k) for k, n in enumerate(SIZES)]
    filler = [_state(model, 5, 99)] * 152  # more segments than one wave of clusters holds
    api.set_tuning(**tuning)
    try:
        many = api.Batch(states + filler)
        try:
            many.push()
            many.run(3)
            general = many.launches_per_step()
            for k, s in enumerate(states):
                one = api.Batch([s])
                try:
                    one.push()
                    one.run(3)
                    assert one.launches_per_step() < general
                    assert many.fetch(k).tobytes() == one.fetch(0).tobytes(), SIZES[k]
                finally:
                    one.close()
        finally:
            many.close()
    finally:
        api.set_tuning()


def test_fixed_box_and_empty_segment(gpu):
    """A fixed box (agents outside it in the edge cells) and a segment without agents."""
    import dataclasses

    def boxed(n, k):
        setup, recs = _state("boids", n, k)
        return dataclasses.replace(setup, fixed_box=((50.0, 50.0, 50.0), (250.0, 250.0, 250.0))), recs

    states = [boxed(3000, 4), (M.boids_setup(mb=4), np.zeros(0, M.BOIDS_RECORD)), boxed(700, 5)]
    few, many = api.Batch(states), api.Batch(states + [_state("boids", 5, 98)] * 152)
    try:
        for b in (few, many):
            b.push()
            b.run(3)
        for k in (0, 2):
            assert few.fetch(k).tobytes() == many.fetch(k).tobytes()
    finally:
        few.close()
        many.close()
