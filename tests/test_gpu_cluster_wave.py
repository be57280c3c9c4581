"""GPU: batches of so many segments that their clusters run at once only with more agents per
thread give the bytes of the general path."""
import pytest

from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _state(n, k):
    ps = W.boids_points(n, seed=160 + k, clusters=3, side=300.0)
    return M.boids_setup(mb=4), M.records(M.BOIDS_RECORD, ps.p, ps.v)


def _run(states):
    b = api.Batch(states)
    try:
        b.push()
        b.run(2)
        return b.launches_per_step(), [b.fetch(k).tobytes() for k in range(3)]
    finally:
        b.close()


# segments, largest segment: 4 agents a thread, 8, 4 a launch per pass, 8, and past every wave
@pytest.mark.parametrize("segments,largest,one_wave", [
    (40, 8192, True), (24, 16384, True), (60, 16380, True), (9, 32768, True), (20, 32768, True), (10, 65536, True),
    (90, 16384, False), (40, 32768, False), (9, 131072, False)])
def test_more_agents_per_thread_for_one_wave(gpu, segments, largest, one_wave):
    first = [_state(largest, 0), _state(largest - 1001, 1), _state(33, 2)]
    filler = [_state(700, 3)]
    launches, got = _run(first + filler * (segments - 3))
    general, want = _run(first + filler * 200)
    assert got == want
    assert (launches < general) == one_wave
