"""GPU: a batch whose cell tables cannot be had says so on every run, launches nothing, and runs
again once they can."""
import numpy as np
import pytest

from tay_gb300 import api
from tay_gb300 import models as M
from tay_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _group(n, side, seed, mb=8192):
    """Agents that see each other, in a box of the given side (two of them in its corners)."""
    ps = W.basic_points(n, seed=seed, side=100.0)
    ps.p[0, :3] = 0.0
    ps.p[1, :3] = side
    return M.test_setup(radius=50.0, part=10.0, passes=("agent_see",), mb=mb), M.records(M.TEST_RECORD, ps.p, ps.v)


def _pairs(groups):
    b = api.Batch(groups)
    try:
        b.push()
        return b.run(1)[1]
    finally:
        b.close()


def test_more_entries_than_an_index_holds(gpu):
    """Five tables of 2^30 entries: refused before anything is allocated, from the first run on."""
    wide = [_group(300, 2e4, k) for k in range(5)]
    small = [_group(300, 200.0, k) for k in range(5)]
    want = _pairs(small)
    assert want > 0
    b = api.Batch(wide)
    try:
        b.push()
        for _ in range(3):
            with pytest.raises(api.TayError, match="too large"):
                b.run(1)
        with pytest.raises(api.TayError, match="too large"):
            b.profile(1)
        b.groups = small
        b.push()
        assert b.run(2)[1] == 2 * want
    finally:
        b.close()


def test_table_that_does_not_fit_in_memory(gpu):
    """A push widens the extent, and the larger table (8 GB) does not fit beside another
    allocation of the process; captured steps of the small table are not run again."""
    torch = pytest.importorskip("torch")
    small, wide = _group(300, 200.0, 7), _group(300, 2e4, 7)
    want_small = _pairs([small])
    b = api.Batch([small])
    hog = None
    try:
        b.push()
        assert b.run(3)[1] == 3 * want_small
        b.groups = [wide]
        b.push()
        want = b.run(1)[1]  # (the budget follows a push one run behind)
        assert want == want_small > 0  # (the far corner sees nothing in either)
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - (4 << 30), dtype=torch.uint8, device="cuda")
        for _ in range(3):
            with pytest.raises(api.TayError, match="cudaMalloc failed"):
                b.run(2)
        hog = None
        torch.cuda.empty_cache()
        assert b.run(2)[1] == 2 * want
        b.groups = [small]
        b.push()
        assert b.run(2)[1] == 2 * want_small
        assert len(b.fetch(0)) == 300
    finally:
        hog = None
        torch.cuda.empty_cache()
        b.close()
