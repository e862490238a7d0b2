"""Possible-pair rows of the cell list, sorted in registers by row length:
equal to the oracle's rows where the longest row lies on either side of each
length class (128, 256, 512, 1024, 2048 entries; beyond the last one the
row is sorted in place)."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 130, 258, 510, 1030, 2060])
@pytest.mark.parametrize("thr", [14.0, 60.0, 1000.0])
def test_rows_of_every_length_class(gpu_ctx, n, thr):
    sp = spec(n, 5, "free", pairs_threshold=thr, max_possiblePairs=n, grid_path=1, cell_list=1)
    g, o = gpu_ctx.job(sp), O.OracleJob(sp)
    g.rebuild(True, True)
    o.rebuild(True, True)
    assert g.status() == 0
    for possible in (True, False):
        cg, rg = g.pairlist(possible)
        co, ro = o.pairlist(possible)
        assert np.array_equal(cg, co) and np.array_equal(rg, ro)
    if thr == 1000.0:      # every bead not bonded to it: lengths just below n
        assert cg.size == n and g.pairlist(True)[0].max() > n - 64
    g.destroy()
