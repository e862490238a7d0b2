"""Exact HI of a job that one cluster of CTAs factorises (up to 128 beads), at
the edges of its 32-row blocks and cluster sizes: one block (10 beads), one
row into the next (11), two to three, three to four blocks and the first
cluster of four (32, 43), the last of four and the first of eight (74, 75,
86), a full last block (128 is 12 whole blocks; 127 is not).  The bounds are
those of the other sizes' tests: the factor within 2e-4 per entry and 2e-6 in
norm of FP64, coordinates within 1e-3 A of the oracle."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 10, 11, 21, 22, 32, 43, 74, 75, 86, 107, 127, 128])
@pytest.mark.parametrize("refresh", [1, 4])
def test_small_exact_hi(gpu_ctx, n, refresh):
    sp = spec(n, 51, "clamp", hi_on=1, hi_a=1.9, hi_exact=1, hi_refresh=refresh, hi_capricious=0)
    g, o = gpu_ctx.job(sp), O.OracleJob(sp)
    x0 = g.read(sopb.COORDS)[:, :3].copy()
    gpu_ctx.run([g], 1)                       # step 0 factorises D at x0
    L = np.tril(g.read(sopb.HIFACTOR).astype(np.float64))
    D = O.rpy_tensor(x0, sp.params.hi_a)
    assert np.max(np.abs(L - np.linalg.cholesky(D))) < 2e-4
    assert np.linalg.norm(L @ L.T - D) / np.linalg.norm(D) < 2e-6
    gpu_ctx.run([g], 8)                       # with a factor of an earlier step, and new ones
    assert o.advance(9) == 0
    assert g.status() == 0
    assert np.array_equal(g.read(sopb.SEEDS), o.read(sopb.SEEDS))
    assert np.max(np.abs(g.read(sopb.COORDS) - o.read(sopb.COORDS))) < 1e-3
    assert np.allclose(g.read(sopb.TEMP), o.read(sopb.TEMP), rtol=1e-3, atol=1e-3)
    g.destroy()
