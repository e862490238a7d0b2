"""The FP64 diagonal tile of the blocked exact-HI factorisation at sizes whose
last tile has few, odd or nearly all of its 128 rows (3 n mod 128 = 3, 126, 1,
127, 2, 120): its factor, and through the solves of the tiles below also its
inverse, against FP64, within the bounds of the other sizes' tests."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 170, 171, 213, 214, 296])
def test_partial_diagonal_tile(gpu_ctx, n):
    sp = spec(n, 57, "free", hi_on=1, hi_a=1.9, hi_exact=1, hi_capricious=0)
    g = gpu_ctx.job(sp)
    for step in range(2):                     # the second factor overwrites the first one's buffers
        x = g.read(sopb.COORDS)[:, :3].copy()
        gpu_ctx.run([g], 1)
        L = np.tril(g.read(sopb.HIFACTOR).astype(np.float64))
        D = O.rpy_tensor(x, sp.params.hi_a)
        assert g.status() == 0
        assert np.max(np.abs(L - np.linalg.cholesky(D))) < 2e-4
        assert np.linalg.norm(L @ L.T - D) / np.linalg.norm(D) < 2e-6
    g.destroy()
