"""The roots and quotients of the small exact-HI factor (estimate, Newton step and
residual correction) lose no more than an ulp each.  Two beads: the factor's
first three columns are the identity and the block B between the beads, the rest
is the Cholesky factor of I - B B^T, whose pivots run from near 0 (beads almost
on top of one another) to 1.

Tolerance: the backward error of Cholesky, |A - L L^T| <= (n + 1) u |L| |L|^T
with n = 6 and u = 2^-24 for correctly rounded roots and quotients; an ulp each
instead of half of one adds u to a quotient and u to a root on both sides of its
square, at most 4 u."""
import numpy as np
import pytest

import sopb
from helpers import plain_params

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
HI_A = 1.9


def test_factor_of_two_beads_to_the_ulp(gpu_ctx):
    rng = np.random.default_rng(5)
    dist = HI_A * np.geomspace(0.02, 200.0, 120)
    worst = pivot = 0.0
    low = 1.0
    for d in dist:
        e = rng.normal(size=3)
        x = np.stack([np.zeros(3), d * e / np.linalg.norm(e)]).astype(np.float32)
        p = plain_params(hi_on=1, hi_exact=1, hi_a=HI_A, hi_capricious=0, el=0.0)
        g = gpu_ctx.job(sopb.JobSpec(x, np.zeros((0, 2)), [], np.zeros((0, 2)), [], [], p, seed=3))
        gpu_ctx.run([g], 1)
        assert g.status() == 0
        L = np.tril(g.read(sopb.HIFACTOR).astype(np.float64).reshape(6, 6))
        assert np.array_equal(L[:3, :3], np.eye(3))
        A = np.eye(6)
        A[3:, :3] = L[3:, :3]
        A[:3, 3:] = L[3:, :3].T
        err = np.abs(A - L @ L.T)[3:, 3:]
        bound = 11 * U * (np.abs(L) @ np.abs(L).T)[3:, 3:]
        assert np.all(err <= bound), d
        worst = max(worst, float(np.max(err / bound)))
        pivot, low = max(pivot, L[3, 3]), min(low, L[5, 5])
        g.destroy()
    assert worst > 0 and pivot > 0.999 and low < 0.2      # the pivots' range was covered
