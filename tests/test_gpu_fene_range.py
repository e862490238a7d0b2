"""The bond force over the range of its parameters: bonds from a third of an
Angstrom to beyond R_limit on either side of r0, R_limit from 0.5 A to values
whose square is no longer a float (a harmonic bond), and a bond torn so far that
the term's denominator overflows.  Isolated dimers along x, so that the bead
distance is exact and the bond is the only force; on the resident and the grid
path, as SOPB_FORCES and as the move of one step without noise.

Tolerance, with u = 2^-24 and t = ((r - r0) / R_limit)^2: the distance carries
1.5 u r (the rounding of its square and of its root) and the difference w = r -
r0 one more u, which the term amplifies by (1 + t) / (1 - t); R^2 - w^2 carries
u t / (1 - t); two products each above and below the line, the root below, the
quotient (an ulp, 2 u) and the product with the separation make 9 u."""
import numpy as np
import pytest

import sopb
from helpers import plain_params

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
KS, R0 = 20.0, 3.8


def dimers(r, **kw):
    m = len(r)
    side = int(np.ceil(np.sqrt(m)))
    x = np.zeros((2 * m, 3), np.float32)
    k = np.arange(m)
    x[0::2, 1] = x[1::2, 1] = 64.0 * (k % side)
    x[0::2, 2] = x[1::2, 2] = 64.0 * (k // side)
    x[1::2, 0] = r
    bonds = np.stack([2 * k, 2 * k + 1], 1)
    p = plain_params(minimization=1, kspring_cov=KS, **kw)
    return sopb.JobSpec(x, bonds, np.full(m, R0, np.float32), np.zeros((0, 2)), [], [], p, seed=3)


def expected(r, R_limit):
    """Force on the dimer's first bead and the bound of its relative error."""
    r, r0 = r.astype(np.float64), np.float64(np.float32(R0))
    with np.errstate(over="ignore"):
        R2 = np.float64(np.float32(R_limit) * np.float32(R_limit))
    w = r - r0
    t = w * w / R2
    f = KS * w / (r * (1 - t)) * r
    g = np.abs(1 - t)
    return f, U * ((1.5 * r / np.abs(w) + 1) * (1 + t) / g + t / g + 9)


@pytest.mark.parametrize("grid", [0, 1])
@pytest.mark.parametrize("R_limit", [0.5, 2.0, 100.0, 1e10, 1e18, 1e19, 1e20, 3e38])
def test_bond_force_over_its_range(gpu_ctx, R_limit, grid):
    reach = min(R_limit, 50.0)
    w = reach * np.concatenate([np.geomspace(1e-3, 0.95, 200), [0.99, 0.999, 1.001, 1.01, 1.5]])
    r = np.concatenate([R0 - w, R0 + w]).astype(np.float32)
    r = r[r > 0.3]
    g = gpu_ctx.job(dimers(r, R_limit=R_limit, grid_path=grid))
    f, rel = expected(r, R_limit)
    got = g.read(sopb.FORCES).astype(np.float64)
    assert np.all(np.abs(got[0::2, 0] - f) <= rel * np.abs(f))
    assert np.all(np.abs(got[1::2, 0] + f) <= rel * np.abs(f))
    assert not got[:, 1:3].any()
    # the move of a step: h / zeta times the force, two roundings there and one of the coordinate
    x0 = g.read(sopb.COORDS).astype(np.float64)
    gpu_ctx.run([g], 1)
    x1 = g.read(sopb.COORDS).astype(np.float64)
    assert g.status() == 0
    d = np.float64(np.float32(0.08) / np.float32(50.0)) * np.stack([f, -f], 1).ravel()
    rel2 = np.repeat(rel, 2) + 4 * U
    assert np.all(np.abs(x1[:, 0] - x0[:, 0] - d) <= rel2 * np.abs(d) + U * np.maximum(np.abs(x0[:, 0]), np.abs(x1[:, 0])))
    g.destroy()


@pytest.mark.parametrize("grid", [0, 1])
def test_a_torn_bond_stays_finite(gpu_ctx, grid):
    r = np.array([1e6, 1e9, 1e13, 1e15], np.float32)
    g = gpu_ctx.job(dimers(r, grid_path=grid))
    got = g.read(sopb.FORCES)
    assert np.isfinite(got).all()
    # beyond R_limit the term pushes on: -ks R^2 / r, or nothing once its denominator is out of range
    assert np.all(np.abs(got[0::2, 0].astype(np.float64)) <= 1.001 * KS * 4.0 / r)
    gpu_ctx.run([g], 1)
    assert g.status() == 0
    g.destroy()
