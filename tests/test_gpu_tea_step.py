"""TEA's step (one cluster of CTAs per 32 or 64 beads) against the oracle at the
edges of its split: fewer beads than a warp or than the cluster's shares,
sizes around whole tiles, the line between one and two beads per lane (1024),
all pairs and listed pairs, and a repeated run bit for bit.

Tolerance: the bound of the TEA parity tests, 1e-4 after a dozen steps."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unlisted", [1, 0])
@pytest.mark.parametrize("n", [2, 7, 33, 64, 1023, 1024, 1025, 1089, 2113])
def test_tea_step_tracks_oracle(gpu_ctx, n, unlisted):
    sp = spec(n, 23, "clamp", hi_on=1, hi_a=1.9, hi_epsilon_freq=10, hi_capricious=0, hi_unlisted=unlisted)
    g, o, r = gpu_ctx.job(sp), O.OracleJob(sp), gpu_ctx.job(sp)
    for chunk in (1, 4):
        gpu_ctx.run([g], chunk)
        assert o.advance(chunk) == 0
        gpu_ctx.run([r], chunk)
    assert g.status() == 0
    assert np.array_equal(g.read(sopb.SEEDS), o.read(sopb.SEEDS))
    assert np.max(np.abs(g.read(sopb.COORDS) - o.read(sopb.COORDS))) < 1e-4
    assert np.array_equal(g.read(sopb.COORDS), r.read(sopb.COORDS))
    g.destroy()
    r.destroy()
