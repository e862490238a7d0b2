"""A job's result does not depend on how many CTAs it gets.  Alone, a resident
job runs on a cluster of two to sixteen CTAs (from 24 beads up); among 160
copies of itself, on one.  Sizes at the edges: the smallest clusters, odd bead
counts (a last pair of one bead), the largest resident job, whose rows do not
all fit one CTA's shared memory; each updater with state of its own; other
lane counts than the usual four.  Bit equality, so no tolerance."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import spec

pytestmark = pytest.mark.gpu

SURFACE = dict(indentationDiscreteSurf=1, indentationSurfaceSize=7, indentationSurfaceStep=3.0, indentationMoveSurface=1)
CASES = {
    "n24": (24, "clamp", {}),
    "n25_odd": (25, "ramp", {}),
    "n97_odd": (97, "free", dict(heating=1, initialT=0.1, deltaT=0.2, tempFreq=20)),
    "n203_ramp": (203, "ramp", {}),
    "n203_pp_between": (203, "clamp", dict(nav=10, pairs_freq=20, possiblepairs_freq=30, pairs_threshold=30.0)),
    "n203_indent": (203, "indent", {}),
    "n203_surface": (203, "indent", SURFACE),
    "n203_lanes2": (203, "clamp", dict(lanes_per_bead=2)),
    "n203_lanes16": (203, "clamp", dict(lanes_per_bead=16)),
    "n1025_odd": (1025, "clamp", {}),
    "n2047_odd": (2047, "ramp", {}),
    "n2048_no_near_list": (2048, "clamp", dict(verlet_skin=-1.0)),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_cluster_equals_one_cta(gpu_ctx, case):
    n, mode, kw = CASES[case]
    sp = spec(n, 41, mode, **kw)
    alone = gpu_ctx.job(sp)
    many = [gpu_ctx.job(sp) for _ in range(160)]
    for chunk in (7, 33):                      # a launch that starts between two rebuilds
        gpu_ctx.run([alone], chunk)
        gpu_ctx.run(many, chunk)
    assert alone.status() == 0 and alone.step() == 40
    ca, ra = alone.pairlist(False, cap=600)
    assert np.array_equal(alone.log(), many[0].log())
    for j in (many[0], many[-1]):
        assert j.status() == 0 and j.step() == 40
        for what in (sopb.COORDS, sopb.SEEDS, sopb.TEMP, sopb.TIPFORCES, sopb.PULLSTATE, sopb.TIPSTATE):
            assert np.array_equal(alone.read(what), j.read(what))
        cj, rj = j.pairlist(False, cap=600)
        assert np.array_equal(ca, cj) and np.array_equal(ra, rj)
    for j in [alone] + many:
        j.destroy()


@pytest.mark.parametrize("n", [25, 2047])
def test_cluster_lists_and_noise_match_oracle(gpu_ctx, n):
    sp = spec(n, 43, "clamp")
    g, o = gpu_ctx.job(sp), O.OracleJob(sp)
    gpu_ctx.run([g], 11)                       # rebuilds at 0 and 10
    assert o.advance(11) == 0
    assert np.array_equal(g.read(sopb.SEEDS), o.read(sopb.SEEDS))
    # one-step bound of the parity tests (1e-5 A) per step
    assert np.max(np.abs(g.read(sopb.COORDS) - o.read(sopb.COORDS))) < 11 * 1e-5
    g.rebuild(True, True)
    x = g.read(sopb.COORDS)
    o.write(sopb.COORDS, x)
    o.rebuild(True, True)
    cg, rg = g.pairlist(False)
    co, ro = o.pairlist(False)
    assert np.array_equal(cg, co) and np.array_equal(rg, ro)
    g.destroy()
