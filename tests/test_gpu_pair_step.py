"""The grid path's step over rows per pair of beads: both group widths on
either side of their boundary (24576 beads), odd sizes, rows that fit a CTA's
shared memory and rows that do not, an odd number of steps (which ends in the
other coordinate buffer) and rebuilds in between, against the oracle.

Tolerance: a step rounds each coordinate once, at most 3e-5 for coordinates
below 512, and the forces agree to 1e-5 of terms that move a bead by far less
than 1 A per step, so n steps stay within n * (6e-5 + 1e-5)."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import FORCE_RTOL, force_error, spec

pytestmark = pytest.mark.gpu

BASE = dict(pairs_threshold=30.0, max_possiblePairs=2048, max_pairs=512)
LONG = dict(pairlist_cutoff=32.0, pairs_cutoff=32.0, pairs_threshold=40.0, max_possiblePairs=4096, max_pairs=2048)
CASES = {
    "two_beads": (2, "free", dict(grid_path=1)),
    "three_beads": (3, "clamp", dict(grid_path=1)),
    "wide_odd": (2051, "clamp", BASE),
    "wide_last": (24576, "free", BASE),
    "narrow_first": (24577, "clamp", BASE),
    "narrow_full_tile": (24640, "free", BASE),
    "wide_long_rows": (2050, "clamp", LONG),
    "narrow_long_rows": (24579, "clamp", LONG),
    "wide_tip": (2049, "indent", BASE),
    "narrow_tip": (24581, "indent", BASE),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_pair_step_tracks_oracle(gpu_ctx, case):
    n, mode, kw = CASES[case]
    sp = spec(n, 7, mode, **kw)
    g, o = gpu_ctx.job(sp), O.OracleJob(sp)
    steps = 0
    for chunk in (1, 4, 8):
        gpu_ctx.run([g], chunk)
        assert o.advance(chunk) == 0
        steps += chunk
        assert g.status() == 0 and g.step() == steps
        assert np.array_equal(g.read(sopb.SEEDS), o.read(sopb.SEEDS))
        assert np.max(np.abs(g.read(sopb.COORDS) - o.read(sopb.COORDS))) <= 7e-5 * steps
    if case == "narrow_long_rows":
        assert g.pairlist(False, cap=2048)[0].mean() > 192      # longer than a CTA's share of shared memory
    g.destroy()


@pytest.mark.parametrize("case", ["narrow_first", "narrow_long_rows", "wide_odd"])
def test_pair_rows_equal_oracle(gpu_ctx, case):
    n, mode, kw = CASES[case]
    sp = spec(n, 7, mode, **kw)
    g, o = gpu_ctx.job(sp), O.OracleJob(sp)
    g.rebuild(True, True)
    o.rebuild(True, True)
    cg, rg = g.pairlist(False, cap=2048)
    co, ro = o.pairlist(False, cap=2048)
    assert np.array_equal(cg, co) and np.array_equal(rg, ro)
    f32, f64, a64 = o.forces()
    assert force_error(g.read(sopb.FORCES), f64, a64) <= FORCE_RTOL
    g.destroy()
