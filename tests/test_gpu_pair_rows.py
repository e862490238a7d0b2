"""Rows per pair of beads, merged from the possible rows of both (grid path
without hydrodynamics): entry for entry the oracle's, whichever way they were
made -- from near rows, from the possible rows (no skin), or with near rows that
overflow (where a later rebuild does not try again until the possible pairs are
new); possible rows and partners beyond what a warp keeps in shared memory (512),
odd bead counts, and both sides of the line between the step's group widths
(14208 beads).  Rows and the trajectories over them are equal bit for bit.  More
partners than max_pairs is an error."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import spec

pytestmark = pytest.mark.gpu

FAR = dict(pairs_threshold=70.0, max_possiblePairs=6001, max_pairs=300)
CASES = {
    "one_pair": (2, dict(grid_path=1)),
    "odd_small": (301, dict(grid_path=1)),
    "far": (6001, FAR),
    "long_rows": (3001, dict(pairlist_cutoff=45.0, pairs_cutoff=45.0, pairs_threshold=60.0, max_possiblePairs=3000,
                             max_pairs=3000)),
    "wide_last": (14208, dict(pairs_threshold=30.0, max_possiblePairs=2048, max_pairs=512)),
    "narrow_first": (14209, dict(pairs_threshold=30.0, max_possiblePairs=2048, max_pairs=512)),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_rows_do_not_depend_on_how_they_were_made(gpu_ctx, case):
    n, kw = CASES[case]
    freq = dict(nav=100, pairs_freq=10, possiblepairs_freq=20)
    # no near rows; the usual ones; ones that overflow where the row capacity allows it
    jobs = [gpu_ctx.job(spec(n, 7, "clamp", verlet_skin=s, **freq, **kw)) for s in (-1.0, 0.0, 40.0)]
    lists = []
    for steps in (1, 10, 34):                 # rebuilds at 0; 10; 20 (new possible pairs), 30, 40
        gpu_ctx.run(jobs, steps)
        assert [j.status() for j in jobs] == [0, 0, 0]
        x = [j.read(sopb.COORDS) for j in jobs]
        rows = [j.pairlist(False, cap=min(n, 3000)) for j in jobs]
        for k in (1, 2):
            assert np.array_equal(x[k], x[0])
            assert np.array_equal(rows[k][0], rows[0][0]) and np.array_equal(rows[k][1], rows[0][1])
        lists.append(rows[0][0])
    if case == "far":
        assert jobs[0].pairlist(True, cap=6001)[0].mean() > 3 * 512
    if case == "long_rows":
        assert lists[0].max() > 512
    # at the same coordinates the oracle's rows
    o = O.OracleJob(spec(n, 7, "clamp", **freq, **kw))
    o.write(sopb.COORDS, x[0])
    o.rebuild(True, True)
    co, ro = o.pairlist(False, cap=min(n, 3000))
    for j in jobs:
        j.rebuild(True, True)
        cg, rg = j.pairlist(False, cap=min(n, 3000))
        assert np.array_equal(cg, co) and np.array_equal(rg, ro)
        j.destroy()


@pytest.mark.parametrize("skin", [-1.0, 0.0])
@pytest.mark.parametrize("n", [2500, 14300])
def test_more_partners_than_max_pairs(gpu_ctx, n, skin):
    base = dict(pairs_threshold=30.0, max_possiblePairs=2048, verlet_skin=skin)
    j = gpu_ctx.job(spec(n, 7, "clamp", max_pairs=512, **base))
    j.rebuild(True, True)
    most = int(j.pairlist(False)[0].max())
    j.destroy()
    for room, status in ((most, 0), (most - 1, 2)):
        j = gpu_ctx.job(spec(n, 7, "clamp", max_pairs=room, **base))
        gpu_ctx.run([j], 1)
        assert j.status() == status
        j.destroy()
