"""Rebuilding a resident job's lists by a call, which a cluster of CTAs shares (one
CTA below 64 beads, four, then eight from 256 on): rows equal the oracle's for
either list and both, the run that follows is the same as without the calls, near
rows that overflow in one CTA's share alone count for all (a job whose first
beads crowd), rows that do not fit the shared memory of a cluster's CTAs, and the
forces over several CTAs are the oracle's."""
import numpy as np
import pytest

import oracle_py as O
import sopb
from helpers import FORCE_RTOL, force_error, plain_params, spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 63, 64, 65, 255, 256, 257, 601, 2047])
def test_rebuild_calls(gpu_ctx, n):
    sp = spec(n, 17, "clamp", pairs_threshold=40.0)
    g, h, o = gpu_ctx.job(sp), gpu_ctx.job(sp), O.OracleJob(sp)
    gpu_ctx.run([g, h], 20)                    # ends before the rebuild at step 20
    x = g.read(sopb.COORDS)
    o.write(sopb.COORDS, x)
    for possible, verlet in ((True, False), (False, True), (True, True)):
        g.rebuild(possible, verlet)
        o.rebuild(possible, verlet)
        for which in (True, False):
            cg, rg = g.pairlist(which)
            co, ro = o.pairlist(which)
            if verlet or which:
                assert np.array_equal(cg, co) and np.array_equal(rg, ro)
    f32, f64, a64 = o.forces()
    assert force_error(g.read(sopb.FORCES), f64, a64) <= FORCE_RTOL
    h.rebuild(True, True)
    gpu_ctx.run([g], 25)
    gpu_ctx.run([h], 25)
    assert g.status() == h.status() == 0
    assert np.array_equal(g.read(sopb.COORDS), h.read(sopb.COORDS))
    g.destroy()
    h.destroy()


def crowd(n, dense, room, skin):
    """n free beads: the first `dense` in a ball of 40 A, the others far apart."""
    rng = np.random.default_rng(3)
    u = rng.normal(size=(dense, 3))
    ball = u / np.linalg.norm(u, axis=1, keepdims=True) * 40.0 * rng.random((dense, 1)) ** (1.0 / 3.0)
    k = np.arange(n - dense)
    rest = np.stack([300.0 + 100.0 * (k % 10), 100.0 * (k // 10 % 10), 100.0 * (k // 100)], 1)
    x = np.concatenate([ball, rest]).astype(np.float32)
    p = plain_params(el=0.0, max_pairs=room, pairs_threshold=70.0, verlet_skin=skin)
    return sopb.JobSpec(x, np.zeros((0, 2)), [], np.zeros((0, 2)), [], [], p, seed=5)


def test_near_rows_that_overflow_in_one_share(gpu_ctx):
    # near rows hold four times max_pairs; a bead in the middle of the ball has all
    # others near at a skin of 40 A, an eighth of them within the cutoff; the last
    # CTAs of the cluster have none
    n, dense = 640, 400
    probe = gpu_ctx.job(crowd(n, dense, n - 1, -1.0))
    probe.rebuild(True, True)
    room = int(probe.pairlist(False)[0].max()) + 10
    probe.destroy()
    assert 4 * room < dense - 1
    jobs = [gpu_ctx.job(crowd(n, dense, room, s)) for s in (-1.0, 0.0, 40.0)]
    many = [gpu_ctx.job(crowd(n, dense, room, 40.0)) for _ in range(160)]
    for c in (5, 30):
        for j in jobs:
            gpu_ctx.run([j], c)
        gpu_ctx.run(many, c)
    for j in jobs[1:] + many[:2]:
        assert j.status() == jobs[0].status() == 0
        assert np.array_equal(j.read(sopb.COORDS), jobs[0].read(sopb.COORDS))
        assert all(np.array_equal(a, b) for a, b in zip(j.pairlist(False), jobs[0].pairlist(False)))
    for j in jobs + many:
        j.destroy()


@pytest.mark.parametrize("skin", [-1.0, 0.0])
def test_rows_beyond_shared_memory_in_a_cluster(gpu_ctx, skin):
    # every bead a partner: 64 rows of 2000 entries per CTA of sixteen, of which its
    # shared memory holds less than half
    n = 2048
    sp = spec(n, 41, "clamp", pairlist_cutoff=300.0, pairs_threshold=400.0, max_pairs=n - 1, verlet_skin=skin)
    g, o = gpu_ctx.job(sp), O.OracleJob(sp)
    many = [gpu_ctx.job(sp) for _ in range(130)]
    for c in (3, 9):                           # a launch that loads its rows, and rebuilds
        gpu_ctx.run([g], c)
        gpu_ctx.run(many, c)
        assert o.advance(c) == 0
    assert g.status() == many[0].status() == 0
    assert g.pairlist(False, cap=8)[0].min() > 1900
    # one-step bound of the parity tests (1e-5 A) per step
    assert np.max(np.abs(g.read(sopb.COORDS) - o.read(sopb.COORDS))) < 12 * 1e-5
    for j in (many[0], many[-1]):
        assert np.array_equal(g.read(sopb.COORDS), j.read(sopb.COORDS))
    for j in [g] + many:
        j.destroy()
