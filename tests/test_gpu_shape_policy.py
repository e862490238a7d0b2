"""The shape policy's limit on CTA sizes and its beads per lane group hold for the
CTAs of clusters too, and change no result: alone (a cluster) and in a batch (one
CTA), from the smallest CTA on, bit for bit those of the default policy."""
import numpy as np
import pytest

import sopb
from helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bpg,most", [(1.0, 64), (1.0, 100), (2.0, 1024), (5.0, 256), (0.0, 512)])
def test_policy_changes_no_result(gpu_ctx, bpg, most):
    sizes = (25, 203, 601, 2047)
    gpu_ctx.set_shape_policy()
    ref = [gpu_ctx.job(spec(n, 19, "clamp")) for n in sizes]
    gpu_ctx.set_shape_policy(4, bpg, most)
    try:
        jobs = [gpu_ctx.job(spec(n, 19, "clamp")) for n in sizes]
        many = [gpu_ctx.job(spec(203, 19, "clamp")) for _ in range(160)]
    finally:
        gpu_ctx.set_shape_policy()
    for c in (11, 20):
        for j in ref + jobs:
            gpu_ctx.run([j], c)
        gpu_ctx.run(many, c)
    for a, b in list(zip(ref, jobs)) + [(ref[1], many[0]), (ref[1], many[-1])]:
        assert a.status() == b.status() == 0
        for what in (sopb.COORDS, sopb.SEEDS, sopb.TEMP):
            assert np.array_equal(a.read(what), b.read(what))
    mixed = [j for pair in zip(ref, jobs) for j in pair]      # both policies in one run
    gpu_ctx.run(mixed, 10)
    for a, b in zip(ref, jobs):
        assert np.array_equal(a.read(sopb.COORDS), b.read(sopb.COORDS))
    for j in ref + jobs + many:
        j.destroy()
