"""Runs that share the GPU -- several streams at once, or more jobs than SMs, with
and without a few large ones -- plan other clusters than a job alone gets, and
again others once they were seen beside one another; the results stay those of a
job alone, bit for bit, over repeated runs."""
import numpy as np
import pytest

import sopb
from helpers import spec

pytestmark = pytest.mark.gpu

SIZES = [60, 97, 150, 203, 301, 450, 600]


def alone(ctx, sizes, chunks):
    out = []
    for n in sizes:
        j = ctx.job(spec(n, 9, "clamp"))
        for c in chunks:
            ctx.run([j], c)
        out.append((j.status(), j.read(sopb.COORDS), j.read(sopb.TEMP)))
        j.destroy()
    return out


@pytest.mark.parametrize("nstreams,per", [(2, 7), (4, 10), (8, 20)])
def test_streams_side_by_side(gpu_ctx, nstreams, per):
    import torch
    chunks = (13, 20, 7)
    ref = alone(gpu_ctx, SIZES, chunks)
    streams = [torch.cuda.Stream() for _ in range(nstreams)]
    groups = [[gpu_ctx.job(spec(SIZES[(k + q) % len(SIZES)], 9, "clamp")) for k in range(per)] for q in range(nstreams)]
    for c in chunks:
        for s, g in zip(streams, groups):
            gpu_ctx.run(g, c, stream=s.cuda_stream)
    torch.cuda.synchronize()
    for q, g in enumerate(groups):
        for k, j in enumerate(g):
            st, x, t = ref[(k + q) % len(SIZES)]
            assert j.status() == st == 0
            assert np.array_equal(j.read(sopb.COORDS), x) and np.array_equal(j.read(sopb.TEMP), t)
            j.destroy()


@pytest.mark.parametrize("large,small", [(0, 119), (1, 148), (8, 140), (100, 100)])
def test_more_jobs_than_sms(gpu_ctx, large, small):
    chunks = (13, 20)
    ref = alone(gpu_ctx, (450, 97), chunks)
    jobs = [gpu_ctx.job(spec(450 if k < large else 97, 9, "clamp")) for k in range(large + small)]
    for c in chunks:
        gpu_ctx.run(jobs, c)
    for k, j in enumerate(jobs):
        st, x, t = ref[0 if k < large else 1]
        assert j.status() == st == 0
        assert np.array_equal(j.read(sopb.COORDS), x) and np.array_equal(j.read(sopb.TEMP), t)
        j.destroy()
