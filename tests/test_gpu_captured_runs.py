"""A run captured in a caller's CUDA graph launches from its stream's plan and table.
Runs of the same jobs outside the graph, beside runs on other streams (which make
such runs plan for a share of the GPU), leave both as they are: the graph's
replays go on advancing every job by its steps, as the jobs alone."""
import numpy as np
import pytest

import sopb
from helpers import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[200] * 10, [60, 203, 450, 97]])
def test_captured_run_keeps_its_plan(gpu_ctx, sizes):
    import torch
    jobs = [gpu_ctx.job(spec(n, 9, "clamp")) for n in sizes]
    others = [[gpu_ctx.job(spec(200, 9, "clamp")) for _ in range(10)] for _ in range(3)]
    s = torch.cuda.Stream()
    so = [torch.cuda.Stream() for _ in others]
    gpu_ctx.run(jobs, 10, stream=s.cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        gpu_ctx.run(jobs, 10, stream=s.cuda_stream)
    for _ in range(4):                         # side by side, the same call outside the graph
        for q, o in zip(so, others):
            gpu_ctx.run(o, 2000, stream=q.cuda_stream)
        gpu_ctx.run(jobs, 10, stream=s.cuda_stream)
    torch.cuda.synchronize()
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    steps = 10 + 4 * 10 + 2 * 10
    for n, j in zip(sizes, jobs):
        r = gpu_ctx.job(spec(n, 9, "clamp"))
        gpu_ctx.run([r], steps)
        assert j.status() == 0 and j.step() == r.step() == steps
        assert np.array_equal(j.read(sopb.COORDS), r.read(sopb.COORDS))
        r.destroy()
    del g
    for j in jobs + [k for o in others for k in o]:
        j.destroy()
