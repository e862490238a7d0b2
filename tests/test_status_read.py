"""Kernels whose job's status another CTA or stream may set while they run decide
as a CTA whether to go on.  A status read by each thread for itself may differ
within a warp, whose collectives (shuffles, votes, mma.sync) would then miss
lanes.  Read from the CUDA sources on the CPU: k_chol_potrf64 and k_chol_tc run
beside one another on several streams, and a CTA of k_g_step may give up its
copy of the rows while the others begin."""
import os
import re

import pytest

from conftest import REPO


def kernel(file, name):
    with open(os.path.join(REPO, "sop-gpu_b200", "csrc", file)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    m = re.search(r"\n%s\s*\([^;{}]*\)\s*\{" % name, src)
    depth, k = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        k += 1
    return src[m.end():k - 1]


# a return on a value that each thread read for itself
OWN_READ = re.compile(r"if\s*\((?:Jp->status|J\.status|status)\)\s*return")


@pytest.mark.parametrize("file,name", [("sopb_chol.cuh", "k_chol_potrf64"), ("sopb_chol.cuh", "k_chol_tc")])
def test_status_is_read_once_per_cta(file, name):
    body = kernel(file, name)
    assert not OWN_READ.search(body)
    assert re.search(r"if\s*\(tid\s*==\s*0\)\s*stop\s*=\s*Jp->status;\s*__syncthreads\(\);\s*if\s*\(stop\)\s*return;", body)


def test_grid_step_votes_on_the_status():
    body = kernel("sopb_grid.cuh", "k_g_step")
    assert not OWN_READ.search(body)
    # only the narrow variant sets the status, and it votes where it waits for its rows
    assert re.search(r"if\s*\(!__syncthreads_and\(\s*there\s*&&\s*!status\s*\)\)\s*\{", body)
    assert body.count("&Jp->status") == 1 and body.index("&Jp->status") < body.index("if (WIDE && status) return;")
