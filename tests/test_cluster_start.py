"""Cluster kernels store into another CTA's shared memory only after a barrier
that every CTA of the cluster has arrived at: before that the other CTA may not
have begun, and its shared memory is not there yet.  Read from the CUDA sources
on the CPU: in every kernel the first cluster wait stands before the first
remote store, in the kernel itself or in a function it calls."""
import os
import re

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "sop-gpu_b200", "csrc")
FILES = ("sopb_resident.cuh", "sopb_grid.cuh", "sopb_hi.cuh", "sopb_chol.cuh")
REMOTE = re.compile(r"st\.async|st\.[a-z.]*shared::cluster")      # stores to a peer's shared memory
WAIT = re.compile(r"barrier\.cluster\.wait")
HEAD = re.compile(r"(?:__global__|__device__)[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*\{")


def functions():
    """name -> (is a kernel, body without comments) of every device function."""
    out = {}
    for name in FILES:
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"//[^\n]*|__launch_bounds__\s*\([^()]*\)", "", f.read())
        for m in HEAD.finditer(src):
            depth, k = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[k], 0)
                k += 1
            out.setdefault(m.group(1), []).append(("__global__" in m.group(0), src[m.end():k - 1]))
    return out


def first_use(body, direct, helpers):
    """Position of the first match of `direct` or call of one of `helpers` (the
    instantiations for one CTA, <false>, left out)."""
    at = [m.start() for m in direct.finditer(body)]
    at += [m.start() for h in helpers for m in re.finditer(r"\b%s\s*(?:<(?!false)[^<>;()]*>)?\s*\(" % h, body)]
    return min(at, default=None)


def closure(fns, direct):
    """Device functions that use `direct` themselves or through others."""
    got = set()
    while True:
        new = {n for n, defs in fns.items() for kernel, body in defs
               if n not in got and not kernel and first_use(body, direct, got) is not None}
        if not new:
            return got
        got |= new


def late_waits(fns):
    """(kernels with remote stores, those that store before their first wait)."""
    senders, waiters = closure(fns, REMOTE), closure(fns, WAIT)
    found, bad = [], []
    for name, defs in fns.items():
        for kernel, body in defs:
            store = first_use(body, REMOTE, senders) if kernel else None
            if store is None:
                continue
            found.append(name)
            # a helper that does both (a rebuild) counts where it is called
            wait = first_use(body, WAIT, waiters - senders)
            if wait is None or wait > store:
                bad.append(name)
    return sorted(set(found)), bad


def test_cluster_kernels_wait_for_their_peers_first():
    found, bad = late_waits(functions())
    assert found == ["k_hi_small", "k_rebuild_lists", "k_resident_steps", "k_tea_eps", "k_tea_step"]
    assert bad == []


@pytest.mark.parametrize("body,ok", [
    ("cluster_arrive(); work(); cluster_wait(); send(p);", True),
    ("if (rank == 0) send(p); cluster_wait();", False),
    ("cluster_arrive(); send(p);", False),
])
def test_reader_tells_the_orders_apart(body, ok):
    fns = {"cluster_wait": [(False, 'asm volatile("barrier.cluster.wait.acquire;");')],
           "cluster_arrive": [(False, 'asm volatile("barrier.cluster.arrive.release;");')],
           "send": [(False, 'asm volatile("st.shared::cluster.u32 [%0], %1;");')],
           "k": [(True, body)]}
    assert (late_waits(fns) == (["k"], [])) == ok
