"""A cluster of the resident kernel gives up as a whole, checked on the CPU.

A CTA whose wait for its peers' coordinates runs out leaves the step loop while
another one may still be stepping, or stand at a barrier of an updater.  The
model below replays the kernel's barriers, sends and waits (k_resident_steps and
run_updaters in sop-gpu_b200/csrc/sopb_resident.cuh) for the CTAs of one cluster
in random interleavings, with CTAs that stall and waits that run out.  Whatever
happens, no CTA may store into the shared memory of one that has left, none may
wait for a barrier that cannot complete, and either all CTAs write their state
back or none does.  The rule that each CTA leaves for itself is the planted
mistake that the model has to find.  The model follows the source line by line;
a change there needs the same change here."""
import os
import random
import re

import pytest

from conftest import REPO

NEVER = 1 << 62


class Cluster:
    def __init__(self, C, chunks, whole, rng):
        self.C, self.chunks, self.whole, self.rng = C, chunks, whole, rng
        self.gave_up = [NEVER] * C              # per CTA: the step at which a chunk that was given up ends
        self.seen = [[set() for _ in range(C)] for _ in range(64)]   # step -> receiver -> senders
        self.gone, self.wrote = set(), {}
        self.arrived, self.passed = set(), 0    # of the current barrier; barriers completed
        self.bad = []

    def store(self, to, what):
        if to in self.gone:
            self.bad.append("%s stored into CTA %d, which has left" % (what, to))

    def barrier(self, r):
        mine = self.passed
        self.arrived.add(r)
        if len(self.arrived) == self.C:
            self.arrived, self.passed = set(), self.passed + 1
        while self.passed == mine:
            yield "wait"

    def cta(self, r):
        """One CTA; yields "wait" while it cannot go on, "go" otherwise."""
        others = [k for k in range(self.C) if k != r]
        yield from self.barrier(r)              # the mbarriers are ready
        step = s = 0
        timed_out = left = False
        for barriers, m in self.chunks:
            for b in range(barriers):           # the updaters of the boundary
                yield from self.barrier(r)
                if self.whole and b == 0 and self.gave_up[r] <= step:
                    left = True                 # that was the last barrier of a CTA that gave up
                    break
                yield "go"
                for k in others:
                    self.store(k, "an updater of CTA %d" % r)
            if left:
                break
            step += m
            for _ in range(m):
                yield "go"
                for k in others:                # integrate and send
                    self.store(k, "step %d of CTA %d" % (s, r))
                    self.seen[s][k].add(r)
                    if self.rng.random() < 0.2:
                        yield "go"
                while len(self.seen[s][r]) < self.C - 1:
                    yield "expire"
                    if self.expired == r:
                        self.expired = None
                        timed_out = True
                        break
                if timed_out:
                    break
                s += 1
            if timed_out:
                break
        if timed_out and self.whole:
            for k in range(self.C):
                self.store(k, "CTA %d giving up" % r)
                self.gave_up[k] = step
        if not left:
            yield from self.barrier(r)
        self.wrote[r] = self.gave_up[r] == NEVER if self.whole else True
        if not self.whole and timed_out:
            self.wrote[r] = "part"
        self.gone.add(r)

    expired = None


def play(seed, whole):
    rng = random.Random(seed)
    C = rng.choice([2, 4, 8])
    chunks = [(rng.choice([0, 0, 1, 2, 3]), rng.randint(1, 3)) for _ in range(rng.randint(1, 4))]
    cl = Cluster(C, chunks, whole, rng)
    run = {r: cl.cta(r) for r in range(C)}
    state = {r: "go" for r in run}
    slow = {r: rng.choice([1, 1, 1, 30]) for r in run}      # a stalled CTA runs rarely
    idle = 0
    while run and not cl.bad:
        ready = [r for r in run if state[r] == "go"] or list(run)
        r = rng.choices(ready, [1.0 / slow[k] for k in ready])[0] if rng.random() < 0.7 else rng.choice(list(run))
        if state[r] == "expire" and rng.random() < (0.03 if idle < 50 * C else 1.0):
            cl.expired = r                       # its wait runs out (in the end every one does)
        before = (cl.passed, len(cl.arrived), len(cl.gone), sum(len(x) for q in cl.seen for x in q))
        try:
            state[r] = next(run[r])
        except StopIteration:
            del run[r]
        after = (cl.passed, len(cl.arrived), len(cl.gone), sum(len(x) for q in cl.seen for x in q))
        idle = 0 if before != after or state[r] == "go" else idle + 1
        if idle > 2000 * C:
            cl.bad.append("CTAs %s wait for ever" % sorted(run))
    if not cl.bad and len(set(cl.wrote.values())) > 1:
        cl.bad.append("state of different steps: %s" % cl.wrote)
    return cl


def test_a_cluster_gives_up_as_a_whole():
    failed = finished = 0
    for seed in range(400):
        cl = play(seed, True)
        assert cl.bad == [], (seed, cl.bad)
        failed += not all(cl.wrote.values())
        finished += all(cl.wrote.values())
    assert failed > 50 and finished > 50       # both ends were reached


def test_ctas_that_leave_alone_are_caught():
    kinds = set()
    for seed in range(400):
        for what in play(seed, False).bad:
            kinds.add("store" if "stored" in what else ("hang" if "wait" in what else "mixed"))
    assert {"store", "mixed"} <= kinds


def body(src, name):
    m = re.search(r"\b%s\s*\([^;{}]*\)\s*\{" % name, src)
    depth, k = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        k += 1
    return src[m.end():k - 1]


def test_the_kernel_follows_the_model():
    with open(os.path.join(REPO, "sop-gpu_b200", "csrc", "sopb_resident.cuh")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    src = re.sub(r"__launch_bounds__\s*\([^()]*\)", "", src)
    # the first barrier of a boundary, whichever updater has it, looks whether a peer gave up
    for fn in ("run_updaters", "rebuild_verlet"):
        assert re.search(r"cluster_sync_all|peers_meet", body(src, fn)).group(0) == "peers_meet", fn
    kernel = body(src, "k_resident_steps")
    # nothing is written back before the last barrier
    last = kernel.rindex("cluster_wait()")
    for write in ("J.x[i] =", "J.seeds[i] =", "J.T[i] =", "Jp->step ="):
        assert kernel.index(write) > last, write
