"""The autotuner times the HI policy on exact-HI jobs above 128 beads alone: TEA and
smaller exact jobs do not depend on it, so a mix without them leaves it as it was
instead of taking one of equal candidates by chance."""
import sopb_autotune as A
from helpers import spec

EXACT = dict(hi_on=1, hi_exact=1, hi_a=1.9, hi_capricious=0)
TEA = dict(hi_on=1, hi_a=1.9, hi_epsilon_freq=10, hi_capricious=0)


class Context:
    def __init__(self):
        self.hi, self.shape = [], []

    def set_hi_policy(self, *p):
        self.hi.append(p)

    def set_shape_policy(self, *p):
        self.shape.append(p)


def tuned(monkeypatch, specs):
    seen = []
    monkeypatch.setattr(A, "time_hi_policy", lambda ctx, s, pol, *a: seen.append([x.n for x in s]) or float(pol[0]))
    monkeypatch.setattr(A, "time_policy", lambda ctx, s, pol, *a: float(pol[0]))
    ctx = Context()
    return ctx, A.autotune(ctx, specs), seen


def test_mix_without_large_exact_jobs_keeps_the_hi_policy(monkeypatch):
    ctx, out, seen = tuned(monkeypatch, [spec(40, 1), spec(300, 2, **TEA), spec(128, 3, **EXACT)])
    assert ctx.hi == [] and seen == [] and out["hi_policy"] is None and out["hi_table"] == []
    assert ctx.shape[-1] == out["policy"]


def test_hi_policy_is_tuned_on_the_largest_exact_job(monkeypatch):
    ctx, out, seen = tuned(monkeypatch, [spec(300, 2, **TEA), spec(129, 3, **EXACT), spec(200, 4, **EXACT)])
    assert all(s == [200] for s in seen) and len(seen) == len(A.DEFAULT_HI_CANDIDATES)
    assert ctx.hi == [out["hi_policy"]] and out["hi_policy"][0] == 2
