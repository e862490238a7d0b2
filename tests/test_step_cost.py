"""The serving loop's first estimate of a grid job's step time against step times
measured alone on a B200 (microseconds, 10 to 200 steps, list rebuilds included).
Within 40 %: it only sizes a job's first quantum and orders jobs until their own
quanta have been timed."""
import types

import pytest

import sopb_serve

MEASURED = [
    # beads, exact, refresh (None: no hydrodynamics), us per step
    (2500, None, None, 8.7), (6000, None, None, 9.8), (12000, None, None, 10.5), (18000, None, None, 13.4),
    (40000, None, None, 19.4), (198000, None, None, 102.0),
    (50, 0, 1, 10.3), (517, 0, 1, 14.4), (1100, 0, 1, 15.8), (4000, 0, 1, 43.6), (12000, 0, 1, 219.0),
    (40, 1, 1, 34.5), (90, 1, 1, 79.0), (128, 1, 1, 112.7), (128, 1, 10, 25.7),
    (129, 1, 1, 332.0), (129, 1, 10, 57.0), (601, 1, 5, 307.0), (4000, 1, 10, 1450.0),
]


@pytest.mark.parametrize("n,exact,refresh,us", MEASURED)
def test_first_estimate_of_a_step(n, exact, refresh, us):
    p = types.SimpleNamespace(hi_on=int(exact is not None), hi_exact=int(bool(exact)), hi_refresh=refresh or 1)
    got = sopb_serve.step_cost(types.SimpleNamespace(n=n, params=p))
    assert us / 1.4 <= got <= us * 1.4
