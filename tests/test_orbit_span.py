"""The time span that the checks of t(f) compare with is the orbit tables' own at the time of the
call, not a copy taken when the orbits were set."""
import numpy as np


def test_span_follows_the_tables():
    from bbhx_b200 import EqualArmlengthOrbits, LISATDIResponse

    resp = LISATDIResponse.__new__(LISATDIResponse)
    resp.orbits = EqualArmlengthOrbits(dt=1e5, t_max_years=1.0)
    t = resp.orbits.t_base
    assert resp.t_span == (0.0, float(t[-1]))
    resp.orbits.t_base = t[:50] + 10.0
    assert resp.t_span == (10.0, float(t[49]) + 10.0)
    resp.orbits.t_base *= 0.5
    assert resp.t_span == (5.0, 0.5 * (float(t[49]) + 10.0))
    resp.orbits = EqualArmlengthOrbits(dt=1e5, t_max_years=2.0)
    assert resp.t_span[1] == float(resp.orbits.t_base[-1])
