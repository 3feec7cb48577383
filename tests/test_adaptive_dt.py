"""The adaptive time step, whose common case skips the divisions, against the rule
written out, over ordinary and odd values of everything it takes."""
import itertools
import math
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from phasefield5d_b200 import _lib
    if not os.path.exists(_lib.LIB_PATH):
        subprocess.run(["make", "-s", "-C", os.path.join(REPO, "phasefield5d_b200", "csrc")], check=True)
    return _lib.load(require_cuda=False)


def _div(a, b):
    try:
        return a / b
    except ZeroDivisionError:
        return math.nan if a == 0 or a != a else math.copysign(math.inf, a)


def _rule(dt, xdotmax, ctld, t_cfl, lower, upper, factor):
    raw = dt
    if not xdotmax <= 0.0:
        lo, hi = _div(lower, xdotmax), _div(upper, xdotmax)
        if lo > hi:
            lo, hi = hi, lo
        if raw < lo:
            raw = lo
        if raw > hi:
            raw = hi
    m = dt * factor
    for bound in (raw, 0.005 * ctld, t_cfl):
        if bound < m:
            m = bound
    return m


def test_equals_the_rule(lib):
    nan, inf = math.nan, math.inf
    dts = [1e-12, 1e-9, 3e-7, 0.0, nan, inf]
    rates = [0.0, -1.0, 1e-300, 1e2, 7e8, 1e11, 1e300, nan, inf]
    caps = [1e-9, 5e-6, nan, inf]
    limits = [1e-5, 1e-3, 2.5e-4, 0.0, -1e-5, nan, inf]
    for dt, x, ctld, cfl, lo, hi, f in itertools.product(dts, rates, caps, caps, limits, limits,
                                                         [2.0, 1.0, 0.5]):
        got, want = lib.pf5d_adaptive_dt(dt, x, ctld, cfl, lo, hi, f), _rule(dt, x, ctld, cfl, lo, hi, f)
        assert got == want or (got != got and want != want), (dt, x, ctld, cfl, lo, hi, f, got, want)
