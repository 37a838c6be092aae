"""The Boys evaluation of the Obara-Saika and nuclear-attraction kernels
(boys_fm in csrc/pfk_os.cuh) restated with the tables the kernels include
(csrc/boys_table_data.inc) and checked against 40-digit values (CPU test).

Bound: a fused multiply-add chain whose terms add up to about the result
leaves 1 to 2 units of 2^-53 relative, the reciprocal square root and the
factors around it another 2: 5e-16 for F_0.  An upward step multiplies the
relative error by (2m+1) F_m / (2T F_{m+1}), largest at T = TS, adds that of
e^-T (3e-16) times e^-T / (2T F_{m+1}), and that of h = 1/(2T) = 0.5 r (s r T):
r enters twice (its argument's two roundings halved and its own: 2.2e-16
each time) and four roundings follow, the product's included: 6e-16.  The next
steps multiply all of it in turn."""
import importlib
import math
import os
import re

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")
special = pytest.importorskip("scipy.special")

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "planck-refactored_b200", "csrc")


def _tables():
    text = open(os.path.join(CSRC, "boys_table_data.inc")).read()
    out = {}
    for name, body in re.findall(r"(\w+)\[[^=;]*\] = (\{.*?\});", text, re.S):
        rows = re.findall(r"\{([^{}]*)\}", body)
        vals = [[float(v) for v in r.split(",") if v.strip()] for r in rows]
        out[name] = vals if len(vals) > 1 else vals[0]
    return out


T_ = _tables()
SHIFT = 16.0


def _fma(a, b, c):
    return float(np.float64(np.longdouble(a) * np.longdouble(b) + np.longdouble(c)))


def _horner(c, x):
    s = c[-1]
    for v in c[-2::-1]:
        s = _fma(s, x, v)
    return s


def _even_odd(c, x):
    return _fma(_horner(c[1::2], x * x), x, _horner(c[0::2], x * x))


def _rsqrt(v):
    return float(1 / mpmath.sqrt(mpmath.mpf(v)))


def _exp(t):
    n = float(np.rint(-t * 1.4426950408889634074))
    r = _fma(n, -5.497923018708371174712471e-14, _fma(n, -0.693147180559890330187045037746429443359375, -t))
    return math.ldexp(_even_odd(T_["kBoysExp"], r), int(n))


def boys(M, T):
    ts, ta, scale = T_["kBoysTS"][M], T_["kBoysTA"][M], T_["kBoysMidScale"][M]
    mid = T_["kBoysMid"][M][:int(T_["kBoysMidDeg"][M]) + 1]
    small = T_["kBoysSmall"][M][:int(T_["kBoysSmallDeg"][M]) + 1]
    near, s = T < ta, T + SHIFT
    if M == 0:
        rs = _rsqrt(s if near else T)
        return [(_even_odd(mid, _fma(T * (rs * rs), scale, -1.0)) if near else 0.88622692545275801365) * rs]
    F = [0.0] * (M + 1)
    if near and T < ts:
        e = _exp(T)
        F[M] = _even_odd(small, T - 0.5 * ts)
        for m in range(M - 1, -1, -1):
            F[m] = _fma(2.0 * T, F[m + 1], e) * (1.0 / (2 * m + 1))
        return F
    r = _rsqrt(T * T * s if near else T)
    if near:
        e, rs = _exp(T), r * T
        h = 0.5 * r * (s * rs)
        F[0] = rs * (_even_odd if M <= 4 else _horner)(mid, _fma(T * (rs * rs), scale, -1.0))
        for m in range(M):
            F[m + 1] = _fma(2 * m + 1.0, F[m], -e) * h
    else:
        F[0] = 0.88622692545275801365 * r
        for m in range(M):
            F[m + 1] = (2 * m + 1) * (0.5 * r * r) * F[m]
    return F


def _exact(m, t):
    a = m + mpmath.mpf(1) / 2
    return 1 / (2 * a) if t < 1e-30 else mpmath.gammainc(a, 0, t) / (2 * t ** a)


def _bound(M):
    err, t = 5e-16, mpmath.mpf(T_["kBoysTS"][M])
    for m in range(M):
        up = float((2 * m + 1) * _exact(m, t) / (2 * t * _exact(m + 1, t)))
        err = err * up + 3e-16 * (up - 1) + 6e-16     # e^-T = (up - 1) 2T F_{m+1}
    return err


@pytest.mark.parametrize("M", range(7))
def test_relative_error(M):
    rng = np.random.default_rng(50 + M)
    ts, ta = T_["kBoysTS"][M], T_["kBoysTA"][M]
    Ts = np.concatenate([rng.uniform(0, 3, 100), rng.uniform(0, 80, 150), rng.uniform(ta - 3, ta + 3, 40),
                         np.logspace(-300, 3, 30),
                         [0.0, ts * (1 - 1e-15), ts, ts * (1 + 1e-15), ta * (1 - 1e-15), ta]])
    worst = 0.0
    with mpmath.workdps(40):
        for T in Ts:
            F, t = boys(M, float(T)), mpmath.mpf(float(T))
            for m in range(M + 1):
                ref = _exact(m, t)
                worst = max(worst, float(abs((F[m] - ref) / ref)))
    assert worst < _bound(M), (worst, _bound(M))


def test_tables_are_the_generators():
    """The committed table is what gen_boys_table.py writes."""
    g = importlib.import_module("planck-refactored_b200.gen_boys_table")
    t = g.tables()
    for M in range(7):
        assert T_["kBoysMid"][M][:g.MID_DEG[M] + 1] == t["mid"][M]
        assert T_["kBoysSmall"][M][:g.SMALL_DEG[M] + 1] == t["small"][M]
    assert T_["kBoysExp"] == t["exp"] and T_["kBoysMidScale"] == t["mid_scale"]
    assert T_["kBoysTA"] == g.TA and T_["kBoysTS"] == g.TS


def _former(M, T):
    """The scheme the polynomials replaced, with the C library's exp and
    scipy's erfcx: the Taylor series of F_M and downward recursion below 1, 2
    or 3, F_0 = sqrt(pi)/2 (1 - e^-T erfcx(sqrt T)) / sqrt T and upward
    recursion above, the large-T limit from TA on."""
    ts, nt = (1.0, 18) if M <= 1 else (2.0, 25) if M <= 4 else (3.0, 32)
    F = [0.0] * (M + 1)
    if T < ts:
        s = 0.0
        for k in range(nt - 1, -1, -1):
            s = s * T + (-1) ** k / (math.factorial(k) * (2 * M + 2 * k + 1))
        F[M], e = s, math.exp(-T)
        for m in range(M - 1, -1, -1):
            F[m] = (2.0 * T * F[m + 1] + e) * (1.0 / (2 * m + 1))
        return F
    ist, near = 1.0 / math.sqrt(T), T < T_["kBoysTA"][M]
    e = math.exp(-T) if near else 0.0
    F[0] = 0.88622692545275801365 * (1.0 - e * special.erfcx(T * ist) if near else 1.0) * ist
    h = 0.5 * ist * ist
    for m in range(M):
        F[m + 1] = ((2 * m + 1) * F[m] - e) * h
    return F


@pytest.mark.parametrize("M", range(7))
def test_no_less_accurate_than_the_former_scheme(M):
    """Largest errors over points that lie densest just above either scheme's
    switch to the upward recursion, where it amplifies most, and in the small
    range.  One unit of 2^-53 for the sample at M = 0, whose errors are two to
    four of them on either side."""
    rng = np.random.default_rng(70 + M)
    ts, ta, old = T_["kBoysTS"][M], T_["kBoysTA"][M], 1.0 if M <= 1 else 2.0 if M <= 4 else 3.0
    Ts = np.concatenate([rng.uniform(ts, ts + 0.3, 500), rng.uniform(old, old + 0.3, 500), rng.uniform(0, ts, 150),
                         rng.uniform(ts, ts + 3, 150), rng.uniform(ts, ta, 150), rng.uniform(ta, ta + 3, 50)])
    new = former = 0.0
    with mpmath.workdps(30):
        for T in map(float, Ts):
            ref = [_exact(m, mpmath.mpf(T)) for m in range(M + 1)]
            err = [max(abs(float((f - r) / r)) for f, r in zip(F, ref)) for F in (boys(M, T), _former(M, T))]
            new, former = max(new, err[0]), max(former, err[1])
    print(f"M = {M}: {new:.2e}, former scheme {former:.2e}")
    assert new <= former + (1.2e-16 if M == 0 else 0.0), (new, former)
