"""log_t32 and exp_t32 (afmm2d_b200/csrc/fast_math.cuh): their tables against the values they stand for, their
steps restated in Python (exact FMA through fractions) against 50-digit values over the whole range of doubles,
and the library's own entries against an 80-bit logarithm."""
import math
import os
import re
import struct
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np
import pytest

from test_fast_math import _exp_table, _table, log_tang

CSRC = os.path.join(os.path.dirname(__file__), "..", "afmm2d_b200", "csrc")
# u and the leading sum are exact up to terms below 2^-63 relative to the result's binade: half an ulp, and
# 2^-60 (the last additions of the small terms) and the polynomial's 2^-59.6 of u beside it
LOG_ULPS = 0.53


def _double(hi, lo=0):
    return struct.unpack("<d", struct.pack("<Q", hi << 32 | lo))[0]


def _words(name):
    s = open(os.path.join(CSRC, "math_tables.cuh")).read()
    s = s[s.index(name + "["):]
    rows = re.findall(r"\{((?:0x[0-9a-f]{8}u(?:, )?){32})\}", s[:s.index("};")])
    return [[int(w[:-1], 16) for w in r.split(", ")] for r in rows]


def log_tables():
    s = open(os.path.join(CSRC, "math_tables.cuh")).read()
    w = _words("kLogT32")
    assert len(w) == 4
    T = [(_double(w[0][j]), _double(w[1][j], w[2][j]), _double(w[3][j])) for j in range(32)]
    Q = [float.fromhex(x) for _, x in sorted(re.findall(r"kLogQ(\d) = (\S+);", s))]
    return T, Q, _table()[2:]


def exp_tables():
    w = _words("kExpT32")
    assert len(w) == 3
    return [(_double(w[0][j], w[1][j]), _double(w[2][j])) for j in range(32)], _exp_table()[1]


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def log_t32(x, tables):
    """The device function's operations in IEEE double, one rounding each."""
    T, Q, (l2h, l2l) = tables
    b = struct.unpack("<Q", struct.pack("<d", x))[0]
    hx, lx = b >> 32, b & 0xffffffff
    t = hx + 0x4000
    j = (t >> 15) & 31
    m = _double(hx - ((t & 0xfff00000) - 0x3ff00000), lx)
    kd = float((t >> 20) - 1023)
    c, Lh, Ll = T[j]
    u = _fma(m, c, -1.0)
    assert Fraction(u) == Fraction(m) * Fraction(c) - 1
    hi, lo = _fma(kd, l2h, Lh), _fma(kd, l2l, Ll)
    assert Fraction(hi) == Fraction(kd) * Fraction(l2h) + Fraction(Lh)
    q = Q[-1]
    for k in reversed(Q[:-1]):
        q = _fma(q, u, k)
    s = hi + u
    return s + ((u - (s - hi)) + _fma(q, u * u, lo))


def exp_t32(x, tables):
    S, c = tables
    shifter = 6755399441055744.0
    nd = _fma(x, c["k32OverLn2"], shifter) - shifter
    N = int(nd)
    r = _fma(-nd, c["kLn2Over32Lo"], _fma(-nd, c["kLn2Over32Hi"], x))
    hi, lo = S[N & 31]
    q = 1.0 / 720.0
    for k in (1.0 / 120.0, 1.0 / 24.0, 1.0 / 6.0, 0.5):
        q = _fma(q, r, k)
    p = _fma(q * r, r, r)
    v = hi + _fma(hi, p, _fma(lo, p, lo))
    return 0.0 if x < -708.0 else v * 2.0 ** (N >> 5)


def _log_error(y, x):
    """|y - ln x| in ulps of the rounded value."""
    getcontext().prec = 50
    L = Decimal(x).ln()
    return abs(float((Decimal(y) - L) / Decimal(math.ulp(float(L))))) if L else abs(y)


def test_log_table_entries():
    T, Q, _ = log_tables()
    getcontext().prec = 60
    largest = Fraction(0)
    for j, (c, Lh, Ll) in enumerate(T):
        assert (Fraction(c) * 64).denominator == 1 or (Fraction(c) * 128).denominator == 1
        assert (Fraction(Lh) * 2 ** 42).denominator == 1
        assert abs(Decimal(Lh) + Decimal(Ll) + Decimal(c).ln()) < Decimal(2) ** -63
        lo, hi = Fraction(2 * (32 + j) - 1, 64), Fraction(2 * (32 + j) + 1, 64)
        u = max(abs(lo * Fraction(c) - 1), abs(hi * Fraction(c) - 1))
        assert u <= (Fraction(1, 32) if (Fraction(c) * 64).denominator == 1 else Fraction(1, 64))
        largest = max(largest, u)
    assert T[0] == (1.0, 0.0, 0.0) and len(Q) == 8
    # (ln(1+u) - u)/u^2 over the polynomial's interval: its Chebyshev remainder h^8 / (10 2^7), and the
    # coefficients' own roundings
    h = Decimal(largest.numerator) / Decimal(largest.denominator)
    for i in range(-64, 65):
        u = h * i / 64
        if i == 0:
            continue
        g = ((1 + u).ln() - u) / (u * u)
        p = sum(Decimal(q) * u ** k for k, q in enumerate(Q))
        assert abs(p - g) < Decimal("1.1") * h ** 8 / 1280 + Decimal(2) ** -54


def test_exp_table_entries():
    S, _ = exp_tables()
    getcontext().prec = 60
    for j, (hi, lo) in enumerate(S):
        v = Decimal(2) ** (Decimal(j) / 32)
        assert hi == float(v)
        assert abs(Decimal(hi) + Decimal(lo) - v) <= abs(v - Decimal(hi)) * Decimal(2) ** -20


def _log_arguments():
    rng = np.random.default_rng(3)
    xs = list(np.exp(rng.uniform(math.log(1e-10), math.log(8.0), 2500)))    # squared distances
    xs += list(np.exp(rng.uniform(-700, 700, 1000)))                        # the whole normal range
    xs += list(rng.uniform(0.9, 1.12, 2500))                                # small logarithms
    xs += [1.0 + d for d in rng.uniform(-2 ** -7, 2 ** -7, 500)]
    xs += [np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), 2.0, 0.5, 1e-10, 2.0 ** -1022, 1.0172843348240832]
    xs += [(1.0 + (j + 0.5) / 32) * (1 + s * 2 ** -40) for j in range(-1, 32) for s in (-1, 0, 1)]  # j's edges
    return [float(x) for x in xs]


def test_log_error_and_the_earlier_functions():
    """At most 0.53 ulp anywhere; no further off than log_tang was, at its worst and on average."""
    tables, earlier = log_tables(), _table()
    xs = _log_arguments()
    now = np.array([_log_error(log_t32(x, tables), x) for x in xs])
    was = np.array([_log_error(log_tang(x, earlier), x) for x in xs])
    assert now.max() <= LOG_ULPS, xs[int(now.argmax())]
    assert now.max() <= was.max() and np.mean(now ** 2) <= np.mean(was ** 2)
    assert log_t32(1.0, tables) == 0.0


def test_exp_error():
    """Within 0.55 ulp: half an ulp, and the last sum's terms of 2^-6 rounded to 2^-59 before it."""
    tables = exp_tables()
    rng = np.random.default_rng(4)
    xs = list(-np.exp(rng.uniform(math.log(1e-12), math.log(700.0), 3000))) + list(rng.uniform(-708.0, 709.0, 1000))
    xs += [0.0, -0.0, 1e-300, -1e-300, -708.0, 709.0, math.log(2) / 64, -math.log(2) / 64]
    xs += [(n + 0.5) * math.log(2) / 32 * (1 + s * 2 ** -45) for n in range(-40, 40) for s in (-1, 1)]
    getcontext().prec = 50
    for x in map(float, xs):
        e = Decimal(x).exp()
        assert abs(Decimal(exp_t32(x, tables)) - e) <= Decimal("0.55") * Decimal(math.ulp(float(e))), x
    assert exp_t32(-708.5, tables) == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(1e-10, 8.0), (0.9, 1.12), (1.0156, 1.0469), (0.96, 0.99), (1e-8, 2.0)])
def test_device_log_error(lo, hi):
    """The library's own FP64 log entries (half the logarithm of a squared distance, exactly) against the 80-bit
    logarithm, whose own error is below 0.001 ulp of a double."""
    import afmm2d_b200 as A
    rng = np.random.default_rng(8)
    d = np.sqrt(np.exp(rng.uniform(np.log(lo), np.log(hi), 400000)))
    x = d * d
    p = np.stack([d, np.zeros_like(d)], axis=1)
    v = 2.0 * A.kernel_eval("log", 2.0 ** -20, p, np.zeros_like(p), mode="fp64")
    ref = np.log(x.astype(np.longdouble))
    ok = (x >= 1e-10) & (x != 1.0)
    err = np.abs(v.astype(np.longdouble) - ref)[ok] / np.spacing(np.abs(ref[ok].astype(np.float64)))
    assert ok.sum() > 0.99 * len(d) and err.max() <= LOG_ULPS + 0.002


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi,ulps", [(1e-6, 1.0 - 1e-9, 0.502), (1.0, 300.0, 0.992)])
def test_device_scaled_entries(lo, hi, ulps):
    """FP64 entries of the scaled 1/r on either side of R = a, of exact squared distances, against 80-bit
    arithmetic: no further off than the square root (R/a) and the square root and division (a/R) that they
    stand for, 0.5 ulp and 0.991."""
    import afmm2d_b200 as A
    rng = np.random.default_rng(9)
    a = 2.0 ** -5
    d = a * np.exp(rng.uniform(np.log(lo), np.log(hi), 400000))
    x = d * d
    p = np.stack([d, np.zeros_like(d)], axis=1)
    v = A.kernel_eval("one_over_r_scaled", a, p, np.zeros_like(p), mode="fp64")
    R = np.sqrt(x.astype(np.longdouble))
    ref = np.where(x < a * a, R / a, a / R)
    err = np.abs(v.astype(np.longdouble) - ref) / np.spacing(ref.astype(np.float64))
    assert err.max() <= ulps


@pytest.mark.gpu
def test_device_scaled_entries_at_the_ends():
    import afmm2d_b200 as A
    a = 2.0 ** -5
    d = np.array([0.0, 1e-100, 1e-30, np.nextafter(a, 0), a, np.nextafter(a, 1), 1e30, 1e150, 1e200])
    p = np.stack([d, np.zeros_like(d)], axis=1)
    got = A.kernel_eval("one_over_r_scaled", a, p, np.zeros_like(p), mode="fp64")
    exact = A.kernel_eval("one_over_r_scaled", a, p, np.zeros_like(p), mode="exact")
    assert np.all(np.abs(got - exact) <= np.spacing(exact)) and got[0] == 0.0 and got[-1] == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["log", "one_over_r_scaled"])
def test_device_entries_of_any_box_size(kernel):
    """kernel_eval takes any box size a: the branch of a separation just below and just above one that is not a
    power of two is the kernel's, at separations that differ from it in their last digits only.  A few ulps:
    a * (1 / a^2) for 1 / a, and the two functions' own."""
    import afmm2d_b200 as A
    for a in (0.3, 0.0123, 0.7 * 2.0 ** -9):
        d = a * (1.0 + np.concatenate([-np.logspace(-15, -4, 60), [0.0], np.logspace(-15, -4, 60)]))
        p = np.stack([d, np.zeros_like(d)], axis=1)
        got = A.kernel_eval(kernel, a, p, np.zeros_like(p), mode="fp64")
        exact = A.kernel_eval(kernel, a, p, np.zeros_like(p), mode="exact")
        assert np.all(np.abs(got - exact) <= 4 * np.spacing(np.abs(exact))), a
