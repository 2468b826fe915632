"""Writes math_tables.cuh: the tables of the setup's correctly rounded logarithm
and exponential (log_cr and exp_cr in exact_math.cuh) and of the FP64 matvec's
(log_t32 and exp_t32 in fast_math.cuh).

log: for j = 0..128 and F = 1 + j/128: 1/F rounded to double, and ln F split
as hi + lo with hi a multiple of 2^-42 (so that k*ln2_hi + hi is exact for
every double exponent k) and lo = ln F - hi rounded to double; ln 2 = entry
128.
exp: 2^(j/32) for j = 0..31 as hi + lo (hi the correctly rounded double), and
ln2/32 as L1 + L2 with L1 a multiple of 2^-42 (N * L1 exact for |N| < 2^16).
log_t32: for j = 0..31 and m in the interval of width 1/32 around 1 + j/32: c near
its inverse, a multiple of 1/64 or of 1/128, so that u = m c - 1 is a double for
every double m (log_centre), and -ln c as hi (a multiple of 2^-42) + lo (21
significant bits); the coefficients of q(u), |u| <= 0.0198 (the largest), the
truncated Chebyshev expansion of (ln(1+u) - u)/u^2.
exp_t32: 2^(j/32) as above, lo to 21 significant bits.
Both as arrays of 32 words, one 128-byte line each: a warp's lookup of one
word touches one line whatever the lanes' indexes are.
Values are computed with 60-digit decimal arithmetic.

Usage: python make_math_tables.py  (rewrites math_tables.cuh beside this file)
"""
import math
import os
import struct
from decimal import Decimal, getcontext
from fractions import Fraction

getcontext().prec = 60
HERE = os.path.dirname(os.path.abspath(__file__))


def split_ln(F):
    ln = Decimal(F).ln()
    hi = Fraction(round(Fraction(ln) * 2 ** 42), 2 ** 42)
    hi_d = float(hi)
    assert Fraction(hi_d) == hi  # 42 fraction bits, magnitude < 1: exact in a double
    lo_d = float(Decimal(ln) - Decimal(hi.numerator) / Decimal(hi.denominator))
    return hi_d, lo_d


def words(x):
    b = struct.unpack("<Q", struct.pack("<d", x))[0]
    return b >> 32, b & 0xffffffff


def round21(x):
    """x (a Decimal or Fraction) to the nearest double with 21 significant bits."""
    x = Fraction(x)
    if x == 0:
        return 0.0
    e = math.frexp(float(x))[1] - 21
    v = float(round(x / Fraction(2) ** e) * Fraction(2) ** e)
    assert words(v)[1] == 0
    return v


def log_centre(j):
    """(c, largest |m c - 1|) for the doubles m in [1 + (j - 1/2)/32, 1 + (j + 1/2)/32).  m is a multiple of
    2^-52 (2^-53 below 1, where c = 1), so m c - 1 is one of 2^-58 for c a multiple of 1/64, exact up to 2^-5,
    and of 2^-59 for a multiple of 1/128, exact up to 2^-6."""
    lo, hi = Fraction(2 * (32 + j) - 1, 64), Fraction(2 * (32 + j) + 1, 64)
    if j == 0:
        return Fraction(1), Fraction(1, 64)
    best = None
    for den, limit in ((64, Fraction(1, 32)), (128, Fraction(1, 64))):
        for a in range(den // 2, den + 1):
            c = Fraction(a, den)
            u = max(abs(lo * c - 1), abs(hi * c - 1))
            if u <= limit and (best is None or u < best[1]):
                best = c, u
    return best


def log_poly(degree, h):
    """Truncated Chebyshev expansion of g(u) = (ln(1+u) - u)/u^2 on [-h, h],
    as monomial coefficients of u rounded to double."""
    n, h = 40, Decimal(h.numerator) / Decimal(h.denominator)

    def g(u):  # its Taylor series: -1/2 + u/3 - u^2/4 + ...
        return sum(Decimal((-1) ** (k + 1)) * u ** k / (k + 2) for k in range(40))

    def cos(x):  # Taylor, |x| <= pi
        t = s = Decimal(1)
        for k in range(1, 60):
            t *= -x * x / ((2 * k - 1) * (2 * k))
            s += t
        return s

    pi = Decimal("3.14159265358979323846264338327950288419716939937510582097494459")
    nodes = [cos(pi * (2 * i + 1) / (2 * n)) for i in range(n)]
    val = [g(h * x) for x in nodes]
    cheb = []
    for k in range(degree + 1):
        tk = []  # T_k at the nodes by the recurrence
        for x in nodes:
            a, b = Decimal(1), x
            for _ in range(k):
                a, b = b, 2 * x * b - a
            tk.append(a)
        cheb.append(sum(v * t for v, t in zip(val, tk)) * 2 / n / (2 if k == 0 else 1))
    T = [[Decimal(1)], [Decimal(0), Decimal(1)]]
    for k in range(2, degree + 1):
        a = [Decimal(0)] + [2 * c for c in T[-1]]
        for i, c in enumerate(T[-2]):
            a[i] -= c
        T.append(a)
    mono = [sum(cheb[k] * T[k][i] for k in range(i, degree + 1)) / h ** i for i in range(degree + 1)]
    return [float(c) for c in mono]


def word_array(name, ws):
    out = [f"    {{{', '.join(f'0x{w:08x}u' for w in row)}}}," for row in ws]
    return [f"static __device__ const __align__(128) unsigned int {name}[{len(ws)}][32] = {{", *out, "};"]


def main():
    inv, lnhi, lnlo = [], [], []
    for j in range(129):
        F = 1.0 + j / 128.0
        inv.append(1.0 / F)  # IEEE division: correctly rounded
        h, lo = split_ln(F)
        lnhi.append(h)
        lnlo.append(lo)
    lines = [
        "// Generated by make_math_tables.py.  Do not edit.",
        "// log_cr: breakpoints F = 1 + j/128 (j = 0..128) -- 1/F, and ln F as hi (a",
        "// multiple of 2^-42) + lo.  exp_cr: 2^(j/32) as hi + lo, ln2/32 as L1 + L2.",
        "// log_t32, exp_t32: 32 entries, each word of an entry in a 128-byte line of its own.",
        "#pragma once",
        "",
        "namespace afmm {",
        "",
        "static __device__ const double kLogInvF[129] = {",
    ]
    lines += [f"    {v.hex()}," for v in inv]
    lines += ["};", "", "// {hi, lo} of ln F", "static __device__ const double2 kLogLnF[129] = {"]
    lines += [f"    {{{h.hex()}, {lo.hex()}}}," for h, lo in zip(lnhi, lnlo)]
    lines += ["};", "", f"constexpr double kLn2Hi = {lnhi[128].hex()};", f"constexpr double kLn2Lo = {lnlo[128].hex()};"]
    # exp: 2^(j/32) as hi + lo
    lines += ["", "// {hi, lo} of 2^(j/32)", "static __device__ const double2 kExp2J32[32] = {"]
    for j in range(32):
        v = Decimal(2) ** (Decimal(j) / Decimal(32))
        hi = float(v)
        lo = float(v - Decimal(hi))
        lines.append(f"    {{{hi.hex()}, {lo.hex()}}},")
    ln2_32 = Decimal(2).ln() / Decimal(32)
    l1 = Fraction(round(Fraction(ln2_32) * 2 ** 42), 2 ** 42)
    l1_d = float(l1)
    assert Fraction(l1_d) == l1
    l2_d = float(ln2_32 - Decimal(l1.numerator) / Decimal(l1.denominator))
    inv = float(Decimal(32) / Decimal(2).ln())
    lines += ["};", "", f"constexpr double kLn2Over32Hi = {l1_d.hex()};", f"constexpr double kLn2Over32Lo = {l2_d.hex()};",
              f"constexpr double k32OverLn2 = {inv.hex()};"]
    # log_t32 and exp_t32
    lw, ew = [[], [], [], []], [[], [], []]
    centres = [log_centre(j) for j in range(32)]
    for j in range(32):
        c = float(centres[j][0])
        L = -Decimal(c).ln()  # (0 for j = 0)
        hi = Fraction(round(Fraction(L) * 2 ** 42), 2 ** 42)
        assert Fraction(float(hi)) == hi
        lo = round21(Fraction(L) - hi)
        for row, w in zip(lw, (words(c)[0], *words(float(hi)), words(lo)[0])):
            row.append(w)
        v = Decimal(2) ** (Decimal(j) / Decimal(32))
        for row, w in zip(ew, (*words(float(v)), words(round21(v - Decimal(float(v))))[0])):
            row.append(w)
    lines += ["", "// high word of c; high, low word of the high part of -ln c; high word of its low part"]
    lines += word_array("kLogT32", lw)
    lines += ["", "// high, low word of the high part of 2^(j/32); high word of its low part"]
    lines += word_array("kExpT32", ew)
    lines += [""] + [f"constexpr double kLogQ{i} = {c.hex()};" for i, c in enumerate(log_poly(7, max(u for _, u in centres)))]
    lines += ["", "}  // namespace afmm", ""]
    with open(os.path.join(HERE, "math_tables.cuh"), "w") as f:
        f.write("\n".join(lines))


if __name__ == "__main__":
    main()
