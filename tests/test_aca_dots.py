"""The dot products of the ACA's stopping test: a double-double sum whose low part is renormalised at every
term.  Terms are chosen so that a low part left to grow rounds the same way again and again."""
import os
import random
import struct
import subprocess
from fractions import Fraction

import pytest

from afmm2d_b200.build import nvcc

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def _terms(n):
    """A large first term, then candidates picked for the low part of an unrenormalised sum: first those that make
    it grow, then those whose addition to it rounds down the most."""
    rng = random.Random(7)
    hi, lo, xs, ys = 0.0, 0.0, [], []
    for k in range(n):
        cand = [(1.25 * 2.0 ** 26, 1.2 * 2.0 ** 26)] if k == 0 else \
            [(rng.uniform(1, 2) * 2.0 ** 10 * rng.choice((1, -1)), rng.uniform(1, 2) * 2.0 ** 9) for _ in range(24)]
        best = None
        for x, y in cand:
            p = x * y
            s = hi + p
            e = float(Fraction(hi) + Fraction(p) - Fraction(s)) + float(Fraction(x) * Fraction(y) - Fraction(p))
            score = e if k < n // 3 else float(Fraction(lo) + Fraction(e) - Fraction(lo + e))
            if best is None or score > best[0]:
                best = score, x, y, s, lo + e
        _, x, y, hi, lo = best
        xs.append(x)
        ys.append(y)
    return xs, ys


@pytest.mark.gpu
def test_accumulation_error(tmp_path):
    exe = tmp_path / "dots_test"
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(NATIVE, "..", "..", "include"), os.path.join(NATIVE, "dots_test.cu"), "-o",
                    str(exe)], check=True, capture_output=True)
    for n in (1, 2, 500, 2000):
        xs, ys = _terms(n)
        path = tmp_path / f"terms{n}"
        path.write_bytes(struct.pack(f"<{1 + 2 * n}d", n, *xs, *ys))
        r = subprocess.run([str(exe), str(path)], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0
        got = sum(Fraction(float.fromhex(v)) for v in r.stdout.split())
        exact = sum(Fraction(x) * Fraction(y) for x, y in zip(xs, ys))
        size = sum(abs(Fraction(x) * Fraction(y)) for x, y in zip(xs, ys))
        assert abs(got - exact) <= 3 * n * size / 2 ** 106, n
