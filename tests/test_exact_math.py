"""The setup's log and exp (exact_math.cuh: a table-driven form with a
rounding test, the double-double series behind it) against 60-digit decimal
arithmetic, at the arguments where the table-driven form changes its terms."""
import numpy as np
import pytest

import afmm2d_b200 as A
from test_gpu_parity import correctly_rounded_kernel

pytestmark = pytest.mark.gpu


def _log_separations():
    """Separations d whose d^2 sits at powers of two, around 1, at and halfway between the table's
    breakpoints 1 + j/128, and at the ends of the kernel's range."""
    rng = np.random.default_rng(3)
    r2 = [2.0 ** k for k in range(-33, 34)] + [1.0 + s * 2.0 ** -k for k in range(1, 53) for s in (1, -1)]
    r2 += [(1.0 + j / 256.0) * 2.0 ** k for j in range(257) for k in (-7, -1, 0, 5)]
    r2 += [1.0e-10, 1.0000001e-10, 1e300, 1e-9]
    d = np.sqrt(np.array(r2))
    return np.concatenate([d, np.nextafter(d, 0), np.nextafter(d, 9e9), rng.uniform(0, 2, 500)])


def _exp_separations():
    """Separations whose -d^2/param is at and beside multiples of ln2/32, and at the ends of the range."""
    p = 0.01
    x = [j * np.log(2.0) / 64 for j in range(200)] + list(np.linspace(0, 720, 300)) + [699.99, 700.0, 700.01, 745.0]
    d = np.sqrt(np.array(x) * p)
    return np.concatenate([d, np.nextafter(d, 0), np.nextafter(d, 9e9)])


@pytest.mark.parametrize("kernel,sep", [("log", _log_separations), ("gaussian", _exp_separations)])
def test_setup_entries_are_correctly_rounded_at_the_edges(kernel, sep):
    d = sep()
    if kernel == "gaussian":
        d = d[d * d / 0.01 < 708]  # below, the result is subnormal: rounded twice by design
    p = np.stack([d, np.zeros_like(d)], axis=1)
    q = np.zeros_like(p)
    a = 2.0 ** -20  # below every separation of interest: the plain branch of the log kernel
    got = A.kernel_eval(kernel, a, p, q, mode="exact")
    for t in range(len(d)):
        assert got[t] == correctly_rounded_kernel(kernel, a, p[t], q[t]), (kernel, d[t])
