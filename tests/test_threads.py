"""Handles of different leaf sizes used by several threads at once: a kernel's shared-memory limit belongs to the
function, so one handle's launch must not find it lowered to another's needs."""
import threading

import numpy as np
import pytest

import afmm2d_b200 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,cols", [("fp64", 1), ("mixed", 1), ("fp64_batched", 3)])
def test_two_leaf_sizes_in_two_threads(precision, cols):
    rng = np.random.default_rng(1)
    jobs = []
    for leaf in (1000, 500):  # 98 and 51 KB in the FP64 near field
        N = 16 * leaf
        a = A.AFMM(N, leaf, 4, rng.uniform(0, 1, (N, 2)), kernel="gaussian", kparam=0.3)
        a.assemble()
        q = np.asfortranarray(rng.standard_normal((N, cols))) if cols > 1 else rng.standard_normal(N)
        jobs.append((a, q, a.computeMatVecProduct(q, precision=precision)))
    failures = []

    def work(a, q, y):
        try:
            for _ in range(400):
                if not np.array_equal(a.computeMatVecProduct(q, precision=precision), y):
                    raise AssertionError("another result")
        except Exception as e:  # noqa: BLE001  (reported by the test's thread)
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


def test_setups_in_two_threads():
    """Set-ups side by side: the ACA's shared memory differs from problem to problem."""
    rng = np.random.default_rng(2)
    cases = [(rng.uniform(0, 1, (n, 2)), m) for n, m in ((2048, 32), (6000, 90))]
    ranks = []
    for p, m in cases:
        a = A.AFMM(len(p), m, 8, p, kernel="log")
        a.assemble()
        ranks.append(a.ranks(a.nLevels))
        a.close()
    failures = []

    def work(k):
        try:
            for _ in range(40):
                a = A.AFMM(len(cases[k][0]), cases[k][1], 8, cases[k][0], kernel="log")
                a.assemble()
                if not np.array_equal(a.ranks(a.nLevels), ranks[k]):
                    raise AssertionError("other ranks")
                a.close()
        except Exception as e:  # noqa: BLE001
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
