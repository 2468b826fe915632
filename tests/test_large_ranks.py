"""Boxes of more rows than the one-column M2L takes at once (1,024): user kernel cos(c r) with waves shorter than
the points' distances, so that boxes keep all of their points."""
import os

import numpy as np
import pytest

import afmm2d_b200 as A
from test_gpu_parity import FP64_BATCHED_TOL

PLUGIN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "plugin", "libafmm_growing.so")
WAVE = 26  # AFMM_KERNEL_USER_FIRST + 10


@pytest.fixture(scope="module")
def plugin():
    if not os.path.exists(PLUGIN):
        pytest.fail("tests/plugin/libafmm_growing.so is missing: run __graft_entry__.build()")
    return A.load_kernel_plugin(PLUGIN)


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["store", "on_the_fly"])
def test_ranks_beyond_one_round_of_rows(plugin, storage):
    """Stored blocks and entries on the fly against the batched passes (every box's own blocks; summation order)
    and against direct sums at some of the points.  Ranks of 1,120 come from level 2 of a tree of 280-point
    leaves."""
    N, M = 17920, 280
    rng = np.random.default_rng(N)
    pts = rng.uniform(0, 1, (N, 2))
    a = A.AFMM(N, M, 8, pts, kernel=WAVE, kparam=4000.0)
    a.set_m2l_storage(storage)
    a.assemble()
    assert a.ranks(2).max() > 1024
    Q = rng.standard_normal((N, 2))
    y = a.computeMatVecProduct(Q[:, 0])
    Yb = a.computeMatVecProduct(Q, precision="fp64_batched")
    assert np.linalg.norm(y - Yb[:, 0]) <= FP64_BATCHED_TOL * np.linalg.norm(y)
    some = rng.choice(N, 50, replace=False)
    R = np.sqrt(((pts[some, None, :] - pts[None, :, :]) ** 2).sum(2))
    direct = np.cos(4000.0 * R) @ Q[:, 0]
    assert np.linalg.norm(y[some] - direct) <= 1e-6 * np.linalg.norm(direct)
