"""User kernels that call the library's FP64 logarithm and exponential by the names first offered to them
(log_tang, exp_tang); tests/plugin/growing_kernels.cu."""
import os

import numpy as np
import pytest

import afmm2d_b200 as A

PLUGIN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "plugin", "libafmm_growing.so")
SPLINE, GAUSS = 24, 25  # AFMM_KERNEL_USER_FIRST + 8, + 9


@pytest.fixture(scope="module")
def plugin():
    if not os.path.exists(PLUGIN):
        pytest.fail("tests/plugin/libafmm_growing.so is missing: run __graft_entry__.build()")
    return A.load_kernel_plugin(PLUGIN)


def test_plugin_registers_both_kernels(plugin):
    assert A.kernel_name(SPLINE) == "PolyharmonicSpline" and A.kernel_name(GAUSS) == "UserGaussian"


@pytest.mark.gpu
def test_entries(plugin):
    """Within the functions' one ulp and the roundings of the products around them (three for the spline; the
    Gaussian's argument has one, as its exact form has)."""
    rng = np.random.default_rng(4)
    xy1 = rng.uniform(0, 1, (20000, 2))
    xy2 = xy1.copy()
    xy2[:, 0] += rng.uniform(0.01, 0.9, 20000)
    for kernel, ulps, param in ((SPLINE, 5.0, 0.0), (GAUSS, 2.0, 0.3)):
        f = A.kernel_eval(kernel, 2.0 ** -7, xy1, xy2, mode="fp64", param=param)
        g = A.kernel_eval(kernel, 2.0 ** -7, xy1, xy2, mode="exact", param=param)
        assert np.all(np.abs(f - g) <= ulps * 2.0 ** -52 * np.abs(g))


@pytest.mark.gpu
@pytest.mark.parametrize("N,M", [(4352, 68), (4160, 65)])
def test_growing_kernel_in_batched_passes(plugin, N, M):
    """r^4 log r overflows at the far-off places that a tile may be padded with: the FP64 batched near field, at
    leaves that do and do not fill a tile of four or eight, gives the one-column product's potentials."""
    rng = np.random.default_rng(N)
    a = A.AFMM(N, M, 6, rng.uniform(0, 1, (N, 2)), kernel=SPLINE)
    a.assemble()
    Q = rng.standard_normal((N, 19))
    for cols in (5, 19):
        Y = a.computeMatVecProduct(np.asfortranarray(Q[:, :cols]), precision="fp64_batched")
        for c in (0, cols - 1):
            y = a.computeMatVecProduct(np.ascontiguousarray(Q[:, c]))
            assert np.linalg.norm(Y[:, c] - y) <= 1e-12 * np.linalg.norm(y)
