"""Calls on a device with little memory left: what only makes calls faster gives way to what they need."""
import numpy as np
import pytest

import afmm2d_b200 as A
from test_gpu_parity import FP64_BATCHED_TOL

pytestmark = pytest.mark.gpu


def test_host_staging_takes_the_place_of_the_near_field_parts():
    """A device call of 16 columns takes the batched near field's parts (168 MB); then 40 MB are left, and a host
    call of 16 columns needs 67 for its staging."""
    torch = pytest.importorskip("torch")
    N = 262144
    rng = np.random.default_rng(2)
    a = A.AFMM(N, 64, 6, rng.uniform(0, 1, (N, 2)), kernel="log")
    a.assemble()
    Q = np.asfortranarray(rng.standard_normal((N, 16)))
    y0 = a.computeMatVecProduct(Q[:, 3])
    qd = torch.from_numpy(np.ascontiguousarray(Q.T)).cuda()
    yd = torch.empty_like(qd)
    free0 = torch.cuda.mem_get_info()[0]
    a.matvec_device(qd.data_ptr(), yd.data_ptr(), 16, N, "fp64_batched")
    assert free0 - torch.cuda.mem_get_info()[0] >= 5 * 16 * 8 * N  # the parts among what it took
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    try:
        Y = a.computeMatVecProduct(Q, precision="fp64_batched")
        Y2 = a.computeMatVecProduct(Q, precision="fp64_batched")
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.linalg.norm(Y[:, 3] - y0) <= FP64_BATCHED_TOL * np.linalg.norm(y0)
    np.testing.assert_array_equal(Y, Y2)
    assert np.linalg.norm(yd[3].cpu().numpy() - y0) <= FP64_BATCHED_TOL * np.linalg.norm(y0)


def test_host_call_after_one_whose_staging_did_not_fit():
    """Growing the staging gives the smaller one up first: when the larger does not fit, the call is refused and
    the next one-column call allocates its own again."""
    torch = pytest.importorskip("torch")
    N = 262144
    rng = np.random.default_rng(3)
    a = A.AFMM(N, 64, 6, rng.uniform(0, 1, (N, 2)), kernel="one_over_r")
    a.assemble()
    q = rng.standard_normal((N, 16))
    qd = torch.from_numpy(np.ascontiguousarray(q.T)).cuda()
    a.matvec_device(qd.data_ptr(), torch.empty_like(qd).data_ptr(), 16, N, "mixed")  # its other buffers exist
    y = a.computeMatVecProduct(q[:, 0])
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (32 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(A.AFMMError):
            a.computeMatVecProduct(np.asfortranarray(q), precision="mixed")
        again = a.computeMatVecProduct(q[:, 0])
    finally:
        del fill
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(again, y)
    assert a.computeMatVecProduct(np.asfortranarray(q), precision="mixed").shape == (N, 16)


def test_batched_near_field_without_room_for_its_parts():
    """With less than twice the parts' bytes free they are not taken, and the call works every pair out twice."""
    torch = pytest.importorskip("torch")
    N = 262144
    parts = 5 * 16 * 8 * N
    rng = np.random.default_rng(4)
    a = A.AFMM(N, 64, 6, rng.uniform(0, 1, (N, 2)), kernel="log")
    a.assemble()
    q = rng.standard_normal((N, 16))
    qd = torch.from_numpy(np.ascontiguousarray(q.T)).cuda()
    yd = torch.empty_like(qd)
    a.matvec_device(qd.data_ptr(), yd.data_ptr(), 16, N, "mixed")  # its other buffers exist
    y = a.computeMatVecProduct(q[:, 5])
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 3 * parts // 2, dtype=torch.uint8, device="cuda")
    try:
        free = torch.cuda.mem_get_info()[0]
        a.matvec_device(qd.data_ptr(), yd.data_ptr(), 16, N, "fp64_batched")
        assert free - torch.cuda.mem_get_info()[0] < parts // 2
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.linalg.norm(yd[5].cpu().numpy() - y) <= FP64_BATCHED_TOL * np.linalg.norm(y)
