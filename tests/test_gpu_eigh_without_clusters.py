"""Orders above 320 where the device holds no cluster of 16 CTAs: the grid kernel
takes them, with the bounds of test_gpu_tridiag.py (4 n eps ||A|| for eigenvalues
and residuals, 1e-6 for the vectors' orthonormality)."""
import ctypes

import numpy as np
import pytest


def test_orders_by_cluster_support():
    from mopac_gpu_b200._lib import lib
    L = lib()
    L.mb_tridiag_cluster_orders.argtypes, L.mb_tridiag_cluster_orders.restype = [ctypes.c_int], ctypes.c_int
    assert [L.mb_tridiag_cluster_orders(k) for k in (0, 1, 9)] == [320, 608, 608]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [321, 400, 512, 513, 608])
def test_grid_takes_the_orders_of_the_large_cluster(n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200._lib import check, lib
    L, P = lib(), ctypes.c_void_p
    L.mb_eigh_cluster_ws.argtypes = [ctypes.c_int, P, ctypes.c_int] + [P] * 4 + [ctypes.c_int, P]
    a = np.random.default_rng(n).normal(size=(n, n))
    a = (a + a.T) / 2
    i, j = np.tril_indices(n)
    f = torch.from_numpy(np.ascontiguousarray(a[i, j])).cuda()
    ws = torch.empty(L.mb_eigh_ws_bytes(n), dtype=torch.uint8, device="cuda")
    c = torch.empty((n, n), dtype=torch.float64, device="cuda")
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    check(L.mb_eigh_cluster_ws(n, f.data_ptr(), 1, c.data_ptr(), e.data_ptr(), ws.data_ptr(), status.data_ptr(),
                               L.mb_tridiag_cluster_orders(0), torch.cuda.current_stream().cuda_stream))
    assert int(status.item()) == 0
    b = a + np.diag(1.0e-10 * np.arange(1, n + 1))
    c, e, want = c.t().cpu().numpy(), e.cpu().numpy(), np.linalg.eigvalsh(b)
    tol = 4.0 * n * np.finfo(float).eps * np.abs(want).max()
    assert np.abs(e - want).max() <= tol
    assert np.abs(b @ c - c * e).max() <= tol
    assert np.abs(c.T @ c - np.eye(n)).max() <= 1.0e-6
