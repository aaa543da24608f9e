"""Eigenvectors of a tridiagonal matrix whose rows are coupled by far less than an
eigenvalue's rounding: where an eigenvalue comes out equal to its diagonal element
the row's pivot is zero, smaller than the coupling, and neither may be divided by.
The Householder reduction leaves such a matrix as it is.  Both forms of the solver:
the one the entry points take and the blocked one of pseudo-diagonalising SCFs.

Bounds: those of a backward stable solver, 4 n eps ||A|| for eigenvalues and
residuals; the eigenvalues are at least 0.4 apart, so orthonormality is held to
4 n eps times the norm over that gap."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _ordered(f, n):
    from mopac_gpu_b200._lib import check, lib
    L, P = lib(), ctypes.c_void_p
    L.mb_eigh_ordered_ws.argtypes = [ctypes.c_int, P, ctypes.c_int] + [P] * 5
    L.mb_eigh_ws_bytes.argtypes, L.mb_eigh_ws_bytes.restype = [ctypes.c_int], ctypes.c_size_t
    ws = torch.empty(L.mb_eigh_ws_bytes(n), dtype=torch.uint8, device="cuda")
    c = torch.empty((n, n), dtype=torch.float64, device="cuda")
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    check(L.mb_eigh_ordered_ws(n, f.data_ptr(), 1, c.data_ptr(), e.data_ptr(), ws.data_ptr(), status.data_ptr(),
                               torch.cuda.current_stream().cuda_stream))
    assert int(status.item()) == 0
    return c.t(), e


@pytest.mark.parametrize("form", ["entry", "ordered"])
@pytest.mark.parametrize("n", [2, 3, 40, 300, 700])
@pytest.mark.parametrize("coupling", [1.0e-20, 1.0e-120, 1.0e-160, 1.0e-200, 1.0e-290, 1.0e-306, 1.0e-310, 5.0e-324])
def test_couplings_below_the_rounding(n, coupling, form):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200 import kernels
    rng = np.random.default_rng(n)
    a = np.diag(rng.permutation(np.arange(n) + rng.uniform(-0.3, 0.3, n)))
    i = np.arange(n - 1)
    a[i, i + 1] = a[i + 1, i] = coupling
    i, j = np.tril_indices(n)
    f = torch.from_numpy(np.ascontiguousarray(a[i, j])).cuda()
    c, e = kernels.eigh_packed(f) if form == "entry" else _ordered(f, n)
    c, e = c.cpu().numpy(), e.cpu().numpy()
    b = a + np.diag(1.0e-10 * np.arange(1, n + 1))
    tol = 4.0 * n * np.finfo(float).eps * np.abs(np.diag(b)).max()
    assert np.abs(e - np.sort(np.diag(b))).max() <= tol
    assert np.abs(b @ c - c * e).max() <= tol
    assert np.abs(c.T @ c - np.eye(n)).max() <= tol / 0.4
