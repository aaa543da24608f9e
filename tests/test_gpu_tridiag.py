"""The eigensolver at the orders where its reduction changes form: one CTA to
64, a cluster of 4, 8 and 16 CTAs to 160, 320 and 608, one CTA per SM with 1 to
4 rows a thread and 8 or 16 columns a CTA to 2048, panels above.

Oracle: LAPACK through numpy.linalg.eigvalsh for the eigenvalues; the vectors by
their residual and orthonormality.  Bounds: a backward stable solver moves an
eigenvalue by p(n) eps ||A||_2 and leaves a residual of that size; p(n) = 4 n
covers the n reflectors' roundings.  Orthonormality of inverse iteration is
eps ||A|| over the smallest gap between vectors it does not orthogonalise
against each other, 1e-8 ||A||: 1e-6 holds for every spectrum here."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [2, 3, 31, 32, 33, 63, 64, 65, 159, 160, 161, 319, 320, 321, 607, 608, 609, 1024, 1025, 1184, 1185, 1537,
          2048, 2049]


@pytest.fixture(autouse=True)
def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def _solve(a):
    import torch
    from mopac_gpu_b200 import kernels
    n = a.shape[0]
    i, j = np.tril_indices(n)
    f = torch.from_numpy(np.ascontiguousarray(a[i, j])).cuda()
    c, e = kernels.eigh_packed(f)
    p = f.cpu().numpy()
    return c.cpu().numpy(), e.cpu().numpy(), p


def _check(a, orth=1.0e-6):
    n = a.shape[0]
    c, e, packed = _solve(a)
    b = a + np.diag(1.0e-10 * np.arange(1, n + 1))
    i, j = np.tril_indices(n)
    assert np.array_equal(packed, b[i, j])  # the perturbed matrix goes back to the caller
    norm = max(np.abs(np.linalg.eigvalsh(b)).max(), np.finfo(float).tiny)
    tol = 4.0 * n * np.finfo(float).eps * norm
    assert np.all(np.diff(e) >= 0.0)
    assert np.abs(e - np.linalg.eigvalsh(b)).max() <= tol
    assert np.abs(b @ c - c * e).max() <= tol
    assert np.abs(c.T @ c - np.eye(n)).max() <= orth


@pytest.mark.parametrize("n", ORDERS)
def test_random_symmetric(n):
    a = np.random.default_rng(n).normal(size=(n, n))
    _check((a + a.T) / 2)


@pytest.mark.parametrize("n,kind", [(40, "identity"), (130, "identity")] + [
    (n, k) for n in (40, 130, 300, 500, 700) for k in ("diagonal", "blocks", "graded", "small", "large")])
def test_special_spectra(n, kind):
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    if kind == "diagonal":        # every reflector is the identity
        a = np.diag(rng.normal(size=n))
    elif kind == "identity":      # eigenvalues apart by the perturbation only
        a = np.eye(n)
    elif kind == "blocks":        # uncoupled blocks, two of them equal
        a = np.zeros((n, n))
        m = n // 4
        x = rng.normal(size=(m, m))
        a[:m, :m] = a[m:2 * m, m:2 * m] = (x + x.T) / 2
        a[2 * m:, 2 * m:] = np.diag(rng.normal(size=n - 2 * m))
    elif kind == "graded":        # nine orders of magnitude
        a = (q * np.logspace(0, -9, n)) @ q.T
        a = (a + a.T) / 2
    else:
        a = (q * rng.normal(size=n)) @ q.T
        a = (a + a.T) / 2 * (1.0e150 if kind == "large" else 1.0e-4)
    _check(a)


def test_status_of_a_matrix_with_nan():
    """A NaN comes back as an error or as NaN values, never as a wait that runs out."""
    import torch
    from mopac_gpu_b200 import kernels
    from mopac_gpu_b200._lib import LibraryError
    for n in (40, 300, 700):
        f = torch.full((n * (n + 1) // 2,), float("nan"), dtype=torch.float64, device="cuda")
        try:
            _, e = kernels.eigh_packed(f)
        except LibraryError as err:
            assert err.code == 6
        else:
            assert torch.isnan(e).any()


def test_orders_the_entries_refuse():
    from mopac_gpu_b200._lib import lib
    L = lib()
    p = ctypes.c_void_p
    L.mb_tridiag_cluster.argtypes = [ctypes.c_int, p, ctypes.c_int] + [p] * 6
    L.mb_tridiag_grid.argtypes = [ctypes.c_int, ctypes.c_int, p, ctypes.c_longlong] + [p] * 7
    for n in (0, 1, 609):
        assert L.mb_tridiag_cluster(n, None, 0, None, None, None, None, None, None) == 1
    for m in (0, 1, 2049):
        assert L.mb_tridiag_grid(m, 148, None, 2, None, None, None, None, None, None, None) == 1
