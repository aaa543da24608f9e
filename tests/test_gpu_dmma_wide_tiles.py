"""The 128-wide tiles of the FP64 GEMM and packed SYRK at odd remainders, with leading
dimensions that allow 16-byte copies and ones that do not, plain and in slices of k
that start at an even and at an odd k.  Which tile a shape takes is asked of the
library, so a change of the rule cannot leave these kernels untested.

Inputs are small integers over 16: every partial sum is exact, and the product is
numpy's bit for bit in any order."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

GEMMS = [(1025, 1985, 1), (1025, 1985, 17), (1409, 1473, 33), (1473, 1409, 15), (1281, 1537, 16)]
SLICED = [(700, 690, 513), (700, 690, 520), (641, 767, 517), (200, 4609, 514)]
SYRKS = [(1857, 1), (1921, 17), (2047, 33), (1920, 16)]


def _lib():
    from mopac_gpu_b200._lib import lib
    L, I, P = lib(), ctypes.c_int, ctypes.c_void_p
    L.mb_dgemm_tile.argtypes, L.mb_dgemm_tile.restype = [I, I, I, ctypes.c_size_t], I
    L.mb_syrk_tile.argtypes, L.mb_syrk_tile.restype = [I], I
    L.mb_dgemm_ws.argtypes = ([ctypes.c_char] * 2 + [I] * 3 + [ctypes.c_double, P, I, P, I, ctypes.c_double, P, I, P,
                              ctypes.c_size_t, P])
    return L


def test_shapes_take_the_wide_tile():
    L = _lib()
    assert [L.mb_dgemm_tile(m, n, k, 0) for m, n, k in GEMMS] == [128] * len(GEMMS)
    assert [L.mb_dgemm_tile(m, n, k, 32 * m * n) for m, n, k in SLICED] == [128] * len(SLICED)
    assert [L.mb_dgemm_tile(m, n, k, 0) for m, n, k in SLICED] == [64] * len(SLICED)  # so they run in slices
    assert [L.mb_syrk_tile(n) for n, _ in SYRKS] == [128] * len(SYRKS)
    assert L.mb_dgemm_tile(64, 300, 40, 0) == L.mb_syrk_tile(64) == 0
    assert L.mb_dgemm_tile(65, 65, 40, 0) == L.mb_syrk_tile(65) == 64


def _integers(shape, seed):
    return torch.from_numpy(np.random.default_rng(seed).integers(-64, 65, size=shape) / 16.0).cuda()


def _column_major(a, pad):
    """a (rows x columns) stored by columns, leading dimension rows + pad."""
    buf = torch.full((a.shape[1], a.shape[0] + pad), float("nan"), dtype=torch.float64, device="cuda")
    buf[:, :a.shape[0]] = a.T
    return buf


def _exact(a, b):
    return torch.from_numpy(a.cpu().numpy() @ b.cpu().numpy()).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", GEMMS + SLICED)
def test_products(ta, tb, m, n, k):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    L = _lib()
    a, b = _integers((m, k), m + k), _integers((k, n), n + k)
    want = _exact(a, b)
    sliced = (m, n, k) in SLICED
    ws = torch.empty(32 * m * n if sliced else 1, dtype=torch.float64, device="cuda")
    for pad in (0, 1, 2):
        da, db = _column_major(a if ta == "N" else a.T, pad), _column_major(b if tb == "N" else b.T, pad)
        c = torch.full((n, m + pad), -7.0, dtype=torch.float64, device="cuda")
        rc = L.mb_dgemm_ws(ta.encode(), tb.encode(), m, n, k, 1.0, da.data_ptr(), da.shape[1], db.data_ptr(),
                           db.shape[1], 0.0, c.data_ptr(), m + pad, ws.data_ptr() if sliced else None,
                           ws.numel() if sliced else 0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        assert torch.equal(c[:, :m].T, want)
        assert bool((c[:, m:] == -7.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", SYRKS)
def test_packed_syrk(n, k):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200._lib import check, lib
    _lib()
    c = _integers((n, k), n)
    i, j = (torch.from_numpy(x).cuda() for x in np.tril_indices(n))
    want = (2.0 * _exact(c, c.T))[i, j]
    for pad in (0, 1):
        d = torch.zeros((n, n + pad), dtype=torch.float64, device="cuda")
        d[:k] = _column_major(c, pad)
        p = torch.full((n * (n + 1) // 2,), float("nan"), dtype=torch.float64, device="cuda")
        check(lib().mb_density_dev(n, k, 2.0, d.data_ptr(), n + pad, p.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream))
        assert torch.equal(p, want)
