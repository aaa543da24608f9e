"""The FP64 GEMM and packed SYRK at the edges of their 64- and 128-wide tiles and
16-deep k blocks, with leading dimensions that allow 16-byte copies and ones
that do not, and k slices that start at an odd k.

Inputs that are small integers over 16 make every partial sum exact, so those
products must be numpy's bit for bit in any order; random ones are held to the
bound k eps |A||B| of a k-term sum."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def _dev(a, lda):
    """Column-major a with leading dimension lda on the device."""
    buf = np.full((a.shape[1], lda), np.nan)
    buf[:, :a.shape[0]] = a.T
    return torch.from_numpy(buf.reshape(-1)).cuda()


def _gemm(ta, tb, a, b, pad, ws):
    from mopac_gpu_b200._lib import check, lib
    L = lib()
    L.mb_dgemm_ws.argtypes = ([ctypes.c_char] * 2 + [ctypes.c_int] * 3 + [ctypes.c_double, ctypes.c_void_p, ctypes.c_int,
                              ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_void_p, ctypes.c_int,
                              ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p])
    m, k = a.shape
    n = b.shape[1]
    sa, sb = (a if ta == "N" else a.T), (b if tb == "N" else b.T)
    da, db = _dev(sa, sa.shape[0] + pad), _dev(sb, sb.shape[0] + pad)
    c = torch.full((n * m,), float("nan"), dtype=torch.float64, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(L.mb_dgemm_ws(ta.encode(), tb.encode(), m, n, k, 1.0, da.data_ptr(), sa.shape[0] + pad, db.data_ptr(),
                        sb.shape[0] + pad, 0.0, c.data_ptr(), m, ws.data_ptr() if ws is not None else None,
                        ws.numel() if ws is not None else 0, s))
    return c.cpu().numpy().reshape(n, m).T


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", [(65, 65, 1), (65, 127, 15), (128, 66, 16), (129, 193, 17), (64, 300, 40),
                                   (1100, 1300, 33), (2000, 2100, 16)])
def test_products_at_tile_edges(ta, tb, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a = rng.integers(-64, 65, size=(m, k)) / 16.0
    b = rng.integers(-64, 65, size=(k, n)) / 16.0
    for pad in (0, 1, 2):
        assert np.array_equal(_gemm(ta, tb, a, b, pad, None), a @ b)


@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
@pytest.mark.parametrize("k", [513, 1031, 2050])
def test_slices_of_k_that_start_anywhere(ta, tb, k):
    rng = np.random.default_rng(k)
    a, b = rng.normal(size=(130, k)), rng.normal(size=(k, 140))
    ws = torch.empty(32 * 130 * 140, dtype=torch.float64, device="cuda")
    bound = k * np.finfo(float).eps * (np.abs(a) @ np.abs(b))
    for pad in (0, 1):
        assert np.all(np.abs(_gemm(ta, tb, a, b, pad, ws) - a @ b) <= bound)


@pytest.mark.parametrize("n,k", [(65, 1), (128, 16), (129, 33), (300, 200), (1300, 17), (2100, 64)])
def test_packed_syrk_at_tile_edges(n, k):
    from mopac_gpu_b200._lib import check, lib
    rng = np.random.default_rng(n)
    c = rng.integers(-64, 65, size=(n, k)) / 16.0
    i, j = np.tril_indices(n)
    want = (2.0 * (c @ c.T))[i, j]
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for pad in (0, 1):
        d = _dev(c, n + pad)
        p = torch.full((n * (n + 1) // 2,), float("nan"), dtype=torch.float64, device="cuda")
        full = torch.cat([d, torch.zeros((n - k) * (n + pad), dtype=torch.float64, device="cuda")])
        check(lib().mb_density_dev(n, k, 2.0, full.data_ptr(), n + pad, p.data_ptr(), s))
        assert np.array_equal(p.cpu().numpy(), want)
