"""The rotation sweep at the edges of its pipeline: fewer than four occupied
blocks, counts that are not multiples of 16 or of 64, single rows and columns,
row counts around 32.  Bit for bit the sequential loop (the oracle's), through
the reference's symbol."""
import numpy as np
import pytest

from oracle import scf_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nocc", [(2, 1), (3, 2), (17, 1), (17, 16), (31, 15), (32, 16), (33, 17), (64, 48), (65, 64),
                                    (100, 99), (129, 65), (200, 64), (201, 81)])
def test_sweep_is_the_sequential_loop(n, nocc):
    from mopac_gpu_b200._lib import lib
    rng = np.random.default_rng(100 * n + nocc)
    c = np.asfortranarray(rng.normal(size=(n, n)) / np.sqrt(n))
    eig = np.sort(rng.normal(size=n) * 10)
    fmo = np.asfortranarray(rng.normal(size=(n - nocc, nocc)) * 0.1)
    tiny = float(np.abs(fmo).max() * 0.3)  # some pairs are skipped
    ref = c.copy(order="F")
    nrot = so.rotation_sweep(ref, fmo, eig, nocc, tiny=tiny)
    got = c.copy(order="F")
    lib().call_rot_cuda_gpu(fmo.ctypes.data, eig.ctypes.data, got.ctypes.data, None, None, nocc, nocc + 1, n,
                            1.5e-7, tiny)
    assert nrot > 0
    assert np.array_equal(got, ref)
