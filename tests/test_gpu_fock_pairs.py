"""The Fock build at the edges of its pair items and fold chunks: heavy-atom
counts around 32, light-atom counts around 32, 96 and 128, one kind of atom only,
light atoms first, single atoms.  Bit for bit the oracle's loop."""
import numpy as np
import pytest

from oracle import scf_oracle as so

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["heavy first", "light first", "mixed"])
@pytest.mark.parametrize("nheavy,nlight", [(0, 2), (0, 130), (1, 0), (1, 2), (2, 0), (31, 32), (32, 96), (33, 98),
                                           (34, 128), (64, 130), (65, 0)])
def test_fock_pair_kinds_bit_identical(nheavy, nlight, order):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200 import kernels as K
    rng = np.random.default_rng(1000 * nheavy + nlight)
    nat = np.array([8] * nheavy + [1] * nlight, np.int32)
    if order == "light first":
        nat = nat[::-1].copy()
    elif order == "mixed":
        nat = rng.permutation(nat)
    side = int(np.ceil(nat.size ** (1 / 3)))
    grid = np.array([(i, j, k) for i in range(side) for j in range(side) for k in range(side)], float)[:nat.size]
    s = so.make_system(nat, 1.6 * grid + rng.uniform(-0.1, 0.1, (nat.size, 3)))
    p = rng.normal(size=s.mpack)
    pa = 0.5 * p + 0.1 * rng.normal(size=s.mpack)  # PA need not be half of P
    f = s.h.copy()
    so.fock2(s, f, p, pa)
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    fd = torch.empty(s.mpack, dtype=torch.float64, device="cuda")
    K.fock2(K.Atoms(s.nfirst, s.nlast), fd, dev(s.h), dev(p), dev(pa), dev(s.w))
    assert np.array_equal(fd.cpu().numpy(), f)
