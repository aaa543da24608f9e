"""Atom layouts whose orbitals do not begin at 1 or leave gaps: the Fock build and
the gradient take any nfirst/nlast, as the reference's loops do.  Rows that belong
to no atom hold NaN in the density and are neither read nor written.  F is the
oracle's loop bit for bit on the same layout; the gradient is that of the compact
layout bit for bit (the same pairs, the same order)."""
import ctypes

import numpy as np
import pytest

from oracle import scf_oracle as so

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _system(nheavy, nlight):
    rng = np.random.default_rng(10 * nheavy + nlight)
    nat = rng.permutation(np.array([8] * nheavy + [1] * nlight, np.int32))
    side = int(np.ceil(nat.size ** (1 / 3)))
    grid = np.array([(i, j, k) for i in range(side) for j in range(side) for k in range(side)], float)[:nat.size]
    return so.make_system(nat, 1.6 * grid + rng.uniform(-0.1, 0.1, (nat.size, 3))), rng


def _spread(s, start, gap):
    """(nfirst, nlast, the packed indices of the compact layout's elements)."""
    nor = s.nlast - s.nfirst + 1
    nfirst = (start + np.concatenate([[0], np.cumsum(nor + gap)[:-1]])).astype(np.int32)
    row = np.concatenate([np.arange(f - 1, f - 1 + k) for f, k in zip(nfirst, nor)])
    i, j = np.tril_indices(s.norbs)
    return nfirst, (nfirst + nor - 1).astype(np.int32), row[i] * (row[i] + 1) // 2 + row[j]


def _place(values, at, size):
    out = np.full(size, np.nan)
    out[at] = values
    return out


@pytest.mark.parametrize("nheavy,nlight", [(0, 2), (2, 0), (5, 8), (33, 40)])
@pytest.mark.parametrize("start,gap", [(4, 0), (1, 3), (7, 1)])
def test_layouts_with_an_offset_or_gaps(nheavy, nlight, start, gap):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200 import kernels as K
    from mopac_gpu_b200._lib import check, lib
    s, rng = _system(nheavy, nlight)
    nfirst, nlast, at = _spread(s, start, gap)
    size = int(nlast[-1]) * (int(nlast[-1]) + 1) // 2
    p = rng.normal(size=s.mpack)
    h, pt, pa = (_place(x, at, size) for x in (s.h, p, 0.5 * p))
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    layout = K.Atoms(nfirst, nlast)

    want = h.copy()
    so.lib().orc_fock2(s.numat, nfirst, nlast, want, pt, pa, s.w)
    f = torch.full((size,), -7.0, dtype=torch.float64, device="cuda")
    K.fock2(layout, f, dev(h), dev(pt), dev(pa), dev(s.w))
    got = f.cpu().numpy()
    assert np.array_equal(got[at], want[at])
    assert np.all(np.delete(got, at) == -7.0)

    nat, xyz = dev(s.nat), dev(s.coord)
    ws = torch.empty(int(lib().mb_dcart_ws_bytes(s.numat)) // 8 + 1, dtype=torch.float64, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def gradient(atoms, density):
        d, g = dev(density), torch.empty(3 * s.numat, dtype=torch.float64, device="cuda")
        check(lib().mb_dcart_dev(nat.data_ptr(), xyz.data_ptr(), ctypes.byref(atoms.s), s.numat, d.data_ptr(),
                                 g.data_ptr(), ws.data_ptr(), 8 * ws.numel(), stream))
        return g.cpu().numpy()

    g = gradient(layout, pt)
    assert np.isfinite(g).all()
    assert np.array_equal(g, gradient(K.Atoms(s.nfirst, s.nlast), p))
