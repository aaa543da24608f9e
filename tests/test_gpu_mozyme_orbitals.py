"""Occupied LMO energies over atoms with one to four orbitals, as a layout takes them,
at the list lengths where the kernel changes.  Bit for bit against the
oracle's sequential loops."""
import numpy as np
import pytest

from mopac_gpu_b200 import workloads
from oracle import mozyme_oracle as mo
from oracle import scf_oracle as so

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def _lmos(iorbs, sizes, pad, rng):
    """LMOs over the given numbers of atoms, drawn without repeats, unit
    coefficients, pad spare atom slots each."""
    ncf, nncf, icocc, ncocc, cocc = [], [], [], [], []
    for size in sizes:
        atoms = rng.permutation(len(iorbs))[:size]
        nncf.append(len(icocc))
        ncocc.append(len(cocc))
        ncf.append(size)
        vec = rng.normal(size=int(iorbs[atoms].sum()))
        icocc.extend((atoms + 1).tolist() + [0] * pad)
        cocc.extend((vec / np.linalg.norm(vec)).tolist() + [0.0] * (4 * pad))
    return (np.array(ncf, np.int32), np.array(nncf, np.int32), np.array(icocc, np.int32),
            np.array(ncocc, np.int32), np.array(cocc, np.float64))


def _system(nwater):
    nat, xyz = workloads.water_lattice(nwater)
    iorbs = np.where(nat == 1, 1, 4).astype(np.int32)
    c1, c2 = mo.cutoffs(len(iorbs), 9.0)
    return nat, xyz, iorbs, c1, c2


@pytest.mark.parametrize("counts", [(2, 3), (1, 2, 3, 4)])
@pytest.mark.parametrize("sizes", [(1, 3, 31, 33), (127, 128, 129), (256, 257)])
def test_occupied_energies_of_atoms_with_any_orbital_count(counts, sizes):
    torch = _torch()
    from mopac_gpu_b200 import mozyme
    nat, xyz = workloads.water_lattice(100)
    c1, c2 = mo.cutoffs(len(nat), 9.0)
    s = so.make_system(nat, xyz, integrals=False)
    rng = np.random.default_rng(sizes[-1] + len(counts))
    iorbs = rng.choice(counts, size=len(nat)).astype(np.int32)
    mp, nb = mo.layout(iorbs, s.coord, c1, c2)
    f, p = rng.normal(size=mp), rng.normal(size=mp)
    occ, vir = _lmos(iorbs, sizes, 2, rng), _lmos(iorbs, (3, 5), 2, rng)
    cap = 4096
    L = mozyme.Layout(iorbs, s.coord, c1, c2)
    D = mozyme.Diagg1(L, mozyme.Lmos(L, occ), mozyme.Lmos(L, vir), cap)
    st = np.array([10.0, 1.0, 0.0, 0.0])
    nfmo, ifmo, fmo = np.zeros(2, np.int32), np.zeros(2 * cap, np.int32), np.zeros(cap)
    nij, eigv, eigs, _ = mo.diagg1(iorbs, nb, f, p, occ, vir, 0, st, nfmo, ifmo, fmo, cap)
    got, done, _ = D(torch.from_numpy(f).cuda(), torch.from_numpy(p).cuda(), 0)
    assert got == nij and done
    np.testing.assert_array_equal(D.eigs.cpu().numpy(), eigs)
    L.close()
