"""diagg2's rotations and diagg1's occupied energies over atom lists at the
lengths where their kernels change: 128 atoms a round, 512 atoms for a
rotation by a CTA (longer lists by one warp), 128 terms a step of the energies.
Bit for bit against the oracle's sequential loops."""
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


@pytest.mark.parametrize("sizes_o,sizes_v,pad", [
    ((1, 2, 3, 32, 33), (1, 31, 4), 2),
    ((127, 128, 129, 40), (126, 128, 130), 400),
    ((127, 128, 129, 40), (126, 128, 130), 1),          # no room: rejected and retried
    ((255, 256, 257), (384, 383, 10), 300),
    ((511, 512, 513, 600), (512, 509, 514), 640),       # either side of the CTA's 512 atoms
])
def test_rotations_over_lists_of_every_form(sizes_o, sizes_v, pad):
    torch = _torch()
    from mopac_gpu_b200 import mozyme
    nat, xyz, iorbs, c1, c2 = _system(216)
    rng = np.random.default_rng(sum(sizes_o))
    occ, vir = _lmos(iorbs, sizes_o, pad, rng), _lmos(iorbs, sizes_v, pad, rng)
    no, nv = len(sizes_o), len(sizes_v)
    pairs = [(i, j) for i in range(nv) for j in range(no)] * 2
    nij = len(pairs)
    ifmo = np.array([[i + 1, j + 1] for i, j in pairs], np.int32).reshape(-1)
    fmo = rng.normal(size=nij) * 0.3
    eigs, eigv = rng.uniform(-20.0, -10.0, no), rng.uniform(1.0, 5.0, nv)
    L = mozyme.Layout(iorbs, xyz, c1, c2)
    qo, qv = mozyme.Lmos(L, occ), mozyme.Lmos(L, vir)
    ro, rv = tuple(x.copy() for x in occ), tuple(x.copy() for x in vir)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    lst = mozyme._HbList(dev(ifmo), dev(fmo), nij, dev(eigs), dev(eigv))
    ctl = [1.0, 0.0, 1.0e-13, 0.0, 50 * np.sqrt(1e-39)]
    nro, nrg = np.zeros(2, np.int32), np.zeros(2, np.int32)
    for idg in (0, 1, 6):
        sb_o, nr_o = mo.diagg2(iorbs, ro, rv, ifmo, fmo, nij, eigs, eigv, idg, ctl, nro)
        sb_g, nr_g = mozyme.diagg2(L, qo, qv, lst, idg, ctl, nrg)
        assert nr_g == nr_o and np.array_equal(nrg, nro)
        assert sb_g == pytest.approx(sb_o, rel=1e-13)
        for ref, q in ((ro, qo), (rv, qv)):
            n, ic, c = q.to_host()
            np.testing.assert_array_equal(n, ref[0])
            np.testing.assert_array_equal(ic, ref[2])
            np.testing.assert_array_equal(c, ref[4])
    L.close()


@pytest.mark.parametrize("sizes", [(1, 3, 31, 33), (127, 128, 129), (256, 257, 600)])
def test_occupied_energies_over_lists_of_every_length(sizes):
    torch = _torch()
    from mopac_gpu_b200 import mozyme
    nat, xyz, iorbs, c1, c2 = _system(200)
    s = so.make_system(nat, xyz)
    rng = np.random.default_rng(sizes[-1])
    mp, nb = mo.layout(iorbs, s.coord, c1, c2)
    f, p = rng.normal(size=mp), rng.normal(size=mp)
    occ, vir = _lmos(iorbs, sizes, 2, rng), _lmos(iorbs, (3, 5), 2, rng)
    cap = 4096
    L = mozyme.Layout(iorbs, s.coord, c1, c2)
    qo, qv = mozyme.Lmos(L, occ), mozyme.Lmos(L, vir)
    D = mozyme.Diagg1(L, qo, qv, cap)
    st = np.array([10.0, 1.0, 0.0, 0.0])
    nfmo, ifmo, fmo = np.zeros(2, np.int32), np.zeros(2 * cap, np.int32), np.zeros(cap)
    nij, eigv, eigs, _ = mo.diagg1(iorbs, nb, f, p, occ, vir, 0, st, nfmo, ifmo, fmo, cap)
    got, done, _ = D(torch.from_numpy(f).cuda(), torch.from_numpy(p).cuda(), 0)
    assert got == nij and done
    np.testing.assert_array_equal(D.eigs.cpu().numpy(), eigs)
    L.close()
