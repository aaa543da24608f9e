"""The batched eigensolver at the edges of its 16-row tiles: molecules of 2, 8,
14, 16, 20, 32, 34, 46, 50, 64, 80, 82, 94, 98, 112, 116 and 128 basis functions, against
the oracle, with the bars of test_gpu_batch.py (heat 1e-4 kcal/mol, density 1e-6)."""
import numpy as np
import pytest

from mopac_gpu_b200 import workloads
from oracle import scf_oracle as so
from tests.helpers import oracle_system

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

_HEADS = {"h2": ([1, 1], [[0, 0, 0], [0.76, 0, 0]]), "co": ([6, 8], [[0, 0, 0], [1.13, 0, 0]]),
          "ch2o": ([6, 8, 1, 1], [[0, 0, 0], [1.21, 0, 0], [-0.58, 0.94, 0], [-0.58, -0.94, 0]])}


def _molecule(head, waters):
    """A head molecule 10 A from a water lattice."""
    nat, xyz = _HEADS[head]
    nat, xyz = np.array(nat, np.int32), np.array(xyz, float)
    if waters:
        wn, wx = workloads.water_lattice(waters)
        nat, xyz = np.concatenate([nat, wn]), np.concatenate([xyz + wx.min(axis=0) - 10.0, wx])
    return nat, xyz


def test_batch_at_tile_edges():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mopac_gpu_b200.batch import Batch
    mols = [_molecule(*m) for m in (("h2", 0), ("h2", 1), ("h2", 2), ("ch2o", 1), ("co", 2), ("co", 4), ("ch2o", 4),
                                    ("ch2o", 6), ("h2", 8), ("ch2o", 9), ("co", 12), ("ch2o", 12), ("ch2o", 14),
                                    ("h2", 16), ("ch2o", 17), ("co", 18), ("co", 20))]
    b = Batch(mols)
    escf, _, conv, _ = b.run()
    assert conv.all()
    for m, (nat, xyz) in enumerate(mols):
        ref = so.iter_scf(oracle_system(nat, xyz))
        assert abs(escf[m] - ref.escf) < 1e-4, (m, escf[m], ref.escf)
        np.testing.assert_allclose(b.density(m), ref.p, atol=1e-6)
    b.close()
