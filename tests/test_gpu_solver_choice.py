"""Which eigensolver an SCF's iterations take: the blocked one (panels) where
pseudo-diagonalisation turns a last bit into a decision, the on-chip one elsewhere.
Camp-King switches the pseudo-diagonalisation off, so such an SCF has nothing to
decide and must give the plain one's result bit for bit."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run(**kw):
    from mopac_gpu_b200 import workloads
    from mopac_gpu_b200._lib import lib
    from mopac_gpu_b200.scf import ScfContext
    L = lib()
    ctx = ScfContext(*workloads.water_lattice(8))
    ctx.hcore()
    L.mb_kstats_read(0, None, None)
    L.mb_kstats_enable(1)
    r = ctx.run(**kw)
    L.mb_kstats_enable(0)
    panels = ctypes.c_longlong(0)
    L.mb_kstats_read(0, ctypes.byref(panels), None)
    p = ctx.density()
    ctx.close()
    return r, p, panels.value


def test_solver_follows_what_the_iterations_do():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    assert _run()[2] == 0
    r, _, panels = _run(pseudo=True)
    assert r.n_pseudo_diag > 0 and panels > 0
    plain, p0, _ = _run(camp=True)
    both, p1, panels = _run(camp=True, pseudo=True)
    assert both.n_pseudo_diag == 0 and both.converged
    assert panels == 0
    assert both.escf == plain.escf and np.array_equal(p0, p1)
