"""Pair integrals and the gradient by kind of pair (two heavy atoms, mixed, two
light ones): molecules without one or two of the kinds, light atoms before and
after the heavy ones, pair counts around a warp's eight, and atoms beyond the
7 A feathering radius, against the oracle.

Tolerances: the integrals agree to rounding (1e-12); the gradient divides
differences of pair energies (1e-13 eV) by 1e-4 A: 23 * 1e-13 / 1e-4 kcal/mol/A a
pair, 1e-5 for the few hundred pairs of the largest."""
import numpy as np
import pytest

from oracle import scf_oracle as so

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _molecule(kinds, spread):
    nat = np.array([{"H": 1, "C": 6, "O": 8}[k] for k in kinds], np.int32)
    rng = np.random.default_rng(len(kinds))
    grid = np.array([(x, y, z) for x in range(4) for y in range(4) for z in range(4)], float)[:len(kinds)]
    return nat, spread * grid + 0.1 * rng.normal(size=(len(kinds), 3))


@pytest.mark.parametrize("spread", [1.4, 4.5])
@pytest.mark.parametrize("kinds", ["HH", "OO", "OC", "HHO", "OHH", "CHHHH", "HHHHC", "OCOCOC", "HHHHHHHH",
                                   "HOHCHOHCHH", "CCCCHHHHHOOHHHHH", "HO" * 12])
def test_integrals_and_gradient_by_kind(kinds, spread):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200.scf import ScfContext
    nat, xyz = _molecule(kinds, spread)
    s = so.make_system(nat, xyz)
    ctx = ScfContext(nat, xyz)
    ctx.hcore()
    h, w, en = ctx.get_hw()
    np.testing.assert_allclose(h, s.h, rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(w, s.w, rtol=1e-12, atol=1e-12)
    assert abs(en - s.enuclr) < 1e-9 * abs(s.enuclr)
    ctx.run()
    g = ctx.gradient()
    ref = so.dcart(s, ctx.density())
    assert np.abs(g - ref).max() < 1e-5
    ctx.close()
