"""The bench's account of the Householder reductions: panels and on-chip kernels
apart, the launches each should have made from the orders and the solver that runs,
and the panels' bytes over the columns they reduce only."""
import os
import sys
from types import SimpleNamespace

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def _result(full, split, n_split=0):
    return SimpleNamespace(n_full_diag=full, exit_split=split, n_split=n_split)


def test_reductions_of_each_mode():
    import bench
    ctx = SimpleNamespace(norbs=3072, nclose=2048)
    fast = bench.reductions(ctx, [_result(2, True), _result(3, False)], pseudo=True)
    assert fast == [(3072, 3071)] * 2 + [(2048, 0), (1024, 0)] + [(3072, 3071)] * 2 + [(3072, 1024)]
    assert bench.reductions(ctx, [_result(2, False)], pseudo=False) == [(3072, 1024)] * 2
    assert bench.reductions(ctx, [_result(4, False, 2)], pseudo=False) == [(3072, 3071)] * 2 + [(3072, 1024)] * 2
    small = SimpleNamespace(norbs=2049, nclose=1366)
    assert bench.reductions(small, [_result(1, False)], pseudo=False) == [(2049, 32)]


def test_panels_and_on_chip_kernels_are_reported_apart():
    import bench
    ctx = SimpleNamespace(norbs=3072, nclose=2048)
    kst = {"tridiag_panel": {"launches": 96 + 32, "total_ms": 100.0}, "tridiag_onchip": {"launches": 2, "total_ms": 16.0}}
    r = bench.panel_roofline(ctx, kst, [3072, 3072], [3071, 1024])
    assert r["launches"] == r["launches_expected"] == 96 + 32
    algo = 8.0 * sum(float(m) ** 2 for m in range(1, 3072)) + 8.0 * sum(float(m) ** 2 for m in range(2048, 3072))
    assert abs(r["achieved"] - algo / 0.1 / 1e9) < 1e-9 * r["achieved"]
    assert "grid" not in r["kernel"]
    o = bench.onchip_reduction(kst, [2048, 1024])
    assert o["launches"] == o["launches_expected"] == 2
    assert abs(o["us_per_column"] - 16.0e3 / (2047 + 1023)) < 1e-9
    assert "hbm" not in o["bound"]
    assert bench.onchip_reduction({"tridiag_onchip": {"launches": 0, "total_ms": 0.0}}, []) is None


@pytest.mark.gpu
@pytest.mark.parametrize("waters,kw", [(8, {}), (120, {}), (8, {"pseudo": True, "pulay": True}), (8, {"precision": 1})])
def test_launches_are_the_expected_ones(waters, kw):
    import ctypes
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import bench
    from mopac_gpu_b200 import workloads
    from mopac_gpu_b200._lib import lib
    from mopac_gpu_b200.scf import ScfContext
    L = lib()
    ctx = ScfContext(*workloads.water_lattice(waters))
    ctx.hcore()
    for k in range(len(bench.KSTATS)):
        L.mb_kstats_read(k, None, None)
    L.mb_kstats_enable(1)
    r = ctx.run(**kw)
    L.mb_kstats_enable(0)
    kst = {}
    for k, name in enumerate(bench.KSTATS):
        n, ms = ctypes.c_longlong(0), ctypes.c_double(0.0)
        L.mb_kstats_read(k, ctypes.byref(n), ctypes.byref(ms))
        kst[name] = {"launches": n.value, "total_ms": ms.value}
    done = bench.reductions(ctx, [r], kw.get("pseudo", False))
    panels = bench.panel_roofline(ctx, kst, [m for m, c in done if c], [c for _, c in done if c])
    chip = bench.onchip_reduction(kst, [m - c for m, c in done if m - c > 1])
    assert (panels is None) == (not kw)
    if panels:
        assert panels["launches"] == panels["launches_expected"]
    assert chip["launches"] == chip["launches_expected"] > 0
    ctx.close()
