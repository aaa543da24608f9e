"""Callers on several threads: a kernel's opt-in to its shared memory is the
function's, so one caller's order must not take it from another's.  Two threads
queue reductions of different orders, which run the same instance of the grid
kernel with 40 and with 56 KB, on one stream (the kernels run one after another; only
the host side overlaps)."""
import ctypes
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

P, I = ctypes.c_void_p, ctypes.c_int


class _Reduction:
    def __init__(self, n, seed):
        a = np.random.default_rng(seed).normal(size=(n, n))
        self.n, self.a = n, torch.from_numpy(a + a.T).cuda()
        self.vall, self.scratch = torch.zeros_like(self.a), torch.empty(8 * n + 2, dtype=torch.float64, device="cuda")
        self.d, self.e, self.tau = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3))
        self.status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def __call__(self, L, stream):
        return L.mb_tridiag_grid(self.n, 148, self.a.data_ptr(), self.n, self.vall.data_ptr(), self.d.data_ptr(),
                                 self.e.data_ptr(), self.tau.data_ptr(), self.scratch.data_ptr(),
                                 self.status.data_ptr(), stream)


def test_two_threads_with_orders_of_different_shared_memory():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from mopac_gpu_b200._lib import lib
    L = lib()
    L.mb_tridiag_grid.argtypes = [I, I, P, ctypes.c_longlong] + [P] * 7
    L.mb_tridiag_grid.restype = I
    stream = torch.cuda.current_stream().cuda_stream
    both = [_Reduction(700, 1), _Reduction(1024, 2)]
    torch.cuda.synchronize()
    alone = []
    for r in both:
        assert r(L, stream) == 0
        alone.append((r.d.clone(), r.e.clone()))
    torch.cuda.synchronize()
    start, codes = threading.Barrier(2), [[], []]

    def work(k):
        start.wait()
        for _ in range(200):
            codes[k].append(both[k](L, stream))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [[0] * 200, [0] * 200]
    for r, (d, e) in zip(both, alone):
        assert int(r.status.item()) == 0
        assert torch.equal(r.d, d) and torch.equal(r.e[:-1], e[:-1])


FIRST = """
import sys, threading, numpy as np, torch
from mopac_gpu_b200 import workloads
from mopac_gpu_b200.scf import ScfContext
done, bad = [], []
start = threading.Barrier(4)
def work(k):
    try:
        ctx = ScfContext(*workloads.water_lattice(24))
        ctx.hcore()
        start.wait()
        r = ctx.run(pseudo=True, pulay=bool(k & 1))
        done.append((k & 1, r.escf, ctx.density().tobytes()))
        ctx.close()
    except Exception as e:
        bad.append(repr(e))
threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not bad, bad
for kind in (0, 1):
    a, b = [d[1:] for d in done if d[0] == kind]
    assert a == b
print("same", len(done))
"""


def test_contexts_that_come_first_together():
    """Four threads whose contexts run the process's first SCFs: what a kernel's
    launcher finds out once (grid sizes, limits) is whole for every one of them."""
    import os
    import subprocess
    import sys
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", FIRST], capture_output=True, text=True, timeout=300, cwd=root)
    assert out.returncode == 0, out.stderr[-2000:]
    assert "same 4" in out.stdout
