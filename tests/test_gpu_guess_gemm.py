"""The networks' BF16 GEMM at the edges of its 64-row tiles, of the weight
gradients' 128-row slices, and on operands that allow no 8-byte copies.

Bound on gradients against the oracle (which rounds at the same places but
sums in another order): a path from an input to a gradient carries at most
twelve BF16 roundings (input, weight and activation of four layers), each
2^-8 at worst, 12/256 = 4.7e-2 of the gradient's norm."""
import numpy as np
import pytest

from oracle import guess_oracle as go

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    x = go.bf16(rng.normal(size=(n, go.DIN)).astype(np.float32))
    return x, rng.normal(size=(n, go.DOUT)).astype(np.float32)


def _bits(x):
    return torch.tensor(go.bf16_bits(x).view(np.int16), device="cuda")


@pytest.mark.parametrize("n", [1, 31, 64, 65, 127, 128, 129, 600, 4097])
def test_gradients_at_tile_and_slice_edges(n):
    from mopac_gpu_b200.guess import Trainer
    blob = go.init_blob(6)
    x, yt = _rows(n, n)
    for t in (0, 1):
        tr = Trainer(blob, n)
        tr.step(t, _bits(x), torch.tensor(yt, device="cuda"), 1e-3, update=False)
        params, grads = tr.get()
        assert np.array_equal(params, blob)  # update=False leaves the weights alone
        _, want, _ = go.loss_and_grads(go.unpack_blob(blob)[t], x, yt, int(go.NOUT[t]))
        got = go.unpack_blob(grads)[t]
        for k in go.TRAINABLE:
            assert np.linalg.norm(got[k] - want[k]) <= 4.7e-2 * np.linalg.norm(want[k]), (t, k)
        tr.close()


@pytest.mark.parametrize("n", [1, 65, 300])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_input_rows_off_an_8_byte_boundary(n, shift):
    from mopac_gpu_b200._lib import lib
    from mopac_gpu_b200.guess import GuessModel
    model = GuessModel(go.init_blob(5))
    xd = _bits(_rows(n, 7)[0])
    moved = torch.empty(n * go.DIN + shift, dtype=torch.int16, device="cuda")
    moved[shift:] = xd.view(-1)
    ws = torch.empty(2 * n * go.HID, dtype=torch.int16, device="cuda")
    y = [torch.empty((n, go.DOUT), dtype=torch.float32, device="cuda") for _ in range(2)]
    s = torch.cuda.current_stream().cuda_stream
    assert lib().mb_guess_forward_dev(model.handle, 0, n, xd.data_ptr(), y[0].data_ptr(), ws.data_ptr(), s) == 0
    assert lib().mb_guess_forward_dev(model.handle, 0, n, moved.data_ptr() + 2 * shift, y[1].data_ptr(),
                                      ws.data_ptr(), s) == 0
    assert torch.equal(y[0], y[1])
    model.close()
