"""The MLP training kernels at the edges of their work split: rows per CTA (8, 16,
32 by batch size on the device's SMs), the 64-row chunks and 8 shares of the
weight gradients, and buffers that are not 16-byte aligned; against the float64
oracle.

Tolerances: an output or gradient is a sum of at most n = batch or 128 products
in float32, through four layers: relative error to its scale below
4 * n * 2^-24, plus the same again for a ReLU that may switch; 1e-4 covers
n = 256 ... 5000 summed in shares with random signs (sqrt(n) growth)."""
import ctypes

import numpy as np
import pytest

from librett_gb300 import _lib
from librett_gb300.learn import train as T
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _run(batch, shift, seed):
    """out, grads of one batch; every buffer starts `shift` floats off 16-byte
    alignment."""
    import torch

    lib = _lib.load()
    nf = lib.librett_c_mlp_feature_count()
    rng = np.random.default_rng(seed)
    params = T.init_params(nf, rng)
    params[-129:-1] = rng.normal(0, 0.3, 128)
    X = rng.normal(size=(batch, nf)).astype(np.float32)
    y = rng.normal(size=batch).astype(np.float32)

    def dev(a):
        buf = torch.full((a.size + 4,), float("nan"), device="cuda")
        buf[shift:shift + a.size] = torch.from_numpy(a.ravel()).cuda()
        return buf, buf.data_ptr() + 4 * shift

    keep = [dev(a) for a in (params, X, y)]
    (_, p), (_, x), (_, yy) = keep
    ws, out, dout, g = (dev(np.full(n, np.nan, np.float32)) for n in (
        lib.librett_c_mlp_workspace_floats(batch), batch, batch, params.size))
    s = torch.cuda.current_stream().cuda_stream
    loss = torch.zeros(1, device="cuda")
    assert lib.librett_c_mlp_forward(p, x, batch, ws[1], out[1], s) == 0
    assert lib.librett_c_mlp_mse_grad(out[1], yy, batch, dout[1], loss.data_ptr(), s) == 0
    assert lib.librett_c_mlp_backward(p, x, batch, ws[1], dout[1], g[1], s) == 0
    torch.cuda.synchronize()
    host = [t[0].cpu().numpy()[shift:shift + n] for t, n in ((out, batch), (g, params.size))]
    # nothing past the ends
    for t, n in ((out, batch), (g, params.size), (ws, lib.librett_c_mlp_workspace_floats(batch))):
        tail = t[0][shift + n:].cpu().numpy()
        assert np.all(np.isnan(tail))
    return params, X, y, host[0], host[1], float(loss.item())


@pytest.mark.parametrize("batch", [1, 7, 8, 9, 63, 65, 512, 513, 1216, 1217, 2432, 2433, 4999])
@pytest.mark.parametrize("shift", [0, 1])
def test_forward_and_gradients(cuda, batch, shift):
    params, X, y, out, g, loss = _run(batch, shift, batch)
    ref_out, _ = M.forward(params, X)
    ref_loss, ref_g = M.mse_gradients(params, X, y)
    assert np.max(np.abs(out - ref_out)) <= TOL * max(1.0, np.abs(ref_out).max())
    assert abs(loss - ref_loss) <= TOL * max(1.0, ref_loss)
    scale = np.abs(ref_g).max()
    # a ReLU input within rounding of zero may switch: one row's share of a
    # gradient is at most a few / batch of the scale
    assert np.max(np.abs(g - ref_g)) <= (TOL + (8.0 / batch if batch > 1000 else 0.0)) * scale


def test_weight_gradients_repeat(cuda):
    """The shares are combined in a fixed order: two runs agree in every bit."""
    a, b = _run(1500, 0, 3)[4], _run(1500, 0, 3)[4]
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
