"""The network kernels layer by layer: each activation, gradient of an activation
and weight gradient against float64 sums of the very float32 numbers that the
kernel had for that layer (its own activations, masks and gradients, which the
workspace holds), so no ReLU can switch between the two.

Bounds: a sum of n products by fused multiply-adds differs from the exact one by at
most n * 2^-24 (and terms of 2^-48) of the sum of their magnitudes.  n is 37 or 128
inputs and the bias for a layer; for a weight gradient the longest serial chain of
the kernel: 32 rows for every 1,024 of the batch, then 4 parts and 8 CTAs.  A bound
counts only if the loss of a single row would exceed it; the test asserts that, too,
for rows whose own gradient is not next to nothing.

Batches: at the edges of the rows per CTA (8, 16, 32 by the device's SMs), of the
128-row chunks, and of the 1,024 rows after which a CTA takes a second chunk."""
import numpy as np
import pytest

from librett_gb300 import _lib
from librett_gb300.learn import train as T

pytestmark = pytest.mark.gpu
H, U = 128, 2.0 ** -24
BATCHES = [1, 7, 8, 9, 127, 128, 129, 895, 896, 897, 1023, 1024, 1025, 1151, 1152, 1153, 1216,
           1217, 2047, 2048, 2049, 2432, 2433, 4999]


def _step(batch, shift):
    """Numbers of one forward and backward pass, every buffer `shift` floats off
    16-byte alignment."""
    import torch

    lib = _lib.load()
    nf = lib.librett_c_mlp_feature_count()
    rng = np.random.default_rng(batch)
    params = T.init_params(nf, rng).astype(np.float32)
    params[-129:-1] = rng.normal(0, 0.3, 128)
    X = rng.normal(size=(batch, nf)).astype(np.float32)
    dout = (rng.normal(size=batch) / batch).astype(np.float32)

    def dev(n, a=None):
        buf = torch.full((n + 4,), float("nan"), device="cuda")
        if a is not None:
            buf[shift:shift + n] = torch.from_numpy(a.ravel()).cuda()
        return buf, buf.data_ptr() + 4 * shift

    p, x, d = dev(params.size, params), dev(X.size, X), dev(batch, dout)
    ws, out, g = dev(5 * batch * H), dev(batch), dev(params.size)
    s = torch.cuda.current_stream().cuda_stream
    assert lib.librett_c_mlp_forward(p[1], x[1], batch, ws[1], out[1], s) == 0
    assert lib.librett_c_mlp_backward(p[1], x[1], batch, ws[1], d[1], g[1], s) == 0
    torch.cuda.synchronize()
    host = [t[0].cpu().numpy()[shift:shift + n] for t, n in
            ((ws, 5 * batch * H), (out, batch), (g, params.size))]
    return nf, params, X, dout, host[0].reshape(5, batch, H), host[1], host[2]


def _split(v, nf):
    W1, b1, W2, b2, W3, b3, W4, b4 = np.split(v, np.cumsum([H * nf, H, H * H, H, H * H, H, H]))
    return [(W1.reshape(H, nf), b1), (W2.reshape(H, H), b2), (W3.reshape(H, H), b3),
            (W4.reshape(1, H), b4)]


def _within(got, want, bound):
    err = np.abs(got.astype(np.float64) - want)
    assert np.all(err <= bound * (1 + 1e-6) + 1e-40), float(np.max(err / (bound + 1e-40)))


@pytest.mark.parametrize("batch", BATCHES)
@pytest.mark.parametrize("shift", [0, 1])
def test_layers(cuda, batch, shift):
    nf, params, X, dout, ws, out, g = _step(batch, shift)
    f64 = np.float64
    layers, grads = _split(params, nf), _split(g, nf)
    acts = [X, ws[0], ws[1], ws[2]]
    for k, (W, b) in enumerate(layers):
        a = acts[k].astype(f64)
        want = a @ W.T.astype(f64) + b.astype(f64)
        size = np.abs(a) @ np.abs(W.T.astype(f64)) + np.abs(b.astype(f64))
        got = acts[k + 1] if k < 3 else out[:, None]
        _within(got, np.maximum(want, 0) if k < 3 else want, (W.shape[1] + 2) * U * size)
    # gradients of the activations
    D3 = np.where(ws[2] > 0, dout[:, None] * layers[3][0], np.float32(0))  # one rounding: equal
    D1, D2 = ws[3], ws[4]
    for got, D, W, mask in ((D2, D3, layers[2][0], ws[1]), (D1, D2, layers[1][0], ws[0])):
        D, W = D.astype(f64), W.astype(f64)
        _within(got, np.where(mask > 0, D @ W, 0), (H + 1) * U * (np.abs(D) @ np.abs(W)))
    # weight gradients
    chain = 32 * -(-batch // 1024) + 4 + 8
    for k, D in enumerate([D1, D2, D3, dout[:, None]]):
        for got, a in zip(grads[k], (acts[k], np.ones((batch, 1), np.float32))):
            D64, a64 = np.abs(D.astype(f64)), np.abs(a.astype(f64))
            want = (D.astype(f64).T @ a.astype(f64)).reshape(got.shape)
            bound = chain * U * (D64.T @ a64).reshape(got.shape)
            _within(got, want, bound)
            for row in {0, batch // 2, max(0, batch - 2), batch - 1, min(1024, batch - 1)}:
                if abs(dout[row]) < 0.05 * np.abs(dout).mean():
                    continue  # a row that hardly counts
                lost = (D64[row][:, None] * a64[row][None, :]).reshape(got.shape)
                assert np.any(lost > 4 * bound), (k, row)
