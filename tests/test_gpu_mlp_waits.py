"""The network kernels' bounded waits: a wait armed with more bytes than its copies
bring runs out after its time limit; the launch then ends with NaN for all results,
and the next launches are right.  Nothing faults: the copies land normally."""
import time

import numpy as np
import pytest

import librett_gb300 as L
from librett_gb300 import _lib
from librett_gb300.learn import train as T

H = 128


def test_arguments():
    """Refused before any launch: no buffers, waits and byte counts out of range."""
    lib = _lib.load()
    p = 16  # never followed
    bad = [(0, 3, 16, p, p, 8, p, p), (1, 2, 16, p, p, 8, p, p), (0, -1, 16, p, p, 8, p, p),
           (0, 0, 0, p, p, 8, p, p), (0, 0, 4097, p, p, 8, p, p), (0, 0, 16, p + 4, p, 8, p, p),
           (0, 0, 16, None, p, 8, p, p), (0, 0, 16, p, None, 8, p, p), (0, 0, 16, p, p, 8, p, None),
           (0, 0, 16, p, p, 0, p, p), (0, 0, 16, p, p, 4097, p, p)]
    for args in bad:
        assert lib.librett_c_mlp_wait_test(*args, None) == L.LIBRETT_INVALID_PARAMETER, args


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [13, 1300])
@pytest.mark.parametrize("backward,wait", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 1)])
def test_wait_runs_out(cuda, batch, backward, wait):
    import torch

    lib = _lib.load()
    nf = lib.librett_c_mlp_feature_count()
    rng = np.random.default_rng(batch)
    p = torch.from_numpy(T.init_params(nf, rng)).cuda()
    X, dout = (torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
               for n in (batch * nf, batch))
    ws = torch.zeros(lib.librett_c_mlp_workspace_floats(batch), device="cuda")
    out = torch.zeros(batch, device="cuda")
    g = torch.zeros(p.numel(), device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def step():
        args = (p.data_ptr(), X.data_ptr(), batch, ws.data_ptr())
        assert lib.librett_c_mlp_forward(*args, out.data_ptr(), s) == 0
        assert lib.librett_c_mlp_backward(*args, dout.data_ptr(), g.data_ptr(), s) == 0
        torch.cuda.synchronize()
        return [t.clone() for t in (out, ws, g)]

    before = step()
    assert not any(bool(torch.isnan(t).any()) for t in before)
    t0 = time.monotonic()
    rc = lib.librett_c_mlp_wait_test(backward, wait, 16, p.data_ptr(), X.data_ptr(), batch,
                                     ws.data_ptr(), (dout if backward else out).data_ptr(), s)
    waited = time.monotonic() - t0
    assert rc == L.LIBRETT_SUCCESS and 0.9 < waited < 30.0, waited
    forward_part = slice(0, 3 * batch * H)
    if backward:
        assert bool(torch.isnan(ws[3 * batch * H:]).all())
        assert torch.equal(ws[forward_part], before[1][forward_part])
    else:
        assert bool(torch.isnan(out).all()) and bool(torch.isnan(ws[forward_part]).all())
        assert torch.equal(ws[3 * batch * H:], before[1][3 * batch * H:])
    for a, b in zip(step(), before):
        assert torch.equal(a, b)
