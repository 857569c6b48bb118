"""The verifier on outputs that are wrong in many places: exact counts and first
index, and a time that stays within a few passes over the tensors."""
import time

import numpy as np
import pytest

import librett_gb300 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# ragged tiles along one to three ranks, units of 4 to 16 bytes on the output
CASES = [([1000, 517], [1, 0]), ([127, 63, 65], [2, 0, 1]), ([129, 65, 33], [2, 1, 0]),
         ([260, 31, 17], [0, 2, 1]), ([2, 3, 2, 5, 2, 3, 2, 3, 2, 4], [9, 7, 5, 3, 1, 0, 2, 4, 6, 8])]


@pytest.mark.parametrize("es", [4, 8, 16])
@pytest.mark.parametrize("dims,perm", CASES)
@pytest.mark.parametrize("share", [0.01, 0.5, 1.0])
def test_counts(cuda, dims, perm, es, share):
    import torch

    vol = int(np.prod(dims))
    rng = np.random.default_rng(vol)
    host = rng.integers(0, 256, vol * es, dtype=np.uint8)
    want = O.transpose_np(host, dims, perm, es).view(np.uint8).copy().reshape(vol, es)
    bad = rng.random(vol) < share
    want[np.flatnonzero(bad), rng.integers(0, es, int(bad.sum()))] ^= 64
    inp, out = torch.from_numpy(host).cuda(), torch.from_numpy(want.reshape(-1)).cuda()
    got = L.verify(dims, perm, es, inp.data_ptr(), out.data_ptr(), torch.cuda.current_stream())
    assert got == (int(bad.sum()), int(np.flatnonzero(bad)[0]))


@pytest.mark.parametrize("dims,perm,es", [([64, 128, 96, 85], [3, 1, 0, 2], 4),
                                          ([127, 63, 65, 33], [3, 1, 2, 0], 4),
                                          ([96, 24, 131, 18, 6], [3, 1, 4, 0, 2], 8),
                                          ([200, 300, 100], [2, 1, 0], 16)])
def test_time_of_a_wrong_output(cuda, dims, perm, es):
    """A wrong output is read a second time, to be counted: at most five times the
    time of a right one (atomics for every wrong element took 8 to 33 times)."""
    import torch

    s = torch.cuda.current_stream()
    vol = int(np.prod(dims))
    inp = torch.randint(0, 2 ** 31 - 1, (vol * es // 4,), dtype=torch.int32, device="cuda")
    out = torch.empty_like(inp)
    with L.Plan(dims, perm, es, s) as p:
        p.execute(inp.data_ptr(), out.data_ptr())

    def best(expected):
        times = []
        for _ in range(7):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            assert L.verify(dims, perm, es, inp.data_ptr(), out.data_ptr(), s) == expected
            times.append(time.perf_counter() - t0)
        return min(times)

    right = best((0, -1))
    out[::es // 4] ^= 1
    assert best((vol, 0)) < 5 * right


@pytest.mark.parametrize("es", [4, 8, 16])
def test_no_tile(cuda, es):
    """A tensor of one element has no tile and goes element by element."""
    import torch

    inp = torch.arange(1, es + 1, dtype=torch.uint8, device="cuda")
    out = inp.clone()
    s = torch.cuda.current_stream()
    assert L.verify([1], [0], es, inp.data_ptr(), out.data_ptr(), s) == (0, -1)
    out[es - 1] ^= 1
    assert L.verify([1], [0], es, inp.data_ptr(), out.data_ptr(), s) == (1, 0)
