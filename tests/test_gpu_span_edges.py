"""Span loads at the length of run from which a tile uses them, 32 4-byte elements
(128 bytes): runs of 31 to 36 elements, whole or merged from leading dims, which take
the most blocks for their bytes; every candidate tile, all positions of the tensors
modulo 16, the tensor filling its buffer.  Results are bytes: they must be equal, and
the bytes around the output unchanged."""
import numpy as np
import pytest

import librett_gb300 as L
from librett_gb300 import _lib
from oracle import oracle as O

CASES = [([r, a, b], [2, 1, 0]) for r in (31, 32, 33, 36) for a, b in ((64, 67), (7, 1030))]
CASES += [([4, 9, 45, 31], [3, 1, 2, 0]), ([3, 11, 50, 29], [2, 0, 3, 1]),
          ([33, 3, 5, 7, 3, 9], [5, 3, 0, 2, 4, 1]), ([32, 128], [1, 0]), ([33, 124], [1, 0])]


@pytest.mark.parametrize("dims,perm", CASES)
def test_addresses(dims, perm):
    """The blocks' addresses on the host: of the tile, and of it in element units."""
    for units in (0, 1):
        for cand in range(20):
            rc = _lib.load().librett_c_slot_check(len(dims), _lib.int_array(dims),
                                                  _lib.int_array(perm), 4, 152, cand, units)
            if rc == L.LIBRETT_INVALID_PARAMETER:
                assert cand > 0
                break
            assert rc == L.LIBRETT_SUCCESS, (cand, units)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,perm", CASES)
@pytest.mark.parametrize("shift_in", [0, 1, 2, 3])
@pytest.mark.parametrize("shift_out", [0, 3])
def test_span_edges(cuda, dims, perm, shift_in, shift_out):
    import torch

    n, a, b = int(np.prod(dims)) * 4, 4 * shift_in, 4 * shift_out
    host = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    want = torch.from_numpy(O.transpose_np(host, dims, perm, 4).view(np.uint8).reshape(-1)).cuda()
    inp = torch.from_numpy(np.concatenate([np.zeros(a, np.uint8), host])).cuda()
    for cand in range(L.describe(dims, perm, 4)["num_candidates"]):
        out = torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        with L.Plan(dims, perm, 4, torch.cuda.current_stream(), candidate=cand) as plan:
            plan.execute(inp.data_ptr() + a, out.data_ptr() + b)
        assert torch.equal(out[b:b + n], want), cand
        assert bool((out[:b] == 0xA5).all()) and bool((out[b + n:] == 0xA5).all())
