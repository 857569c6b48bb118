"""Element-unit inputs loaded by the 16-byte blocks around their runs (4-byte
elements, runs of 256 bytes or more): every candidate tile, runs just below and
above that length, both store units, every rank class, all positions of the
tensors modulo 16.  Results are bytes: they must be equal, and the bytes around
the output unchanged."""
import numpy as np
import pytest

import librett_gb300 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# runs of 63, 64 and 65 elements; 16-byte stores; a stride that is a multiple of
# 16 bytes; merged leading ranks; three to six tile ranks; one whole tensor in a
# tile; one rank
CASES = [([63, 90, 35], [2, 1, 0]), ([64, 45, 67], [2, 1, 0]), ([65, 90, 64], [2, 1, 0]),
         ([256, 20, 72], [2, 1, 0]), ([6, 91, 11, 16, 10], [4, 0, 3, 2, 1]),
         ([187, 2, 7, 25, 8], [0, 2, 4, 1, 3]), ([65, 3, 5, 7, 3, 9], [5, 3, 0, 2, 4, 1]),
         ([129, 2, 3, 2, 5, 2, 3], [6, 4, 2, 0, 5, 3, 1]), ([67, 33], [1, 0]), ([70001], [0])]


@pytest.mark.parametrize("dims,perm", CASES)
@pytest.mark.parametrize("shift_in", [0, 1, 2, 3])
def test_span_loads(cuda, dims, perm, shift_in):
    import torch

    n = int(np.prod(dims)) * 4
    host = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    want = torch.from_numpy(O.transpose_np(host, dims, perm, 4).view(np.uint8).reshape(-1)).cuda()
    a = 4 * shift_in
    b = 4 * ((3 * shift_in) % 4)
    # the tensor fills its buffer but for the shift: blocks at its ends reach past it
    inp = torch.from_numpy(np.concatenate([np.zeros(a, np.uint8), host])).cuda()
    for cand in range(L.describe(dims, perm, 4)["num_candidates"]):
        out = torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        plan = L.Plan(dims, perm, 4, torch.cuda.current_stream(), candidate=cand)
        plan.execute(inp.data_ptr() + a, out.data_ptr() + b)
        assert torch.equal(out[b:b + n], want), cand
        assert bool((out[:b] == 0xA5).all()) and bool((out[b + n:] == 0xA5).all())
        plan.destroy()
