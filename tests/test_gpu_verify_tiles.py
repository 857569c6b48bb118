"""The tiled verifier: planted mismatches are counted once and the first one is
found, also in the overlap of ragged last tiles, for both unit widths, unaligned
pointers and every element size."""
import numpy as np
import pytest

import librett_gb300 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# ragged tiles on one and two ranks, 16-byte and element units on either side,
# small leading dims, one rank, a leading dim that stays, high rank
CASES = [([1000, 517], [1, 0]), ([129, 65, 33], [2, 1, 0]), ([128, 96, 40], [1, 2, 0]),
         ([2, 3, 4, 5, 257], [4, 1, 0, 3, 2]), ([70001], [0]), ([260, 31, 17], [0, 2, 1]),
         ([2, 3, 2, 5, 2, 3, 2, 3, 2, 4], [9, 7, 5, 3, 1, 0, 2, 4, 6, 8])]


@pytest.mark.parametrize("es", [4, 8, 16])
@pytest.mark.parametrize("dims,perm", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_planted_mismatches(cuda, dims, perm, es, shift):
    import torch

    if es == 16 and shift:
        shift = 0  # 16-byte elements are always 16-byte aligned
    vol = int(np.prod(dims))
    rng = np.random.default_rng(vol + es)
    host = rng.integers(0, 256, vol * es, dtype=np.uint8)
    want = O.transpose_np(host, dims, perm, es).view(np.uint8)
    pad = shift * es
    inp = torch.from_numpy(np.concatenate([np.zeros(pad, np.uint8), host])).cuda()
    out = torch.from_numpy(np.concatenate([np.zeros(pad, np.uint8), want])).cuda()

    def verify():
        return L.verify(dims, perm, es, inp.data_ptr() + pad, out.data_ptr() + pad,
                        torch.cuda.current_stream())

    assert verify() == (0, -1)
    # some elements, and all of the last ones (the overlap of the last tiles)
    bad = np.unique(np.concatenate([rng.integers(0, vol, 40), np.arange(max(0, vol - 700), vol)]))
    out[torch.from_numpy(pad + bad * es + int(rng.integers(es))).cuda()] ^= 1
    assert verify() == (len(bad), int(bad[0]))
    # every element
    out[pad::es] ^= 2
    assert verify() == (vol, 0)
