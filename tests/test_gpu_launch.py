"""Launches of single plans: more grid ranks than the small parameter blocks
hold, and chains in which each launch reads what the one before wrote (such
launches may start before their predecessor has ended), plain, captured into a
graph and as one-launch groups (a group's own graph cannot be captured).  Results are bytes: they must be equal."""
import numpy as np
import pytest

import librett_gb300 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# tiles of 2 and 3 ranks over 7 (the small block's last) to 13 grid ranks
MANY = [([17] + [3] * 9 + [19], [10] + list(range(9, 0, -1)) + [0], 4),
        ([40] + [2] * 10 + [40], [11] + list(range(10, 0, -1)) + [0], 8),
        ([70] + [2] * 8 + [3, 70], [10] + list(range(9, 0, -1)) + [0], 16),
        ([70] + [2] * 12 + [70], [13] + list(range(12, 0, -1)) + [0], 4)]


@pytest.mark.parametrize("dims,perm,es", MANY)
@pytest.mark.parametrize("shift", [0, 1])
def test_many_grid_ranks(cuda, dims, perm, es, shift):
    import torch

    shift = shift if es < 16 else 0  # 16-byte elements are always 16-byte aligned
    nbytes = int(np.prod(dims)) * es
    host = np.random.default_rng(es).integers(0, 256, nbytes, dtype=np.uint8)
    want = torch.from_numpy(O.transpose_np(host, dims, perm, es).view(np.uint8).reshape(-1)).cuda()
    pad = shift * es
    inp = torch.from_numpy(np.concatenate([np.zeros(pad, np.uint8), host])).cuda()
    most = 0
    for cand in range(L.describe(dims, perm, es)["num_candidates"]):
        out = torch.zeros_like(inp)
        plan = L.Plan(dims, perm, es, torch.cuda.current_stream(), candidate=cand)
        info = plan.info()
        most = max(most, sum(d > e for d, e in zip(info["fused_dim"], info["tile_extent"])))
        plan.execute(inp.data_ptr() + pad, out.data_ptr() + pad)
        assert torch.equal(out[pad:], want), cand
        plan.destroy()
    assert most >= 7


def _there_and_back(dims, perm, es):
    inverse = [perm.index(i) for i in range(len(perm))]
    return (dims, perm, es), ([dims[p] for p in perm], inverse, es)


# one tile a kernel; several waves; rows; copies; element units; a table tile
CHAINS = [([64, 48, 32], [2, 0, 1], 4), ([127, 63, 65, 9], [3, 1, 2, 0], 4),
          ([300, 200, 60], [2, 1, 0], 8), ([200, 30, 40], [0, 2, 1], 8), ([4099], [0], 16),
          ([2] * 16, list(range(15, -1, -1)), 4)]


@pytest.mark.parametrize("dims,perm,es", CHAINS)
@pytest.mark.parametrize("form", ["plain", "captured", "grouped"])
def test_dependent_chain(cuda, dims, perm, es, form):
    import torch

    nbytes = int(np.prod(dims)) * es
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        a, b = (torch.randint(0, 256, (nbytes,), dtype=torch.uint8, device="cuda")
                for _ in range(2))
        first = a.clone()
        there, back = (L.Plan(*p, stream) for p in _there_and_back(dims, perm, es))
        steps = [(there, a.data_ptr(), b.data_ptr()), (back, b.data_ptr(), a.data_ptr())]
        if form == "grouped":
            groups = [L.Group([p], [i], [o], stream) for p, i, o in steps]
            runs = [g.execute for g in groups]
        else:
            runs = [lambda s=s: s[0].execute(s[1], s[2]) for s in steps]
        stream.synchronize()
    host = first.cpu().numpy()
    want = torch.from_numpy(O.transpose_np(host, dims, perm, es).view(np.uint8).reshape(-1)).cuda()
    torch.cuda.synchronize()

    def chain():
        for _ in range(20):
            runs[0]()
            runs[1]()

    if form == "captured":
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            chain()
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
    else:
        chain()
    stream.synchronize()
    assert torch.equal(a, first) and torch.equal(b, want)
