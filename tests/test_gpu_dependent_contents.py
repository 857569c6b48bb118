"""Chains of launches in which every launch finds other bytes in its input than any
launch of the three before it found or wrote there, so a launch that read before its
predecessor had ended, or read a line from an earlier launch, ends in other bytes.
Launches are small, several of them run at once.  Results are bytes: equal."""
import numpy as np
import pytest

import librett_gb300 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# permutations of order 3 and more over equal dims: register and cp.async tiles in
# 16-byte, 8-byte and element units, rows, a small leading dim, tiles with tables
CHAINS = [([32, 32, 32], [1, 2, 0], 4), ([33, 33, 33], [1, 2, 0], 4), ([65, 65, 65], [1, 2, 0], 4),
          ([24, 24, 24], [1, 2, 0], 8), ([31, 31, 31], [1, 2, 0], 8), ([20, 20, 20], [1, 2, 0], 16),
          ([40, 16, 16, 16], [0, 2, 3, 1], 8), ([3, 17, 17, 17], [0, 2, 3, 1], 4),
          ([2] * 14, [9, 2, 12, 0, 5, 13, 1, 7, 10, 4, 3, 11, 8, 6], 4)]
ROUNDS = 25


def _buffers(n):
    import torch

    return [torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda") for _ in range(2)]


def _after(host, dims, perm, es, times):
    for _ in range(times):
        host = O.transpose_np(host, dims, perm, es).view(np.uint8).reshape(-1)
    return host


@pytest.mark.parametrize("dims,perm,es", CHAINS)
@pytest.mark.parametrize("shift", [0, 1])
def test_transposes(cuda, dims, perm, es, shift):
    """a -> b -> a -> ..., every candidate."""
    import torch

    pad = shift * es if es < 16 else 0
    n = int(np.prod(dims)) * es
    s = torch.cuda.current_stream()
    for cand in range(L.describe(dims, perm, es)["num_candidates"]):
        a, b = _buffers(n + pad)
        first = a[pad:].cpu().numpy()
        pa, pb = a.data_ptr() + pad, b.data_ptr() + pad
        with L.Plan(dims, perm, es, s, candidate=cand) as p:
            for _ in range(ROUNDS):
                p.execute(pa, pb)
                p.execute(pb, pa)
            torch.cuda.synchronize()
        last = _after(first, dims, perm, es, 2 * ROUNDS - 1)
        assert np.array_equal(b[pad:].cpu().numpy(), last), cand
        assert np.array_equal(a[pad:].cpu().numpy(), _after(last, dims, perm, es, 1)), cand


@pytest.mark.parametrize("dims,perm,es", CHAINS[:4])
@pytest.mark.parametrize("units", [0, 1])
def test_copies_between(cuda, dims, perm, es, units):
    """a -> b by a transpose, b -> a by a contiguous copy, both tensors `units`
    elements off 16-byte alignment."""
    import torch

    n, pad = int(np.prod(dims)) * es, units * es
    s = torch.cuda.current_stream()
    a, b = _buffers(n + pad)
    first = a[pad:].cpu().numpy()
    with L.Plan(dims, perm, es, s) as p, L.Plan([n // es], [0], es, s) as copy:
        for _ in range(ROUNDS):
            p.execute(a.data_ptr() + pad, b.data_ptr() + pad)
            copy.execute(b.data_ptr() + pad, a.data_ptr() + pad)
        torch.cuda.synchronize()
    want = _after(first, dims, perm, es, ROUNDS)
    assert np.array_equal(a[pad:].cpu().numpy(), want)
    assert np.array_equal(b[pad:].cpu().numpy(), want)


@pytest.mark.parametrize("policy", [L.Group.LOADS_REGISTERS, L.Group.LOADS_ASYNC,
                                    L.Group.LOADS_PERSISTENT])
@pytest.mark.parametrize("dims,perm,es", CHAINS)
def test_groups(cuda, dims, perm, es, policy):
    """One-member groups: register, mixed and persistent launches sent directly."""
    import torch

    n = int(np.prod(dims)) * es
    s = torch.cuda.current_stream()
    a, b = _buffers(n)
    first = a.cpu().numpy()
    pol = [policy + L.Group.POLICY_WIDEST] * 12
    with L.Plan(dims, perm, es, s) as p, \
            L.Group([p], [a.data_ptr()], [b.data_ptr()], s, policy=pol) as there, \
            L.Group([p], [b.data_ptr()], [a.data_ptr()], s, policy=pol) as on:
        for _ in range(ROUNDS):
            there.execute()
            on.execute()
        torch.cuda.synchronize()
    last = _after(first, dims, perm, es, 2 * ROUNDS - 1)
    assert np.array_equal(b.cpu().numpy(), last)
    assert np.array_equal(a.cpu().numpy(), _after(last, dims, perm, es, 1))
