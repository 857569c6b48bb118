"""Host-side check of the table-free tile kernels' addressing (no GPU).

The flat and bulk-copy kernels form a unit's offsets as the sum of a
per-thread and a per-slot part with carries between the mixed-radix digits.
librett_c_slot_check replays those sums for every unit of a candidate tile and
compares them with the per-unit offset tables, over all candidate tiles of
random problems of every rank class, in vector and in element units.
"""
import numpy as np
import pytest

from librett_gb300 import _lib
from librett_gb300.workloads import grouped_problems
from tests import shapes as S

SUCCESS, INVALID_PARAMETER, INVALID_DEVICE = 0, 2, 3


def _check(dims, perm, es):
    lib = _lib.load()
    dc, pc = _lib.int_array(dims), _lib.int_array(perm)
    n = 0
    for cand in range(16):
        for element_units in (0, 1):
            rc = lib.librett_c_slot_check(len(dims), dc, pc, es, 152, cand, element_units)
            if rc == INVALID_PARAMETER:
                return n
            assert rc in (SUCCESS, INVALID_DEVICE), (dims, perm, es, cand, element_units)
            n += rc == SUCCESS
    return n


def test_random_problems():
    n = 0
    for dims, perm, es in grouped_problems(400, seed=17, log2_lo=3, log2_hi=22, sizes=(4, 8, 16),
                                           max_rank=7):
        n += _check(dims, perm, es)
    assert n > 2000


def test_high_ranks():
    rng = np.random.default_rng(18)
    assert sum(_check(*S.random_problem(rng, max_rank=12, max_vol=1 << 22)) for _ in range(200)) > 300


# offsets near 2^31 elements; a leading run merged over several ranks; one tile
# of a single rank; primes; extents of 2
@pytest.mark.parametrize("dims,perm,es", [([46341, 46340], [1, 0], 4), ([3, 5, 65536, 1087], [3, 1, 0, 2], 4),
                                          ([2, 3, 4, 5, 65536, 16], [5, 3, 1, 4, 0, 2], 4),
                                          ([4099], [0], 8), ([257, 131, 61], [2, 1, 0], 16),
                                          ([2] * 16, list(range(15, -1, -1)), 4)])
def test_named_shapes(dims, perm, es):
    n = _check(dims, perm, es)
    assert n > 0 or len(dims) == 16
