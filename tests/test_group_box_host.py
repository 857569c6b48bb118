"""Host-side check of the grouped mixed launch's box addressing (no GPU).

librett_c_group_box_check replays every thread and slot of a CTA against the
tile's offset tables: each element loaded once, in bounds and aligned, and
stored once where it belongs; over all candidate tiles of random problems, as
they are, in element units, with widened units, and doubled.
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
    done = without = 0
    for cand in range(16):
        for variant in range(4):
            rc = lib.librett_c_group_box_check(len(dims), dc, pc, es, 152, cand, variant)
            if rc == INVALID_PARAMETER:
                return done, without
            assert rc in (SUCCESS, INVALID_DEVICE), (dims, perm, es, cand, variant)
            done += rc == SUCCESS
            without += rc == INVALID_DEVICE
    return done, without


def _check_all(problems):
    done, without = np.sum([_check(*p) for p in problems], axis=0)
    assert done > 1000 and without < 0.05 * done, (done, without)


def test_batch_distribution():
    _check_all(grouped_problems(250, seed=17, log2_lo=3, log2_hi=20, sizes=(4, 8, 16), max_rank=7))


def test_high_ranks():
    rng = np.random.default_rng(18)
    _check_all(S.random_problem(rng, max_rank=14, max_vol=1 << 20) for _ in range(150))


# offsets near 2^31 elements; a leading run over several ranks; one rank; primes
@pytest.mark.parametrize("dims,perm,es", [([46341, 46340], [1, 0], 4), ([3, 5, 65536, 1087], [3, 1, 0, 2], 4),
                                          ([2, 3, 4, 5, 65536, 16], [5, 3, 1, 4, 0, 2], 4),
                                          ([4099], [0], 8), ([257, 131, 61], [2, 1, 0], 16),
                                          ([2] * 16, list(range(15, -1, -1)), 4)])
def test_named_shapes(dims, perm, es):
    assert _check(dims, perm, es)[0] > 0
