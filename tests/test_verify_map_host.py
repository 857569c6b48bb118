"""The verifier's addressing on the host: the map of its tile is the transpose
formula's, its tiles own every element once, and every planted mistake is seen."""
import os
import random
import subprocess
import sys
from pathlib import Path

import pytest

import librett_gb300 as L
from librett_gb300 import _lib

ROOT = Path(__file__).resolve().parents[1]
KNOWN = [([64, 48, 32], [2, 0, 1], 4), ([64, 128, 96, 85], [3, 1, 0, 2], 4),
         ([127, 63, 65, 33], [3, 1, 2, 0], 4), ([1000, 517], [1, 0], 8), ([200, 300, 400], [0, 2, 1], 8),
         ([4, 6, 819, 5, 25], [3, 0, 4, 2, 1], 16), ([70001], [0], 4), ([2] * 16, list(range(15, -1, -1)), 4),
         ([2, 3, 2, 5, 2, 3, 2, 3, 2, 4], [9, 7, 5, 3, 1, 0, 2, 4, 6, 8], 8), ([3, 2], [1, 0], 16),
         ([50000, 3, 60000], [2, 1, 0], 4)]


def _problems(n):
    rng = random.Random(29)
    for _ in range(n):
        rank = rng.randint(2, 9)
        log2 = rng.uniform(4.0, 24.0)
        w = [rng.random() + 0.05 for _ in range(rank)]
        dims = [max(2, round(2.0 ** (x / sum(w) * log2))) for x in w]
        perm = list(range(rank))
        rng.shuffle(perm)
        yield dims, perm, rng.choice([4, 8, 16])


def _check(dims, perm, es, units=0, mistake=0):
    return _lib.load().librett_c_verify_map_check(len(dims), _lib.int_array(dims),
                                                  _lib.int_array(perm), es, 152, units, mistake)


@pytest.mark.parametrize("units", [0, 1])
def test_every_map_is_sound(units):
    for dims, perm, es in KNOWN + list(_problems(300)):
        assert _check(dims, perm, es, units) == L.LIBRETT_SUCCESS, (dims, perm, es)


@pytest.mark.parametrize("mistake", range(1, 10))
@pytest.mark.parametrize("units", [0, 1])
def test_mistakes_are_seen(mistake, units):
    planted = 0
    for dims, perm, es in KNOWN + list(_problems(150)):
        rc = _check(dims, perm, es, units, mistake)
        if rc == L.LIBRETT_INVALID_DEVICE:
            continue  # no place for it
        assert rc == L.LIBRETT_INTERNAL_ERROR, (dims, perm, es)
        planted += 1
    assert planted >= 10


def test_no_tile():
    """A tensor of one element has no tile: it is checked element by element."""
    assert _check([1], [0], 4) == L.LIBRETT_INVALID_DEVICE


def test_arguments():
    assert _check([4, 4], [0, 0], 4) == L.LIBRETT_INVALID_PARAMETER
    assert _check([4, 4], [1, 0], 3) == L.LIBRETT_INVALID_PARAMETER
    assert _check([4, 4], [1, 0], 4, 0, 10) == L.LIBRETT_INVALID_PARAMETER
    assert _check([4, 4], [1, 0], 4, 0, -1) == L.LIBRETT_INVALID_PARAMETER


THROWING_NEW = r"""
#include <cstdlib>
#include <new>
static bool armed;
extern "C" void arm(int on) { armed = on != 0; }
void* operator new(std::size_t n) {
  void* p = armed ? nullptr : std::malloc(n ? n : 1);
  if (p == nullptr) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
"""

NO_MEMORY = r"""
import ctypes, sys
from librett_gb300 import _lib
lib, own = _lib.load(), ctypes.CDLL(sys.argv[1])
dims, perm = _lib.int_array([64, 48, 32]), _lib.int_array([2, 0, 1])
own.arm(1)
rc = lib.librett_c_verify_map_check(3, dims, perm, 4, 152, 0, 0)
own.arm(0)
print(rc, lib.librett_c_verify_map_check(3, dims, perm, 4, 152, 0, 0))
"""


def test_no_host_memory(tmp_path):
    """Without host memory for the choice of a tile there is none (the check then goes
    element by element); no exception leaves the C entry."""
    src, own = tmp_path / "new.cpp", tmp_path / "new.so"
    src.write_text(THROWING_NEW)
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", str(src), "-o", str(own)], check=True)
    r = subprocess.run([sys.executable, "-c", NO_MEMORY, str(own)], cwd=ROOT, text=True,
                       capture_output=True, timeout=300, env={**os.environ, "LD_PRELOAD": str(own)})
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == [str(L.LIBRETT_INVALID_DEVICE), str(L.LIBRETT_SUCCESS)]
