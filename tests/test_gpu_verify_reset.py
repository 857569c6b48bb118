"""Checks go on after a cudaDeviceReset, which ends every registration of host
memory: small and large tiles, errors counted, before and after.  In a process of its
own, without torch, whose buffers would be lost."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
import ctypes, sys
from librett_gb300 import _lib
rt = ctypes.CDLL(sys.argv[1])
lib = _lib.load()
def ok(rc):
    assert rc == 0, rc
def check(dims, perm, es):
    n = es
    for d in dims:
        n *= d
    a, b = ctypes.c_void_p(), ctypes.c_void_p()
    for p in (a, b):
        ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(n)))
        ok(rt.cudaMemset(p, 0, ctypes.c_size_t(n)))
    ok(rt.cudaMemset(ctypes.c_void_p(b.value + 5 * es), 1, ctypes.c_size_t(2 * es)))
    ok(rt.cudaDeviceSynchronize())
    bad, first = ctypes.c_ulonglong(9), ctypes.c_longlong(9)
    ok(lib.librett_c_verify(len(dims), _lib.int_array(dims), _lib.int_array(perm), es, a, b, None,
                            ctypes.byref(bad), ctypes.byref(first)))
    assert (bad.value, first.value) == (2, 5), (bad.value, first.value)
    for p in (a, b):
        ok(rt.cudaFree(p))
for again in range(3):
    for case in (([64, 48, 32], [2, 0, 1], 4), ([200, 60, 100], [2, 1, 0], 16), ([97, 33], [1, 0], 8)):
        check(*case)
        check(*case)
    ok(rt.cudaDeviceReset())
print("checked")
"""


@pytest.mark.gpu
def test_after_a_device_reset(cuda):
    runtime = next((p for d in ("/usr/local/cuda/lib64", "/usr/local/cuda/lib") for p in
                    sorted(Path(d).glob("libcudart.so.*"))), None)
    if runtime is None:
        pytest.skip("no shared CUDA runtime")
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(runtime)], cwd=ROOT, text=True,
                       capture_output=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "checked", r.stdout + r.stderr
