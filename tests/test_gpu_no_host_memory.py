"""Calls that needed no host memory of the library's before still need none: with an
operator new that throws, executing, the network kernels and checks succeed (no
exception leaves a C entry), also as the first call of their kind.  In a process of
its own, without torch."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from tests.test_verify_map_host import THROWING_NEW

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
import ctypes, sys
import numpy as np
from librett_gb300 import _lib
rt, own, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2]), _lib.load()
def ok(rc):
    assert rc == 0, rc
def device(nbytes):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(nbytes)))
    ok(rt.cudaMemset(p, 0, ctypes.c_size_t(nbytes)))
    return p
batch, n = 40, lib.librett_c_mlp_param_count()
p, g, m, v = (device(4 * n) for _ in range(4))
x, out, y, dout = (device(4 * k) for k in (batch * lib.librett_c_mlp_feature_count(),) + (batch,) * 3)
ws = device(4 * lib.librett_c_mlp_workspace_floats(batch))
dims, perm = _lib.int_array([64, 48, 32]), _lib.int_array([2, 0, 1])
a, b = device(4 * 64 * 48 * 32), device(4 * 64 * 48 * 32)
plan = ctypes.c_uint()
if sys.argv[3] == "plan":
    ok(lib.librett_c_plan(ctypes.byref(plan), 3, dims, perm, 4, None))
bad, first = ctypes.c_ulonglong(9), ctypes.c_longlong(9)
own.arm(1)
if sys.argv[3] == "plan":
    rc = [lib.librett_c_execute(plan, a, b)]
elif sys.argv[3] == "verify":
    rc = [lib.librett_c_verify(3, dims, perm, 4, a, b, None, ctypes.byref(bad), ctypes.byref(first))]
else:
    rc = [lib.librett_c_mlp_forward(p, x, batch, ws, out, None),
          lib.librett_c_mlp_mse_grad(out, y, batch, dout, None, None),
          lib.librett_c_mlp_backward(p, x, batch, ws, dout, g, None),
          lib.librett_c_mlp_adam(p, g, m, v, n, 1e-3, 0.9, 0.999, 1e-8, 1, None)]
own.arm(0)
assert not any(rc), rc
ok(rt.cudaDeviceSynchronize())
assert sys.argv[3] != "verify" or (bad.value, first.value) == (0, -1)
print("done")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["plan", "verify", "network"])
def test_throwing_new(cuda, tmp_path, what):
    runtime = next((p for d in ("/usr/local/cuda/lib64", "/usr/local/cuda/lib") for p in
                    sorted(Path(d).glob("libcudart.so.*"))), None)
    if runtime is None:
        pytest.skip("no shared CUDA runtime")
    src, own = tmp_path / "new.cpp", tmp_path / "new.so"
    src.write_text(THROWING_NEW)
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", str(src), "-o", str(own)], check=True)
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(runtime), str(own), what], cwd=ROOT,
                       text=True, capture_output=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": str(own)})
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stdout + r.stderr
