"""Performance cases of the transpose engine: what its users have it do,
through the package's public entry points, from the smallest calls to the
largest.

Transposes are stated in the library's convention: column-major dims (dim 0
varies fastest), output dim i is input dim perm[i], element size 4, 8 or 16
bytes.  Tensors hold random bits and are handed over as 64-bit or 32-bit
words, as every result is a bit copy.  Kinds:

  transpose  a plan kept by the program, executed on its tensors;
             `offset` elements in front of both tensors give views that are
             only aligned to their element
  group      many plans of uneven shapes executed as one group
  verify     the device-side check of a finished transpose
  train      one training step of the plan-selection network
"""
import math
import random

import numpy as np
import torch

import librett_gb300 as L
from librett_gb300 import _lib
from librett_gb300.learn import train as T
from librett_gb300.workloads import grouped_problems, packed_offsets

HIDDEN = 128
LR = 1e-3


def listed():
    return [
        # the smallest calls: one block of a larger computation, launch-bound
        {"name": "small_f32", "kind": "transpose", "dims": "64x48x32", "perm": "2,0,1", "es": 4,
         "offset": 0},
        # an ordinary amplitude-like rank-4 tensor, 32 MiB: fits the L2 cache
        {"name": "mid_f64", "kind": "transpose", "dims": "64x50x40x33", "perm": "2,0,3,1", "es": 8,
         "offset": 0},
        # the random-shape suite's size: 2^27 float64 elements
        {"name": "large_f64", "kind": "transpose", "dims": "96x24x131x18x25", "perm": "3,1,4,0,2",
         "es": 8, "offset": 0},
        # small leading dimensions, complex128, 4 GB in and 4 GB out
        {"name": "small_lead_c128", "kind": "transpose", "dims": "4x6x8192x5x256",
         "perm": "3,0,4,2,1", "es": 16, "offset": 0},
        # small leading dimensions, float32
        {"name": "small_lead_f32", "kind": "transpose", "dims": "2x3x4x5x65536x16",
         "perm": "5,3,1,4,0,2", "es": 4, "offset": 0},
        # odd dims: no run is a multiple of 16 bytes
        {"name": "odd_f32", "kind": "transpose", "dims": "127x63x65x33", "perm": "3,1,2,0", "es": 4,
         "offset": 0},
        # views into larger buffers: tensors aligned to their element only
        {"name": "offset_f32", "kind": "transpose", "dims": "256x128x512", "perm": "2,1,0", "es": 4,
         "offset": 1},
        # the leading dimension stays: rows move
        {"name": "rows_f64", "kind": "transpose", "dims": "200x300x400", "perm": "0,2,1", "es": 8,
         "offset": 0},
        # a batch of many small tensors (latency of one grouped launch)
        {"name": "group_small", "kind": "group", "count": 500, "log2_lo": 10.0, "log2_hi": 16.0},
        # a quarter of the 10,000-tensor batch, the same distribution
        {"name": "group_large", "kind": "group", "count": 2500, "log2_lo": 10.0, "log2_hi": 22.0},
        # checking a 256 MB result on the device
        {"name": "verify_f32", "kind": "verify", "dims": "64x128x96x85", "perm": "3,1,0,2",
         "es": 4},
        # the plan-selection network, the batch that its training uses
        {"name": "train_1024", "kind": "train", "batch": 1024},
    ]


def _split(rng, rank, log2_vol):
    """Dims whose product is about 2^log2_vol, split with random log weights."""
    w = [rng.random() + 0.05 for _ in range(rank)]
    return [max(2, round(2.0 ** (x / sum(w) * log2_vol))) for x in w]


def draw(rng):
    kind = rng.choices(["transpose", "group", "verify", "train"], [6, 2, 1, 1])[0]
    if kind == "train":
        return {"kind": kind, "batch": round(2.0 ** rng.uniform(6.0, 12.0))}
    if kind == "group":
        hi = rng.uniform(13.0, 20.0)
        return {"kind": kind, "count": round(2.0 ** rng.uniform(5.0, 11.0)), "log2_lo": 10.0,
                "log2_hi": round(hi, 2)}
    es = rng.choice([4, 8, 16])
    rank = rng.randint(2, 7)
    log2_bytes = rng.uniform(16.0, 30.0)
    dims = _split(rng, rank, log2_bytes - math.log2(es))
    perm = list(range(rank))
    while perm == sorted(perm):
        rng.shuffle(perm)
    case = {"kind": kind, "dims": "x".join(map(str, dims)), "perm": ",".join(map(str, perm)),
            "es": es}
    if kind == "transpose":
        case["offset"] = rng.choice([0, 0, 0, 0, 1, 3]) if es < 16 else 0
    return case


def _shape(case):
    return ([int(d) for d in case["dims"].split("x")], [int(p) for p in case["perm"].split(",")])


def _problems(case, seed):
    return grouped_problems(case["count"], seed=4711, log2_lo=case["log2_lo"],
                            log2_hi=case["log2_hi"])


def _random_words(nbytes, seed):
    """A device buffer of at least nbytes random bytes, as 64-bit words."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.empty((nbytes + 7) // 8, dtype=torch.int64, device="cuda").random_(generator=g)


def _tensors(nbytes, offset_bytes, seed):
    """Random input and zeroed output of nbytes, offset_bytes into their
    buffers: (address of input, of output, output buffer)."""
    src = _random_words(nbytes + offset_bytes, seed)
    dst = torch.zeros_like(src)
    return src, dst, src.data_ptr() + offset_bytes, dst.data_ptr() + offset_bytes


def prepare(case, seed):
    stream = torch.cuda.current_stream()
    kind = case["kind"]
    if kind == "train":
        rng = np.random.default_rng(seed)
        nf = _lib.load().librett_c_mlp_feature_count()
        params = T.init_params(nf, rng)
        X = torch.from_numpy(rng.normal(size=(case["batch"], nf)).astype(np.float32)).cuda()
        y = torch.from_numpy(rng.normal(size=case["batch"]).astype(np.float32)).cuda()
        return {"kind": kind, "net": T.GpuMlp(params, case["batch"]), "X": X, "y": y}
    if kind == "group":
        problems = _problems(case, seed)
        offs, total = packed_offsets(problems)
        src = _random_words(total, seed)
        dst = torch.zeros_like(src)
        plans = L.plan_batch(problems, stream)
        group = L.Group(plans, [src.data_ptr() + o for o in offs],
                        [dst.data_ptr() + o for o in offs], stream)
        return {"kind": kind, "group": group, "src": src, "dst": dst, "plans": plans}
    dims, perm = _shape(case)
    nbytes = math.prod(dims) * case["es"]
    src, dst, inp, out = _tensors(nbytes, case.get("offset", 0) * case["es"], seed)
    plan = L.Plan(dims, perm, case["es"], stream)
    state = {"kind": kind, "plan": plan, "src": src, "dst": dst, "in": inp, "out": out}
    if kind == "verify":
        # a finished transpose with a few wrong elements
        plan.execute(inp, out)
        words = dst.view(torch.int32)
        rng = random.Random(seed)
        per, vol = case["es"] // 4, math.prod(dims)
        bad = sorted({rng.randrange(vol) for _ in range(rng.randint(1, 200))})
        words[torch.tensor(bad, device="cuda") * per] ^= 1
        state.update(dims=dims, perm=perm, es=case["es"], stream=stream)
    return state


def run(state):
    kind = state["kind"]
    if kind == "transpose":
        state["plan"].execute(state["in"], state["out"])
        return state["dst"]
    if kind == "group":
        state["group"].execute()
        return state["dst"]
    if kind == "verify":
        bad, first = L.verify(state["dims"], state["perm"], state["es"], state["in"], state["out"],
                              state["stream"])
        return {"mismatches": bad, "first": first}
    net = state["net"]
    net.train_step(state["X"], state["y"], LR)
    b = state["X"].shape[0]
    return {"out": net.out[:b], "loss": net.loss, "grads": net.g, "params": net.p, "m": net.m,
            "v": net.v}


def work(case):
    kind = case["kind"]
    if kind == "train":
        b, nf, h = case["batch"], _lib.load().librett_c_mlp_feature_count(), HIDDEN
        params = h * nf + h + 2 * (h * h + h) + h + 1
        macs = b * (h * nf + 2 * h * h + h)  # forward; weight gradients cost the same again
        back = b * (2 * h * h + h)           # gradients of the activations
        # X, y, out once; parameters and both moments read and written, gradients written
        return {"bytes": 4 * (b * (nf + 2) + 7 * params), "flops": 2 * (2 * macs + back)}
    if kind == "group":
        elems = sum(math.prod(d) * es for d, _, es in _problems(case, 0))
        return {"bytes": 2 * elems, "flops": 0}
    dims, _ = _shape(case)
    return {"bytes": 2 * math.prod(dims) * case["es"], "flops": 0}


def exact(case, seed):
    """The training step in 64 bits; the other kinds move bits."""
    if case["kind"] != "train":
        return None
    rng = np.random.default_rng(seed)
    nf, h, b = _lib.load().librett_c_mlp_feature_count(), HIDDEN, case["batch"]
    p = T.init_params(nf, rng).astype(np.float64)
    X = rng.normal(size=(b, nf)).astype(np.float32).astype(np.float64)
    y = rng.normal(size=b).astype(np.float32).astype(np.float64)
    cut = np.cumsum([h * nf, h, h * h, h, h * h, h, h])
    W1, b1, W2, b2, W3, b3, W4, b4 = np.split(p, cut)
    W1, W2, W3 = W1.reshape(h, nf), W2.reshape(h, h), W3.reshape(h, h)
    A1 = np.maximum(X @ W1.T + b1, 0.0)
    A2 = np.maximum(A1 @ W2.T + b2, 0.0)
    A3 = np.maximum(A2 @ W3.T + b3, 0.0)
    out = A3 @ W4 + b4[0]
    loss = np.mean((out - y) ** 2)
    d = 2.0 * (out - y) / b
    D3 = np.outer(d, W4) * (A3 > 0)
    D2 = (D3 @ W3) * (A2 > 0)
    D1 = (D2 @ W2) * (A1 > 0)
    g = np.concatenate([(D1.T @ X).ravel(), D1.sum(0), (D2.T @ A1).ravel(), D2.sum(0),
                        (D3.T @ A2).ravel(), D3.sum(0), A3.T @ d, [d.sum()]])
    m, v = 0.1 * g, 0.001 * g * g  # first step of Adam, beta 0.9 and 0.999
    p = p - LR * (m / 0.1) / (np.sqrt(v / 0.001) + 1e-8)
    return {"out": out, "loss": np.array([loss]), "grads": g, "params": p, "m": m, "v": v}
