"""The calls whose speed this framework is about, as a program makes them.

Each case is one public entry point with the matrices it meets in use: pruned
layers (rows of about equal length), graph-like matrices (Zipf row lengths,
where a few rows are full and many hold one nonzero), single calls and whole
batches, FP16 and E4M3, forward and backward, device and host buffers, and
token counts N as they come. Sizes are those of the reference's own test
(2048 x 512 at 80 %), of the sweep, differentiation, precision and batching
workloads of bench.py and the tests, and odd ones in the same ranges.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath(os.path.join("tca-spmm_b200", "python")))
import tca_spmm  # noqa: E402
from tca_spmm import autograd  # noqa: E402

DEV = "cuda"
E4M3_MAX = 448.0


def listed():
    return [
        # the smallest call: one small pruned layer on a few tokens, where
        # latency and launches are all there is
        dict(name="tiny", kind="spmm", M=512, K=512, N=64, density=0.1, law="binomial", out="f16"),
        # the sweep's middle point as one call: Zipf rows, dense and one-nonzero
        # rows in the same matrix
        dict(name="zipf80", kind="spmm", M=4096, K=1024, N=256, density=0.2, law="zipf", out="f16"),
        # a token count as it comes in serving (N odd, rows of B unaligned),
        # ragged M and K, FP32 output
        dict(name="ragged", kind="spmm", M=3001, K=1777, N=203, density=0.08, law="binomial", out="f32"),
        # the largest single layer: 4096 x 4096 at 90 %, 1024 tokens
        dict(name="large", kind="spmm", M=4096, K=4096, N=1024, density=0.1, law="poisson", out="f16"),
        # the same layer in E4M3 (B quantized in every call)
        dict(name="large_e4m3", kind="fp8", M=4096, K=4096, N=1024, density=0.1, law="poisson", out="f16"),
        # a pattern used once: no plan, straight from CSR
        dict(name="planfree", kind="csr", M=4096, K=1024, N=128, density=0.05, law="zipf", out="f16"),
        # one training step of a sparse layer: forward, gradient of the values
        # and of the activations, 4096 tokens
        dict(name="train", kind="train", M=2048, K=512, N=4096, density=0.1, law="uniform", out="f16"),
        # a network's 24 sparse layers of mixed shapes and token counts as one graph
        dict(name="layers24", kind="layers", layers=24, mix=5, precision="f16"),
        # many problems of one shape per graph replay, the throughput workload of bench.py
        dict(name="batch32", kind="batch", count=32, M=4096, K=1024, N=256, density=0.2, law="zipf",
             precision="f16"),
        dict(name="batch32_e4m3", kind="batch", count=32, M=4096, K=1024, N=256, density=0.2, law="zipf",
             precision="e4m3"),
        # the reference's calling convention: host buffers in, host buffer out
        dict(name="host", kind="host", M=4096, K=1024, N=256, density=0.2, law="zipf", out="f32"),
        # a new pattern per step (dynamic sparsity): plan build and one forward
        dict(name="fresh", kind="fresh", M=2048, K=512, N=256, density=0.2, law="binomial", out="f16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmm", "spmm", "spmm", "fp8", "csr", "train", "layers", "batch", "host", "fresh"])
    if kind == "layers":
        return dict(kind=kind, layers=rng.randint(4, 24), mix=rng.randrange(1 << 20),
                    precision=rng.choice(["f16", "e4m3"]))
    M, K = _log_int(rng, 256, 4096), _log_int(rng, 256, 4096)
    N = _log_int(rng, 32, 1024)
    if kind in ("fp8", "batch") or rng.random() < 0.6:
        N = max(8, N // 8 * 8)  # E4M3 takes multiples of 8; token counts are padded to them as often as not
    case = dict(kind=kind, M=M, K=K, N=N, density=round(math.exp(rng.uniform(math.log(0.02), math.log(0.3))), 4),
                law=rng.choice(["binomial", "zipf", "poisson", "uniform"]))
    if kind == "batch":
        case.update(count=rng.randint(2, 12), N=min(N, 512), M=min(M, 2048), K=min(K, 2048),
                    precision=rng.choice(["f16", "e4m3"]))
    else:
        case["out"] = rng.choice(["f16", "f32"])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _zipf_rows(rng, M, K, total):
    """Row lengths proportional to Zipf(1.2) draws, clipped to [1, K], with
    about `total` nonzeros in all."""
    w = rng.zipf(1.2, size=M).astype(np.float64)
    lo, hi = 0.0, float(K)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        if np.clip(np.rint(w * mid), 1, K).sum() < total:
            lo = mid
        else:
            hi = mid
    return np.clip(np.rint(w * hi), 1, K).astype(np.int64)


def _row_lengths(rng, law, M, K, density):
    if law == "zipf":
        return _zipf_rows(rng, M, K, density * M * K)
    if law == "binomial":
        return rng.binomial(K, density, size=M)
    if law == "poisson":
        return np.clip(rng.poisson(K * density, size=M), 0, K)
    n = int(density * M * K)
    r = np.full(M, n // M, dtype=np.int64)
    r[: n % M] += 1
    return r


def _matrix(seed, M, K, density, law):
    """CSR with distinct uniform columns per row, sorted; values
    N(0, 1 / sqrt(K)); and the generators that made it."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n = torch.from_numpy(np.asarray(_row_lengths(rng, law, M, K, density))).to(DEV)
    order = torch.rand((M, K), generator=g, device=DEV).argsort(dim=1)
    keep = torch.arange(K, device=DEV)[None, :] < n[:, None]
    mask = torch.zeros((M, K), dtype=torch.bool, device=DEV).scatter_(1, order, keep)
    cols = mask.nonzero()[:, 1].to(torch.int32)
    row_ptr = torch.zeros(M + 1, dtype=torch.int32, device=DEV)
    row_ptr[1:] = n.cumsum(0)
    vals = torch.randn(cols.numel(), generator=g, device=DEV) / math.sqrt(K)
    return row_ptr, cols, vals, g


def _uniform(g, K, N):
    return (torch.rand((K, N), generator=g, device=DEV) * 2 - 1).half()


def _specs(case):
    """(M, K, N, density, law) of each of the case's products."""
    if case["kind"] != "layers":
        return [(case["M"], case["K"], case["N"], case["density"], case["law"])] * case.get("count", 1)
    mix = random.Random(case["mix"])
    shapes = [(512, 2048), (2048, 512), (512, 512), (1024, 4096)]
    specs = []
    for i in range(case["layers"]):
        N = mix.choice([64, 128, 256, 512, 1024])
        specs.append((*shapes[i * 4 // case["layers"]], N, 1.0 - mix.uniform(0.5, 0.98), "binomial"))
    return specs


def _inputs(case, seed):
    """The case's matrices: dicts of row_ptr, cols, vals (FP32), M, K, N, B
    (FP16), and dY for a training step."""
    kind = case["kind"]
    specs = _specs(case)
    out, shared = [], []
    for i, (M, K, N, density, law) in enumerate(specs):
        if kind == "batch" and i >= 4:  # four patterns, as bench.py's step has; each problem has its own B
            p = dict(shared[i % 4])
            g = torch.Generator(device=DEV)
            g.manual_seed(seed * 1000 + i)
            p["B"] = _uniform(g, K, N)
        else:
            row_ptr, cols, vals, g = _matrix(seed * 1000 + i, M, K, density, law)
            p = dict(M=M, K=K, N=N, row_ptr=row_ptr, cols=cols, vals=vals)
            if kind in ("train", "fp8"):  # activations
                p["B"] = torch.randn((K, N), generator=g, device=DEV).half()
            else:
                p["B"] = _uniform(g, K, N)
            if kind == "train":
                p["dY"] = torch.randn((M, N), generator=g, device=DEV).half()
            shared.append(p)
        out.append(p)
    return out


def _dtype(case):
    return torch.float32 if case.get("out") == "f32" else torch.float16


def _plan(p):
    return tca_spmm.Plan(p["row_ptr"], p["cols"], p["vals"].half(), p["K"])


def prepare(case, seed):
    kind = case["kind"]
    ps = _inputs(case, seed)
    p = ps[0]
    s = dict(kind=kind, out=_dtype(case))
    if kind in ("layers", "batch"):
        # a serving program captures its batch once and replays it
        plans = [_plan(q) for q in ps]
        s["outs"] = [torch.empty((q["M"], q["N"]), dtype=torch.float16, device=DEV) for q in ps]
        s["graph"] = tca_spmm.BatchGraph(plans, [q["B"] for q in ps], s["outs"], precision=case["precision"])
        return s
    if kind == "host":
        for k, v in (("row_ptr", p["row_ptr"]), ("cols", p["cols"]), ("vals", p["vals"].half()), ("B", p["B"])):
            s[k] = v.cpu().numpy()
        s["K"] = p["K"]
        s["C"] = np.zeros((p["M"], p["N"]), dtype=np.float32 if case["out"] == "f32" else np.float16)
        return s
    s["B"] = p["B"]
    if kind in ("csr", "fresh"):
        s.update(row_ptr=p["row_ptr"], cols=p["cols"], vals=p["vals"].half(), K=p["K"])
        return s
    s["plan"] = _plan(p)
    if kind == "fp8":
        s["plan"].quantize_fp8()
    if kind == "train":
        s["plan"].build_transpose()
        s["vals"] = p["vals"].requires_grad_()  # FP32 master values
        s["B"] = p["B"].requires_grad_()
        s["dY"] = p["dY"].to(s["out"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "spmm":
        return s["plan"].spmm(s["B"], out_dtype=s["out"])
    if kind == "fp8":
        return s["plan"].spmm_fp8(s["B"], out_dtype=s["out"])
    if kind == "csr":
        return tca_spmm.spmm_csr(s["row_ptr"], s["cols"], s["vals"], s["B"], out_dtype=s["out"])
    if kind == "train":
        Y = autograd.spmm(s["plan"], s["vals"], s["B"], out_dtype=s["out"])
        d_vals, d_B = torch.autograd.grad(Y, (s["vals"], s["B"]), s["dY"])
        return Y.detach(), d_vals, d_B
    if kind in ("layers", "batch"):
        s["graph"].launch()
        return s["outs"]
    if kind == "host":
        C, _ = tca_spmm.spmm_host(s["row_ptr"], s["cols"], s["vals"], s["K"], s["B"], C=s["C"])
        return C
    plan = tca_spmm.Plan(s["row_ptr"], s["cols"], s["vals"], s["K"])
    return plan.spmm(s["B"], out_dtype=s["out"])


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its result in 64 bits
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    e4m3 = kind == "fp8" or case.get("precision") == "e4m3"
    c = 4 if case.get("out") == "f32" else 2
    n_bytes = n_flops = 0.0
    for M, K, N, density, _ in _specs(case):
        nnz = density * M * K
        n_bytes += nnz * ((1 if e4m3 else 2) + 4) + (M + 1) * 4 + K * N * 2 + M * N * c
        n_flops += 2 * nnz * N
        if kind == "train":  # FP32 values in, their gradient out, dY in, dB out; two more products
            n_bytes += nnz * (2 + 4) + M * N * c + K * N * 2
            n_flops += 4 * nnz * N
    return {"bytes": n_bytes, "flops": n_flops}


def _dense(p, vals):
    rows = torch.repeat_interleave(torch.arange(p["M"], device=DEV), p["row_ptr"].diff().long())
    A = torch.zeros((p["M"], p["K"]), dtype=torch.float64, device=DEV)
    A[rows, p["cols"].long()] = vals
    return A, rows


def _exact_e4m3(p):
    """The product of the E4M3 operands as the library's header defines them:
    scale max|x| / 448 per row of A and per column of B, A divided by its
    scale, B multiplied by the scale's FP32 reciprocal, nearest even."""
    v = p["vals"].half().float()
    A, rows = _dense(p, v.double())
    a_max = A.abs().amax(1).float()
    b_max = p["B"].float().abs().amax(0)
    # (divided by a tensor: torch multiplies by a rounded reciprocal for a number)
    s_a = torch.where(a_max > 0, a_max / torch.full_like(a_max, E4M3_MAX), torch.ones_like(a_max))
    s_b = torch.where(b_max > 0, b_max / torch.full_like(b_max, E4M3_MAX), torch.ones_like(b_max))
    A[rows, p["cols"].long()] = (v / s_a[rows]).to(torch.float8_e4m3fn).double()
    B = (p["B"].float() * (1.0 / s_b)).to(torch.float8_e4m3fn).double()
    return (A @ B) * s_a.double()[:, None] * s_b.double()[None, :]


def exact(case, seed):
    kind = case["kind"]
    ps = _inputs(case, seed)
    if kind == "fp8" or case.get("precision") == "e4m3":
        outs = [_exact_e4m3(p) for p in ps]
    elif kind == "train":
        p = ps[0]
        A, rows = _dense(p, p["vals"].half().double())
        B, dY = p["B"].double(), p["dY"].double()
        return A @ B, (dY @ B.T)[rows, p["cols"].long()], A.T @ dY
    else:
        outs = [_dense(p, p["vals"].half().double())[0] @ p["B"].double() for p in ps]
    return outs if kind in ("layers", "batch") else outs[0]
