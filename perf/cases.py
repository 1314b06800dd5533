"""The GEMM calls a user of this library makes, as cases that can be timed and compared.

A case is one call through the public Python view of the C ABI (phpc.py) on
inputs the caller already holds:

* ``split``    dgemm_ozaki2_dev: FP64-accurate C += A B, device matrices
* ``plain``    dgemm_dmma_dev: plain FP64 C += A B, device matrices
* ``f32``      sgemm_bf16x3_dev: FP32-accurate C += A B, device matrices
* ``grouped``  GroupedPlan.graph_launch: a planned batch of FP64-accurate GEMMs
* ``host``     gemm_cublas: the reference's own entry point, host matrices

``pad`` is what the leading dimensions exceed the rows by (operands that are
blocks of larger matrices, as SUMMA's are); ``values`` is the distribution of
the FP64 entries: ``uniform`` in [-1, 1), or ``wide``, signed mantissas in
[1, 2) times 2^e with e in -20 .. 20.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "hpc-multigpu-matrixmult_gb300"))
import phpc  # noqa: E402


def _gemm(name, kind, m, k, n, **more):
    return {"name": name, "kind": kind, "m": m, "k": k, "n": n, "pad": 0, "values": "uniform", **more}


def listed():
    return [
        # the smallest calls of the reference's own sweep: launches and latency
        _gemm("split_256", "split", 256, 256, 256),
        # config 1's size, the smallest the tuning table names
        _gemm("split_1024", "split", 1024, 1024, 1024, values="wide"),
        # an odd-sized block of larger matrices
        _gemm("split_ragged", "split", 1537, 1000, 2311, pad=5),
        # one SUMMA k-panel update of a rank's block: large C, short K
        _gemm("split_panel", "split", 4096, 512, 4096, pad=512),
        # ordinary square products, wide-exponent entries (config 3)
        _gemm("split_4096", "split", 4096, 4096, 4096, values="wide"),
        # the benchmark's workload
        _gemm("split_16384", "split", 16384, 16384, 16384, values="wide"),
        # plain FP64 on a small ragged block
        _gemm("plain_ragged", "plain", 250, 514, 302, pad=4, grid=1),
        # config 1: plain FP64 at N = 1024 on one SUMMA block
        _gemm("plain_1024", "plain", 1024, 1024, 1024, grid=1),
        # FP32-accurate product of ordinary, odd sizes
        _gemm("f32_ragged", "f32", 1000, 777, 1530, pad=3),
        # config 4: the rectangular FP32-accurate product
        _gemm("f32_rect", "f32", 32768, 4096, 8192),
        # config 5: 512 problems of log-uniform sizes as one CUDA graph
        {"name": "grouped_512", "kind": "grouped", "count": 512, "lo": 64, "hi": 2048, "multiple": 16, "shapes": 5},
        # the reference's host entry point on pageable host matrices
        _gemm("host_2048", "host", 2048, 2048, 2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["split", "split", "split", "plain", "f32", "f32", "grouped", "host"])
    if kind == "grouped":
        hi = _log(rng, 256, 2048)
        return {"kind": kind, "count": _log(rng, 8, 512), "lo": rng.choice([16, 32, 64]), "hi": hi,
                "multiple": rng.choice([1, 8, 16]), "shapes": rng.randrange(1000)}
    hi = {"split": 8192, "plain": 2048, "f32": 8192, "host": 4096}[kind]
    m, k, n = (_log(rng, 64, hi) for _ in range(3))
    case = {"kind": kind, "m": m, "k": k, "n": n, "pad": rng.choice([0, 0, rng.randrange(1, 65)]),
            "values": rng.choice(["uniform", "wide"])}
    if kind == "plain":
        case["grid"] = rng.choice([1, 2, 4])
    return case


def _values(shape, values, gen):
    x = torch.rand(shape, dtype=torch.float64, device=gen.device, generator=gen)
    if values == "uniform":
        return x.mul_(2).sub_(1)
    e = torch.randint(-20, 21, shape, dtype=torch.int32, device=gen.device, generator=gen)
    s = torch.randint(0, 2, shape, dtype=torch.int32, device=gen.device, generator=gen)
    return torch.ldexp(x.add_(1).mul_(1 - 2 * s), e)


def _block(rows, cols, pad, even, values, gen, dtype=torch.float64):
    """A rows x cols block of a buffer whose rows are `pad` longer (and, with `even`, of even length)."""
    ld = cols + pad
    ld += ld & 1 if even else 0
    if dtype == torch.float32:
        return torch.randn((rows, ld), dtype=dtype, device=gen.device, generator=gen)[:, :cols]
    return _values((rows, ld), values, gen)[:, :cols]


def _shapes(case):
    return phpc.grouped_shapes(case["count"], case["shapes"], case["lo"], case["hi"], case["multiple"])


def _inputs(case, seed):
    """(A, B, C) of one product (device tensors, host arrays for ``host``), or three lists for a batch."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "grouped":
        As, Bs, Cs = [], [], []
        shapes = _shapes(case)
        flat = _values((sum(m * n for m, _, n in shapes),), "uniform", gen)  # every C, one after another
        at = 0
        for m, k, n in shapes:
            As.append(_values((m, k), "uniform", gen))
            Bs.append(_values((k, n), "uniform", gen))
            Cs.append(flat[at:at + m * n].view(m, n))
            at += m * n
        return As, Bs, (flat, Cs)
    m, k, n, pad = case["m"], case["k"], case["n"], case["pad"]
    even = case["kind"] == "plain"  # its operands' rows are 16-byte aligned
    dtype = torch.float32 if case["kind"] == "f32" else torch.float64
    A = _block(m, k, pad, even, case["values"], gen, dtype)
    B = _block(k, n, pad, even, case["values"], gen, dtype)
    C = _block(m, n, pad, False, "uniform", gen, dtype)
    if case["kind"] == "host":
        A, B, C = (x._base.cpu().numpy()[:, :x.shape[1]] for x in (A, B, C))
    return A, B, C


def prepare(case, seed):
    A, B, C = _inputs(case, seed)
    kind = case["kind"]
    s = {"kind": kind, "A": A, "B": B, "C": C}
    if kind == "grouped":
        flat, Cs = C
        probs = [(a.shape[0], a.shape[1], b.shape[1], a, a.stride(0), b, b.stride(0), c, c.stride(0))
                 for a, b, c in zip(A, B, Cs)]
        size = phpc.GroupedPlan.workspace_bytes(probs, 7, moduli=13)
        s["W"] = torch.empty(size, dtype=torch.uint8, device="cuda")
        s["plan"] = phpc.GroupedPlan(probs, 7, s["W"], size, torch.cuda.current_stream(), moduli=13)
        s["C"] = flat
        return s
    m, k, n = case["m"], case["k"], case["n"]
    s["mkn"] = m, k, n
    if kind == "split":
        s["moduli"] = phpc.default_moduli(m, k, n)
        s["size"] = phpc.ozaki2_workspace_bytes(m, k, n, s["moduli"])
    elif kind == "f32":
        s["size"] = phpc.bf16x3_workspace_bytes(m, k, n)
    elif kind == "plain":
        s["grid"] = case["grid"]
    if "size" in s:
        s["W"] = torch.empty(s["size"], dtype=torch.uint8, device="cuda")
    return s


def run(s):
    kind, A, B, C = s["kind"], s["A"], s["B"], s["C"]
    if kind == "grouped":
        s["plan"].graph_launch(torch.cuda.current_stream())
        return C
    m, k, n = s["mkn"]
    if kind == "host":
        phpc.gemm_cublas(A, A.strides[0] // 8, B, B.strides[0] // 8, C, C.strides[0] // 8, m, k, n)
        return C
    lda, ldb, ldc = A.stride(0), B.stride(0), C.stride(0)
    stream = torch.cuda.current_stream()
    if kind == "split":
        phpc.dgemm_ozaki2_dev(m, k, n, A, lda, B, ldb, C, ldc, s["moduli"], s["W"], s["size"], stream)
    elif kind == "plain":
        phpc.dgemm_dmma_dev(m, k, n, A, lda, B, ldb, C, ldc, s["grid"], s["grid"], 256, stream)
    else:
        phpc.sgemm_bf16x3_dev(m, k, n, A, lda, B, ldb, C, ldc, s["W"], s["size"], stream)
    return C


def work(case):
    if case["kind"] == "grouped":
        shapes = _shapes(case)
        return {"bytes": sum(8.0 * (m * k + k * n + 2 * m * n) for m, k, n in shapes),
                "flops": sum(2.0 * m * k * n for m, k, n in shapes)}
    m, k, n = case["m"], case["k"], case["n"]
    item = 4.0 if case["kind"] == "f32" else 8.0
    return {"bytes": item * (m * k + k * n + 2 * m * n), "flops": 2.0 * m * k * n}


def exact(case, seed):
    A, B, C = _inputs(case, seed)
    if case["kind"] == "grouped":
        flat, Cs = C
        for a, b, c in zip(A, B, Cs):
            c.addmm_(a, b)
        return flat
    if case["kind"] == "host":
        A, B, C = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (A, B, C))
        return torch.addmm(C, A, B).cpu().numpy()
    return torch.addmm(C.double(), A.double(), B.double())
