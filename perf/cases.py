"""The GEMM calls whose speed is measured: what a program that uses this library has it do.

A case is one call of one entry point on operands such a program has in hand:

  f64         dgemm, plain FP64 form, device operands (levels 0: classical)
  f64_host    bli_strassen_ab_ex, the FP64 drop-in on host arrays
  f64_batch   batch_dgemm, FP64 problems of uneven sizes
  split       split_dgemm, digit slices on the tensor cores, device operands
  split_host  split_strassen_ab_ex, the same on host arrays
  split_batch batch_dgemm, split problems of uneven sizes

Operands are seeded, uniform in [-1, 1) or, with phi > 0, the wide-range
(u - 0.5) * exp(phi * g). Every call computes C := beta*C + alpha*A*B and
returns C.
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

import fmm_blis_gb300 as fmm
from fmm_blis_gb300 import tune

_COEFFS = Path(fmm.__file__).resolve().parent / "coeffs"
_SHAPES = {"222": (2, 2, 2, 7), "232": (2, 3, 2, 11), "322": (3, 2, 2, 11), "333": (3, 3, 3, 23),
           "444": (4, 4, 4, 49)}          # m~, k~, n~, R
_algs: dict = {}


def _alg(name):
    """the algorithm handle a program reads once and keeps"""
    if name == "classical":
        return None
    if name not in _algs:
        _algs[name] = fmm.new_fmm(_COEFFS / f"{name}.txt")
    return _algs[name]


def _case(kind, m, n, k, alg="classical", levels=0, slices=0, fmt="bf16", alpha=1.0, beta=1.0, pad=0, phi=0.0):
    """one GEMM; pad: rows between the end of a column and the next one (an operand inside a larger array)"""
    return {"kind": kind, "m": m, "n": n, "k": k, "alg": alg, "levels": levels, "slices": slices, "fmt": fmt,
            "alpha": alpha, "beta": beta, "pad": pad, "phi": phi}


def _batch(kind, count, lo, hi, shapes, target=1e-10):
    """count GEMMs, m, n, k log-uniform in [lo, hi] (drawn from the seed `shapes`), each with its tuner plan"""
    return {"kind": kind, "count": count, "lo": lo, "hi": hi, "shapes": shapes, "target": target}


def listed():
    def named(name, c):
        return {"name": name, **c}

    return [
        # the smallest calls: the uneven 97 x 61 x 45 of the parity tests, one Strassen level
        named("f64_tiny", _case("f64", 97, 61, 45, "222", 1)),
        # an ordinary classical FP64 GEMM of a dense solver's block, overwriting C
        named("f64_classical", _case("f64", 1000, 1200, 900, beta=0.0)),
        # small and skinny: a short, wide panel times its transpose-shaped partner (BLIS's "sup" shapes)
        named("f64_skinny", _case("f64", 200, 150, 6000)),
        # the reference's own call, its benchmark configuration: one Strassen level, host operands
        named("f64_dropin_2048", _case("f64_host", 2048, 2048, 2048, "222", 1)),
        # the FP64 sweep's other coefficient files, a size their splits do not divide
        named("f64_333_ragged", _case("f64", 4097, 3001, 3500, "333", 1, alpha=-1.0)),
        # many uneven FP64 problems in one call
        named("f64_batch", _batch("f64_batch", 24, 256, 1024, 1)),
        # a small served request: one split GEMM with the tuner's classical plan
        named("split_small", _case("split", 300, 700, 450, slices=6, beta=0.0)),
        # an ordinary request: one Strassen level, sizes that divide nothing, a sub-array of a larger matrix
        named("split_mid", _case("split", 3000, 2500, 2049, "222", 1, 6, pad=5)),
        # the FP8 format, a rectangular algorithm and shape
        named("split_fp8", _case("split", 4097, 3001, 5000, "322", 1, 10, "fp8")),
        # the headline workload: two Strassen levels at 16384, 6 slices
        named("split_16384", _case("split", 16384, 16384, 16384, "222", 2, 6)),
        # the split form behind the reference's host interface
        named("split_host_4096", _case("split_host", 4096, 4096, 4096, "222", 1, 6)),
        # what a server launches together: uneven split problems, a plan for each
        named("split_batch", _batch("split_batch", 48, 256, 4096, 2)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi, most):
    """m, n, k log-uniform in [lo, hi] with m * n * k at most `most`"""
    while True:
        m, n, k = (_log_int(rng, lo, hi) for _ in range(3))
        if m * n * k <= most:
            return m, n, k


def draw(rng):
    kind = rng.choice(["f64", "f64", "f64_skinny", "f64_host", "f64_batch", "split", "split", "split", "split_host",
                       "split_batch"])
    beta = rng.choice([0.0, 1.0, 1.0, 0.5])
    alpha = rng.choice([1.0, 1.0, -1.0])
    pad = rng.choice([0, 0, rng.randint(1, 40)])
    if kind == "f64_batch":
        return _batch(kind, rng.randint(4, 32), 128, 1024, rng.randint(10, 1 << 20))
    if kind == "split_batch":
        return _batch(kind, rng.randint(4, 60), 128, 4096, rng.randint(10, 1 << 20), rng.choice([1e-8, 1e-10, 1e-10]))
    if kind == "f64_skinny":
        return _case("f64", _log_int(rng, 8, 320), _log_int(rng, 8, 320), _log_int(rng, 512, 16384), alpha=alpha,
                     beta=beta, pad=pad)
    if kind == "f64":
        m, n, k = _dims(rng, 64, 8192, 3.6e10)
        alg, levels = "classical", 0
        if min(m, n, k) >= 192 and rng.random() < 0.7:
            alg, levels = rng.choice(["222", "232", "322", "333", "444"]), 1
            if min(m, n, k) >= 1536 and rng.random() < 0.5:
                levels = 2
        return _case("f64", m, n, k, alg, levels, alpha=alpha, beta=beta, pad=pad)
    if kind == "f64_host":
        m, n, k = _dims(rng, 128, 3000, 1.0e10)
        return _case("f64_host", m, n, k, rng.choice(["222", "232", "322", "333", "444"]), 1, alpha=alpha, beta=beta)
    top = 6000 if kind == "split_host" else 14000
    m, n, k = _dims(rng, 128, top, 1.2e11 if kind == "split_host" else 1.0e12)
    alg, levels = "classical", 0
    if min(m, n, k) >= 1536 and rng.random() < 0.7:
        alg, levels = rng.choice(["222", "222", "232", "322", "333", "444"]), 1
        if alg == "222" and min(m, n, k) >= 4096 and rng.random() < 0.5:
            levels = 2
    fmt = rng.choice(["bf16", "bf16", "fp8"])
    slices = rng.randint(4, 7) if fmt == "bf16" else rng.randint(7, 11)
    return _case(kind, m, n, k, alg, levels, slices, fmt, alpha, beta, 0 if kind == "split_host" else pad,
                 rng.choice([0.0, 0.0, 1.0]))


def _operand(rows, cols, gen, pad=0, phi=0.0):
    """a column-major rows x cols operand on the GPU (leading dimension rows + pad)"""
    x = torch.rand((cols, rows + pad), generator=gen, device="cuda", dtype=torch.float64)
    if phi:
        z = torch.randn((cols, rows + pad), generator=gen, device="cuda", dtype=torch.float64)
        x.sub_(0.5).mul_(z.mul_(phi).exp_())
    else:
        x.mul_(2).sub_(1)
    return x[:, :rows].t()


def _inputs(case, seed):
    """A, B, C of one GEMM, from the seed alone"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    m, n, k, pad, phi = case["m"], case["n"], case["k"], case["pad"], case["phi"]
    return _operand(m, k, g, pad, phi), _operand(k, n, g, pad, phi), _operand(m, n, g, pad)


def _batch_inputs(case, seed):
    """(A, B, C) of every GEMM of a batch: the shapes belong to the case, the values to the seed"""
    r = np.random.default_rng(case["shapes"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    shapes = [tuple(int(round(math.exp(r.uniform(lo, hi)))) for _ in range(3)) for _ in range(case["count"])]
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [(_operand(m, k, g), _operand(k, n, g), _operand(m, n, g)) for m, n, k in shapes]


def _plans(case, ops):
    tuner = tune.Tuner()
    form = "fp64" if case["kind"] == "f64_batch" else "split"
    return [tuner.plan(A.shape[0], B.shape[1], A.shape[1], form, case["target"]) for A, B, _ in ops]


def _host(x):
    """a host copy in the library's pinned host memory, the way its documentation asks for operands"""
    h = fmm.host_empty(*x.shape)
    torch.from_numpy(h).copy_(x)
    return h


def prepare(case, seed):
    kind = case["kind"]
    if kind.endswith("_batch"):
        ops = _batch_inputs(case, seed)
        batch = fmm.make_batch([{"A": A, "B": B, "C": C, "fmm": _alg(p.alg), "levels": p.levels, "slices": p.slices,
                                 "fmt": p.fmt} for (A, B, C), p in zip(ops, _plans(case, ops))])
        ws = torch.empty(max(fmm.batch_workspace_size(batch), 256), dtype=torch.uint8, device="cuda")
        return {"kind": kind, "ops": ops, "batch": batch, "ws": ws}
    A, B, C = _inputs(case, seed)
    s = {**case, "f": _alg(case["alg"])}
    if kind.endswith("_host"):
        return {**s, "A": _host(A), "B": _host(B), "C": _host(C)}
    s.update(A=A, B=B, C=C)
    if kind == "split":
        need = fmm.split_workspace_size(case["m"], case["n"], case["k"], s["f"], case["levels"], case["slices"],
                                        case["fmt"])
        s["ws"] = torch.empty(max(need, 256), dtype=torch.uint8, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind.endswith("_batch"):
        fmm.batch_dgemm(s["batch"], workspace=s["ws"])
        return [C for _, _, C in s["ops"]]
    if kind == "f64":
        fmm.dgemm(s["A"], s["B"], s["C"], s["f"], s["levels"], s["alpha"], s["beta"])
    elif kind == "f64_host":
        fmm.bli_strassen_ab_ex(s["alpha"], s["A"], s["B"], s["beta"], s["C"], s["f"])
    elif kind == "split":
        fmm.split_dgemm(s["A"], s["B"], s["C"], s["f"], s["levels"], s["slices"], s["alpha"], s["beta"], s["ws"],
                        fmt=s["fmt"])
    else:
        fmm.split_strassen_ab_ex(s["alpha"], s["A"], s["B"], s["beta"], s["C"], s["f"], s["levels"], s["slices"],
                                 s["fmt"])
    return s["C"]


def _gemm_work(m, n, k, alg, levels, slices, beta):
    """A, B and C through memory once; the multiplications of the algorithm's products, once for every slice pair"""
    mt, kt, nt, R = (x ** levels for x in _SHAPES[alg]) if alg != "classical" else (1, 1, 1, 1)
    pairs = slices * (slices + 1) // 2 if slices else 1
    nbytes = 8.0 * (m * k + k * n + m * n * (1 if beta == 0.0 else 2))
    return nbytes, 2.0 * pairs * R * -(-m // mt) * -(-n // nt) * -(-k // kt)


def work(case):
    if case["kind"].endswith("_batch"):
        r = np.random.default_rng(case["shapes"])
        lo, hi = math.log(case["lo"]), math.log(case["hi"])
        tuner = tune.Tuner()
        form = "fp64" if case["kind"] == "f64_batch" else "split"
        nbytes = flops = 0.0
        for _ in range(case["count"]):
            m, n, k = (int(round(math.exp(r.uniform(lo, hi)))) for _ in range(3))
            p = tuner.plan(m, n, k, form, case["target"])
            b, f = _gemm_work(m, n, k, p.alg, p.levels, p.slices, 1.0)
            nbytes, flops = nbytes + b, flops + f
    else:
        nbytes, flops = _gemm_work(case["m"], case["n"], case["k"], case["alg"], case["levels"], case["slices"],
                                   case["beta"])
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    if case["kind"].endswith("_batch"):
        return [torch.addmm(C, A, B) for A, B, C in _batch_inputs(case, seed)]
    A, B, C = _inputs(case, seed)
    out = torch.addmm(C, A, B, alpha=case["alpha"], beta=case["beta"])
    return out.cpu().numpy() if case["kind"].endswith("_host") else out
