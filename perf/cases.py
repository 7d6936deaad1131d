"""The work whose speed on one B200 counts, as a serving program gives it to the library.

A tensor-parallel transformer block in inference calls the library for its MLP (prefill and decode),
for the column- and row-parallel projections by themselves, for the reduce + bias + RMSNorm epilogue
between layers, for plain norms and for all-reduces. On one GPU (no process group, world size 1) the
same program makes the same calls. Sizes are those of the benchmark and of the tests (hidden 5120 and
8192, FFN 28672 and its one-eighth shard 3584, decode rows 1 ... 256, messages of 4 KB ... 256 MB)
and, between them, ragged ones.

``listed()`` gives the cases, ``draw(rng)`` more of the same ranges, ``prepare`` what the program holds
before the call, ``run`` one pass, ``work`` the bytes and operations a pass cannot do without and
``tolerance`` how far two correct implementations may differ.
"""
from __future__ import annotations

import math

import torch

from kraken_b200 import comm, fused
from kraken_b200.models import TPMLP
from kraken_b200.parallel import symm_mem

DEVICE = "cuda"


def listed() -> list[dict]:
    return [
        # The benchmark's MLP block: a long prompt batch through up projection, GELU, down projection.
        {"name": "prefill_8192", "kind": "prefill", "m": 8192, "h": 8192, "f": 28672},
        # A prompt of arbitrary length: no dimension is a multiple of the tile sizes but the hidden one.
        {"name": "prefill_777", "kind": "prefill", "m": 777, "h": 5120, "f": 13704},
        # Column-parallel projection, one rank's share of eight; the gathered activations are used again.
        {"name": "all_gather_matmul_2048", "kind": "all_gather_matmul", "m": 2048, "k": 8192, "n": 3584},
        # Row-parallel projection, one rank's share of eight.
        {"name": "gemm_reduce_scatter_8192", "kind": "gemm_reduce_scatter", "m": 8192, "k": 3584, "n": 8192},
        # One token of one request through the down projection's share of eight, with bias and norm.
        {"name": "decode_1", "kind": "decode", "m": 1, "f": 1024, "h": 8192},
        # A small decode batch through the whole down projection.
        {"name": "decode_16", "kind": "decode", "m": 16, "f": 28672, "h": 8192},
        # A large decode batch.
        {"name": "decode_256", "kind": "decode", "m": 256, "f": 8192, "h": 8192},
        # The epilogue between two layers for one token: the smallest call of a decode step.
        {"name": "reduce_bias_norm_1", "kind": "reduce_bias_norm", "rows": 1, "d": 8192, "bias": "row", "form": "one_shot"},
        # The same for a batch, with the bias given for every row as in the tests.
        {"name": "reduce_bias_norm_512", "kind": "reduce_bias_norm", "rows": 512, "d": 5120, "bias": "full", "form": "two_shot"},
        # The norm of a prefill batch.
        {"name": "rms_norm_16384", "kind": "rms_norm", "rows": 16384, "d": 8192},
        # fp32 operands (multiplied as tf32, fp32 result), as in the tests of the GEMM + all-reduce.
        {"name": "gemm_all_reduce_fp32_1000", "kind": "gemm_all_reduce_fp32", "m": 1000, "k": 4096, "n": 4096},
        # The largest message of the all-reduce sweep.
        {"name": "all_reduce_256mb", "kind": "all_reduce", "numel": 128 << 20},
    ]


def _log_int(rng, lo: int, hi: int, unit: int = 1) -> int:
    """A multiple of `unit` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // unit, max(-(-lo // unit), round(v / unit))) * unit


def draw(rng) -> dict:
    kind = rng.choice(["prefill", "all_gather_matmul", "gemm_reduce_scatter", "decode", "decode", "reduce_bias_norm",
                       "rms_norm", "gemm_all_reduce_fp32", "all_reduce"])
    if kind == "prefill":
        return {"kind": kind, "m": _log_int(rng, 65, 8192), "h": _log_int(rng, 1024, 8192, 8), "f": _log_int(rng, 1024, 28672, 8)}
    if kind == "all_gather_matmul":
        return {"kind": kind, "m": _log_int(rng, 65, 8192), "k": _log_int(rng, 1024, 8192, 8), "n": _log_int(rng, 1024, 28672, 8)}
    if kind == "gemm_reduce_scatter":
        return {"kind": kind, "m": _log_int(rng, 65, 8192), "k": _log_int(rng, 1024, 28672, 8), "n": _log_int(rng, 1024, 8192, 8)}
    if kind == "decode":
        return {"kind": kind, "m": _log_int(rng, 1, 256), "f": _log_int(rng, 1024, 28672, 8), "h": _log_int(rng, 1024, 8192, 8)}
    if kind == "reduce_bias_norm":
        rows = _log_int(rng, 1, 2048)
        return {"kind": kind, "rows": rows, "d": _log_int(rng, 1024, 8192, 8), "bias": rng.choice(["row", "full", "none"]),
                "form": rng.choice(["one_shot", "two_shot"]) if rows <= 64 else "two_shot"}
    if kind == "rms_norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 16384), "d": _log_int(rng, 1024, 8192, 8)}
    if kind == "gemm_all_reduce_fp32":
        return {"kind": kind, "m": _log_int(rng, 1, 1024), "k": _log_int(rng, 1024, 8192, 4), "n": _log_int(rng, 1024, 8192, 4)}
    return {"kind": kind, "numel": _log_int(rng, 2 << 10, 128 << 20, 8)}


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _normal(g: torch.Generator, *shape: int, mean: float = 0.0, std: float = 1.0, dtype=torch.bfloat16) -> torch.Tensor:
    return torch.empty(*shape, dtype=dtype, device=DEVICE).normal_(mean, std, generator=g)


def _symmetric(t: torch.Tensor) -> torch.Tensor:
    s = symm_mem.empty(*t.shape, dtype=t.dtype, device=t.device)
    symm_mem.rendezvous(s)
    s.copy_(t)
    return s


def prepare(case: dict, seed: int) -> dict:
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("prefill", "decode"):
        # the block as a program holds it after loading its weights
        h, f = case["h"], case["f"]
        mlp = TPMLP(8, 8, device=DEVICE)
        mlp.hidden, mlp.ffn = h, f
        mlp.w_up_t = _normal(g, f, h, std=0.02) if kind == "prefill" else None
        mlp.w_down_t = _normal(g, h, f, std=0.02)
        mlp.bias = _normal(g, h)
        mlp.norm_w = _normal(g, h, mean=1.0, std=0.1)
        x = mlp.stage_input(_normal(g, case["m"], h)) if kind == "prefill" else _normal(g, case["m"], f)
        return {"kind": kind, "mlp": mlp, "x": x}
    if kind in ("all_gather_matmul", "gemm_reduce_scatter"):
        # weights as nn.Linear keeps them: [N, K], passed as their transpose
        a = _normal(g, case["m"], case["k"])
        return {"kind": kind, "a": _symmetric(a) if kind == "all_gather_matmul" else a,
                "w": _normal(g, case["n"], case["k"], std=0.02)}
    if kind == "gemm_all_reduce_fp32":
        return {"kind": kind, "a": _normal(g, case["m"], case["k"], dtype=torch.float32),
                "w": _normal(g, case["n"], case["k"], std=0.02, dtype=torch.float32)}
    if kind == "reduce_bias_norm":
        rows, d = case["rows"], case["d"]
        x = _normal(g, rows, d)
        bias = {"row": lambda: _normal(g, d), "full": lambda: _normal(g, rows, d), "none": lambda: None}[case["bias"]]()
        return {"kind": kind, "form": case["form"], "x": x, "scratch": _symmetric(torch.zeros_like(x)), "bias": bias,
                "w": _normal(g, d, mean=1.0, std=0.1), "y": torch.empty_like(x)}
    if kind == "rms_norm":
        return {"kind": kind, "x": _normal(g, case["rows"], case["d"]), "w": _normal(g, case["d"], mean=1.0, std=0.1)}
    return {"kind": kind, "x": _symmetric(_normal(g, case["numel"]))}


def run(state: dict):
    kind = state["kind"]
    if kind == "prefill":
        return state["mlp"].prefill(state["x"])
    if kind == "decode":
        return state["mlp"].decode(state["x"])
    if kind == "all_gather_matmul":
        return fused.all_gather_matmul(state["a"], state["w"].t())
    if kind == "gemm_reduce_scatter":
        return fused.gemm_reduce_scatter(state["a"], state["w"].t())
    if kind == "gemm_all_reduce_fp32":
        return fused.gemm_one_shot_all_reduce_fused(state["a"], state["w"].t())
    if kind == "reduce_bias_norm":
        op = fused.one_shot_all_reduce_bias_rms_norm if state["form"] == "one_shot" else fused.two_shot_all_reduce_bias_rms_norm
        op(state["scratch"], state["x"], state["bias"], state["w"], state["y"])
        return state["y"]
    if kind == "rms_norm":
        return fused.rms_norm(state["x"], state["w"])
    return comm.all_reduce(state["x"])


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "prefill":
        m, h, f = case["m"], case["h"], case["f"]
        return {"bytes": 2 * (2 * m * h + 2 * h * f), "flops": 4 * m * h * f}
    if kind == "decode":
        m, f, h = case["m"], case["f"], case["h"]
        return {"bytes": 2 * (m * f + h * f + m * h + 2 * h), "flops": 2 * m * f * h}
    if kind in ("all_gather_matmul", "gemm_reduce_scatter", "gemm_all_reduce_fp32"):
        m, k, n = case["m"], case["k"], case["n"]
        elements = m * k + n * k + m * n + (m * k if kind == "all_gather_matmul" else 0)
        return {"bytes": elements * (4 if kind == "gemm_all_reduce_fp32" else 2), "flops": 2 * m * k * n}
    if kind == "reduce_bias_norm":
        n = case["rows"] * case["d"]
        return {"bytes": 2 * (2 * n + {"row": case["d"], "full": n, "none": 0}[case["bias"]] + case["d"]), "flops": 5 * n}
    if kind == "rms_norm":
        return {"bytes": 2 * (2 * case["rows"] * case["d"] + case["d"]), "flops": 4 * case["rows"] * case["d"]}
    return {"bytes": 4 * case["numel"], "flops": 0}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "all_reduce":
        return "exact"                  # the sum over one rank
    if kind == "gemm_all_reduce_fp32":
        return {"rel": 1e-3}            # operands of 10 mantissa bits, rounded or cut
    if kind in ("prefill", "decode"):
        return {"rel": 1e-2}            # bf16 results with bf16 values in between
    return {"rel": 5e-3}                # bf16 results of fp32 sums
