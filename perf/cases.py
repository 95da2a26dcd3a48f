"""The work that users of this framework have it do, as cases that can be timed and compared on one B200.

A case is a dict of plain values; `op` names the public entry point it goes through:

* `block` / `allreduce`   one rank's whole work of the fused AllReduce (+ residual add + Gemma RMSNorm) of a group of
                          `ranks` GPUs, called eagerly.  One GPU has no peers, so the rank runs alone in compute mode
                          (`SoloRankContext`: every push is looped back into its own window), as `bench.py` does on one GPU.
* `chain`                 a prefill step: 121 such blocks recorded in one CUDA graph, replayed.
* `encode`, `encode_static`, `decode_sum`, `owner_step`, `norm`   the codec and norm ops of `ops/codec.py` (and
                          `torch.ops.fp4ar.add_rms_norm`).
* `gemm`                  the row-parallel linear with NVFP4 output rows.
* `linear`                `torch.ops.fp4ar.linear_nvfp4` and the fused block on its rows (NVFP4 input), one rank of two.

Row counts run from one token to 16384-token prefill chunks, hidden size 6144 everywhere (the only one the row format
has); K is the input width of a row-parallel linear under tensor parallelism.
"""
from __future__ import annotations

import math

import torch

from fp4_all_reduce_b200 import _native as N
from fp4_all_reduce_b200.models.m3_block import BLOCKS_PER_STEP, M3PrefillChain
from fp4_all_reduce_b200.ops import allreduce  # noqa: F401  (registers torch.ops.fp4ar.*)
from fp4_all_reduce_b200.ops import codec
from fp4_all_reduce_b200.ops import gemm as G
from fp4_all_reduce_b200.parallel.context import SoloRankContext
from fp4_all_reduce_b200.utils import timing

H = N.HIDDEN
ROW = 2 * H                       # bytes of a BF16 row
EPI_OUT = {0: ROW, N.EPI_NORM_BF16: ROW, N.EPI_NORM_NVFP4: N.QROW_BYTES, N.EPI_NORM_MXFP8: N.MXROW_BYTES}
MAX_ROWS = 16384
QSCALE = 168.0                    # global scale of the NVFP4 output, the block chain's default


def listed() -> list[dict]:
    return [
        # The headline: the largest prefill chunk at tensor-parallel degree 2, BF16 in and out.
        {"name": "block_tp2_16384", "op": "block", "ranks": 2, "rows": 16384, "inp": "bf16", "epi": 1},
        # An ordinary prefill chunk at degree 4 (two-shot: the rank also owns a quarter of the rows).
        {"name": "block_tp4_4096", "op": "block", "ranks": 4, "rows": 4096, "inp": "bf16", "epi": 1},
        # A ragged chunk at degree 8, normalised activations quantised for an NVFP4 GEMM.
        {"name": "block_tp8_1031_fp4out", "op": "block", "ranks": 8, "rows": 1031, "inp": "bf16", "epi": 2},
        # A decode step of 16 sequences at degree 8: latency, launches and the host path.
        {"name": "block_tp8_16", "op": "block", "ranks": 8, "rows": 16, "inp": "bf16", "epi": 1},
        # A producer that already emits NVFP4 rows, plain AllReduce.
        {"name": "allreduce_tp2_fp4in_2048", "op": "allreduce", "ranks": 2, "rows": 2048, "inp": "nvfp4"},
        # A whole prefill step of 1024 tokens: 121 blocks in one CUDA graph, no host work between them.
        {"name": "chain_tp2_1024", "op": "chain", "ranks": 2, "rows": 1024, "inp": "bf16", "epi": 1},
        # Encode direction: BF16 activations of a prefill chunk to NVFP4 rows with dynamic row scales.
        {"name": "encode_8192", "op": "encode", "rows": 8192},
        # Decode direction: the sum of four ranks' rows, a ragged row count.
        {"name": "decode_sum_4x3001", "op": "decode_sum", "nsrc": 4, "rows": 3001},
        # The two-shot owner step: sum, re-encode, decode of the re-encoding.
        {"name": "owner_step_4x4096", "op": "owner_step", "nsrc": 4, "rows": 4096},
        # Residual add + norm of a decode batch through the custom op.
        {"name": "norm_32", "op": "norm", "rows": 32, "epi": 1},
        # Row-parallel down projection of a prefill chunk, NVFP4 rows out.
        {"name": "gemm_4096_k8192", "op": "gemm", "rows": 4096, "k": 8192},
        # Row-parallel projection, then AllReduce + norm, of a 64-token decode batch: the weights dominate.
        {"name": "linear_64_k2048", "op": "linear", "rows": 64, "k": 2048},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng) -> dict:
    """One more case of the same ranges: any row count from 1 up (log-uniform), any degree, input kind and epilogue."""
    op = rng.choice(["block", "block", "block", "block", "allreduce", "allreduce", "chain", "encode", "decode_sum", "owner_step",
                     "norm", "gemm", "gemm", "linear"])
    rows = _log_int(rng, 1, MAX_ROWS)
    if op in ("block", "allreduce"):
        c = {"op": op, "ranks": rng.choice([2, 4, 8]), "rows": rows, "inp": rng.choice(["bf16", "bf16", "nvfp4"])}
        if op == "block":
            c["epi"] = rng.choice([1, 1, 2, 3])
        return c
    if op == "chain":
        return {"op": op, "ranks": rng.choice([2, 4, 8]), "rows": _log_int(rng, 1, 1024), "inp": "bf16", "epi": 1}
    if op == "encode":
        return {"op": rng.choice(["encode", "encode_static"]), "rows": rows}
    if op in ("decode_sum", "owner_step"):
        return {"op": op, "nsrc": rng.choice([1, 2, 4, 8] if op == "decode_sum" else [2, 4, 8]), "rows": rows}
    if op == "norm":
        return {"op": op, "rows": rows, "epi": rng.choice([1, 2, 3])}
    # K of a row-parallel linear: hidden or intermediate width over the tensor-parallel degree, a multiple of 64
    return {"op": op, "rows": _log_int(rng, 1, 4096), "k": 64 * _log_int(rng, 16, 128)}


def _partial(rows: int, g: torch.Generator) -> torch.Tensor:
    """A rank's partial: N(0,1) times a per-row lognormal scale, 0.1 % of the values 50 times larger."""
    x = torch.randn(rows, H, generator=g, device="cuda") * torch.exp(torch.randn(rows, 1, generator=g, device="cuda"))
    x = torch.where(torch.rand(rows, H, generator=g, device="cuda") < 1e-3, x * 50.0, x)
    return x.to(torch.bfloat16)


def _residual(rows: int, g: torch.Generator) -> torch.Tensor:
    return torch.randn(rows, H, generator=g, device="cuda").to(torch.bfloat16)


def _weight(g: torch.Generator) -> torch.Tensor:
    return (torch.randn(H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)


def prepare(case: dict, seed: int) -> dict:
    g = torch.Generator(device="cuda").manual_seed(seed)
    op, rows = case["op"], case["rows"]
    s: dict = {"case": case}
    if op in ("block", "allreduce"):
        x = _partial(rows, g)
        s["gs"] = None
        if case["inp"] == "nvfp4":
            gs = float(x.abs().max().item()) / 2688.0
            x, s["gs"] = codec.encode_static(x, gs), [gs] * case["ranks"]
        s["x"] = x
        s["ctx"] = SoloRankContext(case["ranks"], rows)
        if op == "block":
            s["residual"], s["weight"] = _residual(rows, g), _weight(g)
    elif op == "chain":
        ctx = SoloRankContext(case["ranks"], rows)
        chain = M3PrefillChain(ctx, rows, epilogue=case["epi"], mode=N.MODE_COMPUTE, nranks=case["ranks"])
        for p in chain.partials:
            p.copy_(_partial(rows, g))
        chain.weight.copy_(_weight(g))
        s["chain"] = chain
        s["graph"] = timing.capture(chain.block, BLOCKS_PER_STEP, chain.device)
        chain.residual.copy_(_residual(rows, g))
    elif op == "encode":
        s["x"] = _partial(rows, g)
    elif op == "encode_static":
        s["x"] = _partial(rows, g)
        s["gs"] = float(s["x"].abs().max().item()) / 2688.0
    elif op in ("decode_sum", "owner_step"):
        rec = [codec.encode(_partial(rows, g)) for _ in range(case["nsrc"])]
        s["q"], s["rs"] = [q for q, _ in rec], [r for _, r in rec]
    elif op == "norm":
        s["x"], s["residual"], s["weight"] = _partial(rows, g), _residual(rows, g), _weight(g)
    else:
        k = case["k"]
        s["x"] = torch.randn(rows, k, generator=g, device="cuda").to(torch.bfloat16)
        s["wt"] = (torch.randn(H, k, generator=g, device="cuda") / math.sqrt(k)).to(torch.bfloat16)
        s["gs"] = 6.0 / 2688.0            # outputs are N(0,1): the largest of a calibration batch is about 6
        if op == "linear":
            s["ctx"] = SoloRankContext(2, rows)
            s["residual"], s["weight"] = _residual(rows, g), _weight(g)
    return s


def run(s: dict):
    case = s["case"]
    op = case["op"]
    if op == "block":
        return s["ctx"].all_reduce_add_rms_norm(s["x"], s["residual"], s["weight"], epilogue=case["epi"], qscale=QSCALE,
                                                gs=s["gs"], mode=N.MODE_COMPUTE)
    if op == "allreduce":
        return s["ctx"].all_reduce(s["x"], gs=s["gs"], mode=N.MODE_COMPUTE)
    if op == "chain":
        s["graph"].replay()
        return s["chain"].out, s["chain"].residual
    if op == "encode":
        return codec.encode(s["x"])
    if op == "encode_static":
        return codec.encode_static(s["x"], s["gs"])
    if op == "decode_sum":
        return codec.decode_sum(s["q"], s["rs"])
    if op == "owner_step":
        return codec.reduce_reencode(s["q"], s["rs"])
    if op == "norm":
        if case["epi"] == N.EPI_NORM_BF16:
            return torch.ops.fp4ar.add_rms_norm(s["x"], s["residual"], s["weight"], 1e-6, 1.0), s["residual"]
        return codec.add_rmsnorm(s["x"], s["residual"], s["weight"], epilogue=case["epi"], qscale=QSCALE, inplace_residual=True)
    if op == "gemm":
        return G.gemm_nvfp4(s["x"], s["wt"], s["gs"])
    q = torch.ops.fp4ar.linear_nvfp4(s["x"], s["wt"], s["gs"])
    return s["ctx"].all_reduce_add_rms_norm(q, s["residual"], s["weight"], gs=[s["gs"]] * 2, mode=N.MODE_COMPUTE)


def work(case: dict) -> dict:
    """Inputs read once, outputs written once; the receive window of the looped-back pushes is not counted."""
    op, rows = case["op"], case["rows"]
    if op in ("block", "allreduce", "chain"):
        epi = case.get("epi", 0)
        b = rows * ((ROW if case["inp"] == "bf16" else N.QROW_BYTES) + EPI_OUT[epi] + (2 * ROW if epi else 0)) + (ROW if epi else 0)
        f = rows * H * (2 * case["ranks"] + 2 + (6 if epi else 0))      # quantise, one multiply-add per source, norm
        n = BLOCKS_PER_STEP if op == "chain" else 1
        return {"bytes": n * b, "flops": n * f}
    if op in ("encode", "encode_static"):
        return {"bytes": rows * (ROW + N.QROW_BYTES + (4 if op == "encode" else 0)), "flops": 2 * rows * H}
    if op == "decode_sum":
        return {"bytes": rows * (case["nsrc"] * (N.QROW_BYTES + 4) + ROW), "flops": 2 * case["nsrc"] * rows * H}
    if op == "owner_step":
        return {"bytes": rows * (case["nsrc"] * (N.QROW_BYTES + 4) + N.REC_STRIDE + ROW),
                "flops": 2 * (case["nsrc"] + 2) * rows * H}
    if op == "norm":
        return {"bytes": rows * (3 * ROW + EPI_OUT[case["epi"]]) + ROW, "flops": 6 * rows * H}
    k = case["k"]
    b = 2 * k * (rows + H)
    b += rows * N.QROW_BYTES if op == "gemm" else rows * 3 * ROW + ROW
    return {"bytes": b, "flops": 2 * rows * H * k}


def tolerance(case: dict):
    """The codec, the AllReduce and the norm are defined bit for bit (IEEE operations in a fixed order, the host model
    of the tests); only the GEMM's FP32 sums may be taken in another order.  Sums that differ by about 1e-6 of their
    size round to another E2M1 value for about 1 in 1e5 of them, and to another block scale (which moves a few of 16
    values) for about 1 in 1e4 blocks."""
    if case["op"] == "gemm":
        return {"differ": 1e-3}
    if case["op"] == "linear":
        return {"rel": 5e-3, "max": 0.5}       # such a value is off by one E2M1 step, up to a third of itself
    return "exact"
