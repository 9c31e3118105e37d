"""The work that a program on one GPU has this library do, as cases with inputs, one pass, and its cost.

Every case goes through the package's public entry points on a one-rank communicator: the tensor-parallel
SwiGLU block and the GEMM under it, the residual + RMSNorm of a layer, the expert dispatch and combine
around an MoE layer, the collectives with a scale / cast epilogue, and a sharded optimizer's pair of
collectives.  Inputs are drawn on the GPU from the seed; weights N(0, 0.02) and activations N(0, 1) as in
``bench.py``.  Sizes are those of ``bench.py``, ``benchmarks/`` and ``tests/``, or generic.
"""
import copy
import functools
import math
import os

import torch

os.environ.setdefault("UCCL_BOOTSTRAP_IFNAME", "lo")

from unified_ccl_b200 import Communicator  # noqa: E402
from unified_ccl_b200.models import TensorParallelMLP  # noqa: E402
from unified_ccl_b200.ops import gemm_bf16  # noqa: E402
from unified_ccl_b200.parallel import MoeDispatcher, allreduce_residual_rmsnorm  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "fp8": torch.float8_e4m3fn}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4, "fp8": 1}


def listed():
    return [
        # the block of bench.py: prefill of 4 sequences of 4096 tokens through one Llama-style MLP
        {"name": "mlp_prefill", "kind": "mlp", "tokens": 16384, "hidden": 4096, "ffn": 14336},
        # the same block in decode: one new token for each of 64 sequences, bound by reading the weights
        {"name": "mlp_decode", "kind": "mlp", "tokens": 64, "hidden": 4096, "ffn": 14336},
        # gate / up projection of a tensor-parallel rank with a quarter of the block, 4096 tokens in flight
        {"name": "gemm_swiglu_rank", "kind": "gemm", "m": 4096, "n": 7168, "k": 4096, "swiglu": True},
        # a chunk of a ragged batch against a weight whose sides are no multiples of a tile
        {"name": "gemm_ragged", "kind": "gemm", "m": 1000, "n": 3592, "k": 4104, "swiglu": False},
        # a small head or adapter: launch latency is all there is
        {"name": "gemm_small", "kind": "gemm", "m": 256, "n": 512, "k": 256, "swiglu": False},
        # residual + RMSNorm of a layer in prefill, new residual in a buffer of its own
        {"name": "norm_prefill", "kind": "norm", "tokens": 8192, "hidden": 8192, "inplace": False},
        # the same in decode with a handful of sequences, residual stream updated in place
        {"name": "norm_decode", "kind": "norm", "tokens": 7, "hidden": 8192, "inplace": True},
        # MoE layer in prefill: tokens leave as fp8 rows, which are then brought into a fixed order
        {"name": "moe_dispatch", "kind": "moe", "part": "dispatch", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8},
        # the other end of that layer: the weighted sum of every token's expert rows
        {"name": "moe_combine", "kind": "moe", "part": "combine", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8},
        # an MoE layer in decode: dispatch, a stand-in for the experts, combine
        {"name": "moe_decode", "kind": "moe", "part": "layer", "tokens": 96, "hidden": 7168, "experts": 32, "topk": 8},
        # activations of a layer leaving for the next stage as block-scaled fp8
        {"name": "cast_fp8", "kind": "cast", "api": "reduce_scatter", "count": 8192 * 8192, "din": "bf16", "dout": "fp8"},
        # sharded optimizer on a small tensor (a bias, a norm weight): calls and launches count, not bytes
        {"name": "shard_small", "kind": "shard", "count": 4096, "din": "bf16"},
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mlp", "gemm", "gemm", "norm", "moe", "cast", "shard"])
    if kind == "mlp":  # the block of bench.py whole, or the slice of it that a rank of 2, 4 or 8 holds
        return {"kind": kind, "tokens": _log(rng, 1, 16384), "hidden": 4096, "ffn": rng.choice([14336, 7168, 3584, 1792])}
    if kind == "gemm":
        swiglu = rng.random() < 0.4
        step = 16 if swiglu else 8
        return {"kind": kind, "m": _log(rng, 1, 16384), "n": step * _log(rng, 1, 14336 // step), "k": 8 * _log(rng, 8, 1536),
                "swiglu": swiglu}
    if kind == "norm":
        return {"kind": kind, "tokens": _log(rng, 1, 8192), "hidden": 8 * _log(rng, 64, 2048), "inplace": rng.random() < 0.5}
    if kind == "moe":
        part = rng.choice(["dispatch", "combine", "layer"])
        return {"kind": kind, "part": part, "tokens": _log(rng, 1, 512 if part == "layer" else 4096), "hidden": 128 * rng.randint(8, 64),
                "experts": rng.choice([8, 16, 32, 64, 256]), "topk": rng.choice([1, 2, 4, 4, 8, 8])}
    if kind == "cast":
        return {"kind": kind, "api": rng.choice(["reduce_scatter", "allreduce"]), "count": 128 * _log(rng, 1, 1 << 19),
                "din": rng.choice(["bf16", "fp32", "fp16"]), "dout": rng.choice(["fp8", "fp8", "bf16", "fp32", "fp16"])}
    return {"kind": kind, "count": _log(rng, 512, 1 << 26), "din": rng.choice(["bf16", "fp16", "fp32"])}


@functools.lru_cache(maxsize=None)
def _comm():
    return Communicator(0, 1)


@functools.lru_cache(maxsize=None)
def _block(hidden, ffn, tokens):
    return TensorParallelMLP(_comm(), hidden, ffn, tokens, seed=0)


_idle = {}  # dispatchers that no state holds any more, by shape: what they returned stays readable


class _Moe:
    """A layer's dispatcher, kept for the next state of the same shape when the state that holds it goes."""

    def __init__(self, case):
        self.shape = (case["tokens"], case["hidden"], case["experts"], case["topk"])
        idle = _idle.setdefault(self.shape, [])
        self.disp = idle.pop(0) if idle else MoeDispatcher(_comm(), *self.shape)

    def __del__(self):
        _idle[self.shape].append(self.disp)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(*shape, device=dev, dtype=dtype).normal_(0.0, std, generator=gen)

    kind = case["kind"]
    s = {"kind": kind, "comm": _comm()}
    if kind == "mlp":
        # a block whose weights have been loaded, with activation buffers of its own
        mlp = copy.copy(_block(case["hidden"], case["ffn"], case["tokens"]))
        mlp.w_gate_up = normal(2 * case["ffn"], case["hidden"], std=0.02)
        mlp.w_down = normal(case["hidden"], case["ffn"], std=0.02)
        mlp.h, mlp.y = torch.empty_like(mlp.h), torch.empty_like(mlp.y)
        s.update(mlp=mlp, x=normal(case["tokens"], case["hidden"]))
    elif kind == "gemm":
        n_out = case["n"] // 2 if case["swiglu"] else case["n"]
        s.update(a=normal(case["m"], case["k"]), b=normal(case["n"], case["k"], std=0.02), swiglu=case["swiglu"],
                 out=torch.empty(case["m"], n_out, device=dev, dtype=torch.bfloat16))
    elif kind == "norm":
        x = normal(case["tokens"], case["hidden"])
        s.update(x=x, residual=normal(case["tokens"], case["hidden"]), gamma=normal(case["hidden"], std=0.02).add_(1.0),
                 out=torch.empty_like(x), residual_out=None if case["inplace"] else torch.empty_like(x))
    elif kind == "moe":
        t, h, k = case["tokens"], case["hidden"], case["topk"]
        moe = _Moe(case)
        weight, idx = torch.softmax(normal(t, case["experts"], dtype=torch.float32), -1).topk(k, dim=-1)
        s.update(moe=moe, part=case["part"], topk=k, x=normal(t, h), idx=idx.to(torch.int32).contiguous(), weight=weight.contiguous())
        if case["part"] == "dispatch":
            s.update(key=torch.empty(t * k, device=dev, dtype=torch.int64), row=torch.arange(t * k, device=dev),
                     at=torch.empty(t * k, device=dev, dtype=torch.int64), rows=torch.empty(t * k, h, device=dev, dtype=torch.uint8),
                     scales=torch.empty(t * k, h // 128, device=dev, dtype=torch.float32))
        else:
            s.update(out=torch.empty(t, h, device=dev, dtype=torch.bfloat16))
        if case["part"] == "combine":
            # the experts' answers: row r belongs to (token, k) of its descriptor
            meta = moe.disp.dispatch(s["x"], s["idx"])[2][0]
            rows = normal(t * k, h)
            torch.index_select(rows, 0, meta[:, 0] * k + meta[:, 2], out=moe.disp.expert_out[0])
    elif kind == "cast":
        fp8 = case["dout"] == "fp8"
        s.update(api=case["api"], x=normal(case["count"], dtype=DTYPES[case["din"]]), factor=0.37,
                 out=torch.empty(case["count"], device=dev, dtype=DTYPES[case["dout"]]),
                 scales=torch.empty(case["count"] // 128, device=dev, dtype=torch.float32) if fp8 else None)
    else:
        grad = normal(case["count"], dtype=DTYPES[case["din"]])
        s.update(grad=grad, shard=torch.empty_like(grad), weight=normal(case["count"], dtype=DTYPES[case["din"]]), full=torch.empty_like(grad))
    return s


def run(s):
    kind, comm = s["kind"], s["comm"]
    if kind == "mlp":
        return s["mlp"](s["x"])
    if kind == "gemm":
        return gemm_bf16(s["a"], s["b"], out=s["out"], swiglu=s["swiglu"])
    if kind == "norm":
        return allreduce_residual_rmsnorm(comm, s["x"], s["residual"], s["gamma"], 1e-6, out=s["out"], residual_out=s["residual_out"])
    if kind == "moe":
        disp = s["moe"].disp
        if s["part"] == "combine":
            return disp.combine(s["weight"], out=s["out"])
        recv_x, recv_scale, recv_meta, recv_counts = disp.dispatch(s["x"], s["idx"])
        if s["part"] == "layer":
            disp.expert_out.copy_(recv_x)  # stands for the experts: one bf16 row for each received row
            return disp.combine(s["weight"], out=s["out"])
        # received rows have no fixed order: here they are laid out by (token, k)
        meta = recv_meta[0]
        torch.add(meta[:, 2], meta[:, 0], alpha=s["topk"], out=s["key"])
        s["at"].scatter_(0, s["key"], s["row"])
        torch.index_select(recv_x[0].view(torch.uint8), 0, s["at"], out=s["rows"])
        torch.index_select(recv_scale[0], 0, s["at"], out=s["scales"])
        return s["rows"], s["scales"], recv_counts
    if kind == "cast":
        fn = comm.reduce_scatter_cast if s["api"] == "reduce_scatter" else comm.allreduce_cast
        return fn(s["x"], s["out"], s["factor"], scales=s["scales"])
    return comm.reduce_scatter(s["grad"], s["shard"]), comm.allgather(s["weight"], s["full"])


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * (2 * t * h + 3 * h * f), "flops": 6 * t * h * f}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * (n // 2 if case["swiglu"] else n)), "flops": 2 * m * n * k}
    if kind == "norm":
        return {"bytes": 2 * case["hidden"] * (4 * case["tokens"] + 1), "flops": 6 * case["tokens"] * case["hidden"]}
    if kind == "moe":
        t, h, rows = case["tokens"], case["hidden"], case["tokens"] * case["topk"]
        row = h + h // 128 * 4  # a received row and its scales
        dispatch = 2 * t * h + rows * (4 + row + 16)
        combine = rows * (2 * h + 4) + 2 * t * h
        if case["part"] == "combine":
            return {"bytes": combine, "flops": 2 * rows * h}
        if case["part"] == "layer":
            return {"bytes": dispatch + rows * 3 * h + combine, "flops": 2 * rows * h + 4 * t * h}
        return {"bytes": dispatch + rows * (2 * row + 16), "flops": 4 * t * h}
    if kind == "cast":
        n = case["count"]
        return {"bytes": n * (BYTES[case["din"]] + BYTES[case["dout"]]) + (n // 32 if case["dout"] == "fp8" else 0), "flops": 2 * n}
    return {"bytes": 4 * case["count"] * BYTES[case["din"]], "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "mlp":
        return {"rel": 8e-3}  # two roundings to bf16, the first of them summed over ffn
    if kind == "gemm":
        return {"rel": 5e-3}  # fp32 sums in another order, one rounding to bf16
    if kind == "norm" or case.get("part") in ("combine", "layer"):
        return {"rel": 4e-3}  # fp32 arithmetic, one rounding to bf16
    return "exact"  # one rank: each value is scaled or quantised with one rounding, or copied
