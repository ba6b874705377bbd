"""The work this framework is used for, as cases that can be timed one pass at a time on one GPU.

Families (``case["op"]``):

``norm``            ``models.RMSNorm`` on row-major activations (decode batches up to long prefills)
``unreorder_norm``  ``models.ReorderRMSNorm`` on the tile-contiguous shard that a fused reduce-scatter leaves
``relayout``        ``ops.reorder`` and ``ops.unreorder``: into the tile-contiguous layout and back
``linear``          ``models.OverlapRowParallelLayer`` with one rank, either collective and either output
                    layout, optionally followed by ``models.ReorderRMSNorm`` (sequence-parallel o_proj)
``add_norm``        ``OverlapImpl.gemm_reducescatter_add_rmsnorm_fused``: projection, residual add and
                    RMSNorm of a pre-norm block
``emulated``        ``ops.fused_loopback``: the fused GEMM + collective kernels with all ranks of the
                    group in one cooperative launch, which is how they run, are tested and are profiled
                    on one GPU
``decoder``         ``models.TPDecoderLayer`` forward with the per-GPU share of the weights

Sizes are the repository's own: the tensor-parallel row-parallel shapes of the benchmark and of the sweep
(M 1024..16384, N 4096 and 8192, K 8192, 14336 or 28672 over 1..8 ranks), a decode batch (the 128 rows
that are the smallest M the GEMM takes), and ragged ones.  Tilings are chosen the way every command line
of the repository chooses them without a tuning run: ``config.default_solution`` of the asked Algo, which
falls back to a kernel that divides the shape.
"""
import math

import torch

from flashoverlap_b200 import ops
from flashoverlap_b200.models import DecoderConfig, OverlapRowParallelLayer, ReorderRMSNorm, RMSNorm, TPDecoderLayer
from flashoverlap_b200.utils import config, layout

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
DEVICE = "cuda"
# Algos the repository's scripts start from: the command lines' default, and those its sweep, its benchmark
# and its single-CTA emulation try.
LINEAR_ALGOS = (1, 17, 19, 3, 0, 16, 2)
EMULATED_ALGOS = (0, 2, 16)
# (hidden, ffn, query heads, KV heads): the tiny test layer; a 4096-wide one; one of eight ranks' share of
# the 8192 / 28672 layer with 64 query and 8 KV heads
DECODERS = ((1024, 2048, 8, 2), (4096, 3584, 8, 2), (8192, 3584, 8, 1))


def listed():
    return [
        # one decoded token's hidden state: nothing but latency
        {"name": "norm_one_token", "op": "norm", "rows": 1, "dim": 8192, "dtype": "bf16"},
        # the norm behind a reduce-scatter over two ranks: 16384 tokens, 64-row slices of every tile
        {"name": "unreorder_norm_tp2_shard", "op": "unreorder_norm", "rows": 8192, "dim": 8192, "bm": 64, "bn": 256,
         "dtype": "bf16"},
        # layout change of an activation matrix, both ways
        {"name": "relayout_fp16", "op": "relayout", "rows": 4096, "dim": 8192, "bm": 128, "bn": 256, "rldn": 1,
         "dtype": "fp16"},
        # down projection of a small decode batch on one of eight ranks: the weights are read once, nothing is reused
        {"name": "linear_decode", "op": "linear", "m": 128, "n": 8192, "k": 3584, "algo": 1, "comm": "all_reduce",
         "layout": "natural", "norm": False, "dtype": "bf16"},
        # smallest shape of the sweep at eight ranks, with the norm of a sequence-parallel block
        {"name": "linear_small_fp16", "op": "linear", "m": 1024, "n": 4096, "k": 1024, "algo": 1,
         "comm": "reduce_scatter", "layout": "reordered", "norm": True, "dtype": "fp16"},
        # odd tile counts in both directions and a K that is no multiple of the k-block
        {"name": "linear_ragged", "op": "linear", "m": 1920, "n": 5376, "k": 1000, "algo": 1, "comm": "all_reduce",
         "layout": "natural", "norm": False, "dtype": "bf16"},
        # attention output projection, residual and norm of a chunk of a prefill
        {"name": "add_norm_chunk", "op": "add_norm", "m": 2048, "n": 8192, "k": 1792, "algo": 17, "dtype": "bf16"},
        # sequence-parallel o_proj + norm, 16384 tokens, one of eight ranks
        {"name": "linear_norm_16k", "op": "linear", "m": 16384, "n": 8192, "k": 1024, "algo": 1,
         "comm": "reduce_scatter", "layout": "reordered", "norm": True, "dtype": "bf16"},
        # the benchmark's headline: the whole MLP down projection on one rank
        {"name": "linear_headline", "op": "linear", "m": 8192, "n": 8192, "k": 28672, "algo": 19,
         "comm": "all_reduce", "layout": "reordered", "norm": False, "dtype": "bf16"},
        # the fused collectives: two ranks all-reducing with the push protocol ...
        {"name": "emulated_allreduce_2", "op": "emulated", "comm": "all_reduce", "ranks": 2, "m": 2048, "n": 4096,
         "k": 2048, "algo": 0, "pull": False, "strided": True, "natural": False, "dtype": "bf16"},
        # ... and eight ranks reduce-scattering with the pull protocol
        {"name": "emulated_reducescatter_8", "op": "emulated", "comm": "reduce_scatter", "ranks": 8, "m": 4096,
         "n": 8192, "k": 1024, "algo": 0, "pull": True, "strided": True, "natural": True, "dtype": "bf16"},
        # prefill of one 4096-token sequence through a decoder layer, one of eight ranks' share of the weights
        {"name": "decoder_prefill", "op": "decoder", "hidden": 8192, "ffn": 3584, "heads": 8, "kv_heads": 1,
         "batch": 1, "seq": 4096},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], spread evenly over the logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi // step, max(-(-lo // step), round(x / step))) * step)


def draw(rng):
    op = rng.choice(("norm", "unreorder_norm", "relayout", "linear", "linear", "linear", "add_norm", "emulated",
                     "emulated", "decoder"))
    dtype = rng.choice(("bf16", "fp16"))
    if op == "norm":
        return {"op": op, "rows": _log(rng, 1, 16384), "dim": _log(rng, 256, 16384, 8), "dtype": dtype}
    if op in ("unreorder_norm", "relayout"):
        bm, bn = rng.choice((16, 32, 64, 128)), rng.choice((128, 256))
        case = {"op": op, "rows": _log(rng, bm, 16384, bm), "dim": _log(rng, bn, 8192, bn), "bm": bm, "bn": bn,
                "dtype": dtype}
        if op == "relayout":
            tiles = (case["rows"] // bm) * (case["dim"] // bn)
            case["rldn"] = rng.choice((1, 2)) if tiles % 2 == 0 else 1
        return case
    if op in ("linear", "add_norm"):
        m, n = _log(rng, 128, 16384, 128), _log(rng, 1024, 8192, 128)
        k = _log(rng, 64, min(28672, 8192 * 8192 * 28672 // (m * n)), 8)
        case = {"op": op, "m": m, "n": n, "k": k, "algo": rng.choice(LINEAR_ALGOS), "dtype": dtype}
        if op == "linear":
            comm = rng.choice(("all_reduce", "reduce_scatter"))
            how = rng.choice(("natural", "reordered"))
            case.update({"comm": comm, "layout": how, "norm": how == "reordered" and comm == "reduce_scatter"})
        return case
    if op == "emulated":
        ranks = rng.choice((2, 4, 8))
        comm = rng.choice(("all_reduce", "reduce_scatter", "all_reduce", "reduce_scatter", "all_to_all"))
        a2a = comm == "all_to_all"
        return {"op": op, "comm": comm, "ranks": ranks, "m": _log(rng, 256, 4096, 128), "n": _log(rng, 512, 8192, 256),
                "k": _log(rng, 128, 4096, 8), "algo": rng.choice(EMULATED_ALGOS), "pull": not a2a and rng.random() < 0.5,
                "strided": rng.random() < 0.5, "natural": a2a or rng.random() < 0.5, "dtype": dtype}
    hidden, ffn, heads, kv_heads = rng.choice(DECODERS)
    batch = rng.choice((1, 2, 4))
    return {"op": op, "hidden": hidden, "ffn": ffn, "heads": heads, "kv_heads": kv_heads, "batch": batch,
            "seq": _log(rng, 128, 8192 // batch, 128 // batch)}


def _randn(seed, *shapes, dtype, scale=1.0):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    return [torch.randn(*s, device=DEVICE, generator=g).mul_(scale).to(dtype) for s in shapes]


def _tiling(case):
    return config.default_solution(case["m"], case["n"], case["algo"])


def prepare(case, seed):
    op = case["op"]
    dt = DTYPES[case.get("dtype", "bf16")]
    torch.manual_seed(seed)                      # the modules draw their weights from torch's own generator
    s = {"op": op, "case": case}
    if op == "norm":
        s["x"], = _randn(seed, (case["rows"], case["dim"]), dtype=dt)
        s["norm"] = RMSNorm(case["dim"], dtype=dt, device=DEVICE, fused=True)
    elif op in ("unreorder_norm", "relayout"):
        rows, dim, bm, bn = case["rows"], case["dim"], case["bm"], case["bn"]
        tiles = (rows // bm) * (dim // bn)
        s["x"], = _randn(seed, (rows, dim), dtype=dt)
        hint = layout.raster_order(rows // bm, dim // bn, 8)         # the order a column-strip GEMM finishes tiles in
        if op == "unreorder_norm":
            s["norm"] = ReorderRMSNorm(dim, rows, bm, bn, hint, eps=1e-5, dtype=dt, device=DEVICE)
        else:
            s["ra"] = layout.reorder_indices(tiles, hint, device=DEVICE)
    elif op == "linear":
        m, n, k, cfg = case["m"], case["n"], case["k"], _tiling(case)
        s["x"], = _randn(seed, (m, k), dtype=dt)
        s["layer"] = OverlapRowParallelLayer(0, 1, k, n, m, cfg, case["comm"], [0] * 16, dtype=dt,
                                             layout_mode=case["layout"])
        if case["norm"]:
            s["norm"] = ReorderRMSNorm(n, m, cfg["BM"], cfg["BN"], cfg["hint"], eps=1e-5, dtype=dt, device=DEVICE)
    elif op == "add_norm":
        m, n, k = case["m"], case["n"], case["k"]
        s["a"], s["x"] = _randn(seed, (m, k), (m, n), dtype=dt)
        s["b"], = _randn(seed + 7919, (n, k), dtype=dt, scale=0.02)
        s["w"] = RMSNorm(n, dtype=dt, device=DEVICE).weight.detach()
        s["algo"] = _tiling(case)["Algo"]
        s["impl"] = ops.OverlapImpl()
        s["impl"].nccl_init(0, 1, [0] * 16)
        s["impl"].cutlass_init()
    elif op == "emulated":
        m, n, k, ranks = case["m"], case["n"], case["k"], case["ranks"]
        s["a"] = _randn(seed, *[(m, k)] * ranks, dtype=dt)
        s["b"] = _randn(seed + 7919, *[(n, k)] * ranks, dtype=dt, scale=0.02)
        cfg = _tiling(case)
        s["algo"], s["mlen"], s["ra"] = cfg["Algo"], None, None
        rows = [m if case["comm"] == "all_reduce" else m // ranks] * ranks
        if case["comm"] == "all_to_all":         # uneven runs: each rank sends at most its m rows in total
            g = torch.Generator().manual_seed(m + n)          # part of the shape: the same for every seed
            s["mlen"] = torch.randint(m // (2 * ranks), m // (ranks - 1) + 1, (ranks, ranks), generator=g, dtype=torch.int32)
            own = torch.eye(ranks, dtype=torch.bool)
            rows = s["mlen"].masked_fill(own, 0).sum(0).tolist()
        elif not case["natural"]:
            s["ra"] = layout.reorder_indices((m // cfg["BM"]) * (n // cfg["BN"]), cfg["hint"], device=DEVICE)
        s["out"] = [torch.zeros(r, n, device=DEVICE, dtype=dt) for r in rows]
    else:
        cfg = DecoderConfig(hidden=case["hidden"], ffn=case["ffn"], n_heads=case["heads"], n_kv_heads=case["kv_heads"])
        s["layer"] = TPDecoderLayer(cfg, 0, 1, case["batch"], case["seq"], impl="fused", dtype=dt, device=DEVICE,
                                    algo=1, seed=seed)
        s["x"], = _randn(seed, (case["batch"] * case["seq"], case["hidden"]), dtype=dt)
    return s


@torch.no_grad()
def run(s):
    op, case = s["op"], s["case"]
    if op in ("norm", "unreorder_norm"):
        return s["norm"](s["x"])
    if op == "relayout":
        bm, bn, rldn = case["bm"], case["bn"], case["rldn"]
        tiled = ops.reorder(s["x"], bm, bn, s["ra"], rldn)
        return tiled, ops.unreorder(tiled, case["rows"], case["dim"], bm, bn, s["ra"], rldn)
    if op == "linear":
        y = s["layer"](s["x"])
        return s["norm"](y) if case["norm"] else y
    if op == "add_norm":
        h = s["x"].clone()                       # the block's input stays: the layer keeps it as its residual
        y = torch.empty_like(h)
        s["impl"].gemm_reducescatter_add_rmsnorm_fused(s["a"], s["b"], h, y, s["w"], 1e-5, s["algo"])
        return h, y
    if op == "emulated":
        status = ops.fused_loopback(case["comm"], s["a"], s["b"], s["out"], RA=s["ra"], algo=s["algo"],
                                    strided_rows=case["strided"], natural_out=case["natural"],
                                    stage_local=case["pull"], mlen=s["mlen"])
        return s["out"], [w[0] for w in status]
    return s["layer"](s["x"])


def work(case):
    op = case["op"]
    if op == "norm":
        e = case["rows"] * case["dim"]
        return {"bytes": 4 * e + 2 * case["dim"], "flops": 4 * e}
    if op == "unreorder_norm":
        e = case["rows"] * case["dim"]
        return {"bytes": 4 * e + 2 * case["dim"], "flops": 4 * e}
    if op == "relayout":
        return {"bytes": 8 * case["rows"] * case["dim"], "flops": 0}
    if op in ("linear", "add_norm"):
        m, n, k = case["m"], case["n"], case["k"]
        out = 3 * m * n if op == "add_norm" else m * n      # residual in, residual and norm out
        return {"bytes": 2 * (m * k + n * k + out), "flops": 2 * m * n * k}
    if op == "emulated":
        m, n, k, ranks = case["m"], case["n"], case["k"], case["ranks"]
        out = ranks * m * n if case["comm"] != "reduce_scatter" else m * n
        return {"bytes": 2 * (ranks * (m + n) * k + out), "flops": 2 * ranks * m * n * k}
    h, f, hd, t = case["hidden"], case["ffn"], 128, case["batch"] * case["seq"]
    qkv = (case["heads"] + 2 * case["kv_heads"]) * hd
    weights = h * (qkv + case["heads"] * hd + 3 * f)
    attention = 2 * case["batch"] * case["heads"] * hd * case["seq"] * case["seq"]      # causal: half of 4 S^2 d
    return {"bytes": 2 * (weights + 2 * t * h), "flops": 2 * t * weights + attention}


def tolerance(case):
    op, fp16 = case["op"], case.get("dtype") == "fp16"
    if op == "relayout":
        return "exact"
    return {"rel": REL[op][1 if fp16 else 0]}


# Relative error that rounding to the data type allows: (bf16, fp16).  Measured against the same computation
# in 64 bits: 1.5e-3 (bf16) and 1.7e-4 (fp16) for a projection alone, up to 3.1e-3 and 4.2e-4 with a norm
# behind it or with partial sums in 16 bits, 8.8e-3 for the decoder layer; about four times that, and the
# decoder's kept at 2e-2.
REL = {
    "norm": (1e-2, 1.2e-3),
    "unreorder_norm": (1e-2, 1.2e-3),
    "linear": (1e-2, 1.2e-3),
    "add_norm": (1e-2, 1.2e-3),
    "emulated": (1e-2, 1.2e-3),
    "decoder": (2e-2, 2e-2),
}
