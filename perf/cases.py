"""Workloads of this library on one GPU, driven through its public entry points.

``listed()`` names the workloads, ``draw(rng)`` gives one more from the ranges they stand for, ``prepare`` builds what
a program holds before the call (inputs, weights, op objects), ``run`` makes one pass and returns everything it
computes, ``work`` counts the bytes and operations a pass cannot do without and ``tolerance`` says how far two
correct implementations of the same precision may be apart.

A process group of one rank stands for the tensor / sequence / expert parallel group: the fused ops then run their
GEMM, epilogue, gather and combine without peers.
"""
import math

import torch
import torch.distributed as dist

import tempname_new_b200 as flux
from tempname_new_b200.models.tp_mlp import TPMLP

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "e4m3": torch.float8_e4m3fn,
          "e5m2": torch.float8_e5m2, "int8": torch.int8}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4, "e4m3": 1, "e5m2": 1, "int8": 1}
DEVICE = "cuda"
MAX_FLOPS = 1.6e12     # bounds of a drawn case; the largest listed ones do 2.5e12
MAX_BYTES = 2.0e9


def listed():
    return [
        # Token generation through a tensor-parallel MLP block (the dimensions of the block's example script): a
        # handful of tokens against all the weights, the smallest calls of a serving loop.
        dict(name="mlp_decode", kind="mlp", tokens=16, hidden=4096, ffn=16384, dtype="bf16", train=False),
        # Prompt processing: one rank's share (ffn / 8) of the headline benchmark's block, all 8192 tokens.
        dict(name="mlp_prefill", kind="mlp", tokens=8192, hidden=12288, ffn=6144, dtype="bf16", train=False),
        # One training step of the example's block: forward, both data gradients, weight and bias gradients.
        dict(name="mlp_train", kind="mlp", tokens=4096, hidden=4096, ffn=16384, dtype="bf16", train=True),
        # A stand-alone fp16 linear with a bias whose sizes fit no tile (variable-length batch, odd vocabulary cut).
        dict(name="linear_fp16_ragged", kind="linear", m=1000, n=3000, k=5000, dtype="fp16", bias=True, kn=False),
        # Per-tensor scaled fp8 linear over a chunk of a prompt.
        dict(name="linear_fp8", kind="linear", m=2048, n=12288, k=4096, dtype="e4m3", bias=False, kn=False),
        # Weight-and-activation int8 linear (one scale per token, one per output channel) while generating.
        dict(name="linear_int8_decode", kind="linear", m=64, n=12288, k=4096, dtype="int8", bias=False, kn=False),
        # Block-scaled fp8 training of one linear layer (the benchmarked shape, N 3584 per rank): the quantisation of
        # activations, weights and output gradients in both orientations, forward, data and weight gradient.
        dict(name="fp8_block_train", kind="fp8_block", m=8192, n=3584, k=8192, train=True),
        # The same layer while generating: the activations of a few sequences are quantised and multiplied.
        dict(name="fp8_block_decode", kind="fp8_block", m=48, n=3584, k=8192, train=False),
        # A mixture-of-experts layer (routing indices, layer 0, SwiGLU, layer 1 with the weighted combine) for a small
        # generation batch: eight rows per expert on average, every expert's weights are read.
        dict(name="moe_decode", kind="moe", tokens=64, hidden=4096, ffn=1536, experts=64, topk=8, dtype="bf16"),
        # The same layer over the 8192 tokens of a prompt or of one rank's training batch.
        dict(name="moe_prefill", kind="moe", tokens=8192, hidden=4096, ffn=1536, experts=64, topk=8, dtype="bf16"),
        # Attention projections of sequence-parallel attention: packed QKV into the head-sharded layout, and the
        # attention output back through the output projection (4096 positions, 32 heads of 128).
        dict(name="ulysses_attention", kind="ulysses", bs=1, seq=4096, heads=32, head_dim=128, dtype="bf16"),
        # Quantisation of a batch whose row count is no multiple of the block, both orientations.
        dict(name="quantize_ragged", kind="quantize", m=5000, k=8192, dtype="bf16", square=False, transpose=True),
    ]


# ------------------------------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi, step=1):
    """Log-uniform between lo and hi, a multiple of step."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, min(int(round(v / step)) * step, hi // step * step))


def draw(rng):
    while True:
        c = _draw_one(rng)
        w = work(c)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= MAX_BYTES:
            return c


def _draw_one(rng):
    kind = rng.choice(["mlp", "mlp", "linear", "linear", "fp8_block", "moe", "moe", "ulysses", "quantize"])
    if kind == "mlp":
        train = rng.random() < 0.3
        # (hidden and ffn of real blocks are multiples of 64; token counts are anything)
        return dict(kind=kind, tokens=_log(rng, 64 if train else 1, 8192), hidden=_log(rng, 1024, 12288, 64),
                    ffn=_log(rng, 1024, 16384, 64), dtype=rng.choice(["bf16", "bf16", "fp16"]), train=train)
    if kind == "linear":
        dtype = rng.choice(["bf16", "fp16", "e4m3", "e5m2", "int8"])
        step = 8 if SIZE[dtype] == 2 else 16
        return dict(kind=kind, m=_log(rng, 1, 8192), n=_log(rng, 256, 16384, 8), k=_log(rng, 256, 16384, step),
                    dtype=dtype, bias=rng.random() < 0.5, kn=SIZE[dtype] == 2 and rng.random() < 0.3)
    if kind == "fp8_block":
        train = rng.random() < 0.4
        m = _log(rng, 512, 8192, 128) if train else _log(rng, 1, 8192)
        return dict(kind=kind, m=m, n=_log(rng, 512, 8192, 128), k=_log(rng, 512, 8192, 128), train=train)
    if kind == "moe":
        experts = rng.choice([8, 16, 32, 64, 128])
        return dict(kind=kind, tokens=_log(rng, 1, 8192), hidden=_log(rng, 1024, 6144, 128),
                    ffn=_log(rng, 512, 3072, 64), experts=experts, topk=rng.choice([1, 2, 4, 6, 8]),
                    dtype=rng.choice(["bf16", "bf16", "fp16", "e4m3"]))
    if kind == "ulysses":
        bs = rng.choice([1, 1, 2])
        return dict(kind=kind, bs=bs, seq=_log(rng, 128, 16384 // bs, 32), heads=rng.choice([8, 16, 24, 32, 40, 64]),
                    head_dim=rng.choice([64, 128]), dtype=rng.choice(["bf16", "fp16"]))
    return dict(kind="quantize", m=_log(rng, 16, 16384), k=_log(rng, 256, 16384, 8),
                dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]), square=rng.random() < 0.4,
                transpose=rng.random() < 0.6)


# ------------------------------------------------------------------------------------------ inputs
def _group():
    if not dist.is_initialized():
        dev = torch.device(DEVICE, torch.cuda.current_device())
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=dev)
    return dist.group.WORLD


class _Inputs:
    """Normal values from one seed, made on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, dtype=torch.bfloat16, std=1.0):
        # (8-bit and odd types are cast from 16-bit values)
        made = dtype if dtype in (torch.bfloat16, torch.float16, torch.float32) else torch.bfloat16
        t = torch.empty(shape, device=DEVICE, dtype=made).normal_(0.0, std, generator=self.g)
        return t if made == dtype else t.to(dtype)

    def int8(self, *shape):
        # what symmetric quantisation of normal values gives: the largest of a row near 127
        t = torch.empty(shape, device=DEVICE, dtype=torch.float16).normal_(0.0, 127.0 / 4, generator=self.g)
        return t.round_().clamp_(-127, 127).to(torch.int8)

    def scale(self, *shape, about=0.01):
        return torch.empty(shape, device=DEVICE).uniform_(0.5 * about, 1.5 * about, generator=self.g)


def prepare(case, seed):
    r = _Inputs(seed)
    s = {"case": case}
    kind = case["kind"]
    dt = DTYPES.get(case.get("dtype", "bf16"))
    if kind == "mlp":
        mlp = TPMLP(case["hidden"], case["ffn"], _group(), dtype=dt, device=DEVICE)
        with torch.no_grad():
            for p in mlp.parameters():
                p.normal_(0.0, 0.02, generator=r.g)
        s["x"] = r.normal(case["tokens"], case["hidden"], dtype=dt)
        if case["train"]:
            s["x"].requires_grad_(True)
            s["dy"] = r.normal(case["tokens"], case["hidden"], dtype=dt)
            s["params"] = list(mlp.parameters())
        else:
            mlp.requires_grad_(False)
        s["mlp"] = mlp
    elif kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        if dt == torch.int8:
            s["x"], s["w"] = r.int8(m, k), r.int8(n, k)
            s["sx"], s["sw"] = r.scale(m, 1), r.scale(1, n)
            out = torch.bfloat16
        elif SIZE[case["dtype"]] == 1:
            s["x"], s["w"] = r.normal(m, k, dtype=dt), r.normal(n, k, dtype=dt)
            s["sx"], s["sw"] = r.scale(1), r.scale(1)
            out = torch.bfloat16
        else:
            s["x"] = r.normal(m, k, dtype=dt)
            s["w"] = r.normal(*((k, n) if case["kn"] else (n, k)), dtype=dt, std=0.02)
            s["sx"] = s["sw"] = None
            out = dt
        s["bias"] = r.normal(1, n, dtype=out) if case["bias"] else None
        s["op"] = flux.GemmOnly(dt, output_dtype=out, transpose_weight=case["kn"], use_fp8_gemm=dt == DTYPES["e4m3"])
    elif kind == "fp8_block":
        m, n, k = case["m"], case["n"], case["k"]
        s["quant"] = flux.Quantization(torch.bfloat16, torch.float8_e4m3fn)
        s["gemm"] = flux.BlockScaleGemm(torch.float8_e4m3fn, torch.float8_e4m3fn, torch.bfloat16)
        s["x"] = r.normal(m, k)
        s["w"] = r.normal(n, k, std=0.02)
        if case["train"]:
            s["dy"] = r.normal(m, n, std=0.1)
        else:      # weights are quantised once, when they are loaded
            s["wq"], s["sw"], _, _ = s["quant"].quantize_square_blockwise(s.pop("w"), False)
    elif kind == "moe":
        t, h, f, e, topk = (case[n] for n in ("tokens", "hidden", "ffn", "experts", "topk"))
        topk = min(topk, e)
        pg = _group()
        out = torch.bfloat16 if dt == torch.float8_e4m3fn else dt
        logits = r.normal(t, e, dtype=torch.float32)
        gate, chosen = torch.softmax(logits, dim=1).topk(topk, dim=1)
        s["chosen"] = chosen.to(torch.int32).contiguous()
        s["gate"] = (gate / gate.sum(1, keepdim=True)).contiguous()
        s["x"] = r.normal(t, h, dtype=dt)
        fp8 = dt == torch.float8_e4m3fn
        s["w_gate"] = r.normal(e, f, h, dtype=dt, std=1.0 if fp8 else 0.02)
        s["w_up"] = r.normal(e, f, h, dtype=dt, std=1.0 if fp8 else 0.02)
        s["w_down"] = r.normal(e, h, f, dtype=dt, std=1.0 if fp8 else 0.02)
        s["s_in"] = [r.scale(e, about=0.02), r.scale(e, about=0.02)] if fp8 else None
        s["s_down"] = r.scale(e, about=0.02) if fp8 else None
        s["h"] = [torch.empty(t * topk, f, device=DEVICE, dtype=out) for _ in range(2)]
        env = flux.DistEnvTPWithEP(pg, 1, None, ep_size=1)
        s["layer0"] = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(t, h, f, e, topk, dt, out))
        s["layer1"] = flux.GemmGroupedV3GatherRS(e, t * topk, h, topk, 0, 1, 1, 1, tp_group=pg, dtype=out)
    elif kind == "ulysses":
        bs, seq, nh, hd = case["bs"], case["seq"], case["heads"], case["head_dim"]
        hidden = nh * hd
        pg = _group()
        s["pre"] = flux.GemmAllToAllTranspose(pg, 1, 1, bs, seq, hidden, hd, 3 * hidden, dt, gqa=1,
                                              comm_op=flux.PreAttnAllToAllCommOp.QKVPackA2A)
        s["post"] = flux.AllToAllTransposeGemm(pg, 1, 1, bs, nh, seq, hd, dt, a2a_only=True)
        s["x"] = r.normal(bs, seq, hidden, dtype=dt)
        s["o"] = r.normal(bs, seq, nh, hd, dtype=dt)
        s["w_qkv"] = r.normal(3 * hidden, hidden, dtype=dt, std=0.02)
        s["w_o"] = r.normal(hidden, hidden, dtype=dt, std=0.02)
    else:
        s["x"] = r.normal(case["m"], case["k"], dtype=dt)
        s["quant"] = flux.Quantization(dt, torch.float8_e4m3fn)
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mlp":
        if not case["train"]:
            with torch.no_grad():
                return s["mlp"](s["x"])
        y = s["mlp"](s["x"])
        grads = torch.autograd.grad(y, [s["x"]] + s["params"], s["dy"])
        return [y.detach(), *grads]
    if kind == "linear":
        return s["op"].forward(s["x"], s["w"], bias=s["bias"], input_scale=s["sx"], weight_scale=s["sw"])
    if kind == "fp8_block":
        q, gemm = s["quant"], s["gemm"]
        xq, sx, xqt, sxt = q.quantize_vector_blockwise(s["x"], case["train"])
        if not case["train"]:
            return gemm.forward(xq, s["wq"], input_scale=sx, weight_scale=s["sw"])
        wq, sw, wqt, swt = q.quantize_square_blockwise(s["w"], True)
        y = gemm.forward(xq, wq, input_scale=sx, weight_scale=sw)
        dyq, sdy, dyqt, sdyt = q.quantize_vector_blockwise(s["dy"], True)
        dx = gemm.forward(dyq, wqt, input_scale=sdy, weight_scale=swt)
        dw = gemm.wgrad(dyqt, xqt, input_scale=sdyt, weight_scale=sxt)
        return [y, dx, dw]
    if kind == "moe":
        splits, _, scatter, gather, tki = flux.moe_index_build(s["chosen"], case["experts"])
        g, u = s["layer0"].forward_multiple_weights(s["x"], [s["w_gate"], s["w_up"]], splits, scatter,
                                                    output_scale=s["s_in"], outputs_buf=s["h"])
        act = torch.nn.functional.silu(g).mul_(u)
        if s["x"].dtype != act.dtype:
            act = act.to(s["x"].dtype)
        row_gate = s["gate"][gather, tki]
        y = s["layer1"].forward_gather_rs(act, s["w_down"], splits, scatter.reshape(-1), weight_scale=s["s_down"],
                                          output_vec_scale=row_gate)
        return [splits, scatter, g, u, y]
    if kind == "ulysses":
        q, k, v = s["pre"].forward(s["x"], s["w_qkv"])
        return [q, k, v, s["post"].forward(s["o"], s["w_o"])]
    op = s["quant"].quantize_square_blockwise if case["square"] else s["quant"].quantize_vector_blockwise
    q, sc, qt, sct = op(s["x"], case["transpose"])
    out = [q.view(torch.uint8), sc]
    return out + [qt.view(torch.uint8), sct] if case["transpose"] else out


# ------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    kind = case["kind"]
    e = SIZE[case.get("dtype", "bf16")]
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        w = 2 * h * f * e
        if not case["train"]:
            return {"bytes": w + 2 * t * h * e, "flops": 4.0 * t * h * f}
        return {"bytes": 2 * w + 4 * t * h * e, "flops": 12.0 * t * h * f}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": (m + n) * k * e + m * n * 2, "flops": 2.0 * m * n * k}
    if kind == "fp8_block":
        m, n, k = case["m"], case["n"], case["k"]
        if not case["train"]:
            return {"bytes": m * k * 2 + n * k + m * n * 2, "flops": 2.0 * m * n * k}
        return {"bytes": 4 * (m * k + n * k + m * n), "flops": 6.0 * m * n * k}
    if kind == "moe":
        t, h, f, x, topk = (case[n] for n in ("tokens", "hidden", "ffn", "experts", "topk"))
        topk = min(topk, x)
        met = x * (1.0 - (1.0 - topk / x) ** t)          # experts that get a row at all
        rows = t * topk
        return {"bytes": met * 3 * h * f * e + t * h * (e + 2) + rows * 2 * f * 2, "flops": 6.0 * rows * h * f}
    if kind == "ulysses":
        t, h = case["bs"] * case["seq"], case["heads"] * case["head_dim"]
        return {"bytes": 4 * h * h * e + 6 * t * h * e, "flops": 8.0 * t * h * h}
    m, k = case["m"], case["k"]
    return {"bytes": m * k * (e + 1 + (1 if case["transpose"] else 0)), "flops": 4.0 * m * k}


def tolerance(case):
    """About four times the 2-norm error of a pass against the same path in 64 bits: one rounding to bf16 shows 1.66e-3,
    one to fp16 2.1e-4; an MLP block rounds its intermediate and its result (2.9e-3, with the unfused activation of
    training 3.4e-3), a MoE layer its intermediate, the activation, the rows of layer 1 and the sum (4.2e-3)."""
    kind = case["kind"]
    if kind == "quantize":
        return "exact"
    dtype = case.get("dtype", "bf16")
    half = dtype == "fp16"
    if kind == "mlp":
        return {"rel": 1.8e-3 if half else 1.4e-2}
    if kind == "moe":
        # (e4m3: an activation next to a rounding boundary falls on the other side when layer 0 differs in its last
        # bit: 1.5e-2)
        return {"rel": {"fp16": 2.1e-3, "bf16": 1.7e-2, "e4m3": 3e-2}[dtype]}
    return {"rel": 8.5e-4 if half else 7e-3}
