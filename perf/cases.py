"""What this library is used for, as measurable cases.

Each case goes through the public entry points (`GpuKernels`, `LlamaU8`, `ClipVisionU`) with the
shapes of the repository's own workloads: the LLaMA-7B/65B and CLIP ViT-L/14 shapes, their
projections one by one, and the call patterns of a caller that uses the kernels directly.
`listed()` names the representative ones, `draw()` gives others of the same ranges.

Kinds of case:

  u8_linear     one u8-weight linear layer, `matmul_nt_fp16u8`: decode (a few tokens) and prefill
  f16_gemm      one fp16 product, `matmul_f16`, weights [K, N] ("rrr") or [N, K] passed permuted ("rrc")
  attention     the three calls of an attention layer on contiguous scores: matmul_f16(Scale, mask),
                softmax_rows_inplace, matmul_f16
  quantize      weight loading: `quantize_absmax_uint8`, then `dequantize_absmax_uint8`
  llama_decode  one captured decode step of the LLaMA-shape decoder with its key/value cache
  llama_prefill a prompt through the same decoder
  clip          the CLIP image encoder on a batch of images
"""
from __future__ import annotations

import functools
import math

import torch

from adrastea_b200 import GpuKernels, MatmulMask, MatmulOptions, MatmulStore, TensorLayout, TensorView
from adrastea_b200.clip import VIT_L_14, ClipVisionU
from adrastea_b200.llama import LLAMA_7B, LLAMA_65B, LlamaU8

SHAPES = {"7b": LLAMA_7B, "65b": LLAMA_65B}
# (n, k) of the projections of the two shapes: q/k/v/o, fused qkv, gate or up, fused gate/up, down,
# output head
PROJECTIONS_7B = [(4096, 4096), (12288, 4096), (11008, 4096), (22016, 4096), (4096, 11008), (32000, 4096)]
PROJECTIONS_65B = [(8192, 8192), (22016, 8192), (8192, 22016)]


def listed():
    return [
        # one projection for one token: the smallest call of the decode path
        dict(name="u8_1x4096x4096", kind="u8_linear", m=1, n=4096, k=4096, block=128, zeros=False),
        # the gate projection for a batch of 16 tokens, with stored zero points
        dict(name="u8_16x11008x4096_zeros", kind="u8_linear", m=16, n=11008, k=4096, block=128, zeros=True),
        # the down projection over a prompt of a length that is no multiple of a tile
        dict(name="u8_300x4096x11008", kind="u8_linear", m=300, n=4096, k=11008, block=128, zeros=False),
        # a few rows against a row-major weight
        dict(name="f16_64x4096x4096_rrr", kind="f16_gemm", m=64, n=4096, k=4096, layout="rrr", store="identity"),
        # a prompt against a weight stored [N, K]
        dict(name="f16_2048x4096x4096_rrc", kind="f16_gemm", m=2048, n=4096, k=4096, layout="rrc", store="identity"),
        # attention of one image (257 tokens, scores rows of 514 bytes) by separate calls
        dict(name="attention_16x257x64", kind="attention", heads=16, tokens=257, head_dim=64, causal=False),
        # loading one matrix of weights
        dict(name="quantize_11008x4096", kind="quantize", rows=11008, k=4096, block=128),
        # a token for one user, and for sixteen, in the middle of a conversation
        dict(name="llama7b_decode_b1", kind="llama_decode", shape="7b", layers=32, batch=1, context=575),
        dict(name="llama7b_decode_b16", kind="llama_decode", shape="7b", layers=32, batch=16, context=575),
        # a prompt of one user, and of sixteen at once
        dict(name="llama7b_prefill_1x512", kind="llama_prefill", shape="7b", layers=32, batch=1, tokens=512),
        dict(name="llama7b_prefill_16x512", kind="llama_prefill", shape="7b", layers=32, batch=16, tokens=512),
        # a batch of images
        dict(name="clip_b64", kind="clip", batch=64),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], evenly spread over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["u8_linear", "u8_linear", "f16_gemm", "attention", "quantize", "llama_decode",
                       "llama_decode", "llama_prefill", "clip"])
    if kind == "u8_linear":
        block = rng.choice([128, 128, 64, 32])
        m = _log(rng, 1, 2048)
        if rng.random() < 0.7:
            n, k = rng.choice(PROJECTIONS_65B if block == 64 else PROJECTIONS_7B)
        else:  # any other layer: rows of any number, whole scale groups
            n, k = _log(rng, 512, 16384), block * _log(rng, 1024 // block, 12288 // block)
        return dict(kind=kind, m=m, n=n, k=k, block=block, zeros=rng.random() < 0.25)
    if kind == "f16_gemm":
        return dict(kind=kind, m=_log(rng, 1, 8192), n=_log(rng, 256, 8192),
                    k=8 * _log(rng, 32, 1024) - (rng.randrange(1, 8) if rng.random() < 0.1 else 0),
                    layout=rng.choice(["rrr", "rrc", "rrc"]),
                    store=rng.choice(["identity", "scale", "bias", "quick_gelu"]))
    if kind == "attention":
        return dict(kind=kind, heads=rng.choice([4, 12, 16, 32]), tokens=_log(rng, 16, 1024),
                    head_dim=rng.choice([64, 128]), causal=rng.random() < 0.5)
    if kind == "quantize":
        block = rng.choice([128, 64, 32])
        return dict(kind=kind, rows=_log(rng, 256, 32000), k=block * _log(rng, 512 // block, 22016 // block),
                    block=block)
    if kind == "llama_decode":
        batch = _log(rng, 1, 16)
        context = _log(rng, 16, min(2040, 16 * 640 // batch))
        shape = rng.choice(["7b", "7b", "65b"])
        return dict(kind=kind, shape=shape, layers=rng.randint(1, 32 if shape == "7b" else 8), batch=batch,
                    context=context)
    if kind == "llama_prefill":
        batch = _log(rng, 1, 16)
        shape = rng.choice(["7b", "7b", "65b"])
        return dict(kind=kind, shape=shape, layers=rng.randint(1, 16 if shape == "7b" else 4), batch=batch,
                    tokens=_log(rng, 16, min(2048, 8192 // batch)))
    return dict(kind=kind, batch=_log(rng, 1, 64))


@functools.lru_cache(maxsize=None)
def _kernels() -> GpuKernels:
    """The library's handle, opened once, with early launch on as the decoder's own program sets it."""
    k = GpuKernels()
    k.set_tunable("pdl", 1)
    return k


def _llama(case, seed, max_seq):
    """The decoder with its seeded weights, scaled to a standard deviation of about 0.02 (seeded as
    they are, with 0.4, the residual stream would overflow fp16 within a few layers)."""
    model = LlamaU8(_kernels(), SHAPES[case["shape"]], max_batch=case["batch"], max_seq=max_seq,
                    n_layers=case["layers"], seed=seed)
    for ly in model.layers:
        for lin in (ly.wqkv, ly.wo, ly.wgu, ly.down):
            lin.w.scales.mul_(0.05)
    model.lm_head.scales.mul_(0.05)
    return model


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    half = dict(dtype=torch.float16, device="cuda")

    def normal(*shape, std=1.0):
        return torch.empty(shape, **half).normal_(0.0, std, generator=g)

    def uniform(*shape, lo, hi):
        return torch.empty(shape, **half).uniform_(lo, hi, generator=g)

    kind = case["kind"]
    s = dict(case=case, kernels=_kernels())
    if kind == "u8_linear":
        m, n, k, groups = case["m"], case["n"], case["k"], case["k"] // case["block"]
        s["x"] = normal(m, k)
        s["q"] = torch.randint(0, 256, (n, k), dtype=torch.uint8, device="cuda", generator=g)
        s["scales"] = uniform(n, groups, lo=0.001, hi=0.01)
        s["zeros"] = uniform(n, groups, lo=120.0, hi=136.0) if case["zeros"] else None
        s["out"] = torch.zeros((m, n), **half)
    elif kind == "f16_gemm":
        m, n, k = case["m"], case["n"], case["k"]
        s["x"] = TensorView.of(normal(m, k, std=0.02))
        s["w"] = (TensorView.of(normal(k, n, std=0.02)) if case["layout"] == "rrr"
                  else TensorView.of(normal(n, k, std=0.02)).permute([1, 0]))
        s["out"] = torch.zeros((m, n), **half)
        bias = TensorView.of(normal(n, std=0.02))
        store = {"identity": MatmulStore.Identity(), "scale": MatmulStore.Scale(0.125),
                 "bias": MatmulStore.BetaBias(0.0, bias), "quick_gelu": MatmulStore.QuickGeluBias(bias)}
        s["options"] = MatmulOptions.new().store(store[case["store"]])
    elif kind == "attention":
        h, t, d = case["heads"], case["tokens"], case["head_dim"]
        heads = TensorLayout.new((t, h, d), (h * d, d, 1))
        s["q"], s["k"], s["v"] = (TensorView(normal(t, h * d), heads) for _ in range(3))
        s["scores"], s["out"] = torch.zeros((h, t, t), **half), torch.zeros((t, h * d), **half)
        s["out_view"] = TensorView(s["out"], heads)
    elif kind == "quantize":
        rows, k = case["rows"], case["k"]
        s["w"] = normal(rows, k, std=0.02)
        s["q"] = torch.zeros((rows, k), dtype=torch.uint8, device="cuda")
        s["scales"] = torch.zeros((rows, k // case["block"]), **half)
        s["back"] = torch.zeros((rows, k), **half)
    elif kind == "llama_decode":
        model = s["model"] = _llama(case, seed, case["context"] + 64)
        model.k_cache.normal_(0.0, 1.3, generator=g)
        model.v_cache.normal_(0.0, 1.3, generator=g)
        s["tokens"] = torch.randint(0, model.shape.vocab, (case["batch"],), device="cuda", generator=g)
        s["pos"] = torch.full((1,), case["context"], dtype=torch.int32, device="cuda")
        model.pos.copy_(s["pos"])
        model.capture()
    elif kind == "llama_prefill":
        model = s["model"] = _llama(case, seed, case["tokens"])
        s["tokens"] = torch.randint(0, model.shape.vocab, (case["batch"], case["tokens"]), device="cuda",
                                    generator=g)
    else:
        s["model"] = ClipVisionU(_kernels(), VIT_L_14, case["batch"], seed=seed)
        s["pixels"] = normal(case["batch"], 3, VIT_L_14.image, VIT_L_14.image)
    return s


def run(s):
    case, k = s["case"], s["kernels"]
    kind = case["kind"]
    if kind == "u8_linear":
        k.matmul_nt_fp16u8(s["out"], s["x"], s["q"], s["scales"], case["block"], zeros=s["zeros"])
        return s["out"]
    if kind == "f16_gemm":
        k.matmul_f16(TensorView.of(s["out"]), s["x"], s["w"], s["options"])
        return s["out"]
    if kind == "attention":
        scores = TensorView.of(s["scores"])
        mask = MatmulMask.Causal if case["causal"] else MatmulMask.None_
        k.matmul_f16(scores, s["q"].permute([1, 0, 2]), s["k"].permute([1, 2, 0]),
                     MatmulOptions.new().store(MatmulStore.Scale(1.0 / math.sqrt(case["head_dim"]))).mask(mask))
        k.softmax_rows_inplace(scores)
        k.matmul_f16(s["out_view"].permute([1, 0, 2]), scores, s["v"].permute([1, 0, 2]))
        return s["scores"], s["out"]
    if kind == "quantize":
        k.quantize_absmax_uint8(s["q"], s["scales"], s["w"])
        k.dequantize_absmax_uint8(s["back"], s["scales"], s["q"])
        return s["q"], s["scales"], s["back"]
    if kind == "llama_decode":
        model = s["model"]
        model.tokens.copy_(s["tokens"])
        model.pos.copy_(s["pos"])
        model.decode_step()
        return model.logits, model.k_cache, model.v_cache
    if kind == "llama_prefill":
        model = s["model"]
        model.prefill(s["tokens"])
        return model.logits, model.k_cache, model.v_cache
    return s["model"].forward(s["pixels"])


def _u8_bytes(n, k, block, zeros=False):
    return n * k + (4 if zeros else 2) * n * (k // block)


def work(case):
    kind = case["kind"]
    if kind == "u8_linear":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=_u8_bytes(n, k, case["block"], case["zeros"]) + 2 * m * (n + k), flops=2 * m * n * k)
    if kind == "f16_gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=2 * (m * k + n * k + m * n), flops=2 * m * n * k)
    if kind == "attention":
        h, t, d = case["heads"], case["tokens"], case["head_dim"]
        pairs = t * (t + 1) // 2 if case["causal"] else t * t
        # q, k, v read and the output written once; the caller's score tensor is written as well
        return dict(bytes=2 * h * (4 * t * d + t * t), flops=4 * h * pairs * d)
    if kind == "quantize":
        rows, k = case["rows"], case["k"]
        return dict(bytes=2 * rows * k + 2 * rows * k + _u8_bytes(rows, k, case["block"]), flops=4 * rows * k)
    if kind == "clip":
        sh, b = VIT_L_14, case["batch"]
        t, d, f = sh.tokens, sh.hidden, sh.mlp
        linears = sh.layers * (4 * d * d + 2 * d * f)
        flops = 2 * b * t * linears + sh.layers * 4 * b * t * t * d + 2 * b * (t - 1) * d * 3 * sh.patch ** 2
        return dict(bytes=2 * linears + 2 * b * (3 * sh.image ** 2 + t * d), flops=flops)
    sh, b, layers = SHAPES[case["shape"]], case["batch"], case["layers"]
    d, f = sh.dim, sh.ffn
    weights = layers * (_u8_bytes(3 * d, d, sh.block) + _u8_bytes(d, d, sh.block)
                        + _u8_bytes(2 * f, d, sh.block) + _u8_bytes(d, f, sh.block))
    head = _u8_bytes(sh.vocab, d, sh.block)
    linears = layers * (4 * d * d + 3 * d * f)
    if kind == "llama_decode":
        t = case["context"] + 1
        cache = layers * b * 2 * (2 * t * d)
        return dict(bytes=weights + head + cache + 2 * b * (d + sh.vocab),
                    flops=2 * b * (linears + sh.vocab * d) + layers * b * 4 * t * d)
    t = case["tokens"]
    return dict(bytes=weights + head + layers * b * 2 * (2 * t * d) + 2 * b * (t * d + sh.vocab),
                flops=2 * b * t * linears + 2 * b * sh.vocab * d + layers * b * 2 * t * (t + 1) * d)


def tolerance(case):
    """About four times the distance from the same computation in 64 bits without intermediate
    rounding, measured on the listed cases and a few others of each kind: a single product 2.1e-4
    to 3.0e-4 (the rounding of its fp16 output, and for u8 prefill of the fp16 weights), attention
    5.6e-4, the image encoder 1.6e-3, a decode step of 32 layers 5.8e-3 and a prompt through 32
    layers 9.8e-3 (fp16 residual stream and activations)."""
    return {"u8_linear": {"rel": 1.2e-3, "max": 6e-3},
            "f16_gemm": {"rel": 1e-3, "max": 4e-3},
            "attention": {"rel": 2.3e-3, "max": 5e-2},
            "quantize": "exact",
            "llama_decode": {"rel": 2.3e-2, "max": 0.12},
            "llama_prefill": {"rel": 3e-2, "max": 0.24},
            "clip": {"rel": 6e-3, "max": 3.5e-2}}[case["kind"]]
