"""The calls that stand for what users of this framework run, with their inputs, least work and tolerances.

`listed()` are fixed cases, `draw(rng)` gives more of the same ranges; `prepare` makes what a program has in hand before the
call, `run` is one pass through the public entry points.  Six families ("kind"):

  attention  one attention call on 16-bit Q, K, V: the framework's main use, through each of its entry points
  chunk      queries of one prefill chunk against keys and values that were quantised once and kept
  video      non-causal self-attention over video latent tokens with NVFP4 score tiles
  quant4     the MXFP4 quantizer pair in the reference project's output format
  quant8     the MXFP8 quantizer pair in the reference project's output format
  gemm       the stand-alone block-scaled matrix product of operands quantised beforehand
"""
import math
import os
import sys

import torch

PKG = os.path.abspath("mp-sparse-attn_b200")
if PKG not in sys.path:
    sys.path.insert(1, PKG)

import mpsa  # noqa: E402
from mpsa.model_hooks import MixedPrecisionAttention  # noqa: E402
from ours.block_scaled_matmul import block_scaled_matmul  # noqa: E402
from ours.mxfp_attn import mxfp_attn  # noqa: E402
from ours.mxfp_attn_kernel import mxfp_attn_kernel  # noqa: E402
from ours.quant_mxint8 import quant_mxfp4, quant_mxfp8e5  # noqa: E402

DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _attention(entry, B, Hq, Hkv, S, D, causal, dtype="bf16", layout="HND", mode="", **name):
    return dict(name, kind="attention", entry=entry, B=B, Hq=Hq, Hkv=Hkv, S=S, D=D, causal=causal, dtype=dtype, layout=layout,
                mode=mode)


def listed():
    return [
        # the README's first call at the plumbing configuration: one short causal layer, where launches and host time count
        _attention("diagonal", 1, 8, 8, 1024, 64, True, name="diagonal_1k_d64"),
        # the reference's `mxfp_attn` with its defaults (MXFP4, smooth K, fp16 out) on a short ragged batch, the smallest calls
        _attention("mxfp_attn", 2, 8, 8, 333, 128, False, "fp16", mode="mxfp4", name="mxfp_attn_ragged_333"),
        # causal prefill of one grouped-query layer with the online router, at the two lengths of the benchmark
        _attention("kernel", 1, 32, 8, 8192, 128, True, mode="online_requant", name="prefill_online_8k"),
        _attention("kernel", 1, 32, 8, 32768, 128, True, mode="online_requant", name="prefill_online_32k"),
        # the reference's MXFP8 mode with fp16 P.V, the comparison with its own kernel
        _attention("kernel", 1, 32, 32, 8192, 128, False, "fp16", mode="mxfp8", name="mxfp8_full_8k"),
        # one video block through the model hook: tokens-first layout, smooth K, a token count that fills no tile
        _attention("hook", 1, 12, 12, 7803, 128, False, layout="NHD", mode="diag_requant", name="hook_video_7803"),
        # a prefill chunk against a long kept prefix (keys and values quantised once)
        dict(name="chunk_512_of_32k", kind="chunk", Hq=32, Hkv=8, S=512, Skv=32768, D=128),
        # the video configuration of the benchmark: 21 x 39 x 40 latent tokens, NVFP4 off the diagonal
        dict(name="video_nvfp4_32760", kind="video", H=40, S=32760),
        # the quantizer pairs as the reference's scripts call them: a long layer; and a ragged mid-size one, tokens first
        dict(name="quant_mxfp4_32k", kind="quant4", B=1, Hq=32, Hkv=8, S=32768, D=128, dtype="bf16", layout="HND"),
        dict(name="quant_mxfp8_4500", kind="quant8", B=2, Hq=16, Hkv=16, S=4500, D=64, dtype="fp16", layout="NHD"),
        # the benchmark's square product, and a ragged NVFP4 one of a projection's size
        dict(name="gemm_mxfp8_8192", kind="gemm", mode="mxfp8", M=8192, N=8192, K=8192, out="bf16"),
        dict(name="gemm_nvfp4_1500", kind="gemm", mode="nvfp4", M=1500, N=4096, K=4096, out="bf16"),
    ]


def _size(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    kind = rng.choice(["diagonal", "mxfp_attn", "online", "online", "kernel", "hook", "chunk", "video", "quant4", "quant8", "gemm",
                       "gemm"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "diagonal":
        H = rng.choice([8, 16, 32])
        return _attention(kind, 1, H, H // rng.choice([1, 2, 4]), _size(rng, 128, 16384), rng.choice([64, 128]), True, dtype)
    if kind == "mxfp_attn":
        H = rng.choice([4, 8, 16])
        return _attention(kind, rng.choice([1, 2, 4]), H, H, _size(rng, 64, 4096), rng.choice([64, 128]), False, dtype,
                          mode=rng.choice(["mxfp4", "mxfp8"]))
    if kind == "online":
        return _attention("kernel", 1, 32, 8, _size(rng, 1024, 32768), 128, True, dtype, mode="online_requant")
    if kind == "kernel":
        H = rng.choice([16, 32])
        return _attention(kind, 1, H, H, _size(rng, 1024, 16384), 128, False, dtype, mode=rng.choice(["mxfp4", "mxfp8"]))
    if kind == "hook":
        return _attention(kind, 1, rng.choice([12, 24, 40]), 0, _size(rng, 1560, 16384), 128, False, dtype, "NHD", "diag_requant")
    if kind == "chunk":
        Skv = _size(rng, 2048, 65536)
        return dict(kind=kind, Hq=32, Hkv=8, S=min(Skv, _size(rng, 16, 2048)), Skv=Skv, D=128)
    if kind == "video":
        return dict(kind=kind, H=rng.choice([12, 24, 40]), S=_size(rng, 1560, 32760))
    if kind in ("quant4", "quant8"):
        H = rng.choice([16, 32])
        return dict(kind=kind, B=rng.choice([1, 2]), Hq=H, Hkv=H // rng.choice([1, 4]), S=_size(rng, 128, 32768 if H == 16 else 16384),
                    D=rng.choice([64, 128]), dtype=dtype, layout=rng.choice(["HND", "NHD"]))
    return dict(kind="gemm", mode=rng.choice(["mxfp8", "mxfp4", "nvfp4"]), M=_size(rng, 64, 8192), N=_size(rng, 512, 8192, 8),
                K=_size(rng, 512, 8192, 128), out=rng.choice(["bf16", "bf16", "fp16"]))


def _randn(g, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _video_tokens(g, H, S, D):
    """N(0,1) plus a smooth component over the token index that correlates neighbouring tokens, as video latents have it."""
    x = _randn(g, 1, H, S, D)
    pos = torch.arange(S, device="cuda", dtype=torch.float32) / S
    for _ in range(8):
        freq = torch.randint(1, 64, (1,), generator=g, device="cuda")
        phase = torch.rand(H, 1, D, generator=g, device="cuda") * (2 * math.pi)
        x += (0.25 * torch.sin(2 * math.pi * freq * pos[None, :, None] + phase)).to(x.dtype)
    return x


def _outlier_channels(g, k):
    """About 4 % of the key channels are twenty times as large, as in the keys of language models."""
    D = k.shape[-1]
    k[..., torch.randperm(D, generator=g, device="cuda")[:max(1, D // 25)]] *= 20.0
    return k


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, st = case["kind"], dict(case)
    if kind == "attention":
        B, Hq, S, D, dt = case["B"], case["Hq"], case["S"], case["D"], DTYPE[case["dtype"]]
        Hkv = case["Hkv"] or Hq
        sizes = [(B, h, S, D) if case["layout"] == "HND" else (B, S, h, D) for h in (Hq, Hkv, Hkv)]
        st["q"], st["k"], st["v"] = (_randn(g, *s, dtype=dt) for s in sizes)
        if case["mode"] == "online_requant":
            _outlier_channels(g, st["k"])
        if case["entry"] == "hook":
            st["module"] = MixedPrecisionAttention(block_scale_type=case["mode"])
    elif kind == "chunk":
        st["q"] = _randn(g, 1, case["Hq"], case["S"], case["D"])
        k, v = (_randn(g, 1, case["Hkv"], case["Skv"], case["D"]) for _ in range(2))
        st["kv"] = mpsa.prepare_kv(_outlier_channels(g, k), v, pv_mode="requant")
    elif kind == "video":
        st["q"], st["k"], st["v"] = (_video_tokens(g, case["H"], case["S"], 128) for _ in range(3))
    elif kind in ("quant4", "quant8"):
        B, S, D = case["B"], case["S"], case["D"]
        st["q"], st["k"] = (_randn(g, *((B, h, S, D) if case["layout"] == "HND" else (B, S, h, D)), dtype=DTYPE[case["dtype"]])
                            for h in (case["Hq"], case["Hkv"]))
        st["k"] = _outlier_channels(g, st["k"])
    else:
        st.update(_gemm_operands(g, case))
    return st


def _gemm_operands(g, case):
    """Weights and activations already in the block-scaled format, as a program that multiplies them keeps them."""
    mode, K = case["mode"], case["K"]
    st, alpha = {}, 1.0
    for side, rows in (("a", case["M"]), ("b", case["N"])):
        x = _randn(g, rows, K)
        if mode == "nvfp4":
            codes, scales, ts = mpsa.quantize_nvfp4(x)
            alpha *= float(ts)
        else:
            q = mpsa.quantize_mx(x.view(1, 1, rows, K), want_fp8=mode == "mxfp8", want_fp4=mode == "mxfp4")
            codes = q.fp8.view(rows, K).view(torch.float8_e5m2) if mode == "mxfp8" else q.fp4.view(rows, K // 2)
            scales = q.fp8_sf if mode == "mxfp8" else q.fp4_sf
        st[side], st[side + "_scale"] = codes, scales
    epb = 1 if mode == "mxfp8" else 2
    st["configs"] = {"ELEM_PER_BYTE_A": epb, "ELEM_PER_BYTE_B": epb, "VEC_SIZE": 16 if mode == "nvfp4" else 32, "alpha": alpha}
    return st


def run(st):
    kind = st["kind"]
    if kind == "attention":
        q, k, v, entry = st["q"], st["k"], st["v"], st["entry"]
        if entry == "diagonal":
            return mpsa.diagonal_tiled_attention(q, k, v, causal=st["causal"])
        if entry == "mxfp_attn":
            return mxfp_attn(q, k, v, is_causal=st["causal"], block_scale_type=st["mode"])
        if entry == "hook":
            return st["module"](q, k, v, is_causal=st["causal"], tensor_layout=st["layout"])
        return mxfp_attn_kernel(q, k, v, is_causal=st["causal"], tensor_layout=st["layout"], output_dtype=q.dtype,
                                block_scale_type=st["mode"])
    if kind == "chunk":
        return mpsa.attention_forward(st["q"], None, None, kv=st["kv"], causal=True, pv_mode="requant")
    if kind == "video":
        return mpsa.attention_forward(st["q"], st["k"], st["v"], causal=False, fp4_kind="nvfp4")
    if kind == "quant4":
        return quant_mxfp4(st["q"], st["k"], tensor_layout=st["layout"])
    if kind == "quant8":
        return quant_mxfp8e5(st["q"], st["k"], tensor_layout=st["layout"])
    return block_scaled_matmul(st["a"], st["a_scale"], st["b"], st["b_scale"], DTYPE[st["out"]], st["M"], st["N"], st["K"],
                               st["configs"])


def work(case):
    """Least bytes (inputs read once, outputs written once) and operations of the two products of one pass."""
    kind = case["kind"]
    if kind == "attention":
        B, Hq, S, D = case["B"], case["Hq"], case["S"], case["D"]
        pairs = S * (S + 1) // 2 if case["causal"] else S * S
        return {"bytes": 2.0 * B * S * D * (2 * Hq + 2 * (case["Hkv"] or Hq)), "flops": 4.0 * B * Hq * pairs * D}
    if kind == "chunk":
        Hq, Hkv, S, Skv, D = case["Hq"], case["Hkv"], case["S"], case["Skv"], case["D"]
        # every key and value in 4 bits with a scale per 32; the 8-bit form is needed for the diagonal tiles only
        kept = 2.0 * Hkv * (Skv * D * (0.5 + 1 / 32) + min(S, Skv) * D)
        return {"bytes": 4.0 * Hq * S * D + kept, "flops": 4.0 * Hq * D * (S * (Skv - S) + S * (S + 1) // 2)}
    if kind == "video":
        H, S = case["H"], case["S"]
        return {"bytes": 8.0 * H * S * 128, "flops": 4.0 * H * S * S * 128}
    if kind in ("quant4", "quant8"):
        n = case["B"] * (case["Hq"] + case["Hkv"]) * case["S"] * case["D"]
        return {"bytes": n * (2 + 1 + 1 / 32), "flops": 0.0}
    M, N, K, bits = case["M"], case["N"], case["K"], {"mxfp8": 8.25, "mxfp4": 4.25, "nvfp4": 4.5}[case["mode"]]
    return {"bytes": (M + N) * K * bits / 8 + 2.0 * M * N, "flops": 2.0 * M * N * K}


def tolerance(case):
    """Codes and scales are whole values and have to match.  Attention and products come in 16 bits; inside attention P is
    rounded to 16 bits or to its tile's 8- or 4-bit format, and a tile at the router's threshold may take either format."""
    if case["kind"] in ("quant4", "quant8"):
        return "exact"
    return {"rel": 5e-3} if case["kind"] == "gemm" else {"rel": 1e-2}
