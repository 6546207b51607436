"""The work that serving a quantised model has this package do, as cases that can be timed one by one.

Every case goes through the public entry points (`custom_esimd_kernels_vllm` and the `torch.ops` it registers) with the
tensors a serving engine holds: weights and scales laid out once at load time, output buffers allocated by the caller,
fresh activations per pass.  Weights are static from then on, so the engine declares that once per thread
(`set_overlap_mode(2)`), as the integration notes recommend.

Kinds of case (`"kind"`):
  int4        one INT4 (group 128) linear: a router, a head, a layer of a small model
  int4_layer  the four INT4 linears of a dense decoder layer with SiLU * mul between them, each fed by the one before
  fp8         one FP8 linear, scale per channel / per tensor / per 128 x 128 block, activations kept in 16 bit
  fp8_layer   the linears of a decoder layer with per-tensor FP8 weights, each residual add + RMSNorm fused in front
  w8a8        dynamic 1 x 128 activation quantisation and the block-scaled FP8 x FP8 GEMM behind it
  moe_int4    routed INT4 experts, from router logits to combined output: prefill pipeline, or (shared = 1) the decode
              pipeline with a sigmoid-gated INT4 shared expert
  moe_fp8     routed FP8 experts with GELU-tanh, from router logits to combined output
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "llm-scaler_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import custom_esimd_kernels_vllm as q  # noqa: E402

DEV = "cuda"
GROUP = 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one small INT4 linear on a decode batch: 9 MB of weights, so launches and latency are what it costs
        {"name": "int4_m16", "kind": "int4", "M": 16, "N": 4096, "K": 4096, "dtype": "bf16", "layout": "int32"},
        # one token through a 70B-class decoder layer: the latency of a single user's stream
        {"name": "int4_layer_m1", "kind": "int4_layer", "M": 1, "H": 8192, "Q": 10240, "I": 28672, "dtype": "fp16", "layout": "uint8"},
        # the same layer for a full decode batch
        {"name": "int4_layer_m64", "kind": "int4_layer", "M": 64, "H": 8192, "Q": 10240, "I": 28672, "dtype": "bf16", "layout": "int32"},
        # and for a prefill chunk
        {"name": "int4_layer_m2048", "kind": "int4_layer", "M": 2048, "H": 8192, "Q": 10240, "I": 28672, "dtype": "bf16", "layout": "int32"},
        # a wide per-channel FP8 projection on a small decode batch
        {"name": "fp8_channel_m8", "kind": "fp8", "M": 8, "N": 27648, "K": 5120, "scale": "channel", "fmt": "e4m3", "dtype": "bf16"},
        # a whole FP8 decoder layer on three tokens, norms included
        {"name": "fp8_layer_m3", "kind": "fp8_layer", "M": 3, "H": 5120, "Q": 7168, "I": 13824, "dtype": "fp16"},
        # block-scaled FP8 (the checkpoint format), an odd decode batch
        {"name": "fp8_block_m27", "kind": "fp8", "M": 27, "N": 17408, "K": 5120, "scale": "block", "fmt": "e4m3", "dtype": "bf16"},
        # block-scaled FP8 prefill with 16-bit activations, a prompt of odd length
        {"name": "fp8_block_m4001", "kind": "fp8", "M": 4001, "N": 17408, "K": 5120, "scale": "block", "fmt": "e4m3", "dtype": "bf16"},
        # the same weights with quantised activations
        {"name": "w8a8_m4096", "kind": "w8a8", "M": 4096, "N": 17408, "K": 5120, "dtype": "bf16"},
        # mixture of experts, prefill: 128 experts, 8 per token
        {"name": "moe_int4_t4096", "kind": "moe_int4", "T": 4096, "E": 128, "k": 8, "H": 2048, "I": 768, "dtype": "bf16", "layout": "nmajor", "shared": 0},
        # the same model decoding 16 tokens, with its shared expert
        {"name": "moe_int4_decode_t16", "kind": "moe_int4", "T": 16, "E": 128, "k": 8, "H": 2048, "I": 768, "dtype": "bf16", "layout": "nmajor", "shared": 1},
        # FP8 experts on a ragged mixed batch
        {"name": "moe_fp8_t257", "kind": "moe_fp8", "T": 257, "E": 64, "k": 4, "H": 2048, "I": 1024, "dtype": "fp16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _near(rng, lo, hi, step):
    """Log-uniform between lo and hi, a multiple of step."""
    return max(step, _log(rng, lo, hi) // step * step)


def _rows(rng, lo, hi):
    """An output width: mostly a multiple of 64, sometimes ragged."""
    n = _near(rng, lo, hi, 64)
    return n + rng.choice((0, 0, 8, 40)) if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(("int4", "int4", "int4_layer", "fp8", "fp8", "fp8_layer", "w8a8", "moe_int4", "moe_int4", "moe_fp8"))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    decode = rng.random() < 0.6
    if kind == "int4":
        return {"kind": kind, "M": _log(rng, 1, 64) if decode else _log(rng, 65, 4096), "N": _rows(rng, 1024, 28672),
                "K": _near(rng, 1024, 16384, 128), "dtype": dtype, "layout": rng.choice(("int32", "uint8", "kmajor"))}
    if kind == "int4_layer":
        H = _near(rng, 2048, 8192, 128)
        return {"kind": kind, "M": _log(rng, 1, 64) if decode else _log(rng, 65, 2048), "H": H, "Q": H + _near(rng, 256, 2048, 128),
                "I": _near(rng, 4096, 28672, 128), "dtype": dtype, "layout": rng.choice(("int32", "uint8"))}
    if kind == "fp8":
        scale = rng.choice(("channel", "tensor", "block", "block"))
        return {"kind": kind, "M": _log(rng, 1, 64) if decode else _log(rng, 65, 4096), "N": _rows(rng, 2048, 28672),
                "K": _near(rng, 2048, 14336, 128), "scale": scale, "fmt": "e5m2" if scale == "tensor" and rng.random() < 0.5 else "e4m3",
                "dtype": dtype}
    if kind == "fp8_layer":
        H = _near(rng, 2048, 8192, 128)
        return {"kind": kind, "M": _log(rng, 1, 64), "H": H, "Q": H + _near(rng, 256, 2048, 128), "I": _near(rng, 4096, 28672, 128),
                "dtype": dtype}
    if kind == "w8a8":
        return {"kind": kind, "M": _log(rng, 16, 4096), "N": _rows(rng, 2048, 17408), "K": _near(rng, 2048, 14336, 128), "dtype": dtype}
    E = rng.choice((32, 64, 128))
    case = {"kind": kind, "T": _log(rng, 1, 64) if decode else _log(rng, 65, 4096), "E": E, "k": rng.choice((2, 4, 8)),
            "H": _near(rng, 1024, 4096, 256), "I": _near(rng, 512, 1536, 128), "dtype": dtype}
    if kind == "moe_int4":
        case["shared"] = 1 if decode else 0
        case["layout"] = rng.choice(("nmajor", "marlin"))
    return case


# ---- inputs -------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _acts(g, M, K, dtype):
    """Activations as a norm leaves them: unit variance, and a few channels that stand out."""
    x = torch.randn(M, K, generator=g, device=DEV)
    x *= 1.0 + 7.0 * (torch.rand(K, generator=g, device=DEV) < 0.005)
    return x.to(dtype)


def _int4(g, lead, N, K, dtype):
    """Packed nibbles int32 [.., N, K/8] and scales [.., N, K/128]; weights of standard deviation about 1 / sqrt(K)."""
    w = torch.randint(-2 ** 31, 2 ** 31, (*lead, N, K // 8), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    s = (0.5 + torch.rand(*lead, N, K // GROUP, generator=g, device=DEV)) / (4.6 * math.sqrt(K))
    return w, s.to(dtype)


def _fp8(g, lead, N, K, fmt="e4m3"):
    """FP8 codes [.., N, K] that fill the format's range as an amax-scaled quantiser leaves them; the scale that goes with them."""
    w = torch.empty(*lead, N, K, dtype=torch.float8_e5m2 if fmt == "e5m2" else torch.float8_e4m3fn, device=DEV)
    rows = w.view(-1, K)
    step = max(1, (1 << 27) // K)
    for i in range(0, rows.shape[0], step):
        r = torch.randn(min(step, rows.shape[0] - i), K, generator=g, device=DEV)
        rows[i:i + step] = (r * 96.0).clamp_(-448.0, 448.0).to(w.dtype)
    return w, 1.0 / (96.0 * math.sqrt(K))


def _jitter(g, shape, value):
    return value * (0.5 + torch.rand(*shape, generator=g, device=DEV))


def _presented(case, w, s):
    """The INT4 weight as the case's layout presents it."""
    if case["layout"] == "uint8":
        return w.view(torch.uint8), s
    if case["layout"] == "kmajor":
        return w.t().contiguous(), s.t().contiguous()
    return w, s


def prepare(case, seed):
    q.set_overlap_mode(2)
    g, kind, dtype = _gen(seed), case["kind"], DTYPES[case["dtype"]]
    st = {"case": case}

    def out(*shape):
        return torch.empty(*shape, dtype=dtype, device=DEV)

    if kind == "int4":
        M, N, K = case["M"], case["N"], case["K"]
        st["x"] = _acts(g, M, K, dtype)
        st["w"], st["s"] = _presented(case, *_int4(g, (), N, K, dtype))
        st["out"] = out(M, N)
    elif kind == "int4_layer":
        M, H = case["M"], case["H"]
        st["x"] = _acts(g, M, H, dtype)
        for name, N, K in _layer_shapes(case):
            st[name] = _presented(case, *_int4(g, (), N, K, dtype))
            st["out_" + name] = out(M, N)
        st["act"] = out(M, case["I"])
    elif kind == "fp8":
        M, N, K = case["M"], case["N"], case["K"]
        st["x"], st["out"] = _acts(g, M, K, dtype), out(M, N)
        st["w"], unit = _fp8(g, (), N, K, case["fmt"])
        shape = {"channel": (N,), "tensor": (1,), "block": ((N + 127) // 128, (K + 127) // 128)}[case["scale"]]
        st["s"] = _jitter(g, shape, unit)
    elif kind == "fp8_layer":
        M, H = case["M"], case["H"]
        st["x"], st["stream"], st["residual"] = _acts(g, M, H, dtype), _acts(g, M, H, dtype), out(M, H)
        st["norms"] = [(1.0 + 0.1 * torch.randn(H, generator=g, device=DEV)).to(dtype) for _ in range(2)]
        st["normed"] = [out(M, H), out(M, H)]
        for name, N, K in _layer_shapes(case):
            w, unit = _fp8(g, (), N, K)
            st[name] = (w, _jitter(g, (1,), unit))
            st["out_" + name] = out(M, N)
        st["act"] = out(M, case["I"])
    elif kind == "w8a8":
        M, N, K = case["M"], case["N"], case["K"]
        st["x"], st["out"] = _acts(g, M, K, dtype), out(M, N)
        st["w"], unit = _fp8(g, (), N, K)
        st["s"] = _jitter(g, ((N + 127) // 128, K // 128), unit)
    else:
        T, E, H, I = case["T"], case["E"], case["H"], case["I"]
        st["x"] = _acts(g, T, H, dtype)
        st["logits"] = torch.randn(T, E, generator=g, device=DEV).to(dtype)
        if kind == "moe_fp8":
            w, unit = _fp8(g, (E,), 2 * I, H)
            st["w13"] = (w, _jitter(g, (E,), unit))
            w, unit = _fp8(g, (E,), H, I)
            st["w2"] = (w, _jitter(g, (E,), unit))
        else:
            st["w13"], st["w2"] = _int4(g, (E,), 2 * I, H, dtype), _int4(g, (E,), H, I, dtype)
            if case["layout"] == "marlin":
                st["w13"], st["w2"] = _marlin(*st["w13"]), _marlin(*st["w2"])
            if case["shared"]:
                # the shared expert as the decode pipeline receives it: scales [K/128, N]
                (gu, gus), (dn, dns) = _int4(g, (), 2 * I, H, dtype), _int4(g, (), H, I, dtype)
                st["shared"] = (gu, gus.t().contiguous(), dn, dns.t().contiguous())
                st["gate"] = (torch.randn(1, H, generator=g, device=DEV) / math.sqrt(H)).to(dtype)
    return st


def _marlin(w, s):
    """Experts K-major: any int32 words are nibbles in some order, so only the shapes change."""
    return w.transpose(1, 2).contiguous(), s.transpose(1, 2).contiguous()


def _layer_shapes(case):
    H, I = case["H"], case["I"]
    return (("qkv", case["Q"], H), ("o", H, H), ("gate_up", 2 * I, H), ("down", H, I))


# ---- one pass -----------------------------------------------------------------------------------------------------

def _linear_int4(x, w, out):
    op = q.esimd_gemv_int4 if x.shape[0] == 1 else q.esimd_gemm_int4_pgrp
    return op(x, w[0], w[1], out)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "int4":
        return _linear_int4(st["x"], (st["w"], st["s"]), st["out"])
    if kind == "int4_layer":
        H, I = case["H"], case["I"]
        qkv = _linear_int4(st["x"], st["qkv"], st["out_qkv"])
        o = _linear_int4(qkv[:, :H], st["o"], st["out_o"])                 # attention itself belongs to the engine
        gate_up = _linear_int4(o, st["gate_up"], st["out_gate_up"])
        q.esimd_moe_silu_mul(gate_up, st["act"], 2 * I, I, case["M"])
        return {"qkv": qkv, "o": o, "gate_up": gate_up, "down": _linear_int4(st["act"], st["down"], st["out_down"])}
    if kind == "fp8":
        if case["scale"] == "channel":
            return q.esimd_gemv_fp8_pern(st["x"], st["w"], st["s"], st["out"], case["N"], case["K"])
        if case["scale"] == "tensor":
            op = q.esimd_gemv_fp8_pert if case["M"] == 1 else q.esimd_gemm_fp8_pert
            return op(st["x"], st["w"], st["s"], st["out"])
        return q.esimd_gemm_fp8_blockscale(st["x"], st["w"], st["s"], st["out"])
    if kind == "fp8_layer":
        H, I = case["H"], case["I"]
        residual = st["residual"].copy_(st["stream"])                     # the residual stream enters the layer
        qkv = q.esimd_resadd_norm_gemv_fp8_pert(st["x"], residual, st["norms"][0], *st["qkv"], st["out_qkv"], st["normed"][0], 1e-6)
        o = q.esimd_gemm_fp8_pert(qkv[:, :H], *st["o"], st["out_o"])
        gate_up = q.esimd_resadd_norm_gemv_fp8_pert(o, residual, st["norms"][1], *st["gate_up"], st["out_gate_up"], st["normed"][1], 1e-6)
        q.esimd_moe_silu_mul(gate_up, st["act"], 2 * I, I, case["M"])
        down = q.esimd_gemm_fp8_pert(st["act"], *st["down"], st["out_down"])
        return {"qkv": qkv, "o": o, "gate_up": gate_up, "down": down, "residual": residual}
    if kind == "w8a8":
        xq, xs = q.act_quant_fp8_1x128(st["x"])
        return q.gemm_fp8_block_w8a8(xq, xs, st["w"], st["s"], st["out"])
    if kind == "moe_fp8":
        return q.moe_forward_full_gelu_tanh(st["x"], st["logits"], *st["w13"], *st["w2"], case["k"], case["E"])
    nmajor = case["layout"] == "nmajor"
    if case["shared"]:
        return q.moe_forward_full_int4(st["x"], st["logits"], *st["w13"], st["shared"][0], st["shared"][1], *st["w2"], st["shared"][2],
                                       st["shared"][3], st["gate"], case["k"], 1, case["E"], nmajor)
    return q.moe_prefill_full_int4(st["x"], st["logits"], *st["w13"], *st["w2"], case["k"], case["E"])


# ---- what a pass cannot do without, and how exact it is --------------------------------------------------------------

def _gemm(M, N, K, wbytes):
    return {"bytes": wbytes + 2 * M * K + 2 * M * N, "flops": 2 * M * N * K}


def _add(*parts):
    return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}


def _int4_bytes(N, K):
    return N * K // 2 + 2 * N * (K // GROUP)


def work(case):
    kind = case["kind"]
    if kind == "int4":
        return _gemm(case["M"], case["N"], case["K"], _int4_bytes(case["N"], case["K"]))
    if kind == "int4_layer":
        return _add(*(_gemm(case["M"], N, K, _int4_bytes(N, K)) for _, N, K in _layer_shapes(case)))
    if kind == "fp8_layer":
        return _add(*(_gemm(case["M"], N, K, N * K) for _, N, K in _layer_shapes(case)))
    if kind in ("fp8", "w8a8"):
        return _gemm(case["M"], case["N"], case["K"], case["N"] * case["K"])
    T, E, k, H, I = (case[n] for n in ("T", "E", "k", "H", "I"))
    touched = E * (1.0 - (1.0 - k / E) ** T)                             # experts that some token chose
    expert = 3 * H * I if kind == "moe_fp8" else _int4_bytes(2 * I, H) + _int4_bytes(H, I)
    w = {"bytes": int(touched * expert) + 2 * T * E + 4 * T * H, "flops": 6 * T * k * H * I}
    if case.get("shared"):
        w = _add(w, {"bytes": _int4_bytes(2 * I, H) + _int4_bytes(H, I), "flops": 6 * T * H * I})
    return w


def tolerance(case):
    """About four times the distance of today's results from the same path in 64 bits.  That distance is the rounding of the
    16-bit output of every stage (2^-9 relative for bf16, 2^-12 for fp16, over the square root of three: 1.7e-3 and 2.1e-4
    measured for one linear), growing along the stages of a layer (2.1e-3, 6.6e-4) or an expert pipeline (4.0e-3, 5.1e-4)."""
    bf16 = case["dtype"] == "bf16"
    if case["kind"] in ("int4", "fp8", "w8a8"):
        return {"rel": 7e-3, "max": 2e-2} if bf16 else {"rel": 1e-3, "max": 4e-3}
    if case["kind"] in ("int4_layer", "fp8_layer"):
        return {"rel": 9e-3, "max": 4e-2} if bf16 else {"rel": 2.6e-3, "max": 1.2e-2}
    return {"rel": 1.6e-2, "max": 1.2e-1} if bf16 else {"rel": 2.6e-3, "max": 2.4e-2}
