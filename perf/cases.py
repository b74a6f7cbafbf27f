"""The work that is timed: what a host of this library has it do, from one small projection to a large prefill chunk.

Every case goes through the public launch functions of `qwen_engine_b200` on tensors with the value distributions of
the benchmark configurations: packed 4-bit weights uniform over 0..15 with fp16 group scales U[0.002, 0.02],
activations N(0, 1), RMSNorm gains around 0.05 (which keeps a random-weight residual stream finite in fp16).
Weights, activations, buffers and plans are made by `prepare`; `run` is one pass over them.
"""
import math

import torch

from qwen_engine_b200 import ops, synth

H, I, NQ, NKV = synth.HIDDEN, synth.INTER, ops.NUM_Q_HEADS, ops.NUM_KV_HEADS
STACK = {"hidden": H, "inter": I, "q_heads": NQ, "kv_heads": NKV}


def listed():
    return [
        # the smallest call of a decode step: one O projection at batch 1 straight from an fp16 activation
        {"name": "projection_o", "kind": "projection", "rows": H, "k": H, "input": "fp16", "residual": True},
        # a batch-1 GEMV over a matrix that fills the chip (the scaled-up shape), Q8_1 activation in hand
        {"name": "projection_large", "kind": "projection", "rows": 28672, "k": 8192, "input": "q8", "residual": False},
        # one decoder layer of a decode step, launch by launch in the order of an engine that runs without a graph
        {"name": "decode_layer", "kind": "decode_layer", "fused": False, **STACK},
        # the whole stack of a decode step as the library's own graph
        {"name": "decode_sweep", "kind": "decode_sweep", "layers": synth.LAYERS, **STACK},
        # the end of a decode step: final norm, lm_head, choice of the next token, logits kept for the host
        {"name": "lm_head_token", "kind": "lm_head", "vocab": synth.VOCAB, "k": H, "temperature": 0.8, "logits": True},
        # one layer's projections for a decode batch: a handful of sequences, a usual batch, an odd larger one
        {"name": "layer_4_tokens", "kind": "layer", "tokens": 4, **STACK},
        {"name": "layer_16_tokens", "kind": "layer", "tokens": 16, **STACK},
        {"name": "layer_47_tokens", "kind": "layer", "tokens": 47, **STACK},
        # one layer's projections for a prompt: short and ragged, a usual chunk, the largest chunk
        {"name": "layer_115_tokens", "kind": "layer", "tokens": 115, **STACK},
        {"name": "layer_1024_tokens", "kind": "layer", "tokens": 1024, **STACK},
        {"name": "layer_4096_tokens", "kind": "layer", "tokens": 4096, **STACK},
        # the scaled-up contraction at the largest chunk
        {"name": "gemm_large", "kind": "gemm", "tokens": 4096, "rows": 28672, "k": 8192, "residual": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _stack(rng):
    heads = rng.randint(2, 8) * 2
    return {"hidden": 128 * heads, "inter": 256 * _log_int(rng, 4, 35), "q_heads": heads, "kv_heads": rng.choice([2, 4])}


def _tokens(rng):
    # decode batches and short prompts, or prompt chunks from 256 tokens on.  Not drawn: 129 to 255 tokens, which the
    # tensor-core dispatch gives a 5-stage ring with two issuing warps that faults, so there is no time to compare with.
    m = _log_int(rng, 2, 4096)
    return m if m <= 128 or m >= 256 else m // 2


def draw(rng):
    kind = rng.choice(["projection", "decode_layer", "decode_sweep", "lm_head", "layer", "layer", "layer", "gemm"])
    if kind == "projection":
        return {"kind": kind, "rows": _log_int(rng, 256, 28672), "k": 256 * _log_int(rng, 2, 35),
                "input": rng.choice(["q8", "fp16", "rmsnorm", "heads"]), "residual": rng.random() < 0.5}
    if kind == "decode_layer":
        return {"kind": kind, "fused": rng.random() < 0.5, **_stack(rng)}
    if kind == "decode_sweep":
        return {"kind": kind, "layers": _log_int(rng, 2, 28), **_stack(rng)}
    if kind == "lm_head":
        return {"kind": kind, "vocab": _log_int(rng, 8000, synth.VOCAB), "k": 256 * rng.randint(2, 8),
                "temperature": rng.choice([0.0, 0.8]), "logits": rng.random() < 0.5}
    if kind == "layer":
        return {"kind": kind, "tokens": _tokens(rng), **_stack(rng)}
    return {"kind": kind, "tokens": _log_int(rng, 256, 4096), "rows": 256 * _log_int(rng, 20, 112), "k": 256 * _log_int(rng, 2, 32),
            "residual": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------------------------------

class _Maker:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def weights(self, rows, k):
        w = torch.randint(-(1 << 31), 1 << 31, (rows, k // 8), dtype=torch.int32, device="cuda", generator=self.gen)
        s = torch.rand((rows, k // 128), device="cuda", generator=self.gen).mul_(0.018).add_(0.002)
        return w, s.to(torch.float16)

    def acts(self, *shape, dtype=torch.float16):
        return torch.randn(shape, device="cuda", generator=self.gen).to(dtype)

    def gain(self, n):
        return torch.rand(n, device="cuda", generator=self.gen).mul_(0.02).add_(0.04).to(torch.float16)

    def layer(self, c):
        hid, inter, qd, kd = c["hidden"], c["inter"], 128 * c["q_heads"], 128 * c["kv_heads"]
        return {"input_norm": self.gain(hid), "q": self.weights(qd, hid), "k": self.weights(kd, hid), "v": self.weights(kd, hid),
                "o": self.weights(hid, qd), "post_norm": self.gain(hid), "gate_up": self.weights(2 * inter, hid),
                "down": self.weights(hid, inter)}


def _half(*shape):
    return torch.empty(shape, dtype=torch.float16, device="cuda")


def _q8(k):
    return (torch.empty(k, dtype=torch.int8, device="cuda"), torch.empty(k // 128, dtype=torch.float32, device="cuda"),
            torch.empty(k // 8, dtype=torch.int32, device="cuda"))


def _qkv_view(layer, q, k, v):
    return ops.QKVProjectionView(layer["q"][0], layer["q"][1], q, layer["k"][0], layer["k"][1], k, layer["v"][0], layer["v"][1], v)


def prepare(case, seed):
    make = _Maker(seed)
    c, s = case, {"case": case}
    kind = c["kind"]
    if kind == "projection":
        rows, k = c["rows"], c["k"]
        s["w"], s["y"] = make.weights(rows, k), _half(rows)
        s["residual"] = make.acts(rows) if c["residual"] else None
        s["x"] = make.acts(k, dtype=torch.float32 if c["input"] == "heads" else torch.float16)
        s["gamma"] = make.gain(k)
        s["act"] = _q8(k)
        if c["input"] == "q8":
            ops.launch_quantize_fp16_to_q8_1(s["x"], *s["act"], k)
    elif kind == "decode_layer":
        hid, inter, qd, kd = c["hidden"], c["inter"], 128 * c["q_heads"], 128 * c["kv_heads"]
        s["layer"] = make.layer(c)
        s["h"], s["h_attn"], s["h_out"] = make.acts(hid), _half(hid), _half(hid)
        s["q"], s["k"], s["v"], s["mlp"] = _half(qd), _half(kd), _half(kd), _half(inter)
        s["view"] = _qkv_view(s["layer"], s["q"], s["k"], s["v"])
        s["act_h"], s["act_q"], s["act_mlp"] = _q8(hid), _q8(qd), _q8(inter)
    elif kind == "decode_sweep":
        s["h"], s["h_out"] = make.acts(c["hidden"]), _half(c["hidden"])
        s["sweep"] = ops.DecodeSweep([make.layer(c) for _ in range(c["layers"])], hidden=c["hidden"], inter=c["inter"],
                                     num_q_heads=c["q_heads"], num_kv_heads=c["kv_heads"])
    elif kind == "lm_head":
        vocab, k = c["vocab"], c["k"]
        s["w"], s["h"], s["gamma"], s["act"] = make.weights(vocab, k), make.acts(k), make.gain(k), _q8(k)
        s["logits"] = _half(vocab) if c["logits"] else None
        slots = ops.sample_slots(vocab)
        s["val"] = torch.empty(slots, dtype=torch.float32, device="cuda")
        s["idx"] = torch.empty(slots, dtype=torch.int32, device="cuda")
        s["control"] = ops.make_sample_control(c["temperature"], seed, 0)
        s["token"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif kind == "layer":
        m, hid, inter, qd, kd = c["tokens"], c["hidden"], c["inter"], 128 * c["q_heads"], 128 * c["kv_heads"]
        s["layer"] = make.layer(c)
        # normed hidden states and attention outputs, which the host's other kernels leave in fp16
        s["x"], s["attn"], s["x_post"], s["h"] = make.acts(m, hid), make.acts(m, qd), make.acts(m, hid), make.acts(m, hid)
        s["q"], s["k"], s["v"] = _half(m, qd), _half(m, kd), _half(m, kd)
        s["h_attn"], s["mlp"], s["h_out"] = _half(m, hid), _half(m, inter), _half(m, hid)
        s["view"] = _qkv_view(s["layer"], s["q"], s["k"], s["v"])
    else:
        m, rows, k = c["tokens"], c["rows"], c["k"]
        s["w"], s["x"], s["y"] = make.weights(rows, k), make.acts(m, k), _half(m, rows)
        s["residual"] = make.acts(m, rows) if c["residual"] else None
    return s


# ---- one pass ---------------------------------------------------------------------------------------

def run(s):
    return {"projection": _projection, "decode_layer": _decode_layer, "decode_sweep": _decode_sweep, "lm_head": _lm_head,
            "layer": _layer, "gemm": _gemm}[s["case"]["kind"]](s)


def _projection(s):
    c, (w, sc) = s["case"], s["w"]
    rows, k = c["rows"], c["k"]
    if c["input"] == "q8":
        ops.launch_gemv_w4a8(w, sc, *s["act"], s["residual"], s["y"], rows, k)
    elif c["input"] == "fp16":
        ops.launch_gemv_w4a16(w, sc, s["x"], s["residual"], s["y"], rows, k)
    elif c["input"] == "rmsnorm":
        ops.launch_gemv_rmsnorm_w4a16(w, sc, s["x"], s["gamma"], s["residual"], s["y"], rows, k)
    else:
        ops.gemv_attn_heads_f32_w4a16(w, sc, s["x"], s["residual"], s["y"], rows, k)
    return s["y"]


def _decode_layer(s):
    c, L = s["case"], s["layer"]
    hid, inter, qd = c["hidden"], c["inter"], 128 * c["q_heads"]
    heads = {"in_features": hid, "num_q_heads": c["q_heads"], "num_kv_heads": c["kv_heads"]}
    # (the q projection stands in for the attention output, as in DecodeSweep)
    if c["fused"]:
        ops.launch_gemv_qkv_rmsnorm_w4a16(s["view"], s["h"], L["input_norm"], **heads)
        ops.launch_gemv_w4a16(*L["o"], s["q"], s["h"], s["h_attn"], hid, qd)
        ops.launch_gemv_dual_gate_up_swiglu_rmsnorm_w4a16(*L["gate_up"], s["h_attn"], L["post_norm"], s["mlp"], hid, inter)
    else:
        ops.launch_rmsnorm_q8_1(s["h"], L["input_norm"], None, *s["act_h"], hidden_size=hid)
        ops.launch_gemv_qkv_w4a8(s["view"], *s["act_h"], **heads)
        ops.launch_quantize_fp16_to_q8_1(s["q"], *s["act_q"], qd)
        ops.launch_gemv_w4a8(*L["o"], *s["act_q"], s["h"], s["h_attn"], hid, qd)
        ops.launch_rmsnorm_q8_1(s["h_attn"], L["post_norm"], None, *s["act_h"], hidden_size=hid)
        ops.launch_gemv_dual_gate_up_swiglu_w4a8(*L["gate_up"], *s["act_h"], s["mlp"], hid, inter)
    ops.launch_quantize_fp16_to_q8_1(s["mlp"], *s["act_mlp"], inter)
    ops.launch_gemv_w4a8(*L["down"], *s["act_mlp"], s["h_attn"], s["h_out"], hid, inter)
    return s["q"], s["k"], s["v"], s["h_attn"], s["mlp"], s["h_out"]


def _decode_sweep(s):
    s["sweep"].run_device(s["h"], s["h_out"])
    return s["h_out"]


def _lm_head(s):
    c = s["case"]
    ops.launch_rmsnorm_q8_1(s["h"], s["gamma"], None, *s["act"], hidden_size=c["k"])
    ops.launch_gemv_w4a8_sample_and_advance(*s["w"], *s["act"], s["logits"], s["val"], s["idx"], s["control"], s["token"], c["vocab"], c["k"])
    return s["token"], s["control"], s["logits"]


def _layer(s):
    c, L = s["case"], s["layer"]
    m, hid, inter, qd = c["tokens"], c["hidden"], c["inter"], 128 * c["q_heads"]
    ops.launch_gemm_prefill_qkv_w4a16(s["view"], s["x"], m, in_features=hid, num_q_heads=c["q_heads"], num_kv_heads=c["kv_heads"])
    ops.launch_gemm_prefill_w4a16(*L["o"], s["attn"], s["h"], s["h_attn"], m, hid, qd)
    ops.launch_gemm_prefill_dual_gate_up_swiglu_w4a16(*L["gate_up"], s["x_post"], s["mlp"], m, hidden_size=hid, intermediate_size=inter)
    ops.launch_gemm_prefill_w4a16(*L["down"], s["mlp"], s["h_attn"], s["h_out"], m, hid, inter)
    return s["q"], s["k"], s["v"], s["h_attn"], s["mlp"], s["h_out"]


def _gemm(s):
    c = s["case"]
    ops.launch_gemm_prefill_w4a16(*s["w"], s["x"], s["residual"], s["y"], c["tokens"], c["rows"], c["k"])
    return s["y"]


# ---- what a pass cannot do without ------------------------------------------------------------------

def _stack_shapes(c):
    hid, inter, qd, kd = c["hidden"], c["inter"], 128 * c["q_heads"], 128 * c["kv_heads"]
    return [(qd + 2 * kd, hid), (hid, qd), (2 * inter, hid), (hid, inter)]


def work(case):
    c, kind = case, case["kind"]
    if kind == "projection":
        rows, k = c["rows"], c["k"]
        act = {"q8": synth.q8_1_bytes(k), "fp16": 2 * k, "rmsnorm": 4 * k, "heads": 4 * k}[c["input"]]
        return {"bytes": synth.weight_bytes(rows, k) + act + rows * (4 if c["residual"] else 2), "flops": 2 * rows * k}
    if kind == "lm_head":
        rows, k = c["vocab"], c["k"]
        return {"bytes": synth.weight_bytes(rows, k) + 4 * k + (2 * rows if c["logits"] else 0), "flops": 2 * rows * k}
    if kind == "gemm":
        m, rows, k = c["tokens"], c["rows"], c["k"]
        return {"bytes": synth.weight_bytes(rows, k) + 2 * m * k + m * rows * (4 if c["residual"] else 2), "flops": 2 * m * rows * k}
    shapes = _stack_shapes(c)
    hid, inter, qd, kd = c["hidden"], c["inter"], 128 * c["q_heads"], 128 * c["kv_heads"]
    layer, flops = sum(synth.weight_bytes(n, k) for n, k in shapes), sum(2 * n * k for n, k in shapes)
    if kind == "decode_sweep":
        return {"bytes": c["layers"] * (layer + 4 * hid) + 4 * hid, "flops": c["layers"] * flops}
    if kind == "decode_layer":
        return {"bytes": layer + 4 * hid + 2 * (hid + qd + 2 * kd + hid + inter + hid), "flops": flops}
    m = c["tokens"]
    return {"bytes": layer + 2 * m * (3 * hid + qd) + 2 * m * (qd + 2 * kd + 2 * hid + inter), "flops": m * flops}


def tolerance(case):
    # fp16 outputs of fp32 sums: two correct implementations round some outputs, and where a kernel rounds its weights to
    # fp16 some weights, to the neighbouring value (2^-11 of it).
    if case["kind"] in ("projection", "gemm", "layer", "lm_head"):
        return {"rel": 1e-3, "max": 8e-3}
    # chained projections at batch 1: such a step can move an activation to the next of its 8-bit values, which is
    # about 1/40 of the activation's root mean square for that one element.
    if case["kind"] == "decode_layer":
        return {"rel": 3e-3, "max": 3e-2}
    return {"rel": 5e-3, "max": 5e-2}
