"""The work that is timed when a change claims to make this framework faster.

Every case is one call (forward, or forward and backward) of a public entry point, at the layer shapes of the model
configurations in ``cornstarch_b200/zoo.py`` (a SigLIP-so400m-shaped encoder, a Llama-3.1-8B-shaped language model, their
projector and optimizer) or, for drawn cases, at generic sizes of the same ranges.  Inputs are synthetic and made on the
GPU from the seed alone.

Ranges that ``draw`` covers: attention with 1..4 sequences of 64..8192 tokens (at most 8192 tokens in all), 8..32 query
heads, GQA groups of 1..8, head widths 64..128, default causal / causal / full / bitfield masks; linear layers with 16..8192
tokens and the projections of the configurations; norms of 1..16384 rows; losses of 64..4096 tokens over 1000..128256
classes; AdamW over 1e6..2e8 parameters; whole encoder and decoder layers of 64..4096 tokens; logits of a small whole model.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from cornstarch_b200.models.llama import DecoderConfig, DecoderLayer, decoder_spec
from cornstarch_b200.models.vision import SiglipEncoderLayer, SiglipVisionConfig
from cornstarch_b200.ops.attention import AttnMask, attention
from cornstarch_b200.ops.cross_entropy import linear_cross_entropy
from cornstarch_b200.ops.elementwise import layer_norm, rms_norm, rope_tables
from cornstarch_b200.ops.linear import linear, multi_linear
from cornstarch_b200.optim.fused_adamw import FusedAdamW, split_decay_groups
from cornstarch_b200.zoo import LLAMA31_8B, SIGLIP_SO400M, Shape, build_model

DEV = "cuda"
BF16 = torch.bfloat16
TEXT = (1 << 62) | 3  # a text token that may see text and the image modality
IMAGE = 2  # a token of the image modality: sees its own kind in both directions


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one short prompt through one attention layer, no gradient (evaluation, greedy generation): the smallest call
        {"name": "attn_prompt", "kind": "attn", "B": 1, "S": 333, "Hq": 32, "Hk": 8, "D": 128, "mask": "default", "image": 0,
         "train": False},
        # text-only training at the benchmark's sequence length: the largest attention call
        {"name": "attn_causal_8k", "kind": "attn", "B": 1, "S": 8192, "Hq": 32, "Hk": 8, "D": 128, "mask": "causal", "image": 0,
         "train": True},
        # multimodal training batch: two ragged sequences with an image span each and padding at the end
        {"name": "attn_multimodal", "kind": "attn", "B": 2, "S": 3571, "Hq": 32, "Hk": 8, "D": 128, "mask": "bitfield",
         "image": 729, "train": True},
        # q|k|v projection of a short prompt, no gradient: weight traffic bounds it
        {"name": "qkv_prompt", "kind": "linear", "T": 77, "K": 4096, "widths": "4096,1024,1024", "bias": False, "train": False},
        # first MLP projection of the vision encoder for four images, with bias
        {"name": "fc1_images", "kind": "linear", "T": 2916, "K": 1152, "widths": "4304", "bias": True, "train": True},
        # gate|up projection of the language model at the benchmark's sequence length: the largest GEMMs of a layer
        {"name": "gate_up_8k", "kind": "linear", "T": 8192, "K": 4096, "widths": "14336,14336", "bias": False, "train": True},
        # residual add + RMSNorm between the sub-layers of the language model
        {"name": "norm_8k", "kind": "norm", "T": 8192, "H": 4096, "layer": False, "residual": True},
        # LM head + cross-entropy over the full vocabulary
        {"name": "lm_loss", "kind": "loss", "T": 4096, "H": 4096, "V": 128256},
        # one encoder layer for four images
        {"name": "encoder_layer", "kind": "encoder", "B": 4, "S": 729, "H": 1152, "I": 4304, "heads": 16},
        # one decoder layer on a multimodal sequence, gradients into the optimizer's flat buffer
        {"name": "decoder_layer", "kind": "decoder", "S": 4096, "H": 4096, "I": 14336, "Hq": 32, "Hk": 8, "image": 729},
        # optimizer step over the parameters of one decoder layer, with gradient clipping
        {"name": "adamw_layer", "kind": "adamw", "N": 218112000},
        # a whole (shallow) model: image and text to logits
        {"name": "vlm_logits", "kind": "vlm", "S": 1531, "layers": 2, "vocab": 32000},
    ]


LINEARS = [  # (K, widths, bias) of the configurations' projections
    (1152, "1152,1152,1152", True), (1152, "1152", True), (1152, "4304", True), (4304, "1152", True), (1152, "4096", True),
    (4096, "4096", True), (4096, "4096,1024,1024", False), (4096, "4096", False), (4096, "14336,14336", False),
    (14336, "4096", False), (1280, "1280,1280,1280", True), (1280, "5120", True), (5120, "1280", True),
]
HEADS = [(32, 8), (16, 16), (20, 20), (32, 32), (12, 12), (8, 1), (16, 4)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn", "attn", "attn", "linear", "linear", "norm", "loss", "encoder", "decoder", "adamw", "vlm"])
    if kind == "attn":
        B = rng.choice([1, 1, 2, 4])
        S = _log(rng, 64, 8192 // B)
        Hq, Hk = rng.choice(HEADS)
        mask = rng.choice(["default", "causal", "full", "bitfield", "bitfield"])
        return {"kind": kind, "B": B, "S": S, "Hq": Hq, "Hk": Hk, "D": rng.choice([64, 72, 80, 96, 128, 128]), "mask": mask,
                "image": rng.randint(S // 16 + 1, S // 2) if mask == "bitfield" else 0, "train": rng.random() < 0.7}
    if kind == "linear":
        K, widths, bias = rng.choice(LINEARS)
        return {"kind": kind, "T": _log(rng, 16, 8192), "K": K, "widths": widths, "bias": bias, "train": rng.random() < 0.7}
    if kind == "norm":
        return {"kind": kind, "T": _log(rng, 1, 16384), "H": rng.choice([768, 1152, 1280, 2048, 4096, 5120]),
                "layer": rng.random() < 0.5, "residual": rng.random() < 0.7}
    if kind == "loss":
        return {"kind": kind, "T": _log(rng, 64, 4096), "H": rng.choice([1024, 2048, 4096]),
                "V": rng.choice([1000, 32000, 50272, 128256])}
    if kind == "encoder":
        H, I, heads = rng.choice([(1152, 4304, 16), (768, 3072, 12), (1024, 4096, 16), (1280, 5120, 20)])
        B = rng.choice([1, 2, 4])
        return {"kind": kind, "B": B, "S": _log(rng, 64, 1500), "H": H, "I": I, "heads": heads}
    if kind == "decoder":
        S = _log(rng, 64, 4096)
        H, I, Hq, Hk = rng.choice([(4096, 14336, 32, 8), (2048, 5632, 16, 4), (4096, 11008, 32, 32)])
        return {"kind": kind, "S": S, "H": H, "I": I, "Hq": Hq, "Hk": Hk, "image": rng.randint(S // 16 + 1, S // 2)}
    if kind == "adamw":
        return {"kind": kind, "N": _log(rng, 1_000_000, 200_000_000)}
    return {"kind": kind, "S": _log(rng, 800, 2048), "layers": rng.choice([1, 2]), "vocab": rng.choice([32000, 64000])}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * std).to(dtype)


def _bits(B, S, image):
    """Text with one span of ``image`` image tokens per sequence, at another place in each; the last sequence of a batch is
    padded at its end."""
    bits = torch.full((B, S), TEXT, dtype=torch.int64, device=DEV)
    for b in range(B):
        start = (b * (S - image)) // (B + 1)
        bits[b, start : start + image] = IMAGE
    if B > 1:
        bits[-1, S - S // 16 :] = 0
    return bits


def _widths(case):
    return [int(w) for w in case["widths"].split(",")]


def _attn_data(case, seed):
    g = _gen(seed)
    B, S, Hq, Hk, D = (case[k] for k in ("B", "S", "Hq", "Hk", "D"))
    # one fused q|k|v buffer, as the projection in front of the attention gives it
    qkv = _randn(g, B, S, (Hq + 2 * Hk) * D)
    do = _randn(g, B, S, Hq, D)
    bits = _bits(B, S, case["image"]) if case["mask"] == "bitfield" else None
    return qkv, do, bits


def _linear_data(case, seed):
    g = _gen(seed)
    T, K, ws = case["T"], case["K"], _widths(case)
    x = _randn(g, T, K)
    w = _randn(g, sum(ws), K, std=0.02)
    b = _randn(g, sum(ws), std=0.02) if case["bias"] else None
    dy = _randn(g, T, sum(ws))
    return x, w, b, dy


def _norm_data(case, seed):
    g = _gen(seed)
    T, H = case["T"], case["H"]
    x, res, dy, dh = (_randn(g, T, H) for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, generator=g, device=DEV)).to(BF16)
    b = _randn(g, H, std=0.1)
    return x, res, dy, dh, w, b


def _loss_data(case, seed):
    g = _gen(seed)
    T, H, V = case["T"], case["H"], case["V"]
    h = _randn(g, T, H)
    w = _randn(g, V, H, std=0.02)
    labels = torch.randint(0, V, (T,), generator=g, device=DEV)
    labels[: T // 11] = -100  # image placeholders do not count
    return h, w, labels


def _fill(module, seed):
    """Weights of a module from the seed: matrices ~ N(0, 0.02), norm weights around 1, biases ~ N(0, 0.02)."""
    g = _gen(seed)
    with torch.no_grad():
        for name, p in module.named_parameters():
            std = 0.02 if p.dim() >= 2 or name.endswith("bias") else 0.1
            v = torch.randn(p.shape, generator=g, device=DEV) * std
            p.copy_(v + 1 if p.dim() == 1 and not name.endswith("bias") else v)
    return g


def _build(make):
    prev = torch.get_default_dtype()
    torch.set_default_dtype(BF16)
    try:
        with torch.device(DEV):
            return make()
    finally:
        torch.set_default_dtype(prev)


def _encoder_module(case):
    cfg = SiglipVisionConfig(hidden_size=case["H"], intermediate_size=case["I"], num_attention_heads=case["heads"],
                             num_hidden_layers=1, hidden_act=SIGLIP_SO400M["hidden_act"])
    return _build(lambda: SiglipEncoderLayer(cfg))


def _decoder_module(case):
    cfg = DecoderConfig(**{**LLAMA31_8B, "hidden_size": case["H"], "intermediate_size": case["I"], "num_hidden_layers": 1,
                           "num_attention_heads": case["Hq"], "num_key_value_heads": case["Hk"]})
    return _build(lambda: DecoderLayer(cfg, decoder_spec(cfg), 0))


def _adamw_shapes(case):
    """Matrices 4096 wide plus the vectors of a layer, about ``N`` parameters in all."""
    rows = max(1, case["N"] // 4096)
    cut = [rows * 5 // 48, rows * 2 // 48, rows // 3, rows // 4]
    cut.append(rows - sum(cut))
    return [(r, 4096) for r in cut if r > 0] + [(4096,), (4096,)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "attn":
        Hq, Hk, D, B, S = (case[k] for k in ("Hq", "Hk", "D", "B", "S"))
        qkv, do, bits = _attn_data(case, seed)
        s["qkv"] = qkv.requires_grad_(case["train"])
        s["do"] = do
        # the mask of a batch is made once and shared by all layers; "default" leaves it to the call
        s["mask"] = {"default": None, "causal": AttnMask.causal(), "full": AttnMask.full(),
                     "bitfield": AttnMask.bitfield(bits) if bits is not None else None}[case["mask"]]
    elif kind == "linear":
        x, w, b, dy = _linear_data(case, seed)
        ws = _widths(case)
        # the projections of one input sit back to back, as the optimizer lays them out
        s["w"] = [t.detach().requires_grad_(case["train"]) for t in torch.split(w, ws)]
        s["b"] = [t.detach().requires_grad_(case["train"]) for t in torch.split(b, ws)] if b is not None else [None] * len(ws)
        s["x"], s["dy"] = x.requires_grad_(case["train"]), dy
    elif kind == "norm":
        x, res, dy, dh, w, b = _norm_data(case, seed)
        s["leaves"] = [t.requires_grad_() for t in ([x, w] + ([res] if case["residual"] else []) + ([b] if case["layer"] else []))]
        s["x"], s["w"], s["res"], s["b"], s["dy"], s["dh"] = x, w, res if case["residual"] else None, b, dy, dh
    elif kind == "loss":
        h, w, labels = _loss_data(case, seed)
        s["h"], s["w"], s["labels"] = h.requires_grad_(), torch.nn.Parameter(w), labels
        s["opt"] = FusedAdamW([s["w"]])  # gives the weight its place in the flat gradient buffer
    elif kind == "encoder":
        m = _encoder_module(case)
        g = _fill(m, seed)
        s["m"], s["opt"] = m, FusedAdamW(split_decay_groups(m))
        s["x"] = _randn(g, case["B"], case["S"], case["H"]).requires_grad_()
        s["dy"] = _randn(g, case["B"], case["S"], case["H"])
        s["mask"] = AttnMask.full()
    elif kind == "decoder":
        m = _decoder_module(case)
        g = _fill(m, seed)
        s["m"], s["opt"] = m, FusedAdamW(split_decay_groups(m))
        s["x"], s["res"] = (_randn(g, 1, case["S"], case["H"]).requires_grad_() for _ in range(2))
        s["dy"], s["dr"] = (_randn(g, 1, case["S"], case["H"]) for _ in range(2))
        s["rope"] = rope_tables(8192, case["H"] // case["Hq"], LLAMA31_8B["rope_theta"], DEV)
        s["mask"] = AttnMask.bitfield(_bits(1, case["S"], case["image"]))
    elif kind == "adamw":
        g = _gen(seed)
        params = [torch.nn.Parameter(_randn(g, *shape, std=0.02)) for shape in _adamw_shapes(case)]
        s["opt"] = FusedAdamW([{"params": [p for p in params if p.dim() == 2], "weight_decay": 0.01},
                               {"params": [p for p in params if p.dim() == 1], "weight_decay": 0.0}], lr=1e-4, max_norm=1.0)
        for p in params:
            p.main_grad.copy_(_randn(g, *p.shape, std=1e-3))
    else:
        llm = {**LLAMA31_8B, "num_hidden_layers": case["layers"], "vocab_size": case["vocab"]}
        vis = {**SIGLIP_SO400M, "num_hidden_layers": case["layers"]}
        shape = Shape("case", seq_len=case["S"], image_tokens=729, image_size=384, vocab=case["vocab"], llm=llm, vision=vis)
        torch.manual_seed(seed)
        m = build_model(shape, device=DEV, dtype=BF16).eval()
        g = _fill(m, seed)
        ids = torch.randint(0, case["vocab"] - 1, (1, case["S"]), generator=g, device=DEV)
        ids[:, :729] = case["vocab"] - 1
        s["m"], s["ids"], s["pixels"] = m, ids, _randn(g, 1, 3, 384, 384)
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "attn":
        B, S, Hq, Hk, D = (case[k] for k in ("B", "S", "Hq", "Hk", "D"))
        qkv = s["qkv"]
        qkv.grad = None
        with torch.set_grad_enabled(case["train"]):
            q = qkv[..., : Hq * D].view(B, S, Hq, D)
            k = qkv[..., Hq * D : (Hq + Hk) * D].view(B, S, Hk, D)
            v = qkv[..., (Hq + Hk) * D :].view(B, S, Hk, D)
            o = attention(q, k, v, s["mask"]) if s["mask"] is not None else attention(q, k, v)
        if not case["train"]:
            return o
        o.backward(s["do"])
        return o.detach(), qkv.grad
    if kind == "linear":
        x, ws, bs = s["x"], s["w"], s["b"]
        for t in [x, *ws, *bs]:
            if t is not None:
                t.grad = None
        with torch.set_grad_enabled(case["train"]):
            y = linear(x, ws[0], bs[0]) if len(ws) == 1 else multi_linear(x, ws, bs)
        if not case["train"]:
            return y
        y.backward(s["dy"])
        return [y.detach(), x.grad] + [t.grad for t in [*ws, *bs] if t is not None]
    if kind == "norm":
        for t in s["leaves"]:
            t.grad = None
        y = layer_norm(s["x"], s["w"], s["b"], 1e-5, s["res"]) if case["layer"] else rms_norm(s["x"], s["w"], 1e-5, s["res"])
        if case["residual"]:
            y, h = y
            torch.autograd.backward([y, h], [s["dy"], s["dh"]])
            return [y.detach(), h.detach()] + [t.grad for t in s["leaves"]]
        y.backward(s["dy"])
        return [y.detach()] + [t.grad for t in s["leaves"]]
    if kind == "loss":
        s["h"].grad = None
        loss = linear_cross_entropy(s["h"], s["w"], s["labels"])
        loss.backward()
        return [loss.detach(), s["h"].grad, s["w"].main_grad]
    if kind == "encoder":
        s["x"].grad = None
        y = s["m"](s["x"], s["mask"])
        y.backward(s["dy"])
        # (softmax does not see a constant added to all keys: the gradient of the k bias is rounding noise around zero)
        return [y.detach(), s["x"].grad] + [p.main_grad for n, p in s["m"].named_parameters() if n != "self_attn.k_proj.bias"]
    if kind == "decoder":
        s["x"].grad = s["res"].grad = None
        y, r, _ = s["m"](s["x"], s["res"], s["rope"], None, s["mask"])
        torch.autograd.backward([y, r], [s["dy"], s["dr"]])
        return [y.detach(), r.detach(), s["x"].grad, s["res"].grad] + [p.main_grad for p in s["m"].parameters()]
    if kind == "adamw":
        opt = s["opt"]
        opt.step()
        return opt.flat_params() + [t for _, r in opt._regions for t in (r.resid, r.exp_avg, r.exp_avg_sq)]
    with torch.no_grad():
        return s["m"](input_ids=s["ids"], pixel_values=s["pixels"]).logits


# ------------------------------------------------------------------------------------------------ floors and tolerances
def _pairs(S, image, mask, B=1):
    """Allowed (query, key) pairs per head over the batch (padding left out of account)."""
    if mask == "full":
        return B * S * S
    # an image token sees its span in both directions and nothing else; every text token sees what comes before it
    total = 0
    for b in range(B):
        start = (b * (S - image)) // (B + 1)
        text = S * (S + 1) // 2 - (image * start + image * (image + 1) // 2)
        total += text + image * image
    return total


def work(case):
    kind = case["kind"]
    if kind == "attn":
        B, S, Hq, Hk, D = (case[k] for k in ("B", "S", "Hq", "Hk", "D"))
        fwd = 4 * D * Hq * _pairs(S, case["image"], case["mask"], B)
        io = B * S * D * 2
        if not case["train"]:
            return {"bytes": io * (2 * Hq + 2 * Hk), "flops": fwd}
        return {"bytes": io * (4 * Hq + 4 * Hk), "flops": fwd * 3.5}
    if kind == "linear":
        T, K, N = case["T"], case["K"], sum(_widths(case))
        if not case["train"]:
            return {"bytes": 2 * (T * K + N * K + T * N), "flops": 2 * T * K * N}
        return {"bytes": 4 * (T * K + N * K + T * N), "flops": 6 * T * K * N}
    if kind == "norm":
        # x (and the residual) in, y (and the sum) out; dy (and its gradient) in, dx out
        n = 6 if case["residual"] else 4
        return {"bytes": 2 * n * case["T"] * case["H"], "flops": 20 * case["T"] * case["H"]}
    if kind == "loss":
        T, H, V = case["T"], case["H"], case["V"]
        return {"bytes": 4 * (T * H + V * H), "flops": 6 * T * H * V}
    if kind == "encoder":
        B, S, H, I = case["B"], case["S"], case["H"], case["I"]
        lin = 4 * H * H + 2 * H * I
        return {"bytes": 4 * (lin + 2 * B * S * H), "flops": 6 * B * S * lin + 14 * H * B * S * S}
    if kind == "decoder":
        S, H, I, Hq, Hk = (case[k] for k in ("S", "H", "I", "Hq", "Hk"))
        lin = 2 * H * H + 2 * H * H * Hk // Hq + 3 * H * I
        return {"bytes": 4 * (lin + 4 * S * H), "flops": 6 * S * lin + 14 * H * _pairs(S, case["image"], "bitfield")}
    if kind == "adamw":
        # parameter, remainder, two moments and the gradient: read and written (the gradient is cleared)
        n = sum(math.prod(s) for s in _adamw_shapes(case))
        return {"bytes": 28 * n + 2 * n, "flops": 20 * n}
    S, L, V = case["S"], case["layers"], case["vocab"]
    llm = L * (2 * 4096 * 4096 + 2 * 4096 * 1024 + 3 * 4096 * 14336) + V * 4096
    vis = L * (4 * 1152 * 1152 + 2 * 1152 * 4304) + 1152 * 4096 + 4096 * 4096 + 588 * 1152
    flops = 2 * S * llm + 2 * 729 * vis + L * (4 * 4096 * _pairs(S, 729, "bitfield") + 4 * 1152 * 729 * 729)
    return {"bytes": 2 * (llm + vis + S * V), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        # 32-bit state; a parameter that sits on the edge between two bf16 values may round the other way
        return {"rel": 2e-4, "max": 0.02, "differ": 0.01}
    if kind == "vlm":
        return {"rel": 0.03, "max": 0.9}  # bf16 activations through all layers
    if kind in ("encoder", "decoder"):
        return {"rel": 0.02, "max": 0.9}  # bf16 activations through the ten kernels of a layer
    return {"rel": 1e-2, "max": 0.5}  # bf16 operands and results, sums in 32 bits


# ------------------------------------------------------------------------------------------------ 64 bits
def _allowed(case, bits, b, S):
    i = torch.arange(S, device=DEV)
    if case["mask"] == "full":
        return torch.ones(S, S, dtype=torch.bool, device=DEV)
    if bits is None:
        return i[None, :] <= i[:, None]
    qb, kb = (bits[b] & ((1 << 62) - 1))[:, None], (bits[b] & ((1 << 62) - 1))[None, :]
    text = (qb & 1) != 0
    ok = torch.where(text, (i[None, :] <= i[:, None]) & ((qb & kb) != 0), qb == kb)
    return ok & (qb != 0) & (kb != 0)


def _head64(q, k, v, ok, scale):
    s = (q @ k.t()) * scale
    s = s.masked_fill(~ok, float("-inf"))
    m = s.max(-1, keepdim=True).values
    p = torch.exp(s - torch.where(torch.isinf(m), torch.zeros_like(m), m))
    z = p.sum(-1, keepdim=True)
    return (p / torch.where(z == 0, torch.ones_like(z), z)) @ v


def _attn64(q, k, v, masks):
    """q [B,S,Hq,D], k and v [B,S,Hk,D] in 64 bits; head by head, scores recomputed in the backward pass."""
    from torch.utils.checkpoint import checkpoint

    B, S, Hq, D = q.shape
    g = Hq // k.shape[2]
    rows = []
    for b in range(B):
        rows.append(torch.stack([checkpoint(_head64, q[b, :, h], k[b, :, h // g], v[b, :, h // g], masks[b], 1 / math.sqrt(D),
                                            use_reentrant=False) for h in range(Hq)], dim=1))
    return torch.stack(rows)


def _norm64(h, w, b, eps, layer):
    if layer:
        return F.layer_norm(h, (h.shape[-1],), w, b, eps)
    return h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + eps) * w


def _leaf(t):
    return t.detach().double().requires_grad_()


def exact(case, seed):
    kind = case["kind"]
    if kind == "attn":
        B, S, Hq, Hk, D = (case[k] for k in ("B", "S", "Hq", "Hk", "D"))
        qkv, do, bits = _attn_data(case, seed)
        masks = [_allowed(case, bits, b, S) for b in range(B)]
        x = _leaf(qkv)
        q, k, v = torch.split(x, [Hq * D, Hk * D, Hk * D], dim=-1)
        with torch.set_grad_enabled(case["train"]):
            o = _attn64(q.view(B, S, Hq, D), k.view(B, S, Hk, D), v.view(B, S, Hk, D), masks)
        if not case["train"]:
            return o
        o.backward(do.double())
        return o.detach(), x.grad
    if kind == "linear":
        x, w, b, dy = _linear_data(case, seed)
        ws = _widths(case)
        x, w, dy = x.double(), w.double(), dy.double()
        y = x @ w.t() + (b.double() if b is not None else 0)
        if not case["train"]:
            return y
        out = [y, dy @ w] + list(torch.split(dy.t() @ x, ws))
        return out + (list(torch.split(dy.sum(0), ws)) if b is not None else [])
    if kind == "norm":
        x, res, dy, dh, w, b = _norm_data(case, seed)
        x, res, w, b = (_leaf(t) for t in (x, res, w, b))
        h = x + res if case["residual"] else x
        y = _norm64(h, w, b, 1e-5, case["layer"])
        leaves = [x, w] + ([res] if case["residual"] else []) + ([b] if case["layer"] else [])
        if case["residual"]:
            torch.autograd.backward([y, h], [dy.double(), dh.double()])
            return [y.detach(), h.detach()] + [t.grad for t in leaves]
        y.backward(dy.double())
        return [y.detach()] + [t.grad for t in leaves]
    if kind == "loss":
        h, w, labels = _loss_data(case, seed)
        h, w = _leaf(h), _leaf(w)
        loss = F.cross_entropy(h @ w.t(), labels, ignore_index=-100)
        loss.backward()
        return [loss.detach(), h.grad, w.grad]
    if kind == "encoder":
        B, S, H = case["B"], case["S"], case["H"]
        m = _encoder_module(case)
        g = _fill(m, seed)
        x = _leaf(_randn(g, B, S, H))
        dy = _randn(g, B, S, H)
        p = {n: _leaf(t) for n, t in m.named_parameters()}
        D = H // case["heads"]

        def lin(t, n):
            return t @ p[n + ".weight"].t() + p[n + ".bias"]

        h = _norm64(x, p["layer_norm1.weight"], p["layer_norm1.bias"], 1e-6, True)
        q, k, v = (lin(h, "self_attn.%s_proj" % n).view(B, S, -1, D) for n in "qkv")
        ok = torch.ones(S, S, dtype=torch.bool, device=DEV)
        r = x + lin(_attn64(q, k, v, [ok] * B).reshape(B, S, H), "self_attn.out_proj")
        h = _norm64(r, p["layer_norm2.weight"], p["layer_norm2.bias"], 1e-6, True)
        y = r + lin(F.gelu(lin(h, "mlp.fc1"), approximate="tanh"), "mlp.fc2")
        y.backward(dy.double())
        return [y.detach(), x.grad] + [t.grad for n, t in p.items() if n != "self_attn.k_proj.bias"]
    if kind == "decoder":
        S, H, Hq, Hk = (case[k] for k in ("S", "H", "Hq", "Hk"))
        D = H // Hq
        m = _decoder_module(case)
        g = _fill(m, seed)
        x, res = (_leaf(_randn(g, 1, S, H)) for _ in range(2))
        dy, dr = (_randn(g, 1, S, H) for _ in range(2))
        p = {n: _leaf(t) for n, t in m.named_parameters()}
        inv = 1.0 / (LLAMA31_8B["rope_theta"] ** (torch.arange(0, D, 2, dtype=torch.float32, device=DEV) / D))
        ang = torch.outer(torch.arange(S, dtype=torch.float32, device=DEV), inv).double()
        cos, sin = ang.cos()[None, :, None], ang.sin()[None, :, None]

        def rot(t):
            a, b = t[..., : D // 2], t[..., D // 2 :]
            return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

        eps = LLAMA31_8B["rms_norm_eps"]
        r = x + res
        h = _norm64(r, p["input_layernorm.weight"], None, eps, False)
        q, k, v = (F.linear(h, p["self_attn.%s_proj.weight" % n]).view(1, S, -1, D) for n in "qkv")
        ok = _allowed({"mask": "bitfield"}, _bits(1, S, case["image"]), 0, S)
        a = F.linear(_attn64(rot(q), rot(k), v, [ok]).reshape(1, S, H), p["self_attn.o_proj.weight"])
        r = r + a
        h = _norm64(r, p["post_attention_layernorm.weight"], None, eps, False)
        y = F.linear(F.silu(F.linear(h, p["mlp.gate_proj.weight"])) * F.linear(h, p["mlp.up_proj.weight"]), p["mlp.down_proj.weight"])
        torch.autograd.backward([y, r], [dy.double(), dr.double()])
        return [y.detach(), r.detach(), x.grad, res.grad] + [t.grad for t in p.values()]
    return None  # the optimizer's state has a layout of its own; a whole model takes too long
