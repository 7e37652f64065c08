"""The work a user of this package has it do, as cases that can be timed and compared.

Every case is one call through a public entry point: a 4-bit linear layer, packed attention, the Mamba2 scan, the
experts of a mixture-of-experts layer, linear + cross-entropy, or a QLoRA training step of a whole (shallow) model.
Sizes are those of the model presets (Mistral-7B, Granite-3B-A800M, Granite-4.0-tiny, Mamba2-2.7B) with token counts from one decoded token to
the packed batches of the benchmark."""
from __future__ import annotations

import math
import random

import torch

from fms_acceleration_b200.models.builder import build_model, quantize_linears_
from fms_acceleration_b200.models.config import preset
from fms_acceleration_b200.nn import Linear4bit, LoraConfig, get_peft_model
from fms_acceleration_b200.ops.attention import doc_bounds_from_cu_seqlens, varlen_attention
from fms_acceleration_b200.ops.cross_entropy import fused_linear_cross_entropy
from fms_acceleration_b200.ops.mamba import ssd_scan
from fms_acceleration_b200.ops.moe import MoEContext, experts_forward

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one decoded token through the output projection of a 4-bit Mistral-7B layer: latency of the smallest call
        {"name": "q4_one_token", "kind": "q4", "rows": 1, "out": 4096, "in": 4096, "train": False, "dtype": "bf16"},
        # a short prompt (odd number of tokens) through the widest 4-bit projection
        {"name": "q4_prompt_77", "kind": "q4", "rows": 77, "out": 14336, "in": 4096, "train": False, "dtype": "bf16"},
        # scoring of one long document: attention forward alone
        {"name": "attn_score_4001", "kind": "attn", "tokens": 4001, "heads": 32, "kv": 8, "dim": 128, "doc_min": 4001,
         "doc_max": 4001, "layout": 0, "train": False, "dtype": "bf16"},
        # small fine-tuning batch of short packed documents, heads of 64 (Granite-3B-A800M)
        {"name": "attn_train_d64_1500", "kind": "attn", "tokens": 1500, "heads": 24, "kv": 8, "dim": 64, "doc_min": 32,
         "doc_max": 700, "layout": 1, "train": True, "dtype": "bf16"},
        # the benchmark's packed batch, one Mistral-7B layer
        {"name": "attn_train_16384", "kind": "attn", "tokens": 16384, "heads": 32, "kv": 8, "dim": 128, "doc_min": 128,
         "doc_max": 4096, "layout": 2, "train": True, "dtype": "bf16"},
        # prompt through the Mamba2 mixer of a Granite-4.0-tiny layer: scan forward, the final state is kept
        {"name": "ssd_prompt_1024", "kind": "ssd", "tokens": 1024, "heads": 48, "train": False, "state": False,
         "dtype": "bf16"},
        # fine-tuning of the hybrid model on a later slice of a document: a state enters
        {"name": "ssd_train_4352", "kind": "ssd", "tokens": 4352, "heads": 48, "train": True, "state": True,
         "dtype": "bf16"},
        # long-sequence training of Mamba2-2.7B
        {"name": "ssd_train_16384", "kind": "ssd", "tokens": 16384, "heads": 80, "train": True, "state": False,
         "dtype": "bf16"},
        # experts of Granite-3B-A800M, a small batch: most experts see a few dozen rows
        {"name": "experts_train_250", "kind": "experts", "tokens": 250, "train": True, "dtype": "bf16"},
        # the benchmark's batch through the experts
        {"name": "experts_train_16384", "kind": "experts", "tokens": 16384, "train": True, "dtype": "bf16"},
        # head and loss of a full fine-tune (vocabulary 49155, weight gradient included)
        {"name": "head_loss_train_8190", "kind": "head", "tokens": 8190, "vocab": 49155, "hidden": 1536, "train": True,
         "dtype": "bf16"},
        # whole call: NF4 QLoRA step of two Mistral-7B layers: loss, logits and adapter gradients
        {"name": "qlora_model_2x1024", "kind": "model", "layers": 2, "batch": 2, "seq": 1024, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["q4", "q4", "attn", "attn", "ssd", "ssd", "experts", "head", "model"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "q4":
        out, inp = rng.choice([(4096, 4096), (1024, 4096), (14336, 4096), (4096, 14336), (8192, 8192)])
        return {"kind": kind, "rows": _log(rng, 1, 4096), "out": out, "in": inp, "train": rng.random() < 0.3,
                "dtype": dtype}
    if kind == "attn":
        heads, kv, dim = rng.choice([(32, 8, 128), (24, 8, 64), (12, 4, 128), (32, 32, 128)])
        tokens = _log(rng, 64, 16384)
        hi = min(4096, max(32, _log(rng, 32, max(33, tokens))))
        return {"kind": kind, "tokens": tokens, "heads": heads, "kv": kv, "dim": dim, "doc_min": max(1, hi // 32),
                "doc_max": hi, "layout": rng.randrange(1 << 20), "train": rng.random() < 0.6, "dtype": dtype}
    if kind == "ssd":
        return {"kind": kind, "tokens": 256 * _log(rng, 1, 64), "heads": rng.choice([48, 80]),
                "train": rng.random() < 0.6, "state": rng.random() < 0.4, "dtype": "bf16"}
    if kind == "experts":
        return {"kind": kind, "tokens": _log(rng, 8, 16384), "train": rng.random() < 0.7, "dtype": "bf16"}
    if kind == "head":
        vocab, hidden, train = rng.choice([(49155, 1536, True), (32000, 4096, False)])
        return {"kind": kind, "tokens": _log(rng, 64, 8192), "vocab": vocab, "hidden": hidden, "train": train,
                "dtype": "bf16"}
    return {"kind": kind, "layers": rng.choice([1, 2]), "batch": rng.choice([1, 2, 3]), "seq": _log(rng, 64, 1024),
            "dtype": "bf16"}


# ------------------------------------------------------------------------------------------------ inputs
P, N, Q = 64, 128, 256  # Mamba2 head dimension, state size and chunk of both presets
E, TOPK, H, I = 40, 8, 1536, 512  # Granite-3B-A800M experts


def _doc_lengths(case):
    r = random.Random(case["layout"])
    left, out = case["tokens"], []
    while left:
        n = min(left, r.randint(case["doc_min"], case["doc_max"]))
        out.append(n)
        left -= n
    return out


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    dt = DTYPES[case["dtype"]]

    def normal(*shape, std=1.0, dtype=dt):
        return (torch.randn(*shape, generator=g, device=DEV) * std).to(dtype)

    kind, s = case["kind"], {"case": case}
    if kind == "q4":
        w = normal(case["out"], case["in"], std=0.02)
        s["layer"] = Linear4bit.from_weight(w, None, "nf4", 64, dt)
        s["x"] = normal(case["rows"], case["in"]).requires_grad_(case["train"])
        s["dy"] = normal(case["rows"], case["out"], std=0.1) if case["train"] else None
    elif kind == "attn":
        T, nh, nkv, d = case["tokens"], case["heads"], case["kv"], case["dim"]
        for name, n in (("q", nh), ("k", nkv), ("v", nkv)):
            s[name] = normal(T, n, d).requires_grad_(case["train"])
        s["dy"] = normal(T, nh, d, std=0.1) if case["train"] else None
        cu = torch.tensor([0] + _doc_lengths(case), device=DEV).cumsum(0)
        s["start"], s["end"] = doc_bounds_from_cu_seqlens(cu, T)
    elif kind == "ssd":
        T, nh = case["tokens"], case["heads"]
        s["x"], s["B"], s["C"] = normal(T, nh, P, std=0.5), normal(T, 1, N, std=0.5), normal(T, 1, N, std=0.5)
        bias = torch.rand(nh, generator=g, device=DEV) * (math.log(1e-1) - math.log(1e-3)) + math.log(1e-3)
        bias = bias.exp() + torch.log(-torch.expm1(-bias.exp()))
        s["dt"] = torch.nn.functional.softplus(normal(T, nh, std=0.5, dtype=torch.float32) + bias)
        s["A"] = -(torch.rand(nh, generator=g, device=DEV) * 15 + 1)
        s["D"] = torch.rand(nh, generator=g, device=DEV) + 0.5
        s["h0"] = normal(nh, P, N, std=0.2, dtype=torch.float32) if case["state"] else None
        s["leaves"] = [s[n] for n in ("x", "dt", "A", "B", "C", "D", "h0") if s[n] is not None]
        if case["train"]:
            for t in s["leaves"]:
                t.requires_grad_(True)
            s["dy"] = normal(T, nh, P, std=0.1)
    elif kind == "experts":
        T = case["tokens"]
        s["x"] = normal(T, H)
        s["w1"], s["w3"] = normal(E, H, I, std=0.02), normal(E, H, I, std=0.02)
        s["w2"] = normal(E, I, H, std=0.02)
        # a router that prefers some experts, as a trained one does
        logits = torch.randn(T, E, generator=g, device=DEV) + torch.randn(E, generator=g, device=DEV) * 0.5
        p, idx = torch.topk(torch.softmax(logits, -1), TOPK, dim=-1)
        s["gates"], s["idx"] = p / p.sum(-1, keepdim=True), idx.to(torch.int32)
        s["ctx"] = MoEContext(H, I, E, TOPK)
        s["leaves"] = [s[n] for n in ("x", "gates", "w1", "w3", "w2")]
        if case["train"]:
            for t in s["leaves"]:
                t.requires_grad_(True)
            s["dy"] = normal(T, H, std=0.1)
    elif kind == "head":
        s["x"] = normal(case["tokens"], case["hidden"]).requires_grad_(True)
        s["w"] = normal(case["vocab"], case["hidden"], std=0.02).requires_grad_(case["train"])
        lab = torch.randint(0, case["vocab"], (case["tokens"],), generator=g, device=DEV)
        s["labels"] = torch.where(torch.rand(case["tokens"], generator=g, device=DEV) < 0.1,
                                  torch.full_like(lab, -100), lab)
        s["leaves"] = [s["x"]] + ([s["w"]] if case["train"] else [])
    else:
        cfg = preset("mistral-7b")
        cfg.num_hidden_layers = case["layers"]
        model = build_model(cfg, device=torch.device(DEV, 0), dtype=dt, seed=seed, layer_hook=lambda layer: quantize_linears_(
            layer, lambda lin: Linear4bit.from_linear(lin, "nf4", 64, dt)))
        model.quantization_method = "bitsandbytes"
        model = get_peft_model(model, LoraConfig(r=16, lora_alpha=16,
                                                 target_modules=["q_proj", "k_proj", "v_proj", "o_proj"]))
        model.get_base_model().enable_fused("fused_ce_liger")
        model.train()
        s["leaves"] = [p for p in model.parameters() if p.requires_grad]
        with torch.no_grad():  # adapters that have been trained a little: both factors non-zero
            for p in s["leaves"]:
                p.copy_(normal(*p.shape, std=0.01, dtype=p.dtype))
        s["model"] = model
        s["ids"] = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), generator=g, device=DEV)
    return s


# ------------------------------------------------------------------------------------------------ the calls
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "q4":
        if not case["train"]:
            with torch.no_grad():
                return s["layer"](s["x"])
        y = s["layer"](s["x"])
        return [y] + list(torch.autograd.grad(y, [s["x"]], s["dy"]))
    if kind == "attn":
        if not case["train"]:
            with torch.no_grad():
                return varlen_attention(s["q"], s["k"], s["v"], s["start"], s["end"])
        y = varlen_attention(s["q"], s["k"], s["v"], s["start"], s["end"])
        return [y] + list(torch.autograd.grad(y, [s["q"], s["k"], s["v"]], s["dy"]))
    if kind == "ssd":
        args = (s["x"], s["dt"], s["A"], s["B"], s["C"], s["D"], s["h0"], Q)
        if not case["train"]:
            with torch.no_grad():
                return list(ssd_scan(*args))
        y, h = ssd_scan(*args)
        return [y, h] + list(torch.autograd.grad(y, s["leaves"], s["dy"]))
    if kind == "experts":
        args = (s["x"], s["gates"], s["idx"], s["w1"], s["w3"], s["w2"], s["ctx"])
        if not case["train"]:
            with torch.no_grad():
                return experts_forward(*args)
        y = experts_forward(*args)
        return [y] + list(torch.autograd.grad(y, s["leaves"], s["dy"]))
    if kind == "head":
        loss = fused_linear_cross_entropy(s["x"], s["w"], s["labels"])
        return [loss] + list(torch.autograd.grad(loss, s["leaves"]))
    out = s["model"](input_ids=s["ids"], labels=s["ids"], return_logits=True)
    return [out.loss, out.logits] + list(torch.autograd.grad(out.loss, s["leaves"]))


# ------------------------------------------------------------------------------------------------ bytes and operations
def work(case):
    kind = case["kind"]
    if kind == "q4":
        m, n, k = case["rows"], case["out"], case["in"]
        passes = 2 if case["train"] else 1
        return {"bytes": passes * (n * k * (0.5 + 1 / 64) + 2 * m * (n + k)), "flops": passes * 2.0 * m * n * k}
    if kind == "attn":
        T, nh, nkv, d = case["tokens"], case["heads"], case["kv"], case["dim"]
        pairs = sum(n * (n + 1) / 2 for n in _doc_lengths(case))
        rows = 2.0 * T * d * (2 * nh + 2 * nkv)
        return {"bytes": rows * (3 if case["train"] else 1), "flops": pairs * nh * d * (14.0 if case["train"] else 4.0)}
    if kind == "ssd":
        T, nh = case["tokens"], case["heads"]
        # per chunk and head: C B^T shared by the heads; G x, C h, x^T B; the lower triangle of G only
        fwd = T * (Q / 2 * 2.0 * N + nh * P * (Q / 2 * 2.0 + 4.0 * N))
        rows = 2.0 * T * (2 * nh * P + 2 * N) + 4.0 * T * nh
        states = 4.0 * nh * P * N * (2 if case["state"] else 1)
        return {"bytes": rows * (2.5 if case["train"] else 1) + states, "flops": fwd * (3 if case["train"] else 1)}
    if kind == "experts":
        T = case["tokens"]
        flops = T * TOPK * 6.0 * H * I
        used = min(E, T * TOPK)
        return {"bytes": 2.0 * used * 3 * H * I * (2 if case["train"] else 1) + 4.0 * T * H * (2 if case["train"] else 1),
                "flops": flops * (3 if case["train"] else 1)}
    if kind == "head":
        T, v, h = case["tokens"], case["vocab"], case["hidden"]
        passes = 3 if case["train"] else 2
        return {"bytes": 2.0 * v * h * (2 if case["train"] else 1) + 4.0 * T * h, "flops": passes * 2.0 * T * v * h}
    T, L, hid, mid, vocab = case["batch"] * case["seq"], case["layers"], 4096, 14336, 32000
    per_layer = hid * (hid * 2 + 2 * 1024) + 3 * hid * mid
    att = case["batch"] * case["seq"] * (case["seq"] + 1) / 2 * 32 * 128
    # frozen weights: forward and input gradient; the head runs for the loss (with its gradient) and for the logits
    return {"bytes": L * per_layer * 0.52 * 2 + 2.0 * vocab * hid * 3 + 2.0 * T * vocab,
            "flops": L * (4.0 * T * per_layer + 14.0 * att) + 6.0 * T * vocab * hid}


def tolerance(case):
    return {"q4": {"rel": 0.01, "max": 0.06},
            "attn": {"rel": 0.015, "max": 0.3},
            "ssd": {"rel": 0.015, "max": 0.3},
            "experts": {"rel": 0.015, "max": 0.3},
            "head": {"rel": 0.015, "max": 0.3},
            "model": {"rel": 0.03, "max": 1.0}}[case["kind"]]


# ------------------------------------------------------------------------------------------------ 64 bits
def _dequant64(layer):
    """The weight a 4-bit layer stands for, from its stored buffers."""
    scale = layer.code2.double()[layer.absmax_q.long()] * layer.absmax2.double().repeat_interleave(256)[:layer.absmax_q.numel()]
    scale = scale + layer.offset.double()
    packed = layer.weight.reshape(-1).long()
    vals = layer.code.double()[torch.stack([packed >> 4, packed & 15], dim=1).reshape(-1)]
    return (vals.view(-1, 64) * scale[:, None]).view(layer.out_features, layer.in_features)


def _attention64(q, k, v, lengths, scale):
    rep, outs, t = q.shape[1] // k.shape[1], [], 0
    for n in lengths:
        qd, kd, vd = q[t:t + n].transpose(0, 1), k[t:t + n].transpose(0, 1), v[t:t + n].transpose(0, 1)
        kd, vd = kd.repeat_interleave(rep, 0), vd.repeat_interleave(rep, 0)
        sc = qd @ kd.transpose(1, 2) * scale
        sc = sc.masked_fill(torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1), float("-inf"))
        outs.append((torch.softmax(sc, -1) @ vd).transpose(0, 1))
        t += n
    return torch.cat(outs)


def _scan64(x, dt, A, B, C, D, h0):
    T, nh = dt.shape
    c = 64
    n = T // c
    xc, dtc = x.view(n, c, nh, P), dt.view(n, c, nh)
    Bc, Cc = B.view(n, c, N), C.view(n, c, N)
    L = (dtc * A).cumsum(1).transpose(1, 2)  # [n, nh, c]
    keep = torch.ones(c, c, dtype=torch.bool, device=x.device).tril()
    decay = torch.exp((L[..., :, None] - L[..., None, :]).masked_fill(~keep, float("-inf")))
    G = (Cc @ Bc.transpose(1, 2))[:, None] * decay * dtc.transpose(1, 2)[:, :, None, :]
    xh = xc.transpose(1, 2)  # [n, nh, c, P]
    y = G @ xh
    w = torch.exp(L[..., -1:] - L) * dtc.transpose(1, 2)
    S = (xh * w[..., None]).transpose(2, 3) @ Bc[:, None]  # [n, nh, P, N]
    h = torch.zeros(nh, P, N, dtype=x.dtype, device=x.device) if h0 is None else h0
    entering = []
    for i in range(n):
        entering.append(h)
        h = torch.exp(L[i, :, -1])[:, None, None] * h + S[i]
    y = y + torch.exp(L)[..., None] * (Cc[:, None] @ torch.stack(entering).transpose(2, 3))
    return y.transpose(1, 2).reshape(T, nh, P) + D[:, None] * x, h


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _model64(s):
    cfg, base = s["model"].get_base_model().config, s["model"].get_base_model()
    B, S = s["ids"].shape
    grads = {id(p): p.detach().double().requires_grad_(True) for p in s["leaves"]}

    def proj(x, mod):
        if not hasattr(mod, "lora_A"):
            return x @ _dequant64(mod).t()
        a, b = (grads[id(m["default"].weight)] for m in (mod.lora_A, mod.lora_B))
        return x @ _dequant64(mod.base_layer).t() + x @ a.t() @ b.t() * float(mod.scaling["default"])

    d = cfg.head_dim
    inv = 1.0 / cfg.rope_theta ** (torch.arange(0, d, 2, dtype=torch.float64, device=DEV) / d)
    ang = torch.arange(S, dtype=torch.float64, device=DEV).repeat(B)[:, None] * inv
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def rope(t):
        a, b = t[..., : d // 2], t[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = base.model.embed_tokens.weight.double()[s["ids"].reshape(-1)]
    for layer in base.model.layers:
        att, mlp = layer.self_attn, layer.mlp
        y = _norm64(x, layer.input_layernorm.weight.double(), cfg.rms_norm_eps)
        q = rope(proj(y, att.q_proj).view(B * S, -1, d))
        k = rope(proj(y, att.k_proj).view(B * S, -1, d))
        v = proj(y, att.v_proj).view(B * S, -1, d)
        x = x + proj(_attention64(q, k, v, [S] * B, d ** -0.5).reshape(B * S, -1), att.o_proj)
        y = _norm64(x, layer.post_attention_layernorm.weight.double(), cfg.rms_norm_eps)
        x = x + proj(torch.nn.functional.silu(proj(y, mlp.gate_proj)) * proj(y, mlp.up_proj), mlp.down_proj)
    logits = _norm64(x, base.model.norm.weight.double(), cfg.rms_norm_eps) @ base.lm_head.weight.double().t()
    logits = logits.view(B, S, -1)
    loss = torch.nn.functional.cross_entropy(logits[:, :-1].reshape(B * (S - 1), -1), s["ids"][:, 1:].reshape(-1))
    return [loss.detach(), logits.detach()] + list(torch.autograd.grad(loss, [grads[id(p)] for p in s["leaves"]]))


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]

    def leaf(t):
        return t.detach().double().requires_grad_(t.requires_grad)

    if kind == "q4":
        w, x = _dequant64(s["layer"]), s["x"].detach().double()
        return [x @ w.t(), s["dy"].double() @ w] if case["train"] else x @ w.t()
    if kind == "attn":
        q, k, v = leaf(s["q"]), leaf(s["k"]), leaf(s["v"])
        y = _attention64(q, k, v, _doc_lengths(case), case["dim"] ** -0.5)
        return [y.detach()] + list(torch.autograd.grad(y, [q, k, v], s["dy"].double())) if case["train"] else y
    if kind == "ssd":
        names = [n for n in ("x", "dt", "A", "B", "C", "D", "h0") if s[n] is not None]
        t = {n: leaf(s[n]) for n in names}
        y, h = _scan64(t["x"], t["dt"], t["A"], t["B"], t["C"], t["D"], t.get("h0"))
        if not case["train"]:
            return [y, h]
        return [y.detach(), h.detach()] + list(torch.autograd.grad(y, [t[n] for n in names], s["dy"].double()))
    if kind == "experts":
        names = ("x", "gates", "w1", "w3", "w2")
        t = {n: leaf(s[n]) for n in names}
        out = torch.zeros_like(t["x"])
        for e in range(E):
            tok, slot = torch.nonzero(s["idx"] == e, as_tuple=True)
            xe = t["x"][tok]
            h = torch.nn.functional.silu(xe @ t["w1"][e]) * (xe @ t["w3"][e])
            out = out.index_add(0, tok, (h @ t["w2"][e]) * t["gates"][tok, slot][:, None])
        if not case["train"]:
            return out.detach()
        return [out.detach()] + list(torch.autograd.grad(out, [t[n] for n in names], s["dy"].double()))
    if kind == "head":
        x, w = leaf(s["x"]), leaf(s["w"])
        loss = torch.nn.functional.cross_entropy(x @ w.t(), s["labels"], ignore_index=-100)
        return [loss.detach()] + list(torch.autograd.grad(loss, [x] + ([w] if case["train"] else [])))
    return _model64(s)
