"""The work that programs built on this package have it do, as cases that can be timed and compared.

A case is a dict of plain values.  `kind` picks the model family, `mode` what one pass is:

  steps     next tokens of sequences whose context is already cached (a chat server's inner loop, or a replay)
  prompt    one prompt, or the next turn of a conversation, through the many-row path
  request   a whole request: the prompt, then some tokens one by one
  train     one optimiser step of a small network through the drop-in tensor operations

Tokens are given and not sampled, so that a pass always does the same work; every decode step still makes its own pick and
brings it to the host, as a generation loop does.  Weights are normal with deviation 0.02, gains near one, biases small.
`exact` computes the same outputs in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

from deepj_b200.decoder import DecoderConfig, Q8Decoder
from deepj_b200.hybrid import HybridConfig, HybridDecoder
from deepj_b200.tensor import CudaBackend, Tensor

Q8_KINDS = ("llama", "deepseek", "gpt")
RMS_EPS, LN_EPS = 1e-6, 1e-5
LOG_ROWS = 32                                   # rows of a learned distance-bias table
DECAY_RANK = 64                                 # rank of a delta layer's decay projection


# ───────────── cases ─────────────

def _q8(kind, mode, vocab, width, heads, layers, ff, batch, context, tokens, kv="f32", q_rank=0, kv_rank=0, **more):
    return dict(kind=kind, mode=mode, vocab=vocab, width=width, heads=heads, layers=layers, ff=ff, batch=batch, context=context, tokens=tokens,
                kv=kv, q_rank=q_rank, kv_rank=kv_rank, **more)


def _punilix(mode, vocab, width, layers, every, delta_heads, delta_dim, heads, dim, rot, vdim, q_rank, kv_rank, ff, experts, top, context, tokens,
             dtype="bf16", **more):
    return dict(kind="punilix", mode=mode, vocab=vocab, width=width, layers=layers, every=every, delta_heads=delta_heads, delta_dim=delta_dim, heads=heads,
                dim=dim, rot=rot, vdim=vdim, q_rank=q_rank, kv_rank=kv_rank, ff=ff, experts=experts, top=top, batch=1, context=context, tokens=tokens,
                dtype=dtype, **more)


def _somipel(mode, vocab, width, layers, heads, kv_heads, dim, lstm_heads, lstm_dim, lstm_vdim, ff, context, tokens, dtype="bf16", **more):
    return dict(kind="somipel", mode=mode, vocab=vocab, width=width, layers=layers, heads=heads, kv_heads=kv_heads, dim=dim, lstm_heads=lstm_heads,
                lstm_dim=lstm_dim, lstm_vdim=lstm_vdim, ff=ff, batch=1, context=context, tokens=tokens, dtype=dtype, **more)


def listed():
    return [
        # the smallest model of the benchmark: every step is launches and latency
        _q8("llama", "steps", 256, 256, 8, 4, 688, 1, 32, 16, name="llama_tiny_steps"),
        # blocks of the 7B model behind a full context, one user
        _q8("llama", "steps", 32000, 4096, 32, 8, 11008, 1, 2048, 8, name="llama_7b_steps"),
        # the same blocks serving sixteen users at once
        _q8("llama", "steps", 32000, 4096, 32, 4, 11008, 16, 1000, 4, name="llama_7b_steps_16"),
        # a long prompt through blocks of the 7B model
        _q8("llama", "prompt", 32000, 4096, 32, 8, 11008, 1, 0, 2048, name="llama_7b_prompt"),
        # the next turn of a conversation: a short message behind cached context, half-precision cache
        _q8("llama", "prompt", 32000, 2048, 32, 11, 5632, 1, 700, 123, kv="f16", name="llama_1b_turn"),
        # latent projections, a request of ordinary length
        _q8("deepseek", "request", 32000, 2048, 16, 8, 5632, 1, 300, 16, q_rank=1024, kv_rank=512, name="deepseek_request"),
        # GPT-2 XL's width, whose projections are no multiple of 128 long
        _q8("gpt", "request", 50257, 1600, 25, 12, 6400, 1, 200, 16, name="gpt2xl_request"),
        # layer-list models at real widths: a long prompt, and requests where single steps count
        _punilix("prompt", 32000, 4096, 4, 4, 32, 128, 32, 128, 64, 128, 1536, 512, 11008, 0, 0, 0, 2048, name="punilix_prompt"),
        _punilix("request", 32000, 2048, 4, 4, 32, 64, 16, 128, 64, 128, 1024, 512, 1408, 64, 4, 90, 24, name="punilix_experts_request"),
        _somipel("prompt", 32000, 4096, 4, 32, 8, 128, 16, 128, 256, 11008, 0, 2048, name="somipel_prompt"),
        _somipel("request", 32000, 2048, 8, 32, 32, 64, 8, 128, 256, 5632, 60, 24, name="somipel_request"),
        # the unchanged reference program on the drop-in backend: forward, loss, backward and AdamW of two layers
        dict(kind="mlp", mode="train", rows=1024, width=384, ff=1536, classes=1000, name="dropin_train_step"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("llama", "llama", "llama", "deepseek", "gpt", "punilix", "punilix", "somipel", "somipel", "mlp"))
    if kind == "mlp":
        return dict(kind="mlp", mode="train", rows=_log(rng, 32, 1200), width=_log(rng, 64, 512), ff=_log(rng, 128, 1536), classes=_log(rng, 10, 1200))
    mode = rng.choice(("steps", "prompt", "request")) if kind in Q8_KINDS else rng.choice(("prompt", "request"))
    vocab = rng.choice((256, 1000, 5003, 12345, 32000))
    if kind in Q8_KINDS:
        head_dim = rng.choice((32, 64, 64, 128, 128))
        heads = max(2, _log(rng, 256, 4096) // head_dim)
        width = heads * head_dim
        unit = rng.choice((16, 128))
        ff = min(unit * max(1, int(width * rng.uniform(2.5, 3.0)) // unit), 11008)
        layers = rng.randint(2, 4) if width > 2048 else rng.randint(2, 8)
        batch = 1 if mode == "request" else rng.choice((1, 1, 1, 2, 3, 4, 7, 8, 12, 16))
        context = _log(rng, 16, 2000) // (1 if batch < 4 else 4)
        tokens = rng.randint(3, 16) if mode != "prompt" else max(2, _log(rng, 16, 2048) // batch)
        if mode == "prompt" and rng.random() < 0.5:
            context = 0
        if mode == "request":
            context = max(2, context)
        ranks = (width // 2 // 32 * 32, max(32, width // 4 // 32 * 32)) if kind == "deepseek" else (0, 0)
        return _q8(kind, mode, vocab, width, heads, layers, ff, batch, context, tokens, rng.choice(("f32", "f32", "f16")), *ranks)
    context = 0 if mode == "prompt" else _log(rng, 4, 1500)
    tokens = _log(rng, 16, 2048) if mode == "prompt" else rng.randint(3, 24)
    width = 64 * _log(rng, 8, 48)
    dtype = rng.choice(("bf16", "bf16", "bf16", "f32"))
    if dtype == "f32":
        width, tokens, context = min(width, 1024), min(tokens, 600), min(context, 600)
    ff = 8 * max(8, int(width * rng.uniform(2.2, 2.8)) // 8)
    if kind == "punilix":
        dim = rng.choice((64, 128))
        routed = rng.random() < 0.5
        return _punilix(mode, vocab, width, rng.randint(2, 4), rng.choice((1, 2, 4)), max(1, width // dim), dim, max(1, width // 128), 128, 64, 128,
                        max(64, width // 2 // 32 * 32), rng.choice((256, 512)), ff // 4 if routed else ff, rng.choice((8, 16, 32)) if routed else 0,
                        rng.choice((2, 4)) if routed else 0, context, tokens, dtype)
    dim = rng.choice((64, 128))
    heads = max(2, width // dim // 2 * 2)
    return _somipel(mode, vocab, width, rng.randint(3, 8), heads, rng.choice((1, 2, heads)) if heads % 2 == 0 else 1, dim, rng.randint(2, 8),
                    rng.choice((64, 128)), rng.choice((64, 128, 256)), ff, context, tokens, dtype)


# ───────────── weights, the same for the package and for the plain computation ─────────────

def _generator(seed, name):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    return g


def _normal(seed, name, shape, std=0.02, mean=0.0):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=_generator(seed, name))


def _tokens(case, seed):
    n = case["context"] + case["tokens"]
    return torch.randint(0, case["vocab"], (case["batch"], n), generator=_generator(seed, "tokens"), device="cuda")


def _q8_shape(case, name):
    v, d, f, n = case["vocab"], case["width"], case["ff"], case["context"] + case["tokens"]
    return {"emb": (v, d), "pos": (n, d), "Wlm": (d, v), "blm": (v,), "W1": (d, f), "W2": (f, d), "Wg": (d, f), "Wu": (d, f), "Wd": (f, d),
            "Wdq": (d, case["q_rank"]), "Wuq": (case["q_rank"], d), "Wdkv": (d, case["kv_rank"]), "Wuk": (case["kv_rank"], d), "Wuv": (case["kv_rank"], d),
            "bg": (f,), "bu": (f,), "c1": (f,)}.get(name, (d, d) if name[0] == "W" else (d,))


def _q8_weight(case, seed, name, layer):
    shape = _q8_shape(case, name)
    if len(shape) == 2:
        return _normal(seed, f"{name}.{layer}", shape)
    return _normal(seed, f"{name}.{layer}", shape, 0.1, 1.0 if name[0] == "g" else 0.0)


def _list_weight(seed, name, shape, case):
    """A tensor of a layer-list checkpoint; matrices hold bf16 values, as such checkpoints do."""
    last = name.split(".", 1)[-1]
    if last == "mlp.table":
        return torch.rand((shape[0], case["experts"]), generator=_generator(seed, name), device="cuda").argsort(dim=1)[:, :shape[1]]
    if last == "mix.w0":
        t = _normal(seed, name, shape, 1.5, -2.0)           # decays from almost none to fast
    elif last == "mix.f.b":
        t = _normal(seed, name, shape, 0.5, 4.5)            # forget gates start open
    elif last == "mix.rel":
        t = _normal(seed, name, shape, 0.5)
    elif name == "embed":
        t = _normal(seed, name, shape, 1.0)                 # of the size of a sublayer's normed output: tokens stay distinct
    elif len(shape) == 1:
        t = _normal(seed, name, shape, 0.1, 1.0 if last.endswith(("norm", "norm1", "norm2")) else 0.0)
    else:
        t = _normal(seed, name, shape)
    return t.bfloat16().float()


def _record(case):
    """config.json of a layer-list model."""
    c, layers = case, []
    for i in range(c["layers"]):
        if c["kind"] == "punilix":
            if (i + 1) % c["every"] == 0:
                L = {"type": "latent_attention", "mixer": {
                    "heads": c["heads"], "dim": c["dim"], "rot_dim": c["rot"], "vdim": c["vdim"], "q_rank": c["q_rank"], "kv_rank": c["kv_rank"],
                    "scale": (c["dim"] + c["rot"]) ** -0.5,
                    "rot": {"base": 10000.0, "dims": c["rot"], "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
            else:
                L = {"type": "general_delta", "mixer": {"heads": c["delta_heads"], "dim": c["delta_dim"]}}
            if c["experts"] and i % 2 == 1:
                L["mlp"] = {"kind": "moe", "router": {"experts": c["experts"], "top": c["top"]}, "expert": {"ff": c["ff"], "limit": 7.0}}
            else:
                L["mlp"] = {"kind": "dense", "ff": 4 * c["ff"] if c["experts"] else c["ff"], "limit": 7.0}
        else:
            attn = {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": c["dim"], "vdim": c["dim"], "scale": c["dim"] ** -0.5}
            if i % 4 == 3:
                L = {"type": "mlstm", "mixer": {"heads": c["lstm_heads"], "dim": c["lstm_dim"], "vdim": c["lstm_vdim"], "gate_cap": 15.0}}
            elif i % 4 == 2:
                L = {"type": "attention_2", "mixer": dict(attn, q_temp={"coef": 0.1, "every": 1024})}
            else:
                L = {"type": "attention", "mixer": dict(attn, bias_max=128, **({"kv_from": i - 1} if i % 4 == 1 else {}))}
            L["mlp"] = {"kind": "dense", "ff": c["ff"]}
        layers.append(L)
    rec = {"architecture": c["kind"].capitalize(), "vocab": c["vocab"], "width": c["width"], "layers": layers}
    return dict(rec, norm={"groups": 4, "eps": 1e-5}, logit_softcap=30.0) if c["kind"] == "punilix" else dict(rec, norm={"eps": 1e-5}, residual_mult=0.5)


def _list_config(case):
    return HybridConfig.parse(_record(case), case["context"] + case["tokens"] + 8, lambda n: LOG_ROWS if n.endswith(".rel") else DECAY_RANK)


# ───────────── the package's side ─────────────

_next_ids = [1 << 24]
_staging = []


def _host(t):
    """A device tensor as numpy in page-locked memory that the next call uses again."""
    t = t.float()
    torch.cuda.synchronize()
    if not _staging or _staging[0].numel() < t.numel():
        _staging[:] = [torch.empty(max(t.numel(), 1 << 24), dtype=torch.float32, pin_memory=True)]
    view = _staging[0][:t.numel()].view(t.shape)
    view.copy_(t)
    return view.numpy()


class _Model:
    """A decoder with its weights loaded and, for "steps", its context cached."""

    def __init__(self, case, seed):
        self.case = case
        base = _next_ids[0]
        _next_ids[0] += 1 << 14
        size = case["context"] + case["tokens"] + 8
        if case["kind"] in Q8_KINDS:
            cfg = DecoderConfig(case["kind"], case["vocab"], size if case["kind"] != "gpt" else size - 8, case["width"], case["heads"], case["layers"],
                                case["ff"], case["q_rank"], case["kv_rank"])
            self.dec = Q8Decoder(cfg, batch=case["batch"], id_base=base, kv_dtype=case["kv"])
            self.dec.load_weights(lambda name, layer: _host(_q8_weight(case, seed, name, layer)))
        else:
            cfg = _list_config(case)
            shapes = cfg.tensors()
            self.dec = HybridDecoder(cfg, id_base=base, dtype=case["dtype"])
            self.dec.load_weights(lambda name: _host(_list_weight(seed, name, shapes[name], case)))
        torch.cuda.synchronize()
        self.tokens = _tokens(case, seed).cpu().numpy()
        self.at = case["context"]
        if case["mode"] != "request" and self.at:
            self.dec.reset()
            self.dec.prefill(self.tokens[:, :self.at])

    def __del__(self):
        if hasattr(self, "dec"):
            self.dec.close()


class _Network:
    """Two linear layers with GELU between them and softmax cross-entropy behind, in the middle of their training."""

    def __init__(self, case, seed):
        if Tensor._backend is None:
            Tensor.setBackend(CudaBackend())
        self.case = case
        host = {n: t.cpu().numpy() for n, t in _network(case, seed).items()}
        self.x, self.targets = host.pop("x"), host.pop("targets")
        self.t = {n: Tensor(a.shape[0], a.shape[1], a) for n, a in host.items()}


def _network(case, seed):
    n, d, f, c = case["rows"], case["width"], case["ff"], case["classes"]
    out = {"x": _normal(seed, "x", (n, d), 1.0), "targets": torch.randint(0, c, (n,), generator=_generator(seed, "targets"), device="cuda")}
    for name, shape in (("w1", (d, f)), ("b1", (1, f)), ("w2", (f, c)), ("b2", (1, c))):
        out[name] = _normal(seed, name, shape, 0.05)
        out["m." + name] = _normal(seed, "m." + name, shape, 1e-3)
        out["v." + name] = _normal(seed, "v." + name, shape, 1e-3).abs().add_(1e-3).square_()
    return out


ADAM = (1e-3, 0.9, 0.999, 1e-8, 0.01, 1.0 - 0.9 ** 10, 1.0 - 0.999 ** 10)


def prepare(case, seed):
    return _Network(case, seed) if case["kind"] == "mlp" else _Model(case, seed)


def _wanted(case):
    """Places of a replayed prompt whose logits are asked for.  (Not the first token's: a matrix memory of one token gives
    its value times the sign of one product, which no precision pins down when that product is near zero.)"""
    n = case["tokens"]
    return sorted({n // 4, n // 2, 3 * n // 4, n - 1})


def run(state):
    case = state.case
    if case["kind"] == "mlp":
        return _train_step(state)
    dec, tok, at = state.dec, state.tokens, state.at
    if case["mode"] == "prompt":
        if at:
            dec.set_position(at)
        else:
            dec.reset()
        if case["kind"] not in Q8_KINDS:
            return dec.feed(tok[0], _wanted(case))
        dec.prefill(tok[:, at:])
        return dec.logits()
    if case["mode"] == "request":
        dec.reset()
        dec.prefill(tok[:, :at])
    else:
        dec.set_position(at)
    for t in range(at, tok.shape[1]):
        dec.step(tok[:, t])
    return dec.logits()


def _train_step(s):
    T, rows = s.t, s.case["rows"]
    be = Tensor.backend()
    x = Tensor(rows, s.case["width"], s.x)
    z = x.matmul(T["w1"]).addRowVector(T["b1"])
    h = z.geluActivation()
    logits = h.matmul(T["w2"]).addRowVector(T["b2"])
    g = be.crossEntropyGradient(logits, s.targets)
    dh = g.matmul(T["w2"].transpose())
    dz = be.geluBackward(z, dh)
    grads = {"w1": x.transpose().matmul(dz), "b1": dz.sumRows(), "w2": h.transpose().matmul(g), "b2": g.sumRows()}
    for n, gr in grads.items():
        be.adamWUpdate(T[n], gr, T["m." + n], T["v." + n], *ADAM)
    out = {"loss": be.crossEntropyLoss(logits, s.targets)}
    out.update({"grad_" + n: gr.numpy() for n, gr in grads.items()})
    out["w2"] = T["w2"].numpy().copy()
    return out


# ───────────── what a pass cannot do without ─────────────

def _matrices(case):
    """Weights of the projections one token goes through, by layer, as numbers of elements; and the whole model's."""
    d = case["width"]
    if case["kind"] in Q8_KINDS:
        qr, kr = case["q_rank"], case["kv_rank"]
        attn = 4 * d * d if case["kind"] != "deepseek" else d * (qr + kr) + qr * d + 2 * kr * d + d * d
        one = case["layers"] * (attn + (2 if case["kind"] == "gpt" else 3) * d * case["ff"])
        return one, one
    cfg = _list_config(case)
    one = whole = 0
    for name, shape in cfg.tensors().items():
        if len(shape) != 2 or name in ("embed", "head") or name.endswith((".table", ".rel")):
            continue
        n = shape[0] * shape[1]
        whole += n
        one += n * case["top"] / case["experts"] if ".mlp.e" in name else n
    return one, whole


def work(case):
    if case["kind"] == "mlp":
        n, d, f, c = case["rows"], case["width"], case["ff"], case["classes"]
        w = d * f + f * c + f + c
        return {"bytes": 4 * (n * d + 7 * w), "flops": 6 * n * (d * f + f * c) - 2 * n * d * f}
    B, at, n, d, V = case["batch"], case["context"], case["tokens"], case["width"], case["vocab"]
    one, whole = _matrices(case)
    per = 1.125 if case["kind"] in Q8_KINDS else 2.0
    # cached state per position and sequence, in bytes, and attention's multiply-adds per (query, key) pair
    if case["kind"] in Q8_KINDS:
        cached, pair = 2 * d * case["layers"] * (2 if case["kv"] == "f16" else 4), 2 * d * case["layers"]
    elif case["kind"] == "punilix":
        k = case["layers"] // case["every"]
        cached, pair = k * (case["kv_rank"] + case["rot"]) * 2, k * case["heads"] * (case["dim"] + case["rot"] + case["vdim"])
    else:
        k = sum(i % 4 != 3 for i in range(case["layers"]))
        cached, pair = k * 2 * case["kv_heads"] * case["dim"] * 2, k * 2 * case["heads"] * case["dim"]
    b = f = 0.0
    if case["mode"] != "steps":
        lo, rows = (at, n) if case["mode"] == "prompt" else (0, at)
        b += per * (min(whole, one * rows) + d * V) + B * cached * (lo + rows) + 4 * B * rows * d
        f += 2 * B * (rows * one + d * V) + 2 * B * pair * (rows * lo + rows * (rows + 1) / 2)
    if case["mode"] != "prompt":
        b += n * (per * (one + d * V) + B * (cached * (at + n / 2) + 4 * V))
        f += n * (2 * B * (one + d * V) + 2 * B * pair * (at + n / 2))
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the error against 64 bits that is seen over these ranges."""
    if case["kind"] == "mlp":
        return {"rel": 5e-6, "max": 1e-3}               # 32-bit sums
    if case["kind"] in Q8_KINDS:                        # up to five rows go through 24-bit operands, more through 16-bit ones
        return {"rel": 2.4e-3 if case["kv"] == "f16" else 6e-4}
    return {"rel": 2e-2} if case["dtype"] == "bf16" else {"rel": 2e-5}


# ───────────── the same in 64 bits ─────────────

def _dequantised(w):
    """int8 codes with one scale per 32 rows of a column, as 64-bit values."""
    K, N = w.shape
    p = torch.nn.functional.pad(w, (0, 0, 0, -K % 32)).view(-1, 32, N)
    scale = p.abs().amax(dim=1, keepdim=True) / 127.0
    q = torch.where(scale > 0, torch.round(p / scale), torch.zeros((), device=w.device)).clamp_(-127, 127)
    return (q.double() * scale.double()).view(-1, N)[:K]


def _rms(x, eps, groups=1):
    p = x.view(*x.shape[:-1], groups, x.shape[-1] // groups)
    return (p / torch.sqrt(p.square().mean(-1, keepdim=True) + eps)).view(x.shape)


def _attend(q, k, v, scale, bias=None, sink=False):
    """Causal attention of q [H, T, n] over k [G, T, n] and v [G, T, m]; bias [H, distance]."""
    H, T, _ = q.shape
    out = torch.empty((H, T, v.shape[2]), dtype=torch.float64, device="cuda")
    part = max(1, (1 << 27) // (H * T))
    k, v = (t.repeat_interleave(H // t.shape[0], dim=0) for t in (k, v))
    for lo in range(0, T, part):
        hi = min(T, lo + part)
        s = torch.matmul(q[:, lo:hi], k[:, :hi].transpose(1, 2)) * scale
        back = torch.arange(lo, hi, device="cuda")[:, None] - torch.arange(hi, device="cuda")[None, :]
        if bias is not None:
            s = s + bias[:, back.clamp(0, bias.shape[1] - 1)]
        s = s.masked_fill(back < 0, -math.inf)
        m = s.amax(-1, keepdim=True)
        m = m.clamp(min=0) if sink else m
        e = torch.exp(s - m)
        total = e.sum(-1, keepdim=True)
        out[:, lo:hi] = torch.matmul(e, v[:, :hi]) / (total + torch.exp(-m) if sink else total)
    return out


def _rotate(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * cos - b * sin, a * sin + b * cos), dim=-1).view(x.shape)


def _q8_tables(hd, n):
    """The rotary tables as the model defines them: angles and their cosines are 32-bit values."""
    i = np.arange(hd // 2, dtype=np.float32)
    inv = np.float64(10000.0) ** ((np.float32(2.0) * i) / np.float32(hd)).astype(np.float64)
    theta = (np.arange(n, dtype=np.float64)[:, None] / inv[None, :]).astype(np.float32).astype(np.float64)
    return [torch.from_numpy(f(theta).astype(np.float32)).double().cuda() for f in (np.cos, np.sin)]


def _layer_norm(x, g, b):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + LN_EPS) * g + b


def _exact_q8(case, seed):
    B, T, d, H = case["batch"], case["context"] + case["tokens"], case["width"], case["heads"]
    hd, gpt = d // H, case["kind"] == "gpt"
    tok = _tokens(case, seed)
    mat = lambda n, l: _dequantised(_q8_weight(case, seed, n, l))       # noqa: E731
    vec = lambda n, l: _q8_weight(case, seed, n, l).double()            # noqa: E731
    x = vec("emb", -1)[tok.reshape(-1)]
    if gpt:
        x = x + vec("pos", -1)[:T].repeat(B, 1)
        norm = lambda x, n, l: _layer_norm(x, vec("g" + n, l), vec("b" + n, l))     # noqa: E731
    else:
        cos, sin = _q8_tables(hd, T)
        norm = lambda x, n, l: _rms(x, RMS_EPS) * vec("g" + n, l)                   # noqa: E731
    for l in range(case["layers"]):
        h = norm(x, "1", l)
        if case["kind"] == "deepseek":
            cq, ckv = h @ mat("Wdq", l), h @ mat("Wdkv", l)
            q, k, v = cq @ mat("Wuq", l), ckv @ mat("Wuk", l), ckv @ mat("Wuv", l)
        else:
            q, k, v = (h @ mat(n, l) for n in ("Wq", "Wk", "Wv"))
        o = torch.empty_like(x)
        for b in range(B):
            at = slice(b * T, (b + 1) * T)
            qb, kb, vb = (t[at].view(T, H, hd).transpose(0, 1) for t in (q, k, v))
            if not gpt:
                qb, kb = _rotate(qb, cos, sin), _rotate(kb, cos, sin)
            o[at] = _attend(qb, kb, vb, hd ** -0.5).transpose(0, 1).reshape(T, d)
        x = x + o @ mat("Wo", l)
        h = norm(x, "2", l)
        if gpt:
            h = h @ mat("W1", l) + vec("c1", l)
            x = x + torch.nn.functional.gelu(h, approximate="tanh") @ mat("W2", l) + vec("c2", l)
        else:
            h = torch.nn.functional.silu(h @ mat("Wg", l) + vec("bg", l)) * (h @ mat("Wu", l) + vec("bu", l))
            x = x + h @ mat("Wd", l) + vec("bd", l)
    x = x.view(B, T, d)[:, -1]
    return (norm(x, "F", -1) @ mat("Wlm", -1) + vec("blm", -1)).cpu().numpy()


def _yarn(m, T):
    r = m["rot"]
    dims, base, s = r["dims"], r["base"], r["scaling"]
    i = np.arange(dims // 2)
    f = base ** (-2.0 * i / dims)
    turning = lambda n: dims * math.log(s["original"] / (2.0 * math.pi * n)) / (2.0 * math.log(base))      # noqa: E731
    lo, hi = max(math.floor(turning(s["fast"])), 0), min(math.ceil(turning(s["slow"])), dims - 1)
    ramp = np.clip((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    f = f / s["factor"] * ramp + f * (1.0 - ramp)
    angle = np.arange(T)[:, None] * f[None, :]
    gain = 0.1 * math.log(s["factor"]) + 1.0
    return [torch.from_numpy(fn(angle) * gain).cuda() for fn in (np.cos, np.sin)]


def _delta(h, W, m, eps):
    H, n, T = m["heads"], m["dim"], h.shape[0]
    r, k, v = ((h @ W("mix." + s).T).view(T, H, n) for s in "rkv")
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ W("mix.w1").T) @ W("mix.w2").T + W("mix.w0"))).view(T, H, n)
    removal = torch.sigmoid(h @ W("mix.a").T + W("mix.a.b")).view(T, H, n)
    u = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    out, S, ru = torch.empty_like(r), torch.zeros((H, n, n), dtype=torch.float64, device="cuda"), removal * u
    for t in range(T):
        S = decay[t, :, :, None] * S - ru[t, :, :, None] * (u[t, :, None] @ S) + k[t, :, :, None] * v[t, :, None]
        out[t] = (r[t, :, None] @ S)[:, 0]
    return _rms(out, eps).view(T, H * n) * W("mix.norm") * torch.sigmoid(h @ W("mix.g").T)


def _latent(h, W, m, eps):
    H, dim, rd, vd, R, T = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], h.shape[0]
    cos, sin = _yarn(m, T)
    q = ((_rms(h @ W("mix.dq").T, eps) * W("mix.dq.norm")) @ W("mix.uq").T).view(T, H, dim + rd).transpose(0, 1)
    kv = h @ W("mix.dkv").T
    c = _rms(kv[:, :R].contiguous(), eps) * W("mix.dkv.norm")
    kr = _rotate(kv[:, R:].contiguous(), cos, sin)
    k = torch.cat(((c @ W("mix.uk").T).view(T, H, dim).transpose(0, 1), kr[None].expand(H, T, rd)), dim=-1)
    q = torch.cat((q[..., :dim], _rotate(q[..., dim:].contiguous(), cos, sin)), dim=-1)
    o = _attend(q, k, (c @ W("mix.uv").T).view(T, H, vd).transpose(0, 1), m["scale"])
    return o.transpose(0, 1).reshape(T, H * vd) * torch.sigmoid(h @ W("mix.g").T)


def _pair(g, u, limit):
    g = g.clamp(max=limit)
    return g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1.0)


def _grouped(x, W, m, eps, kind, cache, l):
    H, G, n, T = m["heads"], m["kv_heads"], m["dim"], x.shape[0]
    first = kind == "attention"
    heads = lambda t, k: t.view(T, k, n).transpose(0, 1)        # noqa: E731
    q = x @ W("mix.q").T + (W("mix.q.b") if first else 0.0)
    q = _rms(heads(q, H).contiguous(), eps) * W("mix.q.norm")
    src = m.get("kv_from")
    if src is None:
        raw = heads(x @ W("mix.k").T + (W("mix.k.b") if first else 0.0), G).contiguous()
        v = heads(x @ W("mix.v").T + W("mix.v.b"), G) if first else raw
        cache[l] = (_rms(raw, eps) * W("mix.k.norm"), v)
    k, v = cache[l if src is None else src]
    if not first:
        t = m["q_temp"]
        q = q * (1.0 + t["coef"] * torch.log(torch.floor((torch.arange(T, device="cuda", dtype=torch.float64) + 1) / t["every"]) + 1.0))[None, :, None]
        return _attend(q, k, v, m["scale"], sink=True).transpose(0, 1).reshape(T, H * n)
    half = LOG_ROWS // 2
    row = [i if i < half else min(LOG_ROWS - 1, half + math.floor(math.log(i / half) / math.log(m["bias_max"] / half) * (LOG_ROWS - half) + 1e-9))
           for i in range(T)]
    o = _attend(q, k, v, m["scale"], W("mix.rel")[torch.tensor(row, device="cuda")].T.contiguous())
    return o.transpose(0, 1).reshape(T, H * n) * torch.sigmoid(x @ W("mix.g").T)


def _memory(x, W, m, eps):
    H, n, p, cap, T = m["heads"], m["dim"], m["vdim"], m["gate_cap"], x.shape[0]
    q, k, v = (x @ W("mix.q").T).view(T, H, n) * n ** -0.5, (x @ W("mix.k").T).view(T, H, n), (x @ W("mix.v").T).view(T, H, p)
    i = cap * torch.tanh((x @ W("mix.i").T + W("mix.i.b")) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((x @ W("mix.f").T + W("mix.f.b")) / cap))
    S, z = torch.zeros((H, n, p), dtype=torch.float64, device="cuda"), torch.zeros((H, n), dtype=torch.float64, device="cuda")
    top, out = torch.zeros(H, dtype=torch.float64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(f[t] + top, i[t])
        keep, add = torch.exp(f[t] + top - new), torch.exp(i[t] - new)
        S = keep[:, None, None] * S + (add[:, None] * k[t])[:, :, None] * v[t, :, None]
        z, top = keep[:, None] * z + add[:, None] * k[t], new
        under = torch.maximum((z * q[t]).sum(-1).abs(), torch.exp(-new)) + 1e-6
        out[t] = (q[t, :, None] @ S)[:, 0] / under[:, None]
    return _rms(out, eps).view(T, H * p) * W("mix.norm") * torch.sigmoid(x @ W("mix.g").T)


def _exact_list(case, seed):
    rec, shapes = _record(case), _list_config(case).tensors()
    get = lambda n: _list_weight(seed, n, shapes[n], case)      # noqa: E731
    tok = _tokens(case, seed)[0]
    eps, cache = rec["norm"]["eps"], {}
    punilix = case["kind"] == "punilix"
    groups = rec["norm"].get("groups", 1)
    x = get("embed").double()[tok]
    for l, L in enumerate(rec["layers"]):
        W = lambda n, l=l: get(f"l{l}.{n}").double()            # noqa: E731
        m, f = L["mixer"], L["mlp"]
        if not punilix:
            y = _memory(x, W, m, eps) if L["type"] == "mlstm" else _grouped(x, W, m, eps, L["type"], cache, l)
            x = x + rec["residual_mult"] * _rms(y @ W("mix.o").T, eps) * W("norm1")
            y = (torch.nn.functional.silu(x @ W("mlp.gate").T) * (x @ W("mlp.up").T)) @ W("mlp.down").T
            x = x + rec["residual_mult"] * _rms(y, eps) * W("norm2")
            continue
        h = _rms(x, eps, groups) * W("norm1")
        y = (_delta if L["type"] == "general_delta" else _latent)(h, W, m, eps) @ W("mix.o").T
        if f["kind"] == "dense":
            y = y + _pair(h @ W("mlp.gate").T, h @ W("mlp.up").T, f["limit"]) @ W("mlp.down").T
        else:
            chosen = get(f"l{l}.mlp.table").long()[tok]
            for e in range(case["experts"]):
                rows = (chosen == e).any(dim=1).nonzero()[:, 0]
                if rows.numel():
                    z = _pair(h[rows] @ W(f"mlp.e{e}.gate").T, h[rows] @ W(f"mlp.e{e}.up").T, f["expert"]["limit"]) @ W(f"mlp.e{e}.down").T
                    y[rows] += z / case["top"]
        x = x + y
    x = x[_wanted(case)] if case["mode"] == "prompt" else x[-1:]
    logits = (_rms(x, eps, groups) * get("final.norm").double()) @ get("head").double().T
    cap = rec.get("logit_softcap")
    return (cap * torch.tanh(logits / cap) if cap else logits).cpu().numpy()


def _exact_network(case, seed):
    t = {n: a if n == "targets" else a.double() for n, a in _network(case, seed).items()}
    rows = case["rows"]
    z = (t["x"] @ t["w1"] + t["b1"]).requires_grad_()
    h = torch.nn.functional.gelu(z, approximate="tanh")
    logits = h.detach() @ t["w2"] + t["b2"]
    loss = torch.nn.functional.cross_entropy(logits, t["targets"])
    g = torch.softmax(logits, dim=1)
    g[torch.arange(rows, device="cuda"), t["targets"]] -= 1.0
    g = g / rows
    dz, = torch.autograd.grad(h, z, g @ t["w2"].T)
    grads = {"w1": t["x"].T @ dz, "b1": dz.sum(0, keepdim=True), "w2": h.detach().T @ g, "b2": g.sum(0, keepdim=True)}
    lr, b1, b2, eps, wd, c1, c2 = ADAM
    m, v = (b * t[p + "w2"] + (1 - b) * q for b, p, q in ((b1, "m.", grads["w2"]), (b2, "v.", grads["w2"].square())))
    out = {"loss": float(loss), "w2": t["w2"] - lr * (m / c1) / (torch.sqrt(v / c2) + eps) - lr * wd * t["w2"]}
    out.update({"grad_" + n: a for n, a in grads.items()})
    return {n: a if isinstance(a, float) else a.detach().cpu().numpy() for n, a in out.items()}


def exact(case, seed):
    with torch.no_grad() if case["kind"] != "mlp" else torch.enable_grad():
        return (_exact_network if case["kind"] == "mlp" else _exact_q8 if case["kind"] in Q8_KINDS else _exact_list)(case, seed)
