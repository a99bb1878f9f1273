"""What users of lmrs_b200 have it compute, as cases that can be timed and compared.

Kinds of cases:
  lmrs_decode     one forward(token, pos) of a quantized LMRS model whose cache holds the tokens before pos
  lmrs_prefill    get_embeddings + fill_kv_cache of a prompt (the batched pass; Q8_0)
  linear          a product with a quantized weight matrix kept in HBM (ResidentWeights: the layers of a vision tower)
  folder_prefill  forward_tokens of a whole prompt, logits of its last rows (folder models, bf16 or f32)
  folder_decode   one forward(token, pos) of a folder model whose cache holds the tokens before pos
  folder_replay   token after token from position 0 (models with recurrent state cannot repeat a position)

Models carry the layer shapes of the real ones with fewer layers and random weights, so that a case is a few blocks and the
head.  Weights are made here from the seed; exact() computes from the same numbers in 64 bits with plain torch.
"""
import json
import math
import os
import shutil
import struct
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lm.rs_b200"))
import lmrs_b200  # noqa: E402
from lmrs_b200 import functional, lmrs_file, quantization  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
GROUP = 128   # quantization group of LMRS files

# width, feed-forward, heads, KV heads, head size: the layer shapes of the models the framework is used with, and small ones
SHAPES = {
    "llama-3.2-1b": (2048, 8192, 32, 8, 64),
    "llama-3.2-3b": (3072, 8192, 24, 8, 128),
    "phi-3.5-mini": (3072, 8192, 32, 32, 96),
    "small": (1024, 2048, 16, 4, 64),
    "tiny": (256, 512, 4, 2, 64),
}


def listed():
    return [
        # a chat turn on the flagship model: one token of decode, full vocabulary (latency of many small launches + HBM)
        dict(name="q8_decode_1b", kind="lmrs_decode", shape="llama-3.2-1b", q=1, layers=4, vocab=128256, pos=512),
        # the same on 4-bit weights
        dict(name="q4_decode_3b", kind="lmrs_decode", shape="llama-3.2-3b", q=2, layers=3, vocab=32064, pos=200),
        # a system prompt or a pasted document before the first answer
        dict(name="q8_prefill_1b_512", kind="lmrs_prefill", shape="llama-3.2-1b", layers=8, vocab=4096, tokens=512),
        # one projection of an image encoder over all of an image's patches (24 x 24 + 1 rows)
        dict(name="q8_vision_linear", kind="linear", q=1, rows=577, n=1024, o=4096),
        # decode of an unquantized model: HBM-bound, one sequence
        dict(name="genetar_decode_1b", kind="folder_decode", arch="genetar", shape="llama-3.2-1b", dtype="bfloat16", layers=6, vocab=32064, pos=512),
        # decode of a small draft-sized model: nothing but launch latency
        dict(name="genetar_decode_tiny", kind="folder_decode", arch="genetar", shape="tiny", dtype="bfloat16", layers=3, vocab=512, pos=40),
        # an ordinary prompt of an unquantized model
        dict(name="genetar_prefill_1b_512", kind="folder_prefill", arch="genetar", shape="llama-3.2-1b", dtype="bfloat16", layers=3, vocab=4096, tokens=512, rows=1),
        # a long document, scored over its tail: attention grows with the square of the length
        dict(name="genetar_prefill_3b_2048", kind="folder_prefill", arch="genetar", shape="llama-3.2-3b", dtype="bfloat16", layers=2, vocab=4096, tokens=2048, rows=64),
        # full precision with several wanted rows (scoring a continuation), a ragged length
        dict(name="genetar_prefill_f32_301", kind="folder_prefill", arch="genetar", shape="llama-3.2-1b", dtype="float32", layers=2, vocab=4096, tokens=301, rows=16),
        # delta rule, windowed and latent attention, routed experts: a prompt, scored over its tail
        dict(name="tudatar_prefill_512", kind="folder_prefill", arch="tudatar", shape="llama-3.2-1b", dtype="bfloat16", layers=3, vocab=4096, tokens=512, rows=32),
        # the same model fed token by token (a short chat replayed)
        dict(name="tudatar_replay_16", kind="folder_replay", arch="tudatar", shape="llama-3.2-1b", dtype="bfloat16", layers=3, vocab=4096, tokens=16),
        # state-space layers and sink attention, a ragged length
        dict(name="rupenex_prefill_1000", kind="folder_prefill", arch="rupenex", shape="llama-3.2-1b", dtype="bfloat16", layers=2, vocab=4096, tokens=1000, rows=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lmrs_decode", "lmrs_prefill", "linear", "folder_prefill", "folder_prefill", "folder_prefill", "folder_decode", "folder_replay"])
    if kind == "linear":
        return dict(kind=kind, q=rng.choice([1, 1, 2]), rows=_log_int(rng, 1, 1200), n=128 * _log_int(rng, 2, 32), o=4 * _log_int(rng, 32, 1024))
    shape = rng.choice(["llama-3.2-1b", "llama-3.2-3b", "small", "tiny"])
    if kind == "lmrs_decode":
        return dict(kind=kind, shape=shape, q=rng.choice([1, 2]), layers=rng.randint(1, 3), vocab=4 * _log_int(rng, 128, 8000), pos=_log_int(rng, 4, 700))
    if kind == "lmrs_prefill":
        return dict(kind=kind, shape=shape, layers=rng.randint(1, 2), vocab=4 * _log_int(rng, 128, 1024), tokens=_log_int(rng, 2, 900))
    shape = rng.choice(["llama-3.2-1b", "llama-3.2-3b", "phi-3.5-mini", "small", "tiny"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
    c = dict(kind=kind, shape=shape, dtype=dtype, vocab=_log_int(rng, 300, 8000))
    if kind == "folder_decode":
        c.update(arch="genetar", layers=rng.randint(1, 4), pos=_log_int(rng, 3, 1500))
    elif kind == "folder_replay":
        c.update(arch=rng.choice(["genetar", "tudatar", "rupenex"]), layers=rng.randint(1, 2), tokens=rng.randint(2, 24))
    else:
        c.update(arch=rng.choice(["genetar", "tudatar", "rupenex"]), layers=rng.randint(1, 2),
                 tokens=_log_int(rng, 2, 1800 if dtype == "bfloat16" else 400))
        c["rows"] = min(c["tokens"], rng.randint(1, 24) if c["arch"] == "genetar" else rng.randint(16, 32))
    return c


# ---- LMRS models ------------------------------------------------------------------------------------------------------------------------
def _lmrs_args(case):
    dim, ff, H, G, hs = SHAPES[case["shape"]]
    return lmrs_file.LmrsArgs(dim=dim, hidden_dim=ff, n_layers=case["layers"], n_heads=H, head_size=hs, n_kv_heads=G, vocab_size=case["vocab"],
                              seq_len=2048, rms_norm_eps=1e-5, rope_theta=500000.0, q_type=case.get("q", 1), model_type=lmrs_file.LLAMA)


def _quant_codes(gen, o, n, q, sigma):
    """uniform codes with group scales around the standard deviation: int8 [o][n], or 0 .. 15 as uint8; scales f32 [o][n / 128]"""
    s = torch.rand((o, n // GROUP), generator=gen, device=DEV) + 0.5
    if q == 1:
        c = torch.randint(-127, 128, (o, n), generator=gen, device=DEV, dtype=torch.int8)
        return c, s * (sigma / 73.3)
    c = torch.randint(0, 16, (o, n), generator=gen, device=DEV, dtype=torch.uint8)
    return c, s * (-sigma / 4.61)


def _pack(c, q):
    """codes as the file holds them: bytes, or nibble pairs with the even element low"""
    flat = c.reshape(-1)
    return flat.view(torch.uint8) if q == 1 else flat[0::2] | (flat[1::2] << 4)


def _dequant(c, s, q):
    v = c.double() - (0 if q == 1 else 8)
    return (v.reshape(c.shape[0], -1, GROUP) * s.double()[..., None]).reshape(c.shape)


def _lmrs_weights(case, seed):
    """name -> per layer f32 vector, or (codes, scales)"""
    dim, ff, H, G, hs = SHAPES[case["shape"]]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    q, L = case.get("q", 1), case["layers"]
    W = {"emb": [_quant_codes(gen, case["vocab"], dim, q, 0.05)]}
    for name, o, n in (("wq", H * hs, dim), ("wk", G * hs, dim), ("wv", G * hs, dim), ("wo", dim, H * hs), ("w1", ff, dim), ("w2", dim, ff), ("w3", ff, dim)):
        W[name] = [_quant_codes(gen, o, n, q, n ** -0.5) for _ in range(L)]
    for name, n in (("rms_att", L), ("rms_post_att", L), ("rms_final", 1)):
        W[name] = [1.0 + 0.1 * torch.randn(dim, generator=gen, device=DEV) for _ in range(n)]
    return W


def _lmrs_file(case, seed):
    a, W = _lmrs_args(case), _lmrs_weights(case, seed)
    offs, end = lmrs_file.tensor_offsets(a)
    buf = np.zeros(end, np.uint8)
    buf[:lmrs_file.HEADER_BYTES] = np.frombuffer(a.pack(), np.uint8)
    for name, parts in W.items():
        for where, part in zip(offs[name], parts):
            pieces = [(where, part.view(torch.uint8))] if torch.is_tensor(part) else \
                     [(where[0], _pack(part[0], a.q_type)), (where[1], part[1].reshape(-1).view(torch.uint8))]
            for off, data in pieces:
                torch.from_numpy(buf[off:off + data.numel()]).copy_(data)
    return buf


def _tokens(case, seed, n):
    return np.random.default_rng([seed, 77]).integers(0, case["vocab"], n).astype(np.uint32)


def _requant(x, q):
    """a row quantized group by group the way LMRS activations are, and dequantized again"""
    g = x.reshape(*x.shape[:-1], -1, GROUP)
    if q == 1:
        s = g.abs().amax(-1, keepdim=True) / 127.0
        r = g / s
        v = torch.sign(r) * torch.floor(r.abs() + 0.5)
    else:
        s = g.abs().amax(-1, keepdim=True) / -8.0
        v = torch.floor(g / s + 8.5).clamp(0, 15) - 8.0
    return (v * s).reshape(x.shape)


def _lmrs_exact(case, seed, tokens, logits):
    """residual stream [T][dim] after the last layer, or the logits of the last token"""
    dim, ff, H, G, hs = SHAPES[case["shape"]]
    W, q, eps = _lmrs_weights(case, seed), case.get("q", 1), 1e-5
    t = torch.as_tensor(tokens.astype(np.int64), device=DEV)
    T = len(t)

    def mm(x, w):
        return _requant(x, q) @ _dequant(*w, q).T

    def norm(x, w):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()
    codes, scales = W["emb"][0]
    x = _dequant(codes[t], scales[t], q)
    f = 500000.0 ** (-torch.arange(0, hs, 2, device=DEV, dtype=torch.float64) / hs)
    wl = 2 * math.pi / f
    smooth = (8192.0 / wl - 1.0) / 3.0
    f = torch.where(wl > 8192.0, f / 32.0, torch.where(wl >= 2048.0, (1 - smooth) * f / 32.0 + smooth * f, f))
    ang = torch.arange(T, device=DEV, dtype=torch.float64)[:, None] * f[None]
    c, s = ang.cos()[:, None], ang.sin()[:, None]

    def rope(v):
        a, b = v[..., : hs // 2], v[..., hs // 2:]
        return torch.cat([a * c - b * s, a * s + b * c], -1)
    for i in range(case["layers"]):
        h = norm(x, W["rms_att"][i])
        qq, k, v = rope(mm(h, W["wq"][i]).view(T, H, hs)), rope(mm(h, W["wk"][i]).view(T, G, hs)), mm(h, W["wv"][i]).view(T, G, hs)
        x = x + mm(_attend(qq, k, v, hs ** -0.5, T).reshape(T, -1), W["wo"][i])
        h = norm(x, W["rms_post_att"][i])
        g = mm(h, W["w1"][i])
        x = x + mm(g * torch.sigmoid(g) * mm(h, W["w3"][i]), W["w2"][i])
    return mm(norm(x[-1:], W["rms_final"][0]), W["emb"][0])[0] if logits else x


def _attend(q, k, v, scale, T, softcap=0.0, window=0, keep=0, penalty=None, sink=None):
    """q [T][H][d], k / v [T][G][d] in 64 bits: causal softmax attention with the options the folder models use"""
    H, G = q.shape[1], k.shape[1]
    pos = torch.arange(T, device=q.device)
    dist = pos[:, None] - pos[None]
    vis = dist >= 0
    if window:
        vis &= (dist < window) | (pos[None] < keep)
    out = []
    for g in range(G):
        hs = slice(g * (H // G), (g + 1) * (H // G))
        s = torch.einsum("thd,nd->htn", q[:, hs], k[:, g]) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if penalty is not None:
            s = s - penalty[0][hs, None, None] * torch.log1p(penalty[1][hs, None, None] * dist.clamp(min=0).double())
        s = s.masked_fill(~vis, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[hs, None, None].expand(-1, T, 1)], -1)
        a = torch.softmax(s, -1)[..., :T]
        out.append(torch.einsum("htn,nd->thd", a, v[:, g]))
    return torch.cat(out, 1)


# ---- folder models ------------------------------------------------------------------------------------------------------------------------
def _genetar_config(case):
    w, ff, H, G, d = SHAPES[case["shape"]]
    layers = []
    for i in range(case["layers"]):
        m = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "softcap": 50.0, "v_mix": True}
        if i % 2:
            m["rot"] = {"base": 500000.0, "dims": d // 2, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
        layers.append({"type": "attention_2" if i % 2 else "attention", "mixer": m, "mlp": {"kind": "dense", "ff": ff}})
    return {"architecture": "Genetar", "width": w, "vocab": case["vocab"], "norm": {"eps": 1e-5}, "logit_scale": 1.0,
            "embedding": {"bigram": {"buckets": 1021, "mul_prev": 8191, "mul_cur": 127}}, "layers": layers}


def _genetar_tensors(cfg):
    w = cfg["width"]
    t = [("embed", (cfg["vocab"], w), "table"), ("bigram", (cfg["embedding"]["bigram"]["buckets"] + 1, w), "table")]
    for i, L in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", L["mixer"], L["mlp"]["ff"]
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        t += [(p + "norm1", (w,), "ones"), (p + "mix.q", (H * d, w), "matrix"), (p + "mix.k", (G * d, w), "matrix"), (p + "mix.v", (G * d, w), "matrix"),
              (p + "mix.vmix", (), "quarter"), (p + "mix.o", (w, H * d), "matrix"), (p + "ls1", (w,), "small"), (p + "mlp.gate", (ff, w), "matrix"),
              (p + "mlp.up", (ff, w), "matrix"), (p + "mlp.down", (w, ff), "matrix"), (p + "ls2", (w,), "small")]
        if L["type"] == "attention_2":
            t.append((p + "mix.g", (H, w), "matrix"))
    return t + [("final.norm", (w,), "ones"), ("head", (cfg["vocab"], w), "matrix")]


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _genetar_exact(cfg, W, tokens):
    eps, T = cfg["norm"]["eps"], len(tokens)
    bg = cfg["embedding"]["bigram"]
    t = [int(v) for v in tokens]
    rows = [bg["buckets"]] + [(t[i - 1] * bg["mul_prev"] + t[i] * bg["mul_cur"]) % bg["buckets"] for i in range(1, T)]
    x = W("embed")[t] + W("bigram")[rows]
    first = None
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.", L["mixer"]
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        h = _rms(x, eps) * W(p + "norm1")
        q, k, v = (h @ W(p + "mix.q").T).view(T, H, d), (h @ W(p + "mix.k").T).view(T, G, d), (h @ W(p + "mix.v").T).view(T, G, d)
        if L["type"] == "attention":
            q, k = _rms(q, eps), _rms(k, eps)
        else:
            r, sc = m["rot"], m["rot"]["scaling"]
            half = r["dims"] // 2
            f = r["base"] ** (-2.0 * torch.arange(half, device=DEV, dtype=torch.float64) / r["dims"])
            wl = 2 * math.pi / f
            s = (sc["original"] / wl - sc["low"]) / (sc["high"] - sc["low"])
            f = torch.where(wl > sc["original"] / sc["low"], f / sc["factor"], torch.where(wl < sc["original"] / sc["high"], f, (1 - s) * f / sc["factor"] + s * f))
            q, k = _rotate_halves(q, f), _rotate_halves(k, f)
        lam = W(p + "mix.vmix")
        if first is None:
            first = v
        else:
            v = (1 - lam) * v + lam * first
        o = _attend(q, k, v, m["scale"], T, softcap=m["softcap"])
        if L["type"] == "attention_2":
            o = o * torch.sigmoid(h @ W(p + "mix.g").T)[..., None]
        g = h @ W(p + "mlp.gate").T
        x = x + (o.reshape(T, -1) @ W(p + "mix.o").T) * W(p + "ls1") + ((g * torch.sigmoid(g) * (h @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T) * W(p + "ls2")
    return _rms(x, eps) * W("final.norm")


def _rotate_halves(z, f):
    T, half = z.shape[0], f.numel()
    ang = torch.arange(T, device=z.device, dtype=torch.float64)[:, None] * f[None]
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    u, w = z[..., :half], z[..., half:2 * half]
    return torch.cat([u * c - w * s, w * c + u * s, z[..., 2 * half:]], -1)


def _tudatar_config(case):
    w, ff, H, G, d = SHAPES[case["shape"]]
    kinds, layers = ("channel_delta", "attention", "latent_attention"), []
    mlp = {"kind": "moe", "expert": {"ff": ff // 8}, "router": {"experts": 16, "top": 4, "scale": 1.0}}
    for i in range(case["layers"]):
        kind = kinds[i % 3]
        if kind == "channel_delta":
            n = max(1, w // 128)
            m = {"heads": n, "kv_heads": n, "dim": 128, "vdim": 128, "conv": 4}
        elif kind == "attention":
            m = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": 1024}}
        else:
            m = {"heads": H, "dim": d, "rot_dim": 64, "vdim": d, "kv_rank": 256, "q_rank": 768, "scale": (d + 64) ** -0.5,
                 "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "fast": 32.0, "slow": 1.0, "original": 4096}}}
        layers.append({"type": kind, "mixer": m, "mlp": mlp})
    return {"architecture": "Tudatar", "width": w, "vocab": case["vocab"], "norm": {"eps": 1e-5}, "logit_scale": 1.0, "layers": layers}


def _tudatar_tensors(cfg):
    w = cfg["width"]

    def norm(n):
        return [(n, (w,), "ones"), (n + ".b", (w,), "shift"), (n + ".alpha", (), "half")]
    t = [("embed", (cfg["vocab"], w), "table")]
    for i, L in enumerate(cfg["layers"]):
        p, q, m = f"l{i}.", f"l{i}.mix.", L["mixer"]
        t += norm(p + "norm1") + norm(p + "norm1b") + norm(p + "norm2") + norm(p + "norm2b")
        H, d = m["heads"], m["dim"]
        if L["type"] == "channel_delta":
            for n in ("q", "k", "v"):
                t += [(q + n, (H * d, w), "matrix"), (q + n + ".conv", (H * d, m["conv"]), "conv")]
            t += [(q + "b", (H, w), "matrix"), (q + "A_log", (H,), "rate"), (q + "norm", (d,), "ones"), (q + "a1", (64, w), "matrix"),
                  (q + "a2", (H * d, 64), "matrix"), (q + "dt_bias", (H * d,), "shift"), (q + "g1", (64, w), "matrix"), (q + "g2", (H * d, 64), "matrix")]
        elif L["type"] == "attention":
            G = m["kv_heads"]
            for n, k in (("q", H), ("k", G), ("v", G)):
                t += [(q + n, (k * d, w), "matrix"), (q + n + ".b", (k * d,), "shift")]
            t += [(q + "q.norm", (H * d,), "ones"), (q + "k.norm", (G * d,), "ones"), (q + "r1", (H,), "small"), (q + "r2", (H,), "small")]
        else:
            rk, rq, dr = m["kv_rank"], m["q_rank"], m["rot_dim"]
            t += [(q + "dq", (rq, w), "matrix"), (q + "dq.norm", (rq,), "ones"), (q + "uq", (H * (d + dr), rq), "matrix"), (q + "dkv", (rk + dr, w), "matrix"),
                  (q + "dkv.norm", (rk,), "ones"), (q + "uk", (H * d, rk), "matrix"), (q + "uv", (H * d, rk), "matrix")]
        t.append((q + "o", (w, H * d), "matrix"))
        f = L["mlp"]
        t += [(p + "mlp.router", (16, w), "matrix"), (p + "mlp.correction", (16,), "shift")]
        for e in range(16):
            b = f"{p}mlp.e{e}."
            t += [(b + "gate", (f["expert"]["ff"], w), "matrix"), (b + "up", (f["expert"]["ff"], w), "matrix"), (b + "down", (w, f["expert"]["ff"]), "matrix")]
    return t + norm("final.norm") + [("head", (cfg["vocab"], w), "matrix")]


def _causal_conv(x, w, bias=None):
    """depth-wise over the last taps rows, the last column of w on the current one"""
    taps, T = w.shape[1], x.shape[0]
    full = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x], 0)
    y = sum(full[j:j + T] * w[:, j] for j in range(taps))
    return y if bias is None else y + bias


def _silu(z):
    return z * torch.sigmoid(z)


def _tudatar_exact(cfg, W, tokens):
    eps, T = cfg["norm"]["eps"], len(tokens)

    def norm(v, n):
        return torch.tanh(W(n + ".alpha") * v) * W(n) + W(n + ".b")
    x = W("embed")[[int(v) for v in tokens]]
    for i, L in enumerate(cfg["layers"]):
        p, q_, m = f"l{i}.", f"l{i}.mix.", L["mixer"]
        H, d = m["heads"], m["dim"]
        h = norm(x, p + "norm1")
        if L["type"] == "channel_delta":
            q, k, v = (_silu(_causal_conv(h @ W(q_ + n).T, W(q_ + n + ".conv"))).view(T, H, d) for n in ("q", "k", "v"))
            q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            q = q * d ** -0.5
            beta = torch.sigmoid(h @ W(q_ + "b").T)
            a = ((h @ W(q_ + "a1").T) @ W(q_ + "a2").T + W(q_ + "dt_bias")).view(T, H, d)
            g = torch.exp(-torch.exp(W(q_ + "A_log"))[None, :, None] * torch.nn.functional.softplus(a, threshold=50.0))
            S, o = x.new_zeros(H, d, d), x.new_zeros(T, H, d)
            for t in range(T):
                S = S * g[t][..., None]
                u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
                S = S + k[t][..., None] * u[:, None]
                o[t] = torch.einsum("hkv,hk->hv", S, q[t])
            gate = torch.sigmoid((h @ W(q_ + "g1").T) @ W(q_ + "g2").T).view(T, H, d)
            o = _rms(o, eps) * W(q_ + "norm") * gate
        elif L["type"] == "attention":
            G = m["kv_heads"]
            q = (_rms(h @ W(q_ + "q").T + W(q_ + "q.b"), eps) * W(q_ + "q.norm")).view(T, H, d)
            k = (_rms(h @ W(q_ + "k").T + W(q_ + "k.b"), eps) * W(q_ + "k.norm")).view(T, G, d)
            v = _rms((h @ W(q_ + "v").T + W(q_ + "v.b")).view(T, G, d), eps)
            o = _attend(q, k, v, m["scale"], T, window=m["mask"]["size"], penalty=(W(q_ + "r1"), W(q_ + "r2")))
        else:
            rk, dr, r = m["kv_rank"], m["rot_dim"], m["rot"]
            sc = r["scaling"]

            def where(turns):
                return dr * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(r["base"]))
            lo, hi = max(math.floor(where(sc["fast"])), 0), min(math.ceil(where(sc["slow"])), dr - 1)
            n = torch.arange(dr // 2, device=DEV, dtype=torch.float64)
            f, ramp = r["base"] ** (-2 * n / dr), ((n - lo) / max(hi - lo, 0.001)).clamp(0, 1)
            ang = torch.arange(T, device=DEV, dtype=torch.float64)[:, None] * (f / sc["factor"] * ramp + f * (1 - ramp))[None]
            mult = 0.1 * math.log(sc["factor"]) + 1.0
            c, s = (ang.cos() * mult)[:, None], (ang.sin() * mult)[:, None]

            def rot(z):
                u, w = z[..., 0::2], z[..., 1::2]
                return torch.stack([u * c - w * s, w * c + u * s], -1).flatten(-2)
            qq = ((_rms(h @ W(q_ + "dq").T, eps) * W(q_ + "dq.norm")) @ W(q_ + "uq").T).view(T, H, d + dr)
            ckr = h @ W(q_ + "dkv").T
            lat = _rms(ckr[:, :rk], eps) * W(q_ + "dkv.norm")
            kr = rot(ckr[:, None, rk:]).expand(T, H, dr)
            q = torch.cat([qq[..., :d], rot(qq[..., d:])], -1)
            k = torch.cat([(lat @ W(q_ + "uk").T).view(T, H, d), kr], -1)
            o = _attend(q, k, (lat @ W(q_ + "uv").T).view(T, H, d), m["scale"], T)
        x = x + norm(o.reshape(T, -1) @ W(q_ + "o").T, p + "norm1b")
        x = x + norm(_routed(norm(x, p + "norm2"), W, p + "mlp.", L["mlp"]), p + "norm2b")
    return norm(x, "final.norm")


def _routed(h, W, p, f):
    """Tudatar: sigmoid router, choice with a correction, SiLU GLU experts.  Rupenex: softmax router with identity experts, squared
    ReLU experts and a shared one."""
    r = f["router"]
    E, top, rup = r["experts"], r["top"], "identity" in r
    z = h @ W(p + "router").T
    s = torch.softmax(z, -1) if rup else torch.sigmoid(z)
    idx = torch.topk(s + W(p + "correction"), top, dim=-1).indices
    w = torch.zeros_like(s).scatter(1, idx, s.gather(1, idx))
    w = w / (w.sum(-1, keepdim=True) + 1e-20) * r.get("scale", 1.0)

    def expert(v, b):
        if rup:
            return torch.relu(v @ W(b + "up").T) ** 2 @ W(b + "down").T
        return (_silu(v @ W(b + "gate").T) * (v @ W(b + "up").T)) @ W(b + "down").T
    y = expert(h, p + "shared.") if rup else torch.zeros_like(h)
    for e in range(E):
        t = (w[:, e] > 0).nonzero()[:, 0]
        if t.numel():
            y[t] += w[t, e, None] * expert(h[t], f"{p}e{e}.")
    return y + w[:, E:].sum(-1, keepdim=True) * h if rup else y


def _rupenex_config(case):
    w, ff, H, G, d = SHAPES[case["shape"]]
    layers = []
    for i in range(case["layers"]):
        if i % 2 == 0:
            layers.append({"type": "mamba2", "mixer": {"heads": 2 * w // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8},
                           "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}})
        else:
            layers.append({"type": "attention",
                           "mixer": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": 1024, "keep_first": 4},
                                     "rot": {"base": 500000.0, "dims": d, "scaling": {"factor": 8.0}}},
                           "mlp": {"kind": "moe", "expert": {"ff": ff // 4}, "router": {"experts": 16, "identity": 2, "top": 4}, "shared": {"ff": ff // 2}}})
    return {"architecture": "Rupenex", "width": w, "vocab": case["vocab"], "norm": {"eps": 1e-5}, "logit_scale": 1.0, "layers": layers}


def _rupenex_tensors(cfg):
    w = cfg["width"]
    t = [("embed", (cfg["vocab"], w), "table"), ("embed.norm", (w,), "ones")]
    for i, L in enumerate(cfg["layers"]):
        p, q, m, f = f"l{i}.", f"l{i}.mix.", L["mixer"], L["mlp"]
        H = m["heads"]
        t += [(p + "norm1", (w,), "ones"), (p + "ls1", (w,), "small"), (p + "norm2", (w,), "ones"), (p + "ls2", (w,), "small")]
        if L["type"] == "attention":
            G, d = m["kv_heads"], m["dim"]
            t += [(q + "q", (H * d, w), "matrix"), (q + "k", (G * d, w), "matrix"), (q + "v", (G * d, w), "matrix"), (q + "q.norm", (d,), "ones"),
                  (q + "k.norm", (d,), "ones"), (q + "sink", (H,), "shift"), (q + "g", (H * d, w), "matrix"), (q + "o", (w, H * d), "matrix")]
        else:
            inner, gn = H * m["vdim"], m["groups"] * m["state"]
            t += [(q + "in", (2 * inner + 2 * gn + H, w), "matrix"), (q + "conv", (inner + 2 * gn, m["conv"]), "conv"), (q + "conv.b", (inner + 2 * gn,), "shift"),
                  (q + "dt_bias", (H,), "shift"), (q + "A_log", (H,), "rate"), (q + "D", (H,), "ones"), (q + "norm", (inner,), "ones"), (q + "o", (w, inner), "matrix")]
        if f["kind"] == "dense":
            t += [(p + "mlp.gate", (f["ff"], w), "matrix"), (p + "mlp.up", (f["ff"], w), "matrix"), (p + "mlp.down", (w, f["ff"]), "matrix")]
        else:
            n = f["router"]["experts"] + f["router"]["identity"]
            t += [(p + "mlp.router", (n, w), "matrix"), (p + "mlp.correction", (n,), "tenth")]
            for b, ff in [(f"e{e}.", f["expert"]["ff"]) for e in range(f["router"]["experts"])] + [("shared.", f["shared"]["ff"])]:
                t += [(p + "mlp." + b + "up", (ff, w), "matrix"), (p + "mlp." + b + "down", (w, ff), "matrix")]
    return t + [("final.norm", (w,), "ones"), ("head", (cfg["vocab"], w), "matrix")]


def _rupenex_exact(cfg, W, tokens):
    eps, T = cfg["norm"]["eps"], len(tokens)

    def norm(v, n):
        c = v - v.mean(-1, keepdim=True)
        return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps) * W(n)
    x = norm(W("embed")[[int(v) for v in tokens]], "embed.norm")
    for i, L in enumerate(cfg["layers"]):
        p, q_, m, f = f"l{i}.", f"l{i}.mix.", L["mixer"], L["mlp"]
        H = m["heads"]
        if L["type"] == "attention":
            G, d, r = m["kv_heads"], m["dim"], m["rot"]
            fr = r["base"] ** (-2.0 * torch.arange(r["dims"] // 2, device=DEV, dtype=torch.float64) / r["dims"]) / r["scaling"]["factor"]
            q = _rotate_halves(_rms((x @ W(q_ + "q").T).view(T, H, d), eps) * W(q_ + "q.norm"), fr)
            k = _rotate_halves(_rms((x @ W(q_ + "k").T).view(T, G, d), eps) * W(q_ + "k.norm"), fr)
            o = _attend(q, k, (x @ W(q_ + "v").T).view(T, G, d), m["scale"], T, window=m["mask"]["size"], keep=m["mask"]["keep_first"], sink=W(q_ + "sink"))
            y = (o.reshape(T, -1) * torch.sigmoid(x @ W(q_ + "g").T)) @ W(q_ + "o").T
        else:
            P, N, G = m["vdim"], m["state"], m["groups"]
            inner = H * P
            z, xbc, dt = (x @ W(q_ + "in").T).split([inner, inner + 2 * G * N, H], -1)
            xs, B, C = _silu(_causal_conv(xbc, W(q_ + "conv"), W(q_ + "conv.b"))).split([inner, G * N, G * N], -1)
            xs = xs.reshape(T, H, P)
            B, C = (v.reshape(T, G, 1, N).expand(T, G, H // G, N).reshape(T, H, N) for v in (B, C))
            dt = torch.nn.functional.softplus(dt + W(q_ + "dt_bias"), threshold=50.0)
            decay = torch.exp(-torch.exp(W(q_ + "A_log")) * dt)
            S, o = x.new_zeros(H, N, P), x.new_zeros(T, H, P)
            for t in range(T):
                S = S * decay[t][:, None, None] + (dt[t][:, None] * B[t])[..., None] * xs[t][:, None]
                o[t] = torch.einsum("hnp,hn->hp", S, C[t])
            o = (o + W(q_ + "D")[:, None] * xs).reshape(T, inner) * _silu(z)
            y = (_rms(o.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * W(q_ + "norm")) @ W(q_ + "o").T
        x = x + W(p + "ls1") * norm(y, p + "norm1")
        if f["kind"] == "dense":
            g, u = (x @ W(p + "mlp.gate").T).clamp(max=f["limit"]), (x @ W(p + "mlp.up").T).clamp(-f["limit"], f["limit"])
            y = (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W(p + "mlp.down").T
        else:
            y = _routed(x, W, p + "mlp.", f)
        x = x + W(p + "ls2") * norm(y, p + "norm2")
    return norm(x, "final.norm")


ARCH = {"genetar": (_genetar_config, _genetar_tensors, _genetar_exact), "tudatar": (_tudatar_config, _tudatar_tensors, _tudatar_exact),
        "rupenex": (_rupenex_config, _rupenex_tensors, _rupenex_exact)}
# mean and deviation of the weights that are not matrices
KINDS = {"table": (0.0, 1.0), "ones": (1.0, 0.1), "small": (0.3, 0.05), "shift": (0.0, 0.1), "tenth": (0.0, 0.05), "conv": (0.0, 0.5), "rate": (-1.0, 0.5),
         "quarter": (0.25, 0.0), "half": (0.5, 0.0)}


def _tensor(name, shape, kind, seed):
    """one bf16 weight tensor, from the seed and its name alone"""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed * 1000003 + sum((i + 1) * ord(ch) for i, ch in enumerate(name)))
    mean, dev = (0.0, shape[-1] ** -0.5) if kind == "matrix" else KINDS[kind]
    return (mean + dev * torch.randn(shape, generator=gen, device=DEV)).to(torch.bfloat16)


def _open_folder(case, seed):
    make_config, tensors, _ = ARCH[case["arch"]]
    cfg = make_config(case)
    table = tensors(cfg)
    header, off = {}, 0
    for name, shape, _k in table:
        n = 2 * math.prod(shape)
        header[name] = {"dtype": "BF16", "shape": list(shape), "data_offsets": [off, off + n]}
        off += n
    hj = json.dumps(header).encode()
    hj += b" " * (-len(hj) % 8)
    folder = tempfile.mkdtemp(prefix="lmrs_case_", dir="/dev/shm" if os.access("/dev/shm", os.W_OK) else None)
    try:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(cfg, f)
        with open(os.path.join(folder, "model.safetensors"), "wb") as f:
            f.write(struct.pack("<Q", len(hj)) + hj)
            for name, shape, kind in table:
                f.write(_tensor(name, shape, kind, seed).reshape(-1).view(torch.uint8).cpu().numpy())
        return lmrs_b200.Transformer.open(folder, dtype=case["dtype"], max_tokens=max(64, _positions(case)))
    finally:
        shutil.rmtree(folder, ignore_errors=True)


def _positions(case):
    return case["pos"] + 3 if "pos" in case else case["tokens"]


def _folder_exact(case, seed, tokens, rows):
    make_config, tensors, forward = ARCH[case["arch"]]
    cfg = make_config(case)
    table = {n: (s, k) for n, s, k in tensors(cfg)}

    def W(name):
        return _tensor(name, *table[name], seed).double()
    return forward(cfg, W, tokens)[-rows:] @ W("head").T


# ---- the interface ------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        q, n, o = case["q"], case["n"], case["o"]
        wc, ws = _quant_codes(gen, o, n, q, n ** -0.5)
        xc, xs = _quant_codes(gen, case["rows"], n, q, 1.0)

        def host(c, s):
            return quantization.QuantizedTensor(_pack(c, q).cpu().numpy().view(np.int8 if q == 1 else np.uint8), s.reshape(-1).cpu().numpy())
        return dict(w=functional.ResidentWeights(host(wc, ws), n, o, GROUP, q), x=host(xc, xs), out=np.zeros(case["rows"] * o, np.float32))
    if kind in ("lmrs_decode", "lmrs_prefill"):
        m, _ = lmrs_b200.Transformer.new(_lmrs_file(case, seed))
        if kind == "lmrs_prefill":
            return dict(m=m, tokens=_tokens(case, seed, case["tokens"]))
        p, t = case["pos"], _tokens(case, seed, case["pos"] + 1)
        m.fill_kv_cache(m.get_embeddings(t[:p]), 0)
        return dict(m=m, token=int(t[p]), pos=p)
    m = _open_folder(case, seed)
    if kind == "folder_prefill":
        n = case["tokens"]
        return dict(m=m, tokens=_tokens(case, seed, n), want=np.arange(n - case["rows"], n, dtype=np.uint32))
    if kind == "folder_replay":
        return dict(m=m, tokens=_tokens(case, seed, case["tokens"]))
    p, t = case["pos"], _tokens(case, seed, case["pos"] + 3)
    m.forward_tokens(t[:p], 0)
    for i in (p, p + 1):   # a generation that is under way
        m.forward(int(t[i]), i)
    return dict(m=m, token=int(t[p + 2]), pos=p + 2)


class _Logits(np.ndarray):
    """a model's own logits buffer, which lives as long as the model"""
    model = None


def _forward(m, token, pos):
    logits = m.forward(token, pos).view(_Logits)
    logits.model = m
    return logits


def run(state):
    if "w" in state:
        state["w"].matmul(state["out"], state["x"])
        return state["out"]
    m = state["m"]
    if "pos" in state:
        return _forward(m, state["token"], state["pos"])
    if "want" in state:
        return m.forward_tokens(state["tokens"], 0, state["want"])
    if m.args.q_type:
        emb = m.get_embeddings(state["tokens"])
        m.fill_kv_cache(emb, 0)
        return emb
    t = state["tokens"]
    for i in range(len(t) - 1):
        m.forward_device(int(t[i]), i)
    return _forward(m, int(t[-1]), len(t) - 1)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        r, n, o = case["rows"], case["n"], case["o"]
        per = (1.0 if case["q"] == 1 else 0.5) + 4.0 / GROUP
        return {"bytes": int((r * n + o * n) * per + 4 * r * o), "flops": 2 * r * n * o}
    w, ff, H, G, d = SHAPES[case["shape"]]
    L, vocab = case["layers"], case["vocab"]
    if kind in ("lmrs_decode", "lmrs_prefill"):
        per = (1.0 if case.get("q", 1) == 1 else 0.5) + 4.0 / GROUP
        mats = L * (w * (2 * H + 2 * G) * d + 3 * w * ff)
        if kind == "lmrs_decode":
            n = case["pos"] + 1
            return {"bytes": int((mats + vocab * w) * per + L * n * G * d * 8 + 4 * vocab), "flops": 2 * (mats + vocab * w) + 4 * L * H * d * n}
        n = case["tokens"]
        return {"bytes": int(mats * per + 8 * n * w), "flops": 2 * mats * n + 2 * L * H * d * n * (n + 1)}
    cfg = ARCH[case["arch"]][0](case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    steps = case["tokens"] if kind == "folder_replay" else 1
    n = 1 if kind != "folder_prefill" else case["tokens"]   # tokens a step
    ctx = case["pos"] + 3 if kind == "folder_decode" else n
    head = [(name, shape) for name, shape, k in ARCH[case["arch"]][1](cfg) if name == "head"][0][1]
    nbytes, flops = head[0] * head[1] * size + 4 * vocab * case.get("rows", 1), 2 * case.get("rows", 1) * head[0] * head[1]
    if kind == "folder_replay":
        flops, nbytes = flops / steps, nbytes / steps   # only the last step's logits are asked for
    for name, shape, k in ARCH[case["arch"]][1](cfg):
        if k != "matrix" or name == "head":
            continue
        share = 1.0   # of the rows that meet this matrix
        if ".mlp.e" in name:
            r = cfg["layers"][int(name[1:name.index(".")])]["mlp"]["router"]
            share = r["top"] / (r["experts"] + r.get("identity", 0))
        nbytes += math.prod(shape) * size * min(1.0, n * share)
        flops += 2 * math.prod(shape) * share * n
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] in ("channel_delta", "mamba2"):
            flops += 6 * m["heads"] * m.get("state", m["dim"] if "dim" in m else 0) * m["vdim"] * n
            nbytes += 8 * m["heads"] * m.get("state", m["dim"] if "dim" in m else 0) * m["vdim"]
        else:
            pairs = ctx * n - n * (n - 1) / 2
            flops += 2 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]) * pairs
            nbytes += 4 * ctx * ((m["kv_rank"] + m["rot_dim"]) if "kv_rank" in m else m["kv_heads"] * (m["dim"] + m["vdim"]))
    return {"bytes": int(nbytes * steps), "flops": int(flops * steps)}


def tolerance(case):
    if case["kind"] in ("linear", "lmrs_decode", "lmrs_prefill"):
        return "exact"   # the quantized path keeps the CPU arithmetic's order of operations bit for bit
    if case["dtype"] == "float32":
        return {"rel": 4e-6}   # seen against 64 bits: 0.9e-6
    # seen against 64 bits: 1.8e-3 to 2.2e-3 (bf16 operands, rounded once per product).  Routed experts: two scores that are closer than
    # that rounding may change places (about one decision in 200), which moves that token's row by 10 to 20 percent: one of 32 rows
    return {"rel": 8e-3 if case["arch"] == "genetar" else 4e-2}


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        q, n, o = case["q"], case["n"], case["o"]
        w, x = _quant_codes(gen, o, n, q, n ** -0.5), _quant_codes(gen, case["rows"], n, q, 1.0)
        return (_dequant(*x, q) @ _dequant(*w, q).T).reshape(-1).cpu().numpy()
    if kind == "lmrs_decode":
        return _lmrs_exact(case, seed, _tokens(case, seed, case["pos"] + 1), True).cpu().numpy()
    if kind == "lmrs_prefill":
        return _lmrs_exact(case, seed, _tokens(case, seed, case["tokens"]), False).reshape(-1).cpu().numpy()
    if kind == "folder_prefill":
        return _folder_exact(case, seed, _tokens(case, seed, case["tokens"]), case["rows"]).cpu().numpy()
    return _folder_exact(case, seed, _tokens(case, seed, _positions(case)), 1)[0].cpu().numpy()
