"""The work that this framework is measured on: single-stream decode steps and prompt batches of GGUF LLaMA models, prompts and short
requests of layer-stack models, all through booster_b200.engine as a program calls it (Model, Context, decode, decode_rows).

Models are synthetic (booster_b200.gguf_io / stack_io write them), with the layer shapes of the configurations that the repository
names. Depth and vocabulary of the 8B-class models are cut to a quarter together, so that layers and head keep their shares of a
token. A model is loaded once in a process, as a server loads it, and every prepared state is a context of its own on it, with the
tokens and the cached rows that the seed gives.

`exact` is the same model in 64 bits from the file's weights, in plain torch. The LLaMA path's data types are part of it: a product's
activations are 8-bit blocks there, and cached rows 16 bits. A value that falls on the other side of a rounding step in 64 bits moves all that follows by
as much as that step, so a whole model's logits agree to a few percent and not better.
"""
from __future__ import annotations

import json
import math
import os
import shutil
import struct
import tempfile

import numpy as np
import torch

from booster_b200 import engine, gguf_io, stack_io

# LLaMA layer shapes: name -> configuration. "8b" and "mistral" are an 8B and a 7B model at a quarter of their depth and (8b) vocabulary, "70b"
# two layers of a 70B model, "tiny" is the small test model.
LLAMA = {
    "8b": dict(n_layer=8, n_vocab=32064, rope_freq_base=500000.0),
    "mistral": dict(n_layer=8, n_vocab=8000, rope_freq_base=10000.0, n_ctx_train=32768),
    "70b": dict(n_layer=2, n_embd=8192, n_head=64, n_head_kv=8, n_ff=28672, n_vocab=8192),
    "tiny": dict(n_layer=3, n_embd=512, n_head=4, n_head_kv=1, n_ff=768, n_vocab=512, n_ctx_train=512),
}
STACK = {"matulorn": stack_io.matulorn_config, "bozisun": stack_io.bozisun_config}


def listed():
    return [
        # one generated token of a chat in the middle of its context: the headline workload
        dict(name="decode-8b-q4km-at-2000", path="llama", shape="8b", ftype="Q4_K_M", past=2000, tokens=1),
        # one generated token early in a conversation, the 8-bit file type
        dict(name="decode-8b-q8_0-at-333", path="llama", shape="8b", ftype="Q8_0", past=333, tokens=1),
        # one generated token at the end of an 8k context
        dict(name="decode-mistral-q5km-at-8123", path="llama", shape="mistral", ftype="Q5_K_M", past=8123, tokens=1),
        # the smallest call: a toy model's token, nothing but launches
        dict(name="decode-tiny-q4km-at-100", path="llama", shape="tiny", ftype="Q4_K_M", past=100, tokens=1),
        # a full prompt batch
        dict(name="prompt-8b-q4km-512", path="llama", shape="8b", ftype="Q4_K_M", past=0, tokens=512),
        # the next user turn of a chat: a short, ragged batch behind a conversation
        dict(name="prompt-8b-q4km-77-at-1234", path="llama", shape="8b", ftype="Q4_K_M", past=1234, tokens=77),
        # a full prompt batch of the 8-bit file type
        dict(name="prompt-8b-q8_0-512", path="llama", shape="8b", ftype="Q8_0", past=0, tokens=512),
        # a late batch of a long document
        dict(name="prompt-mistral-q5km-512-at-6000", path="llama", shape="mistral", ftype="Q5_K_M", past=6000, tokens=512),
        # layer stacks: a long prompt scored at eight places
        dict(name="stack-matulorn-prompt-2048", path="stack", design="matulorn", width=2048, dtype="bfloat16", tokens=2048, steps=0),
        # a short request: a question, then the answer token by token
        dict(name="stack-matulorn-request-64-32", path="stack", design="matulorn", width=2048, dtype="bfloat16", tokens=64, steps=32),
        # a ragged prompt through grouped attention and a routed mixture, and the first tokens after it
        dict(name="stack-bozisun-prompt-701-8", path="stack", design="bozisun", width=2048, dtype="bfloat16", tokens=701, steps=8),
        # the 32-bit mode, as used to check a model
        dict(name="stack-matulorn-f32-300-4", path="stack", design="matulorn", width=1024, dtype="float32", tokens=300, steps=4),
    ]


def _spread(rng, lo, hi):
    """a whole number from lo to hi, spread over its logarithm"""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    if rng.random() < 2.0 / 3.0:
        shape = rng.choice(["8b", "8b", "mistral", "70b", "tiny"])
        room = {"8b": 4096, "mistral": 8192, "70b": 4096, "tiny": 500}[shape]
        ftype = rng.choice(["Q4_K_M", "Q5_K_M", "Q8_0"])
        tokens = 1 if rng.random() < 0.4 else _spread(rng, 2, 512 if room > 512 else 100)
        past = _spread(rng, 1, room - tokens - 1) - 1
        return dict(path="llama", shape=shape, ftype=ftype, past=past, tokens=tokens)
    design = rng.choice(sorted(STACK))
    dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
    width = rng.choice([512, 1024, 2048] if dtype == "bfloat16" else [512, 1024])
    return dict(path="stack", design=design, width=width, dtype=dtype, tokens=_spread(rng, 5, 2048 if dtype == "bfloat16" else 600), steps=rng.randrange(0, 17))


# ---- models ------------------------------------------------------------------------------------------------------------------
def _llama_config(case):
    return gguf_io.LlamaConfig(name="synthetic-" + case["shape"], **LLAMA[case["shape"]])


def _stack_config(case):
    w = case["width"]
    if case["design"] == "matulorn":
        return stack_io.matulorn_config(w, 4, 4 * w, max(2, w // 128), vocab=16000, kv_rank=min(512, w // 2), groups=8)
    return stack_io.bozisun_config(w, 4, 4 * w, max(2, w // 128), vocab=16000, buckets=4093)


def _model_key(case):
    return tuple((k, case[k]) for k in ("path", "shape", "ftype", "design", "width", "dtype") if k in case)


def _write_model(case, folder):
    if case["path"] == "llama":
        path = os.path.join(folder, "model.gguf")
        gguf_io.synth_llama(path, _llama_config(case), case["ftype"], seed=20, share_period=2)
        return path
    path = os.path.join(folder, "model")
    stack_io.synth_stack(path, _stack_config(case), seed=20)
    return path


_models = {}


def _model(case):
    key = _model_key(case)
    if key not in _models:
        folder = tempfile.mkdtemp(prefix="cases_")
        try:
            path = _write_model(case, folder)
            _models[key] = engine.Model(path) if case["path"] == "llama" else engine.Model(path, dtype=case["dtype"])
        finally:
            shutil.rmtree(folder)
    return _models[key]


class _Context(engine.Context):
    """a context that is given back with the state that holds it"""

    def __del__(self):
        if getattr(self, "h", None):
            self.close()


def _tokens(case, seed):
    n = case["tokens"] + case.get("steps", 0)
    vocab = LLAMA[case["shape"]]["n_vocab"] if case["path"] == "llama" else 16000
    return np.random.default_rng([seed, 1]).integers(0, vocab, size=n).astype(np.int32)


def _cached_rows(case, seed, layer, device):
    """the rows of earlier positions in one layer's cache: [past, kv heads * head dim] f16, keys and values"""
    c = _llama_config(case)
    g = torch.Generator(device=device).manual_seed(1000003 * seed + layer)
    kv = torch.randn((2, case["past"], c.n_head_kv * c.head_dim), generator=g, device=device, dtype=torch.float32)
    return kv.half()


def prepare(case, seed):
    model = _model(case)
    tokens = _tokens(case, seed)
    if case["path"] == "llama":
        need = case["past"] + case["tokens"]
        ctx = _Context(model, (need + 255) // 256 * 256)
        if case["past"]:
            for layer in range(model.n_layer):
                kv = _cached_rows(case, seed, layer, "cuda").cpu().numpy()
                ctx.kv_write(layer, 0, kv[0], kv[1])
        return dict(kind="llama", ctx=ctx, tokens=tokens, past=case["past"])
    ctx = _Context(model, (len(tokens) + 63) // 64 * 64)
    return dict(kind="stack", ctx=ctx, prompt=tokens[:case["tokens"]], answer=[tokens[case["tokens"] + i:][:1] for i in range(case["steps"])], rows=_rows(case))


def _rows(case):
    """places of a stack's prompt whose logits are wanted: eight along it when it is scored, the last when it is answered"""
    n = case["tokens"]
    return [n - 1] if case["steps"] else sorted({n * (i + 1) // 8 - 1 for i in range(8)} - {-1})


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "llama":
        return ctx.decode(state["tokens"], state["past"])
    ctx.kv_clear()
    out = [ctx.decode_rows(state["prompt"], 0, state["rows"])]
    pos = len(state["prompt"])
    for token in state["answer"]:
        out.append(ctx.decode(token, pos))
        pos += 1
    return [out[0], np.stack(out[1:])] if len(out) > 1 else out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------
def work(case):
    if case["path"] == "llama":
        c, T, past = _llama_config(case), case["tokens"], case["past"]
        attended = T * past + T * (T + 1) // 2
        per_layer = 2 * c.n_embd * c.n_embd + 2 * c.n_embd * c.n_head_kv * c.head_dim + 3 * c.n_embd * c.n_ff
        return {"bytes": gguf_io.weight_bytes_per_token(c, case["ftype"]) + gguf_io.kv_bytes_per_token(c, past + T) + 4 * c.n_vocab + 4 * T,
                "flops": 2 * T * c.n_layer * per_layer + 2 * c.n_embd * c.n_vocab + 4 * c.n_layer * c.n_head * c.head_dim * attended}
    cfg, T, steps = _stack_config(case), case["tokens"], case["steps"]
    size = 2 if case["dtype"] == "bfloat16" else 4
    order = list(range(len(cfg["layers"])))
    if cfg.get("loop"):
        lp = cfg["loop"]
        order = order[:lp["start"]] + order[lp["start"]:lp["stop"]] * lp["times"] + order[lp["stop"]:]
    shapes = stack_io.tensor_shapes(cfg)
    head = cfg["vocab"] * cfg["width"]
    every = used = 0                                    # a layer pass's matrix entries: all of them, and those one token meets
    for i in order:
        mlp = cfg["layers"][i].get("mlp") or {}
        for name, shp in shapes.items():
            if name.startswith(f"l{i}.") and len(shp) == 2 and not name.endswith(".conv"):
                n = shp[0] * shp[1]
                every += n
                used += n * mlp["router"]["top"] / mlp["router"]["experts"] if f"l{i}.mlp.e" in name else n
    rows = len(_rows(case))
    hit = every if T >= 64 else min(every, used * T)
    attention = 0
    for i in order:
        mx = cfg["layers"][i]["mixer"]
        if cfg["layers"][i]["type"] in ("latent_attention", "attention"):
            window = (mx.get("mask") or {}).get("size", T + steps)
            keys = sum(min(p + 1, window) for p in range(T + steps))
            attention += 2 * mx["heads"] * keys * ((2 * mx["kv_rank"] + mx["rot_dim"]) if "kv_rank" in mx else mx["dim"] + mx["vdim"])
    return {"bytes": size * (hit + head + steps * (used + head)) + 4 * cfg["vocab"] * (rows + steps),
            "flops": 2 * used * (T + steps) + 2 * head * (rows + steps) + attention}


def tolerance(case):
    # The LLaMA path promises the CPU implementation's bits: every variant of its kernels gives the same ones.
    if case["path"] == "llama":
        return "exact"
    # Layer stacks: seen against 64 bits are up to 6e-3 (bfloat16 products) and 2.4e-6 (float32); four times that.
    return {"rel": 2.4e-2} if case["dtype"] == "bfloat16" else {"rel": 1e-5}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------------
def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    folder = tempfile.mkdtemp(prefix="cases_")
    try:
        path = _write_model(case, folder)
        with torch.no_grad():
            if case["path"] == "llama":
                return _llama_exact(case, seed, path, device)
            return _stack_exact(case, seed, path, device)
    finally:
        shutil.rmtree(folder)


D = torch.float64


def _f16(raw, at):
    return raw[:, at:at + 2].contiguous().view(torch.float16).to(D)


def _six_bit(s):
    """the eight 6-bit scales and minimums of a 12-byte field [n, 12]"""
    s = s.to(torch.int32)
    sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | (s[:, 0:4] >> 6 << 4)], 1)
    mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | (s[:, 4:8] >> 6 << 4)], 1)
    return sc.to(D), mn.to(D)


def _dequantized(t, device):
    """a GGUF tensor's weights [rows, k]"""
    k, rows = t.ne[0], (t.ne[1] if len(t.ne) > 1 else 1)
    raw = torch.from_numpy(np.array(t.data)).to(device)
    if t.type == gguf_io.F32:
        return raw.view(torch.float32).to(D).reshape(rows, k)
    raw = raw.reshape(-1, gguf_io.BLOCK[t.type][1])
    if t.type == gguf_io.Q8_0:
        return (raw[:, 2:].contiguous().view(torch.int8).to(D) * _f16(raw, 0)).reshape(rows, k)
    if t.type in (gguf_io.Q4_K, gguf_io.Q5_K):
        sc, mn = _six_bit(raw[:, 4:16])
        qs = raw[:, -128:].reshape(-1, 4, 1, 32)
        q = torch.cat([qs & 15, qs >> 4], 2).reshape(-1, 8, 32).to(D)
        if t.type == gguf_io.Q5_K:
            bit = torch.arange(8, device=device, dtype=torch.uint8).reshape(1, 8, 1)
            q += 16.0 * ((raw[:, None, 16:48] >> bit) & 1).to(D)
        return ((_f16(raw, 0) * sc)[:, :, None] * q - (_f16(raw, 2) * mn)[:, :, None]).reshape(rows, k)
    if t.type == gguf_io.Q6_K:
        ql, qh = raw[:, :128].reshape(-1, 2, 2, 32), raw[:, 128:192].reshape(-1, 2, 1, 32)
        shift = torch.tensor([0, 2, 4, 6], device=device, dtype=torch.uint8).reshape(1, 1, 4, 1)
        q = (torch.cat([ql & 15, ql >> 4], 2) | (((qh >> shift) & 3) << 4)).reshape(-1, 16, 16).to(D) - 32.0
        sc = raw[:, 192:208].contiguous().view(torch.int8).to(D)
        return ((_f16(raw, 208) * sc)[:, :, None] * q).reshape(rows, k)
    raise ValueError(t.type)


def _eight_bit(x, ftype):
    """activations as a product takes them: blocks of 8-bit values, 32 with a 16-bit scale (Q8_0) or 256 with a 32-bit one (the K types)"""
    n = 32 if ftype == "Q8_0" else 256
    b = x.reshape(-1, n)
    if n == 32:
        d = b.abs().amax(1, keepdim=True) / 127.0
        q = torch.where(d > 0, torch.round(b / d), 0.0)
        return (q * d.half().to(D)).reshape(x.shape)
    top = b.gather(1, b.abs().argmax(1, keepdim=True))
    q = torch.where(top != 0, torch.round(b * (-127.0 / top)).clamp(max=127.0), 0.0)
    return (q * (top / -127.0)).reshape(x.shape)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, first, window=None, sink=None):
    """q [T, heads, D] at positions first.., k, v [n, kv heads, D]: causal soft-max attention -> [T, heads, D of v]"""
    T, H, n, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=D, device=q.device)
    back = torch.arange(first, first + T, device=q.device)[:, None] - torch.arange(n, device=q.device)[None, :]
    hidden = (back < 0) if window is None else (back < 0) | (back >= window)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :n] @ v[:, g]
    return out


def _llama_exact(case, seed, path, device):
    c, past = _llama_config(case), case["past"]
    f = gguf_io.read_gguf(path)
    tokens = torch.from_numpy(_tokens(case, seed)).long().to(device)
    T, hd, kvd = len(tokens), c.head_dim, c.n_head_kv * c.head_dim
    W = lambda name: _dequantized(f.tensors[name], device)  # noqa: E731
    x = W("token_embd.weight")[tokens]
    angle = torch.arange(past, past + T, device=device, dtype=D)[:, None] * c.rope_freq_base ** (-torch.arange(0, hd, 2, device=device, dtype=D) / hd)[None, :]
    cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]

    def rope(y):
        a, b = y[..., 0::2], y[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).reshape(y.shape)
    product = lambda h, name: _eight_bit(h, case["ftype"]) @ W(name).T  # noqa: E731
    for i in range(c.n_layer):
        p = f"blk.{i}."
        h = _unit(x, c.rms_eps) * W(p + "attn_norm.weight")
        q = rope(product(h, p + "attn_q.weight").reshape(T, c.n_head, hd))
        if T > 1:                                       # a batch of several tokens takes its queries in 16 bits
            q = q.half().to(D)
        k = rope(product(h, p + "attn_k.weight").reshape(T, c.n_head_kv, hd)).reshape(T, kvd).half().to(D)
        v = product(h, p + "attn_v.weight").half().to(D)
        old = _cached_rows(case, seed, i, device).to(D)
        k, v = torch.cat([old[0], k]).reshape(-1, c.n_head_kv, hd), torch.cat([old[1], v]).reshape(-1, c.n_head_kv, hd)
        x = x + product(_attend(q, k, v, hd ** -0.5, past).reshape(T, -1), p + "attn_output.weight")
        h = _unit(x, c.rms_eps) * W(p + "ffn_norm.weight")
        x = x + product(torch.nn.functional.silu(product(h, p + "ffn_gate.weight")) * product(h, p + "ffn_up.weight"), p + "ffn_down.weight")
    return product(_unit(x[-1:], c.rms_eps) * W("output_norm.weight"), "output.weight")[0]


def _stack_weights(path, device):
    with open(os.path.join(path, "model.safetensors"), "rb") as f:
        head = json.loads(f.read(struct.unpack("<Q", f.read(8))[0]))
        data = np.frombuffer(f.read(), dtype=np.uint8)
    out = {}
    for name, d in head.items():
        a, b = d["data_offsets"]
        out[name] = torch.from_numpy(data[a:b].copy()).to(device).view(torch.bfloat16).reshape(d["shape"])
    return out


def _stack_exact(case, seed, path, device):
    cfg, tokens = _stack_config(case), _tokens(case, seed)
    raw = _stack_weights(path, device)
    x = (_matulorn if case["design"] == "matulorn" else _bozisun)(cfg, lambda name: raw[name].to(D), tokens, raw)
    wanted = torch.tensor(_rows(case) + list(range(case["tokens"], len(tokens))), device=device)
    logits = x[wanted] @ raw["head"].to(D).T
    if cfg.get("logit_softcap"):
        logits = cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])
    rows = len(_rows(case))
    return [logits[:rows], logits[rows:]] if case["steps"] else [logits]


def _yarn(rot, n, device):
    """(cos, sin) [n, dims / 2] of positions 0..n-1 under YaRN"""
    dims, base, sc = rot["dims"], rot["base"], rot.get("scaling")
    i = torch.arange(dims // 2, device=device, dtype=D)
    f, mag = base ** (-2.0 * i / dims), 1.0
    if sc:
        index = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(index(sc["fast"])), 0), min(math.ceil(index(sc["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, mag = f * (ramp / sc["factor"] + 1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    a = torch.arange(n, device=device, dtype=D)[:, None] * f[None, :]
    return torch.cos(a) * mag, torch.sin(a) * mag


def _rotate(x, cos, sin):
    """x [T, heads, n]: the first dims entries in half-split pairs"""
    m = cos.shape[1]
    u, v, cos, sin = x[..., :m], x[..., m:2 * m], cos[:, None, :], sin[:, None, :]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., 2 * m:]], -1)


def _matulorn(cfg, W, tokens, raw):
    G, eps = cfg["norm"]["groups"], cfg["norm"]["eps"]
    sig, silu, T = torch.sigmoid, torch.nn.functional.silu, len(tokens)
    grouped = lambda x, w: _unit(x.reshape(T, G, -1), eps).reshape(T, -1) * w  # noqa: E731
    x = raw["embed"][torch.from_numpy(tokens).long().to(raw["embed"].device)].to(D)
    for i, layer in enumerate(cfg["layers"]):
        p, mx = f"l{i}.", layer["mixer"]
        m = p + "mix."
        h = grouped(x, W(p + "norm1"))
        if layer["type"] == "mingru":
            z, u = sig(h @ W(m + "z").T + W(m + "z.b")), h @ W(m + "x").T + W(m + "x.b")
            cand = torch.where(u >= 0, u + 0.5, sig(u))
            y, s = torch.empty_like(z), torch.zeros_like(z[0])
            for t in range(T):
                s = (1.0 - z[t]) * s + z[t] * cand[t]
                y[t] = s
            y = (y * silu(h @ W(m + "g").T)) @ W(m + "o").T
        elif layer["type"] == "latent_attention":
            H, Dm, R, rank = mx["heads"], mx["dim"], mx["rot_dim"], mx["kv_rank"]
            cos, sin = _yarn(mx["rot"], T, h.device)
            q, dkv = (h @ W(m + "q").T).reshape(T, H, Dm + R), h @ W(m + "dkv").T
            lat = _unit(dkv[:, :rank], eps) * W(m + "dkv.norm")
            shared = _rotate(dkv[:, None, rank:], cos, sin).expand(T, H, R)
            k = torch.cat([(lat @ W(m + "uk").T).reshape(T, H, Dm), shared], -1)
            q = torch.cat([q[..., :Dm], _rotate(q[..., Dm:], cos, sin)], -1)
            v = (lat @ W(m + "uv").T).reshape(T, H, -1)
            y = _attend(q, k, v, mx["scale"], 0, mx["mask"]["size"], W(m + "sink")).reshape(T, -1) @ W(m + "o").T
        else:
            H, KH, Dm, V, taps = mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"], mx["conv"]

            def conv(name, heads, n):
                u = torch.cat([torch.zeros((taps - 1, heads * n), dtype=D, device=h.device), h @ W(m + name).T])
                w = W(m + name + ".conv")
                return silu(sum(u[j:j + T] * w[:, j] for j in range(taps))).reshape(T, heads, n)
            q, k, v = conv("q", KH, Dm), conv("k", KH, Dm), conv("v", H, V)
            q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * Dm ** -0.5).repeat_interleave(H // KH, 1)
            k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // KH, 1)
            beta = sig(h @ W(m + "b").T)
            g = torch.exp(-torch.exp(W(m + "A_log")) * torch.nn.functional.softplus(h @ W(m + "a").T + W(m + "dt_bias")))
            S, o = torch.zeros((H, Dm, V), dtype=D, device=h.device), torch.empty((T, H, V), dtype=D, device=h.device)
            for t in range(T):
                S = S * g[t][:, None, None]
                u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
                S = S + k[t][:, :, None] * u[:, None, :]
                o[t] = torch.einsum("hdv,hd->hv", S, q[t])
            y = (_unit(o, eps) * W(m + "norm") * silu(h @ W(m + "g").T).reshape(T, H, V)).reshape(T, H * V) @ W(m + "o").T
        x = x + grouped(y, W(p + "norm1b"))
        f, lim = p + "mlp.", layer["mlp"]["limit"]
        h = grouped(x, W(p + "norm2"))
        g, u = (h @ W(f + "gate").T + W(f + "gate.b")).clamp(max=lim), (h @ W(f + "up").T + W(f + "up.b")).clamp(-lim, lim)
        x = x + grouped((g * sig(1.702 * g) * (u + 1.0)) @ W(f + "down").T + W(f + "down.b"), W(p + "norm2b"))
    return grouped(x, W("final.norm"))


def _bozisun(cfg, W, tokens, raw):
    eps, dim, T = cfg["norm"]["eps"], cfg["token_side"]["dim"], len(tokens)
    sig, silu = torch.sigmoid, torch.nn.functional.silu
    device = raw["embed"].device
    ids, pairs = torch.from_numpy(tokens).long().to(device), cfg["embedding"]["bigram"]
    row = torch.cat([torch.tensor([pairs["buckets"]], device=device), (ids[:-1] * pairs["mul_prev"] + ids[1:] * pairs["mul_cur"]) % pairs["buckets"]])
    x = raw["embed"][ids].to(D) + raw["bigram"][row].to(D)
    own = raw["side.embed"][ids].to(D)
    lp = cfg["loop"]
    order = list(range(lp["start"])) + list(range(lp["start"], lp["stop"])) * lp["times"] + list(range(lp["stop"], len(cfg["layers"])))

    def unit_of(h, p):
        return (silu(h @ W(p + "gate").T) * (h @ W(p + "up").T)) @ W(p + "down").T
    for i in order:
        p, mx, mlp = f"l{i}.", cfg["layers"][i]["mixer"], cfg["layers"][i]["mlp"]
        m, H, G, Dm = p + "mix.", mx["heads"], mx["kv_heads"], mx["dim"]
        h = _unit(x, eps) * W(p + "norm1")
        cos, sin = _yarn(mx["rot"], T, device)
        q = _rotate(_unit((h @ W(m + "q").T).reshape(T, H, Dm), eps) * W(m + "q.norm"), cos, sin)
        k = _rotate(_unit((h @ W(m + "k").T).reshape(T, G, Dm), eps) * W(m + "k.norm"), cos, sin)
        v = (h @ W(m + "v").T).reshape(T, G, -1)
        y = (_attend(q, k, v, mx["scale"], 0).reshape(T, -1) * sig(h @ W(m + "g").T)) @ W(m + "o").T
        if mlp["kind"] == "dense":
            y = y + unit_of(h, p + "mlp.")
        else:
            z = h @ W(p + "mlp.router").T + W(p + "mlp.router.b")
            best, sel = torch.topk(z, mlp["router"]["top"], dim=-1)
            weight = torch.softmax(best, -1)
            for e in range(mlp["router"]["experts"]):
                t, j = torch.nonzero(sel == e, as_tuple=True)
                if len(t):
                    y[t] += weight[t, j][:, None] * unit_of(h[t], f"{p}mlp.e{e}.")
        x = x + y
        gate = torch.nn.functional.gelu(x @ W(p + "side.gate").T, approximate="tanh")
        x = x + _unit((gate * own[:, i * dim:(i + 1) * dim]) @ W(p + "side.proj").T, eps) * W(p + "side.norm")
    return _unit(x, eps) * W("final.norm")
