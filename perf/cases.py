"""The calls whose speed counts, as a user's program makes them, with inputs, sizes and 64-bit results.

The framework serves quantised decoders behind `ForwardEngine`, the dequant-fused matmul on its own, and layer-plan designs.
A case is one call of that surface on a model of the shapes in `synth.CONFIGS`. So that a model is made in a second or two, the
two large ones have half of their layers, and layers share four random sets of weights (every layer has its own copy on the device):

  op       `Weight.matmul_nt_dev`: one quantised linear on device rows
  decode   one token of one sequence, logits to the host (a chat with sampling on the host)
  verify   the k + 1 rows of a speculative round, logits of each
  batch    one token of many sequences of unequal lengths
  serve    a portion of a prompt beside decoded tokens of other sequences: a step of a server that admits while it decodes
  prefill  a prompt from its first token
  request  a layer-plan design (bf16): prompts of several sequences, then some decoded tokens of all of them

A pass that appends to a cache starts by cutting it back to where it stood, so that every pass is the same call.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sapient_b200 import ops, synth
from sapient_b200.engine import ForwardEngine

FORMATS = {"q4_k": synth.Q4_K, "q6_k": synth.Q6_K, "q8_0": synth.Q8_0}
POOL = 4  # distinct sets of layer weights of a model
MODELS = {name: dict(synth.CONFIGS[name], n_layers=n) for name, n in (("qwen05b", 24), ("qwen15b", 28), ("phi2", 16), ("llama8b", 16))}
TEDELIX_RANK = 64


def listed():
    return [
        # the smallest call: an attention projection of one token
        {"name": "op_q4k_4096x4096_m1", "kind": "op", "fmt": "q4_k", "n": 4096, "k": 4096, "rows": 1},
        # a down projection for an odd number of rows
        {"name": "op_q6k_4096x14336_m37", "kind": "op", "fmt": "q6_k", "n": 4096, "k": 14336, "rows": 37},
        # chat with a small model: launches and latency
        {"name": "decode_qwen05b", "kind": "decode", "model": "qwen05b", "ctx": 130},
        # chat with the headline model
        {"name": "decode_llama8b", "kind": "decode", "model": "llama8b", "ctx": 517},
        # the Phi block (LayerNorm, GELU, biases, head size 80), 8-bit blocks
        {"name": "decode_phi2", "kind": "decode", "model": "phi2", "ctx": 645},
        # a draft of four tokens verified
        {"name": "verify_qwen15b", "kind": "verify", "model": "qwen15b", "ctx": 309, "rows": 5},
        # a small server's step: few sequences
        {"name": "batch_qwen15b_13", "kind": "batch", "model": "qwen15b", "seqs": 13, "ctx": 700},
        # a full server's step on the headline model
        {"name": "batch_llama8b_32", "kind": "batch", "model": "llama8b", "seqs": 32, "ctx": 1000},
        # a prompt's portion admitted beside running sequences
        {"name": "serve_qwen15b", "kind": "serve", "model": "qwen15b", "seqs": 11, "ctx": 400, "rows": 181},
        # prompts: of the headline model, and a ragged one of the Phi block
        {"name": "prefill_llama8b_512", "kind": "prefill", "model": "llama8b", "rows": 512},
        {"name": "prefill_phi2_389", "kind": "prefill", "model": "phi2", "rows": 389},
        # a layer-plan design: state mixers, grouped attention, bf16 products; prompts and decoding
        {"name": "request_tedelix", "kind": "request", "width": 2048, "heads": 16, "ff": 6144, "seqs": 4, "rows": 301, "steps": 8},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["op", "op", "decode", "verify", "batch", "serve", "prefill", "request"])
    if kind == "op":
        fmt = rng.choice(sorted(FORMATS))
        k = 32 * log(27, 448) if fmt == "q8_0" else 256 * log(4, 56)
        return {"kind": kind, "fmt": fmt, "n": log(1000, 40000), "k": k, "rows": log(1, 512)}
    if kind == "request":
        heads = rng.choice([8, 16])
        return {"kind": kind, "width": 128 * heads, "heads": heads, "ff": 384 * heads, "seqs": rng.randint(1, 8), "rows": log(33, 500), "steps": rng.randint(4, 12)}
    model = rng.choice(sorted(MODELS))
    ctx = 16 * log(4, 64) + rng.randint(1, 6)  # room for the call's rows on the sequence's last page or the next ones
    if kind == "decode":
        return {"kind": kind, "model": model, "ctx": ctx}
    if kind == "verify":
        return {"kind": kind, "model": model, "ctx": ctx, "rows": rng.randint(2, 9)}
    if kind == "batch":
        return {"kind": kind, "model": model, "ctx": min(ctx, 900), "seqs": log(2, 30)}
    if kind == "serve":
        return {"kind": kind, "model": model, "ctx": min(ctx, 500), "seqs": rng.randint(2, 12), "rows": log(17, 250)}
    return {"kind": kind, "model": model, "rows": log(20, 500)}


# ── inputs ──────────────────────────────────────────────────────────────────
def _op_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    fmt, n, k = FORMATS[case["fmt"]], case["n"], case["k"]
    blocks = synth.quantize(fmt, torch.randn(n, k, generator=g, device="cuda") * 0.02)
    x = torch.randn(case["rows"], k, generator=g, device="cuda")
    return fmt, blocks, x


def _model(case, seed, max_ctx):
    """(cfg, weights by name) of a quantised model, uint8 tensors on the GPU; layer l has the weights of set l % POOL."""
    full = MODELS[case["model"]]
    cfg, W = synth.build_model(dict(full, n_layers=POOL), seed=seed, device="cuda", max_ctx=max_ctx)
    cfg["n_layers"] = full["n_layers"]
    for name in [n for n in W if n.startswith("model.layers.")]:
        _, _, l, rest = name.split(".", 3)
        for j in range(int(l) + POOL, cfg["n_layers"], POOL):
            W[f"model.layers.{j}.{rest}"] = W[name]
    return cfg, W


def _lengths(case, rng):
    """Cached tokens of each sequence: unequal, the longest is ctx; never a whole number of pages."""
    if case["kind"] in ("decode", "verify"):
        return [case["ctx"]]
    n = [max(2, int(case["ctx"] * f)) for f in rng.uniform(0.25, 1.0, case["seqs"])]
    n[0] = case["ctx"]
    return [v if v % 16 else v - 1 for v in n]


def _tokens(case, seed, vocab):
    """(cached prompt of every slot, the call's own tokens)."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "prefill":
        return [], rng.integers(0, vocab, case["rows"]).astype(np.uint32)
    if case["kind"] == "request":
        return [rng.integers(0, vocab, case["rows"] - 3 * s).astype(np.uint32) for s in range(case["seqs"])], rng.integers(0, vocab, (case["steps"], case["seqs"])).astype(np.uint32)
    cached = [rng.integers(0, vocab, n).astype(np.uint32) for n in _lengths(case, rng)]
    own = case.get("rows", 0) if case["kind"] in ("verify", "serve") else 0
    return cached, rng.integers(0, vocab, own + (0 if case["kind"] == "verify" else len(cached))).astype(np.uint32)


def _tedelix(case):
    h = case["heads"]
    return synth.tedelix_config(layers=["general_delta", "general_delta", "attention", "lightning"] * 2, width=case["width"], heads=h, kv_heads=h // 4, dim=128, vdim=128,
                                state_heads=2 * h, state_dim=64, state_vdim=64, window=1024, ff=case["ff"], vocab=32768)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "op":
        fmt, blocks, x = _op_inputs(case, seed)
        return {"kind": kind, "w": ops.Weight(fmt, case["n"], case["k"], blocks.cpu().numpy()), "x": x, "y": torch.empty(case["rows"], case["n"], device="cuda")}
    if kind == "request":
        cfg = _tedelix(case)
        weights = synth.tedelix_weights(cfg, seed, TEDELIX_RANK, device="cuda")
        eng = ForwardEngine.from_config(cfg, weights, max_ctx=1024, max_batch=case["seqs"], max_tokens=512)
        prompts, steps = _tokens(case, seed, cfg["vocab"])
        return {"kind": kind, "eng": eng, "prompts": prompts, "steps": steps, "slots": list(range(case["seqs"]))}
    vocab = MODELS[case["model"]]["vocab"]
    cached, own = _tokens(case, seed, vocab)
    cfg, W = _model(case, seed, max_ctx=case.get("ctx", 0) + case.get("rows", 0) + 64)
    host = {}  # layers of a set share one host copy
    weights = {name: (dt, dims, host.setdefault(t.data_ptr(), t.cpu().numpy())) for name, (dt, dims, t) in W.items()}
    del W
    torch.cuda.empty_cache()
    slots = len(cached) + (kind == "serve")
    eng = ForwardEngine.from_weights(cfg, weights, max_batch=max(1, slots), max_tokens=512)
    for s, ids in enumerate(cached):
        eng.forward_slot(s, ids)
    return {"kind": kind, "eng": eng, "lengths": [len(c) for c in cached], "own": own, "rows": case.get("rows", 0), "slots": list(range(len(cached)))}


def run(s):
    kind = s["kind"]
    if kind == "op":
        s["w"].matmul_nt_dev(s["x"].data_ptr(), s["x"].shape[0], s["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return s["y"]
    eng = s["eng"]
    if kind == "request":
        eng.reset_cache()
        first = [eng.forward_slot(i, ids) for i, ids in zip(s["slots"], s["prompts"])]
        return first + [eng.decode_batch(ids, s["slots"])[0] for ids in s["steps"]]
    if kind == "prefill":
        return eng.forward_logits(s["own"], False)
    for slot, n in zip(s["slots"], s["lengths"]):
        eng.truncate_cache(n, slot)
    if kind == "decode":
        return eng.forward_logits(s["own"])
    if kind == "verify":
        return eng.forward_all_logits_cached(s["own"])
    if kind == "batch":
        return eng.decode_batch(s["own"], s["slots"])[0]
    n, new = len(s["slots"]), len(s["slots"])
    eng.reset_cache(new)
    return eng.forward_mixed([(new, s["own"][n:], [s["rows"] - 1])] + [(i, s["own"][i:i + 1], [0]) for i in s["slots"]])


# ── what a pass cannot do without ───────────────────────────────────────────
def _matrices(cfg):
    """(format, rows, columns) of the matrices a row goes through, the head last."""
    H, G, D, hid, ffn = cfg["n_heads"], cfg["n_kv_heads"], cfg["head_dim"], cfg["hidden"], cfg["ffn"]
    out = []
    for l in range(cfg["n_layers"]):
        roles = [("q", H * D, hid), ("k", G * D, hid), ("v", G * D, hid), ("o", hid, H * D)]
        roles += [("up", ffn, hid), ("down", hid, ffn)] + ([] if cfg["arch"] == "phi2" else [("gate", ffn, hid)])
        out += [(synth.weight_dtype(cfg, r, l % POOL, k), n, k) for r, n, k in roles]
    return out + [(synth.weight_dtype(cfg, "embed" if cfg.get("tied") else "output", 0, hid), cfg["vocab"], hid)]


def work(case):
    kind = case["kind"]
    if kind == "op":
        n, k, m = case["n"], case["k"], case["rows"]
        return {"bytes": synth.byte_count(FORMATS[case["fmt"]], n * k) + 4 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "request":
        w, h, ff, B, T, S = case["width"], case["heads"], case["ff"], case["seqs"], case["rows"], case["steps"]
        hd, V = 128 * h, 32768
        mats = 8 * 2 * ff * w + 2 * (2 * hd + 2 * hd // 4) * w + 2 * 5 * hd * w + 4 * (6 * hd * w + TEDELIX_RANK * (w + hd))
        state = 6 * 2 * h * 64 * 64 * 8 * B  # read and written once per call
        return {"bytes": (B + S) * 2 * (mats + V * w) + (1 + S) * state + 4 * V * B * (1 + S),
                "flops": 2 * mats * B * (T + S) + 2 * V * w * B * (1 + S)}
    cfg = MODELS[case["model"]]
    mats = _matrices(cfg)
    lengths = [] if kind == "prefill" else _lengths(case, np.random.default_rng(0))
    rows = {"decode": 1, "verify": case.get("rows"), "batch": len(lengths), "serve": case.get("rows", 0) + len(lengths), "prefill": case.get("rows")}[kind]
    heads = {"verify": rows, "serve": len(lengths) + 1, "prefill": 1}.get(kind, rows)
    kv = 2 * cfg["n_layers"] * cfg["n_kv_heads"] * cfg["head_dim"] * 2
    q = 4 * cfg["n_layers"] * cfg["n_heads"] * cfg["head_dim"]
    new = case.get("rows", 0)
    pairs = {"verify": sum(lengths) * new + new * (new + 1) // 2, "prefill": new * (new + 1) // 2, "serve": sum(lengths) + new * (new + 1) // 2}.get(kind, sum(lengths))
    return {"bytes": sum(synth.byte_count(f, n * k) for f, n, k in mats) + kv * (sum(lengths) + rows) + 4 * cfg["vocab"] * heads,
            "flops": sum(2 * n * k for _, n, k in mats[:-1]) * rows + 2 * cfg["vocab"] * cfg["hidden"] * heads + q * pairs}


def tolerance(case):
    """Four times the distance from exact() that was measured. Products: f32 sums over k. Models whose head size is a multiple
    of 32 keep keys and values in eight-bit blocks, and a value near the edge of a step moves by a whole step for the last bit
    of a sum before it; deeper and wider models move more. Phi-2's cache has no such steps."""
    if case["kind"] == "op":
        return {"rel": 5e-5}
    if case["kind"] == "request":
        return {"rel": 0.016}
    return {"rel": {"phi2": 1.2e-4, "qwen05b": 6e-3, "qwen15b": 7e-3, "llama8b": 0.025}[case["model"]]}


# ── the same in 64 bits ─────────────────────────────────────────────────────
def _half(b):
    return b.contiguous().view(torch.float16).double()


def _values(fmt, raw, n, k):
    """[n, k] float64 of a matrix of ggml blocks."""
    if fmt == synth.F32:
        return raw.view(torch.float32).double().reshape(n, k)
    if fmt == synth.Q8_0:
        b = raw.reshape(-1, 34)
        return (_half(b[:, :2]) * b[:, 2:].contiguous().view(torch.int8).double()).reshape(n, k)
    if fmt == synth.Q4_K:
        b = raw.reshape(-1, 144)
        d, dmin, s = _half(b[:, 0:2]), _half(b[:, 2:4]), b[:, 4:16].int()
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1)
        q = b[:, 16:].reshape(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32).double()
        return ((d * sc).unsqueeze(-1) * q - (dmin * mn).unsqueeze(-1)).reshape(n, k)
    b = raw.reshape(-1, 210)
    ql, qh = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 1, 32)
    lo = torch.cat([ql & 15, ql >> 4], 2).int()
    hi = torch.cat([(qh >> sh) & 3 for sh in (0, 2, 4, 6)], 2).int()
    q = (lo | (hi << 4)).double().reshape(-1, 16, 16) - 32
    sc = b[:, 192:208].contiguous().view(torch.int8).double()
    return ((_half(b[:, 208:210]) * sc).unsqueeze(-1) * q).reshape(n, k)


def _rotate(x, pos, dims, base):
    """x [T, heads, D]: coordinates i and i + dims / 2 turn together."""
    a = pos.double()[:, None, None] * base ** (-torch.arange(0, dims, 2, device=x.device, dtype=torch.float64) / dims)
    u, v, rest = x[..., : dims // 2], x[..., dims // 2:dims], x[..., dims:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), rest], -1)


def _cache_rounded(x):
    """Rows as the reference's cache holds them: blocks of 32, eight bits and a half-precision scale."""
    b = x.reshape(*x.shape[:-1], -1, 32)
    top = b.abs().amax(-1, keepdim=True)
    q = b * torch.where(top > 0, 127.0 / top, 0.0)
    return ((torch.sign(q) * torch.floor(q.abs() + 0.5)).clamp(-127, 127) * (top / 127.0).half().double()).reshape(x.shape)


def _attend(q, k, v, scale, window=None):
    """q [T, H, D] are the last T positions of k, v [S, G, D]; causal."""
    T, H, _ = q.shape
    S, G, _ = k.shape
    out = q.new_empty(T, H, v.shape[-1])
    at = torch.arange(S - T, S, device=q.device)[:, None] - torch.arange(S, device=q.device)[None]
    seen = at >= 0 if window is None else (at >= 0) & (at < window)
    for h in range(H):
        z = (q[:, h] @ k[:, h * G // H].T) * scale
        out[:, h] = torch.softmax(z.masked_fill(~seen, -torch.inf), -1) @ v[:, h * G // H]
    return out


def _exact_quantised(case, seed):
    vocab = MODELS[case["model"]]["vocab"]
    cached, own = _tokens(case, seed, vocab)
    cfg, W = _model(case, seed, max_ctx=case.get("ctx", 0) + case.get("rows", 0) + 64)
    n = len(cached)
    if case["kind"] == "prefill":
        seqs, wanted = [own], [[len(own) - 1]]
    elif case["kind"] == "verify":
        seqs, wanted = [np.concatenate([cached[0], own])], [list(range(len(cached[0]), len(cached[0]) + len(own)))]
    else:
        seqs = [np.concatenate([c, own[i:i + 1]]) for i, c in enumerate(cached)]
        wanted = [[len(c)] for c in cached]
        if case["kind"] == "serve":
            seqs, wanted = [own[n:]] + seqs, [[case["rows"] - 1]] + wanted
    H, G, D, eps, phi = cfg["n_heads"], cfg["n_kv_heads"], cfg["head_dim"], cfg["norm_eps"], cfg["arch"] == "phi2"
    get = lambda name: W[name][2].view(torch.float32).double()  # noqa: E731
    sets = {}

    def linear(x, name):
        """Dequantised in pieces of rows; the layers of a set share their values."""
        fmt, (rows, k), raw = W[name + ".weight"]
        raw, out = raw.reshape(rows, -1), []
        key = raw.data_ptr()
        for r in range(0, rows, 16384):
            if (key, r) not in sets:
                sets[key, r] = _values(fmt, raw[r:r + 16384].reshape(-1), min(16384, rows - r), k).float()
            out.append(x @ sets[key, r].double().T)
        y = torch.cat(out, -1)
        return y + get(name + ".bias") if name + ".bias" in W else y

    def norm(x, name):
        if phi:
            c = x - x.mean(-1, keepdim=True)
            return c / (c.square().mean(-1, keepdim=True) + eps).sqrt() * get(name + ".weight") + get(name + ".bias")
        return x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * get(name + ".weight")

    def mix(h, p):
        q, k, v = (linear(h, p + f"self_attn.{c}_proj").reshape(len(h), -1, D) for c in "qkv")
        q, k = _rotate(q, pos, cfg["rotary_dim"], cfg["rope_theta"]), _rotate(k, pos, cfg["rotary_dim"], cfg["rope_theta"])
        if D % 32 == 0:
            k, v = _cache_rounded(k), _cache_rounded(v)
        o = torch.cat([_attend(q[a:b], k[a:b], v[a:b], D ** -0.5) for a, b in zip(ends, ends[1:])])
        return linear(o.reshape(len(h), H * D), p + "self_attn.o_proj")

    ends = np.concatenate([[0], np.cumsum([len(s) for s in seqs])]).tolist()
    pos = torch.cat([torch.arange(len(s)) for s in seqs]).cuda()
    ids = torch.from_numpy(np.concatenate(seqs).astype(np.int64)).cuda()
    fmt, (_, k), raw = W["model.embed_tokens.weight"]
    x = _values(fmt, raw.reshape(vocab, -1)[ids].reshape(-1), len(ids), k)
    for l in range(cfg["n_layers"]):
        p = f"model.layers.{l}."
        h = norm(x, p + "input_layernorm")
        if phi:
            x = x + mix(h, p) + linear(torch.nn.functional.gelu(linear(h, p + "mlp.fc1"), approximate="tanh"), p + "mlp.fc2")
        else:
            x = x + mix(h, p)
            h = norm(x, p + "post_attention_layernorm")
            x = x + linear(torch.nn.functional.silu(linear(h, p + "mlp.gate_proj")) * linear(h, p + "mlp.up_proj"), p + "mlp.down_proj")
    rows = [a + r for a, want in zip(ends, wanted) for r in want]
    z = linear(norm(x[rows], "model.norm"), "model.embed_tokens" if cfg.get("tied") else "lm_head").cpu().numpy()
    return z[0] if case["kind"] in ("decode", "prefill") else z


def _exact_tedelix(case, seed):
    cfg = _tedelix(case)
    W = {n: w.double() for n, w in synth.tedelix_weights(cfg, seed, TEDELIX_RANK, device="cuda").items()}
    prompts, steps = _tokens(case, seed, cfg["vocab"])
    eps = cfg["norm"]["eps"]
    rms = lambda x: x / (x.square().mean(-1, keepdim=True) + eps).sqrt()  # noqa: E731

    def mix(kind, m, h, p, pos):
        T, n, D = len(h), m["heads"], m["dim"]
        V = m.get("vdim", D)
        part = lambda name, d: (h @ W[p + name].T).reshape(T, -1, d)  # noqa: E731
        if kind == "attention":
            base = m["rot"]["base"]
            q, k, v = (_rotate(part(c, D), pos, D, base) for c in "qkv")
            return _rotate(_attend(q, k, v, m["scale"], m["mask"]["size"]), -pos, V, base).reshape(T, n * V)
        S, o = h.new_zeros(n, D, V), []
        if kind == "lightning":
            q, k, v = (torch.nn.functional.silu(part(c, d)) for c, d in (("q", D), ("k", D), ("v", V)))
            decay = torch.tensor(m["decay"], device="cuda", dtype=torch.float64)[:, None, None]
            for t in range(T):
                S = decay * S + k[t, :, :, None] * v[t, :, None, :]
                o.append((S * q[t, :, :, None]).sum(1))
            y = rms(torch.stack(o).reshape(T, n * V))
        else:
            r, k, v = (part(c, D) for c in "rkv")
            w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ W[p + "w1"].T) @ W[p + "w2"].T + W[p + "w0"])).reshape(T, n, D)
            a = torch.sigmoid(h @ W[p + "a"].T + W[p + "a.b"]).reshape(T, n, D)
            u = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
            for t in range(T):
                held = (S * u[t, :, :, None]).sum(1, keepdim=True)
                S = w[t, :, :, None] * S - (a[t] * u[t])[:, :, None] * held + k[t, :, :, None] * v[t, :, None, :]
                o.append((S * r[t, :, :, None]).sum(1))
            y = rms(torch.stack(o)).reshape(T, n * V)
        return y * W[p + "norm"] * torch.sigmoid(h @ W[p + "g"].T)

    out = []
    for s, prompt in enumerate(prompts):
        ids = torch.from_numpy(np.concatenate([prompt, steps[:, s]]).astype(np.int64)).cuda()
        pos, x = torch.arange(len(ids), device="cuda"), W["embed"][ids]
        for i, layer in enumerate(cfg["layers"]):
            h = rms(x) * W[f"l{i}.norm1"]
            y = mix(layer["type"], layer["mixer"], h, f"l{i}.mix.", pos) @ W[f"l{i}.mix.o"].T
            x = x + y + torch.relu(h @ W[f"l{i}.mlp.up"].T).square() @ W[f"l{i}.mlp.down"].T
        z = (rms(x[len(prompt) - 1:]) * W["final.norm"]) @ W["embed"].T * cfg["logit_scale"]
        out.append((cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])).cpu().numpy())
    return [z[0] for z in out] + [np.stack([z[1 + t] for z in out]) for t in range(len(steps))]


def exact(case, seed):
    if case["kind"] == "op":
        fmt, blocks, x = _op_inputs(case, seed)
        return x.double() @ _values(fmt, blocks.reshape(-1), case["n"], case["k"]).T
    return (_exact_tedelix if case["kind"] == "request" else _exact_quantised)(case, seed)
