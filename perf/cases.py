"""What this engine is timed on: whole passes through ``Engine``, ``Engine.step`` and ``Engine.generate``.

A case is one pass of a serving program.  Three kinds:

``step``      one batch through ``Engine.step``: ``decoding`` requests with about ``context`` cached tokens bring one
              token each, ``portions`` requests bring a portion of a prompt of up to ``portion`` tokens (the first of
              them continues a prompt of which ``start`` tokens are cached).  The requests and their caches are there
              before; afterwards the step's tokens are taken back, so that the next pass does the same.  Returned:
              the logits of every last token, and of ``score`` more places of a portion.
``session``   ``requests`` requests from the first token to the last: open, one step with all prompts (up to
              ``prompt`` tokens each), ``steps`` decode steps of given tokens, close.  Returned: all logits.
``generate``  the same through ``Engine.generate``: greedy, the generated ids are returned.

Sizes are those of the repository's configurations and benchmark: the two tiny models of its tests, TinyLlama 1.1B (22
layers), layers of Llama-2 7B and Llama-3 8B, and a Senulix model of 2048 channels for the designs with other mixers than
Llama's (mixed-score window attention, latent attention, linear attention).  Weights are random (N(0, 0.02), drawn on the
device from the seed), token ids uniform.
"""
from __future__ import annotations

import hashlib
import math
import random

import torch

PAGE = 64


def _llama(layers, hidden, heads, kv, head_dim, inter, vocab, theta, tied=False, eps=1e-5):
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": head_dim, "intermediate_size": inter,
            "vocab_size": vocab, "rope_theta": theta, "rms_norm_eps": eps, "max_position_embeddings": 8192,
            "tie_word_embeddings": tied}


def _senulix(layers, width=2048, heads=32, kv=4, dim=64, ff=5632, vocab=32000, rank=128, rot=32, window=1024, side=128):
    mixers = [("attention", {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                             "mask": {"size": window}, "rot": {"base": 50000.0, "dims": dim // 2}}),
              ("latent_attention", {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": dim, "kv_rank": rank,
                                    "scale": (dim + rot) ** -0.5, "rot": {"base": 50000.0, "dims": rot}}),
              ("lightning", {"heads": heads, "dim": dim, "vdim": dim,
                             "decay": [1.0 - 2.0 ** (-1.0 - 7.0 * h / (heads - 1)) for h in range(heads)]})]
    out = []
    for i in range(layers):
        k = i % 4
        kind, m = mixers[1 if k == 3 else k]
        out.append({"type": kind, "mixer": dict(m, kv_from=i - 2) if k == 3 else dict(m),
                    "mlp": None if k == 2 else {"kind": "dense", "ff": ff}})
    return {"architecture": "Senulix", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "token_side": {"dim": side},
            "logit_softcap": 30.0, "layers": out}


MODELS = {
    "tiny-a": _llama(2, 64, 4, 2, 16, 172, 256, 10000.0),
    "tiny-b": _llama(3, 96, 3, 1, 32, 256, 512, 500000.0, tied=True, eps=1e-6),
    "tinyllama-1.1b": _llama(22, 2048, 32, 4, 64, 5632, 32000, 10000.0),
    # eight of the 32 layers: every layer is alike, the step's time is their sum
    "llama2-7b": _llama(8, 4096, 32, 32, 128, 11008, 32000, 10000.0),
    "llama3-8b": _llama(8, 4096, 32, 8, 128, 14336, 128256, 500000.0),
    "senulix-2048": _senulix(8),
}


def _step(model, dtype="bfloat16", decoding=0, context=0, portions=0, portion=0, start=0, score=0):
    return {"kind": "step", "model": model, "dtype": dtype, "decoding": decoding, "context": context, "portions": portions,
            "portion": portion, "start": start, "score": score}


def _session(model, dtype="bfloat16", requests=1, prompt=64, steps=16, kind="session"):
    return {"kind": kind, "model": model, "dtype": dtype, "requests": requests, "prompt": prompt, "steps": steps}


def listed():
    return [
        # the smallest calls: the test model through generate(), all launches and host work
        dict(_session("tiny-a", "float32", requests=4, prompt=64, steps=16, kind="generate"), name="tiny-generate"),
        # one user chatting: a prompt of 64 tokens and the first 16 tokens of the answer
        dict(_session("tinyllama-1.1b", requests=1, prompt=64, steps=16), name="chat-b1"),
        # the headline: decoding at batch 8 with 2048 tokens of context
        dict(_step("tinyllama-1.1b", decoding=8, context=2047), name="decode-b8"),
        # a busy server: 64 requests with 512-token prompts in the middle of 256-token answers
        dict(_step("tinyllama-1.1b", decoding=64, context=640), name="decode-b64"),
        # time to the first token of a long prompt
        dict(_step("tinyllama-1.1b", portions=1, portion=2048, score=15), name="prompt-2048"),
        # short ragged prompts arriving together while others decode: continuous batching
        dict(_step("tinyllama-1.1b", decoding=11, context=700, portions=3, portion=333, start=129), name="mixed-small"),
        # the 32-bit path: decoding, and a prompt of odd length
        dict(_step("tinyllama-1.1b", "float32", decoding=8, context=2047), name="decode-b8-f32"),
        dict(_step("tinyllama-1.1b", "float32", portions=1, portion=1003, score=15), name="prompt-1003-f32"),
        # large layers: 64 requests at 1024 to 1280 tokens, a whole long prompt, and the mixed workload's steps
        dict(_step("llama3-8b", decoding=64, context=1280), name="decode-b64-8b"),
        dict(_step("llama3-8b", portions=1, portion=8192, score=15), name="prompt-8192-8b"),
        dict(_step("llama2-7b", decoding=24, context=1500, portions=2, portion=1700, start=1000), name="mixed-7b"),
        # another design: two prompts and the first tokens of the answers
        dict(_session("senulix-2048", requests=2, prompt=1100, steps=8), name="senulix-session"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: any batch, context and prompt length up to the listed ones."""
    pick = rng.random()
    if pick < 0.06:
        return _session(rng.choice(["tiny-a", "tiny-b"]), "float32", rng.randint(1, 6), _log(rng, 3, 128), rng.randint(2, 24),
                        kind="generate")
    if pick < 0.22:
        model = rng.choice(["tinyllama-1.1b", "senulix-2048"])
        return _session(model, "bfloat16", rng.randint(1, 3), _log(rng, 9, 1100), rng.randint(2, 16))
    model, dtype = rng.choice([("tinyllama-1.1b", "bfloat16"), ("tinyllama-1.1b", "bfloat16"), ("tinyllama-1.1b", "float32"),
                               ("llama3-8b", "bfloat16"), ("llama2-7b", "bfloat16")])
    long = {"tinyllama-1.1b": 2047, "llama3-8b": 8191, "llama2-7b": 4095}[model]
    if pick < 0.62:
        batch = _log(rng, 1, 64 if dtype == "bfloat16" else 16)
        most = {"tinyllama-1.1b": 64 * 2048, "llama3-8b": 64 * 1280, "llama2-7b": 32 * 1536}[model] // batch
        return _step(model, dtype, decoding=batch, context=_log(rng, 33, min(long, most)))
    if pick < 0.82:
        most = 1003 if dtype == "float32" else 2048 if model != "llama3-8b" else 8192
        return _step(model, dtype, portions=1, portion=_log(rng, 17, most), score=15)
    scale = 4 if dtype == "float32" else 1
    return _step(model, dtype, decoding=rng.randint(1, 24), context=_log(rng, 65, min(long, 2000)), portions=rng.randint(1, 4 // scale),
                 portion=_log(rng, 17, 1000 // scale), start=rng.choice([0, 0, rng.randint(1, 900)]))


# ---- what a case consists of -------------------------------------------------------------

def _entries(case):
    """(cached tokens, new tokens) of every request of a step, as the case's numbers give them."""
    B, P = case["decoding"], case["portions"]
    out = [(case["context"] - (case["context"] // 4) * i // max(1, B - 1), 1) for i in range(B)]
    for j in range(P):
        out.append((case["start"] if j == 0 else 0, max(2, case["portion"] - (case["portion"] // 2) * j // P)))
    return out


def _places(case, new):
    """The places of a portion whose logits are wanted: the last, and ``score`` more spread over it."""
    n = min(case["score"], new - 1) if new > 1 else 0
    return sorted({(i * (new - 1)) // n for i in range(n)} | {new - 1}) if n else [new - 1]


def _prompts(case):
    R, T = case["requests"], case["prompt"]
    return [max(1, T - (T // 3) * i // R) for i in range(R)]


def _vocab(model):
    return MODELS[model].get("vocab_size") or MODELS[model]["vocab"]


def _ids(rng, n, vocab):
    return [rng.randrange(vocab) for _ in range(n)]


def _tokens(case, seed):
    """Token ids: per request of a step (cached, new); per request of a session (prompt, decoded)."""
    rng, vocab = random.Random(int(seed)), _vocab(case["model"])
    if case["kind"] == "step":
        return [(_ids(rng, c, vocab), _ids(rng, n, vocab)) for c, n in _entries(case)]
    return [(_ids(rng, n, vocab), _ids(rng, case["steps"], vocab)) for n in _prompts(case)]


# ---- prepare and run ---------------------------------------------------------------------

def prepare(case, seed):
    """An engine with its weights bound and its kernels and decode graph in use, as a server keeps it, and the
    requests of the pass with their tokens cached."""
    from kllm_b200 import Engine, Options
    tokens = _tokens(case, seed)
    if case["kind"] == "step":
        total = [len(c) + len(n) for c, n in tokens]
        budget = max(2048, sum(len(n) for _, n in tokens))
    else:
        total = [len(p) + case["steps"] for p, _ in tokens]
        budget = max(256, sum(len(p) for p, _ in tokens))
    pages = sum(-(-t // PAGE) + 1 for t in total)
    engine = Engine(None, Options(max_seq=max(max(total), 256), block_size=PAGE, num_blocks=pages, max_batch=len(tokens),
                                  max_step_tokens=budget, dtype=case["dtype"]),
                    config=MODELS[case["model"]], random_seed=int(seed))
    state = {"case": case, "engine": engine, "tokens": tokens}
    if case["kind"] == "step":
        state["requests"] = [_fill(engine, cached, budget) for cached, _ in tokens]
    run(state)
    return state


def _fill(engine, cached, budget):
    from kllm_b200 import StepEntry
    request = engine.cache.open()
    for i in range(0, len(cached), budget):
        engine.step([StepEntry(request, cached[i:i + budget])])
    return request


def run(state):
    case, engine, tokens = state["case"], state["engine"], state["tokens"]
    from kllm_b200 import StepEntry
    if case["kind"] == "generate":
        return engine.generate([prompt for prompt, _ in tokens], max_new_tokens=case["steps"])
    if case["kind"] == "session":
        requests = [engine.cache.open() for _ in tokens]
        logits = [engine.step([StepEntry(r, prompt, [len(prompt) - 1]) for r, (prompt, _) in zip(requests, tokens)])]
        for i in range(case["steps"]):
            logits.append(engine.step([StepEntry(r, [answer[i]], [0]) for r, (_, answer) in zip(requests, tokens)]))
        for r in requests:
            engine.cache.close(r)
        return logits
    requests = state["requests"]
    held = [r.length for r in requests]
    logits = engine.step([StepEntry(r, new, _places(case, len(new))) for r, (_, new) in zip(requests, tokens)])
    for r, length in zip(requests, held):
        r.length = length
        engine.cache.trim_reservation(r)
    return logits


# ---- what a pass cannot do without ---------------------------------------------------------

def _mixers(cfg):
    """Per layer: (matrix parameters, numbers cached per token, sum of query/key and value sizes over the heads, window)."""
    if "num_hidden_layers" in cfg:
        d, H, G, hd, f = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                           "intermediate_size"))
        return [(d * (H + 2 * G) * hd + H * hd * d + 3 * d * f, 2 * G * hd, 2 * H * hd, None)] * cfg["num_hidden_layers"]
    d, out = cfg["width"], []
    for L in cfg["layers"]:
        m, H = L["mixer"], L["mixer"]["heads"]
        side = 2 * d * cfg["token_side"]["dim"] + (2 * d * L["mlp"]["ff"] if L["mlp"] else 0)
        if L["type"] == "attention":
            n = d * (H * m["dim"] + m["kv_heads"] * (m["dim"] + m["vdim"])) + d * H * m["vdim"]
            out.append((n + side, m["kv_heads"] * (m["dim"] + m["vdim"]), H * (m["dim"] + m["vdim"]), m["mask"]["size"]))
        elif L["type"] == "latent_attention":
            R, dr, own = m["kv_rank"], m["rot_dim"], m.get("kv_from") is None
            n = d * H * (m["dim"] + dr) + H * (m["dim"] + m["vdim"]) * R + d * H * m["vdim"] + (d * (R + dr) if own else 0)
            out.append((n + side, R + dr, H * (m["dim"] + dr + m["vdim"]), None))
        else:
            out.append((5 * d * H * m["dim"] + side, 0, 0, None))
    return out


def _step_work(cfg, dtype, entries, rows):
    e = 2 if dtype == "bfloat16" else 4
    d, vocab = cfg.get("hidden_size") or cfg["width"], cfg.get("vocab_size") or cfg["vocab"]
    n = sum(new for _, new in entries)
    bytes_ = vocab * d * e + n * d * e + 4.0 * rows * vocab
    flops = 2.0 * rows * vocab * d
    for params, cached, sizes, window in _mixers(cfg):
        bytes_ += params * e
        flops += 2.0 * n * params
        for c, new in entries:
            seen = min(c, window) if window else c
            bytes_ += (seen + new) * cached * e
            whole = c * new + new * (new + 1) // 2 if not window else sum(min(window, c + i + 1) for i in range(new))
            flops += 2.0 * sizes * whole
    return bytes_, flops


def work(case):
    cfg = MODELS[case["model"]]
    if case["kind"] == "step":
        entries = _entries(case)
        steps = [(entries, sum(len(_places(case, n)) for _, n in entries))]
    else:
        prompts = _prompts(case)
        more = case["steps"] - (1 if case["kind"] == "generate" else 0)       # generate: the prompt gives the first token
        steps = [([(0, p) for p in prompts], len(prompts))]
        steps += [([(p + i, 1) for p in prompts], len(prompts)) for i in range(more)]
    parts = [_step_work(cfg, case["dtype"], entries, rows) for entries, rows in steps]
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"            # greedy ids of the 32-bit path
    # measured between two ways of cutting the same prompt (portions of 7 tokens against the whole: other kernels, sums in
    # another order), four times what was seen: float32 4.3e-6 (max 1.8e-5), bfloat16 7.9e-3 (max 3.7e-2)
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 8e-5}
    return {"rel": 0.03, "max": 0.15}


# ---- the same numbers in 64 bits -----------------------------------------------------------

def _weights(cfg, seed, dtype):
    """name, shape -> the tensor as the engine draws it: N(0, 0.02) from a stream keyed by (seed, name), rounded to the
    dtype it is stored in; norms' gains are 1."""
    def get(name, *shape):
        key = hashlib.sha256(f"{int(seed)}:{name}".encode()).digest()
        g = torch.Generator(device="cuda")
        g.manual_seed(int.from_bytes(key[:8], "little") & ((1 << 63) - 1))
        t = 0.02 * torch.randn(shape, generator=g, dtype=torch.float32, device="cuda")
        return t.to(torch.bfloat16 if dtype == "bfloat16" else torch.float32).double()
    return get


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _turn(x, pos, dims, base):
    """x [T, heads, size]: the pairs (i, i + dims / 2) of the first ``dims`` values turned by pos * base^(-2i / dims)."""
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    a = pos.double()[:, None, None] * f
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., dims:]], dim=-1)


def _spread(lengths, fn, *tensors):
    """fn on every sequence's rows of the concatenated tensors."""
    return torch.cat([fn(*parts) for parts in zip(*(t.split(lengths) for t in tensors))])


def _attend(q, k, v, scale, window=None, sink=False):
    """q [T, H, dk] over k [T, G, dk] and v [T, G, dv]; causal, a window, a sink of score 0."""
    T, H = q.shape[:2]
    k, v = (t.repeat_interleave(H // t.shape[1], dim=1).transpose(0, 1) for t in (k, v))
    out = torch.empty((T, H, v.shape[-1]), dtype=q.dtype, device=q.device)
    chunk = max(1, min(T, (1 << 27) // max(1, H * T)))
    for a in range(0, T, chunk):
        b = min(T, a + chunk)
        lo = max(0, a - window + 1) if window else 0
        i = torch.arange(a, b, device=q.device)[:, None]
        j = torch.arange(lo, b, device=q.device)[None, :]
        see = (j <= i) & (i - j < window if window else j <= i)
        s = (q[a:b].transpose(0, 1) @ k[:, lo:b].transpose(1, 2) * scale).masked_fill(~see, -math.inf)
        top = s.amax(dim=-1, keepdim=True)
        if sink:
            top = top.clamp(min=0.0)
        e = (s - top).exp()
        den = e.sum(dim=-1, keepdim=True) + ((-top).exp() if sink else 0.0)
        out[a:b] = ((e / den) @ v[:, lo:b]).transpose(0, 1)
    return out


def _rows(x, *matrices, fn=None):
    """fn(x A^T, ...) or x A^T, in slices of rows."""
    fn = fn or (lambda y: y)
    return torch.cat([fn(*(part @ m.T for m in matrices)) for part in x.split(8192)])


def _llama_exact(cfg, seed, dtype, sequences, wanted):
    w, eps = _weights(cfg, seed, dtype), cfg["rms_norm_eps"]
    d, H, G, hd, f, V = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                          "intermediate_size", "vocab_size"))
    lengths = [len(s) for s in sequences]
    ids = torch.tensor([t for s in sequences for t in s], device="cuda")
    pos = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    embed = w("model.embed_tokens.weight", V, d)
    x = embed[ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}"
        h = _rms(x, eps)
        q, k, v = (_rows(h, w(f"{p}.self_attn.{n}_proj.weight", heads * hd, d)).view(-1, heads, hd)
                   for n, heads in (("q", H), ("k", G), ("v", G)))
        q, k = _turn(q, pos, hd, cfg["rope_theta"]), _turn(k, pos, hd, cfg["rope_theta"])
        a = _spread(lengths, lambda q, k, v: _attend(q, k, v, hd ** -0.5), q, k, v).reshape(-1, H * hd)
        x = x + _rows(a, w(f"{p}.self_attn.o_proj.weight", d, H * hd))
        del h, q, k, v, a
        h = _rows(_rms(x, eps), w(f"{p}.mlp.gate_proj.weight", f, d), w(f"{p}.mlp.up_proj.weight", f, d),
                  fn=lambda g, u: torch.nn.functional.silu(g) * u)
        x = x + _rows(h, w(f"{p}.mlp.down_proj.weight", d, f))
        del h
    head = embed if cfg["tie_word_embeddings"] else w("lm_head.weight", V, d)
    return _rms(x[torch.tensor(wanted, device="cuda")], eps) @ head.T


def _senulix_exact(cfg, seed, dtype, sequences, wanted):
    w, eps, d, V = _weights(cfg, seed, dtype), cfg["norm"]["eps"], cfg["width"], cfg["vocab"]
    P, n_layers = cfg["token_side"]["dim"], len(cfg["layers"])
    lengths = [len(s) for s in sequences]
    ids = torch.tensor([t for s in sequences for t in s], device="cuda")
    pos = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    x = w("embed", V, d)[ids]
    side = w("side.embed", V, P * n_layers)[ids]
    latents = {}
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix", L["mixer"]
        H = m["heads"]
        if L["type"] == "attention":                     # the mixing matrix is drawn as the identity
            G, dk = m["kv_heads"], m["dim"]
            q = _rms(x @ w(p + ".q", H * dk, d).T, eps).view(-1, H, dk)
            k = _rms(x @ w(p + ".k", G * dk, d).T, eps).view(-1, G, dk)
            v = (x @ w(p + ".v", G * m["vdim"], d).T).view(-1, G, m["vdim"])
            q, k = (_turn(t, pos, m["rot"]["dims"], m["rot"]["base"]) for t in (q, k))
            y = _spread(lengths, lambda q, k, v: _attend(q, k, v, m["scale"], m["mask"]["size"], sink=True), q, k, v)
        elif L["type"] == "latent_attention":
            dk, dr, R = m["dim"], m["rot_dim"], m["kv_rank"]
            q = (x @ w(p + ".q", H * (dk + dr), d).T).view(-1, H, dk + dr)
            q = torch.cat([q[..., :dk], _turn(q[..., dk:], pos, dr, m["rot"]["base"])], dim=-1)
            if m.get("kv_from") is None:
                down = x @ w(p + ".dkv", R + dr, d).T
                latents[i] = (_rms(down[:, :R], eps), _turn(down[:, None, R:], pos, dr, m["rot"]["base"]))
            c, kr = latents[i if m.get("kv_from") is None else m["kv_from"]]
            k = torch.cat([(c @ w(p + ".uk", H * dk, R).T).view(-1, H, dk), kr.expand(-1, H, dr)], dim=-1)
            v = (c @ w(p + ".uv", H * m["vdim"], R).T).view(-1, H, m["vdim"])
            y = _spread(lengths, lambda q, k, v: _attend(q, k, v, m["scale"]), q, k, v)
        else:
            q, k, v = (torch.nn.functional.silu(x @ w(f"{p}.{n}", H * m["dim"], d).T).view(-1, H, m["dim"]) for n in "qkv")
            decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda").float().double()

            def scan(q, k, v):
                o, S = torch.empty_like(v), torch.zeros((H, m["dim"], m["vdim"]), dtype=v.dtype, device="cuda")
                for a in range(0, v.shape[0], 64):       # within 64 rows the products, before them the state
                    qc, kc, vc = (t[a:a + 64].transpose(0, 1) for t in (q, k, v))
                    n = qc.shape[1]
                    t = torch.arange(n, dtype=torch.float64, device="cuda")
                    gap = t[:, None] - t[None, :]
                    mask = torch.where(gap >= 0, decay[:, None, None] ** gap.clamp(min=0), torch.zeros_like(gap))
                    o[a:a + 64] = ((qc @ kc.transpose(1, 2) * mask) @ vc + qc @ S * decay[:, None, None] ** (t + 1)[:, None]
                                   ).transpose(0, 1)
                    S = S * decay[:, None, None] ** n + (kc * decay[:, None, None] ** (n - 1 - t)[:, None]).transpose(1, 2) @ vc
                return o
            y = _rms(_spread(lengths, scan, q, k, v).reshape(-1, H * m["vdim"]), eps) * torch.sigmoid(
                x @ w(p + ".g", H * m["vdim"], d).T)
        x = x + _rms(y.reshape(-1, H * m["vdim"]) @ w(p + ".o", d, H * m["vdim"]).T, eps)
        if L["mlp"]:
            ff = L["mlp"]["ff"]
            y = torch.nn.functional.gelu(x @ w(f"l{i}.mlp.up", ff, d).T) @ w(f"l{i}.mlp.down", d, ff).T
            x = x + _rms(y, eps)
        g = torch.nn.functional.gelu(x @ w(f"l{i}.side.gate", P, d).T, approximate="tanh") * side[:, i * P:(i + 1) * P]
        x = x + _rms(g @ w(f"l{i}.side.proj", d, P).T, eps)
    z = _rms(x[torch.tensor(wanted, device="cuda")], eps) @ w("head", V, d).T
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def exact(case, seed):
    if case["kind"] == "generate":
        return None               # whole numbers
    cfg = MODELS[case["model"]]
    tokens = _tokens(case, seed)
    sequences = [a + b for a, b in tokens]
    if 2.0 * sum(len(s) for s in sequences) * sum(m[0] for m in _mixers(cfg)) > 2.5e14:
        return None               # over about 20 seconds in 64 bits
    begin, n = [], 0
    for s in sequences:
        begin.append(n)
        n += len(s)
    forward = _llama_exact if "num_hidden_layers" in cfg else _senulix_exact
    with torch.no_grad():
        if case["kind"] == "step":
            wanted = [at + len(a) + w for at, (a, b) in zip(begin, tokens) for w in _places(case, len(b))]
            return forward(cfg, seed, case["dtype"], sequences, wanted)
        wanted = [at + len(a) - 1 + i for i in range(case["steps"] + 1) for at, (a, _) in zip(begin, tokens)]
        return list(forward(cfg, seed, case["dtype"], sequences, wanted).split(len(tokens)))
