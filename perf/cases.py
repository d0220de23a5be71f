"""Performance cases of the library: the calls that a program makes which generates text, scores given text or serves several
sequences at once with it, over the three model families. Sizes are those of the repository's own configurations
(puppygrad_b200/synthetic.py, puppygrad_b200/layered_bench.py, bench.py).

A program keeps a loaded model for all its requests, so a model is loaded once per process, with weights of a fixed seed; what
`prepare` makes from its seed is the request: token ids, and the cache that they run in. Every pass starts its sequences
anew. Continuations are given token ids where a choice that hangs on the last bit would change all that follows (sampled
tokens, BF16 products); single-sequence and FP32-grade greedy decoding feed their own tokens back.
"""
import functools
import json
import math
import os
import tempfile

import numpy as np
import torch

import puppygrad_b200 as pg

TOP_K = 40
VOCAB = 32000  # of the layered models; GPT-2 has 50257
GPT2_SIZES = {"small": (768, 12, 12), "medium": (1024, 24, 16), "xl": (1600, 48, 25)}  # width, layers, heads
GPT2_VOCAB, GPT2_POSITIONS = 50257, 1024
LAYERED_DEPTH, LAYERED_CONTEXT = 8, 9216


# ------------------------------------------------------------------ the cases
def _case(name, model, mode, path, batch, prompt, steps, ragged=False):
    """`prompt` is the longest prompt; `ragged`: the others are shorter, each by another amount."""
    return {"name": name, "model": model, "mode": mode, "path": path, "batch": batch, "prompt": prompt, "steps": steps, "ragged": ragged}


def listed():
    return [
        # the first token of a short question, one user, the library's default arithmetic: nothing but latency
        _case("small_first_token", "gpt2-small", "fp32", "prefill", 1, 11, 0),
        # one user's greedy completion (the repository's first benchmark configuration)
        _case("small_b1_greedy", "gpt2-small", "fp32", "greedy", 1, 32, 64),
        # several prompts at once: scoring, or the first tokens of a batch (second benchmark configuration)
        _case("small_prefill_8x1024", "gpt2-small", "tf32x3", "prefill", 8, 1024, 0),
        # a small server with two-byte weights: prompts of different lengths, top-k lists to the host's sampler
        _case("medium_b8_bf16_topk", "gpt2-medium", "bf16", "topk", 8, 75, 32, True),
        # a loaded server, greedy (third benchmark configuration: the headline number)
        _case("medium_b64_greedy", "gpt2-medium", "tf32x3", "greedy", 64, 128, 48),
        # the largest GPT-2, long prompts, top-k lists to the host's sampler (fourth benchmark configuration)
        _case("xl_b32_topk", "gpt2-xl", "tf32x3", "topk", 32, 512, 24),
        # one user of a recurrent design: a prompt, then token by token
        _case("dirurax1024_b1_topk", "dirurax-1024", "bf16", "topk", 1, 512, 64),
        # a batch of prompts through the scans and the block-local attention
        _case("dirurax2048_prefill_8x1024", "dirurax-2048", "bf16", "prefill", 8, 1024, 0),
        # a loaded server with short prompts of different lengths
        _case("dirurax2048_b64_topk", "dirurax-2048", "bf16", "topk", 64, 70, 24, True),
        # continuous batching: in every call some sequences append a piece of their prompt and the others one token
        _case("sanesun1024_b12_portions", "sanesun-1024", "bf16", "portions", 12, 257, 10, True),
        # a loaded server with prompts longer than the attention window
        _case("sanesun2048_b64_topk", "sanesun-2048", "bf16", "topk", 64, 70, 24, True),
        # one long document
        _case("sanesun2048_prefill_1x8192", "sanesun-2048", "bf16", "prefill", 1, 8192, 0),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    """Sequences, lengths, paths and arithmetic over the ranges between the listed cases; at most about 8192 prompt tokens."""
    family = rng.choice(("gpt2", "gpt2", "dirurax", "sanesun"))
    if family == "gpt2":
        size, mode = rng.choice(("small", "medium")), rng.choice(("fp32", "tf32x3", "tf32x3", "bf16", "int8"))
        model, longest, paths = "gpt2-" + size, GPT2_POSITIONS - 64, ("prefill", "greedy", "topk")
    else:
        mode = "bf16"
        model, longest, paths = "%s-%d" % (family, rng.choice((1024, 2048))), 8192, ("prefill", "topk", "portions")
    path = rng.choice(paths)
    batch = rng.choice((1, _log_int(rng, 2, 8), _log_int(rng, 9, 64)))
    prompt = _log_int(rng, 7, max(8, min(longest, (2048 if mode == "fp32" else 8192) // batch)))
    steps = 0 if path == "prefill" else _log_int(rng, 4, 12) if path == "portions" else _log_int(rng, 8, 48)
    case = _case("", model, mode, path, batch, prompt, steps, rng.random() < 0.6)
    del case["name"]
    return case


def _lengths(case):
    """Tokens of each sequence's prompt: from the case alone, so that every seed is the same work."""
    n = case["prompt"]
    if not case["ragged"]:
        return [n] * case["batch"]
    return [n - (i * 37 + i * i) % max(1, n // 2 + 1) for i in range(case["batch"])]


def _portion_plan(case):
    """Calls of the path "portions": [(slot, from, to)] each. Sequence i appends its prompt in i % 3 + 1 pieces, then one token a call."""
    lens, at, plan = _lengths(case), [0] * case["batch"], []
    for _ in range(case["steps"]):
        call = []
        for i, n in enumerate(lens):
            piece = -(-n // (i % 3 + 1))
            to = min(n, at[i] + piece) if at[i] < n else at[i] + 1
            call.append((i, at[i], to))
            at[i] = to
        plan.append(call)
    return plan, at


# ------------------------------------------------------------------ weights (on the GPU, from the model's name alone)
def _generator(model):
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(ord(c) * 131 ** (i % 5) for i, c in enumerate(model)) % (1 << 31))
    return g


def _gpt2_config(model):
    c, layers, heads = GPT2_SIZES[model.split("-")[1]]
    return dict(vocab_size=GPT2_VOCAB, n_positions=GPT2_POSITIONS, n_embd=c, n_layer=layers, n_head=heads, n_inner=4 * c, layer_norm_epsilon=1e-5)


def _gpt2_weights(model):
    """Yields (name, FP32 tensor): random init as in the benchmark configurations."""
    cfg, g = _gpt2_config(model), _generator(model)
    c, f = cfg["n_embd"], cfg["n_inner"]

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda") * 0.02

    def pair(name, n):
        yield name + ".weight", torch.ones(n, device="cuda")
        yield name + ".bias", torch.zeros(n, device="cuda")

    yield "wte.weight", normal(GPT2_VOCAB, c)
    yield "wpe.weight", normal(GPT2_POSITIONS, c)
    yield from pair("ln_f", c)
    for i in range(cfg["n_layer"]):
        p = "h.%d." % i
        yield from pair(p + "ln_1", c)
        for name, rows, cols in (("attn.c_attn", c, 3 * c), ("attn.c_proj", c, c)):
            yield p + name + ".weight", normal(rows, cols)
            yield p + name + ".bias", torch.zeros(cols, device="cuda")
        yield from pair(p + "ln_2", c)
        for name, rows, cols in (("mlp.c_fc", c, f), ("mlp.c_proj", f, c)):
            yield p + name + ".weight", normal(rows, cols)
            yield p + name + ".bias", torch.zeros(cols, device="cuda")


def _layered_config(model):
    """The layers of the repository's benchmark of layered models."""
    family, width = model.split("-")[0], int(model.split("-")[1])
    ff = {"kind": "dense", "ff": 4 * width}
    if family == "dirurax":
        gla = {"type": "gla", "mixer": {"heads": width // 128, "dim": 64, "vdim": 128, "tau": 16.0}, "mlp": ff}
        left = {"heads": width // 64, "kv_heads": width // 256, "dim": 64, "vdim": 64, "mask": {"size": 512}, "scale": 0.125}
        both = {"type": "parallel", "mlp": ff, "mixer": {"left": left, "right": {"heads": width // 64, "dim": 64}, "left_scale": 0.7, "right_scale": 0.7}}
        cycle, more = (gla, gla, gla, both), {"architecture": "Dirurax"}
    else:
        att = {"type": "attention", "mlp": ff,
               "mixer": {"heads": width // 64, "kv_heads": width // 256, "dim": 64, "vdim": 64, "scale": 0.125,
                         "rot": {"dims": 32, "base": 1e4}, "mask": {"size": 512, "keep_first": 4}}}
        delta = {"type": "channel_delta", "mlp": ff, "mixer": {"heads": width // 128, "kv_heads": width // 128, "dim": 128, "vdim": 128, "conv": 4}}
        latent = {"type": "latent_attention", "mlp": ff,
                  "mixer": {"heads": width // 128, "dim": 128, "vdim": 128, "kv_rank": 512, "q_rank": 3 * width // 8, "scale": 128 ** -0.5}}
        cycle, more = (att, delta, latent, delta), {"architecture": "Sanesun", "embedding": {"scale": 1.0}}
    return dict(more, vocab=VOCAB, width=width, norm={"eps": 1e-5}, layers=[cycle[i % 4] for i in range(LAYERED_DEPTH)])


def _layered_shapes(cfg):
    """{tensor name: (shape, mean, deviation)}: inputs of products of unit size, norms around 1, decays near 1."""
    W, out = cfg["width"], {}

    def mat(name, n, k, gain=1.0):
        out[name] = ((n, k), 0.0, gain / math.sqrt(k))

    def vec(name, n, mean=1.0, dev=0.1):
        out[name] = ((n,), mean, dev)

    def norm(name):  # LayerNorm
        vec(name, W)
        vec(name + ".b", W, 0.0)

    out["embed"] = ((cfg["vocab"], W), 0.0, 1.0)
    if cfg["architecture"] == "Dirurax":
        norm("final.norm")
    else:
        mat("head", cfg["vocab"], W)
        vec("final.norm", W)
    for i, layer in enumerate(cfg["layers"]):
        p, m, kind = "l%d.mix." % i, layer["mixer"], layer["type"]
        if cfg["architecture"] == "Dirurax":
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                norm("l%d.%s" % (i, n))
        else:
            vec("l%d.norm1" % i, W)
            vec("l%d.mlp.act" % i, 2, 0.5)
        if kind == "gla":
            K, V = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            for n, r in (("k", K), ("q", K), ("v", V), ("g", V), ("a1", 64)):
                mat(p + n, r, W)
            mat(p + "a2", K, 64)
            vec(p + "a2.b", K, 3.0)
            vec(p + "norm", m["vdim"])
            mat(p + "o", W, V)
        elif kind == "parallel":
            a, r = m["left"], m["right"]
            for n, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                mat(p + "left." + n, rows, W)
            vec(p + "left.q.norm", a["dim"])
            vec(p + "left.k.norm", a["dim"])
            mat(p + "left.o", W, a["heads"] * a["vdim"])
            K = r["heads"] * r["dim"]
            for n in "krvga":
                mat(p + "right." + n, K, W)
            mat(p + "right.w1", 64, W)
            mat(p + "right.w2", K, 64)
            vec(p + "right.w0", K, -4.0)
            vec(p + "right.a.b", K, -1.0)
            vec(p + "right.norm", K)
            mat(p + "right.o", W, K)
        elif kind == "attention":
            H = m["heads"]
            for n, rows in (("q", H * m["dim"]), ("k", m["kv_heads"] * m["dim"]), ("v", m["kv_heads"] * m["vdim"])):
                mat(p + n, rows, W)
                vec(p + n + ".b", rows, 0.0)
            mat(p + "talk", H, H, 0.4)  # beside the unit matrix, below
            vec(p + "sink", H)
            mat(p + "o", W, H * m["vdim"])
        elif kind == "channel_delta":
            H, Q, V = m["heads"], m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
            for n, rows in (("q", Q), ("k", Q), ("v", V)):
                mat(p + n, rows, W)
                mat(p + n + ".conv", rows, m["conv"])
            for n, rows, k in (("b", H, W), ("a1", 128, W), ("a2", H * m["dim"], 128), ("g1", 128, W), ("g2", V, 128)):
                mat(p + n, rows, k)
            vec(p + "A_log", H, -1.0)
            vec(p + "dt_bias", H * m["dim"], -3.0)
            vec(p + "norm", m["vdim"])
            mat(p + "o", W, V)
        else:
            H, V = m["heads"], m["heads"] * m["vdim"]
            for n, rows, k in (("dq", m["q_rank"], W), ("uq", H * m["dim"], m["q_rank"]), ("dkv", m["kv_rank"], W),
                               ("uk", H * m["dim"], m["kv_rank"]), ("uv", V, m["kv_rank"]), ("g", H, W), ("o", W, V)):
                mat(p + n, rows, k)
            vec(p + "dq.norm", m["q_rank"])
            vec(p + "dkv.norm", m["kv_rank"])
        mat("l%d.mlp.up" % i, 4 * W, W)
        mat("l%d.mlp.down" % i, W, 4 * W)
    return out


def _layered_weights(model):
    """Yields (name, BF16 tensor). Queries of Dirurax's recurrences lie partly along the keys: what a first token reads back is
    normalised, so with independent ones its direction would hang on the last bits of a product near zero."""
    g, keys = _generator(model), None
    for name, (shape, mean, dev) in _layered_shapes(_layered_config(model)).items():
        a = torch.randn(shape, generator=g, device="cuda") * dev + mean
        if name.endswith(".talk"):
            a += torch.eye(shape[0], device="cuda")
        if model.startswith("dirurax") and name.endswith((".mix.k", ".right.k")):
            keys = a
        if model.startswith("dirurax") and name.endswith((".mix.q", ".right.r")):
            a = (a + keys) * math.sqrt(0.5)
        yield name, a.bfloat16()


@functools.lru_cache(maxsize=16)
def _model(name, mode):
    if name.startswith("gpt2"):
        weights = {n: a.cpu().numpy() for n, a in _gpt2_weights(name)}
        return pg.Gpt2Model(_gpt2_config(name), weights, pg.Gpt2CudaConfig(math_mode="fp32" if mode == "int8" else mode, quantized_weights=mode == "int8"))
    with tempfile.TemporaryDirectory() as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(_layered_config(name), f)
        header, at = {}, 0
        for n, (shape, _, _) in _layered_shapes(_layered_config(name)).items():
            size = 2 * math.prod(shape)
            header[n] = {"dtype": "BF16", "shape": list(shape), "data_offsets": [at, at + size]}
            at += size
        text = json.dumps(header).encode()
        text += b" " * (-len(text) % 8)
        with open(os.path.join(folder, "model.safetensors"), "wb") as f:
            f.write(len(text).to_bytes(8, "little") + text)
            for _, a in _layered_weights(name):
                f.write(a.view(torch.int16).cpu().numpy().tobytes())
        return pg.load_model(folder, pg.CudaConfig(math_mode=mode, max_context=LAYERED_CONTEXT))


# ------------------------------------------------------------------ inputs and passes
def _tokens(case, seed):
    """Every sequence's ids, prompt and continuation."""
    vocab = GPT2_VOCAB if case["model"].startswith("gpt2") else VOCAB
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocab, n + max(1, case["steps"])) for n in _lengths(case)]


def prepare(case, seed):
    model = _model(case["model"], case["mode"])
    ids, lens = _tokens(case, seed), _lengths(case)
    state = {"case": case, "model": model, "cache": model.new_kv_cache(max_batch=case["batch"])}
    if case["path"] == "portions":
        plan, _ = _portion_plan(case)
        # the logits at the end of every piece
        state["calls"] = [([s for s, _, _ in call], [ids[s][a:b] for s, a, b in call], np.cumsum([b - a for _, a, b in call]) - 1) for call in plan]
    else:
        state["prompts"] = [a[:n] for a, n in zip(ids, lens)]
        state["steps"] = [np.array([a[n + t] for a, n in zip(ids, lens)]) for t in range(max(1, case["steps"]))]
    return state


def run(state):
    case, model, cache = state["case"], state["model"], state["cache"]
    if case["path"] == "portions":
        cache.clear()
        return [model.extend(slots, portions, cache, want) for slots, portions, want in state["calls"]]
    if case["path"] == "prefill":
        logits, _ = model.prefill_batch(state["prompts"], cache, want_logits=True)
        return {"logits": logits}
    model.prefill_batch(state["prompts"], cache)
    if case["path"] == "greedy":
        logits, first, _, _ = model.forward_one_batch(state["steps"][0], cache, want_logits=True)
        return {"logits": logits, "tokens": model.decode_greedy(first, cache, case["steps"])}
    # top-k lists of every step, the last step's logits too
    lists = [model.forward_one_batch(ids, cache, top_k=TOP_K) for ids in state["steps"][:-1]]
    logits, _, values, at = model.forward_one_batch(state["steps"][-1], cache, want_logits=True, top_k=TOP_K)
    out = {"logits": logits, "top": np.stack([x[2] for x in lists] + [values])}
    if case["mode"] != "bf16" or case["model"].startswith("gpt2"):  # FP32-grade logits: their order is worth comparing
        out["top_ids"] = np.stack([x[3] for x in lists] + [at])
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _mixer_work(cfg, layer):
    """(weights, state bytes of a sequence, FLOPs of a token beside the weights', keys' bytes of a visible position, FLOPs of
    a (query, key) pair, (block or window) size or 0) of one layer's mixer."""
    W, m, kind = cfg["width"], layer["mixer"], layer["type"]
    if kind == "gla":
        K, V = m["heads"] * m["dim"], m["heads"] * m["vdim"]
        return W * (2 * K + 3 * V + 64) + 64 * K, 4 * K * m["vdim"], 6 * K * m["vdim"], 0, 0, 0
    if kind == "parallel":
        a, r = m["left"], m["right"]
        K = r["heads"] * r["dim"]
        weights = W * (2 * a["heads"] * a["dim"] + 2 * a["kv_heads"] * a["dim"] + 6 * K + 64) + 64 * K
        return weights, 4 * K * r["dim"], 10 * K * r["dim"], 4 * a["kv_heads"] * a["dim"], 4 * a["heads"] * a["dim"], a["mask"]["size"]
    if kind == "attention":
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        return W * (2 * H * d + 2 * G * d) + H * H, 0, 0, 4 * G * d, 4 * H * d + 2 * H * H, m["mask"]["size"]
    H, V = m["heads"], m["heads"] * m["vdim"]
    if kind == "channel_delta":
        K, Q = H * m["dim"], m["kv_heads"] * m["dim"]
        return W * (2 * Q + 2 * V + H + 256) + 128 * (K + V), 4 * K * m["vdim"], 8 * K * m["vdim"], 0, 0, 0
    weights = W * (m["q_rank"] + m["kv_rank"] + H + V) + H * m["dim"] * m["q_rank"] + H * (m["dim"] + m["vdim"]) * m["kv_rank"]
    return weights, 0, 0, 2 * m["kv_rank"], 2 * H * (m["dim"] + m["vdim"]), 0


def work(case):
    """Weights once for every dependent call, states and visible keys and values in and out, logits and lists out."""
    lens, gpt2 = _lengths(case), case["model"].startswith("gpt2")
    if case["path"] == "portions":
        calls = [[(a, b) for _, a, b in call] for call in _portion_plan(case)[0]]
    else:
        calls = [[(0, n) for n in lens]] + [[(n + t, n + t + 1) for n in lens] for t in range(case["steps"] + (case["path"] == "greedy"))]
    if gpt2:
        c, layers, _ = GPT2_SIZES[case["model"].split("-")[1]]
        vocab, size = GPT2_VOCAB, {"fp32": 4, "tf32x3": 4, "bf16": 2, "int8": 1}[case["mode"]]
        mixers, dense, head = [(4 * c * c, 0, 0, 8 * c, 4 * c, 0)] * layers, layers * 8 * c * c, vocab * c
    else:
        cfg = _layered_config(case["model"])
        vocab, size, head = VOCAB, 2, VOCAB * cfg["width"]
        mixers, dense = [_mixer_work(cfg, layer) for layer in cfg["layers"]], LAYERED_DEPTH * 8 * cfg["width"] ** 2
    weights = dense + sum(m[0] for m in mixers)
    flops = moved = 0.0
    for call in calls:
        rows = sum(b - a for a, b in call)
        flops += 2.0 * rows * weights + 2.0 * len(call) * head
        moved += size * (weights + head) + 4.0 * len(call) * (vocab if case["path"] in ("prefill", "portions") else 2 * TOP_K)
        for _, state, token, key, pair, span in mixers:
            flops += token * rows
            for a, b in call:
                before = min(a, span) if span else a
                n = b - a
                flops += pair * (n * before + n * (n + 1) / 2.0 if not span or n + before <= span else n * min(span, before + n))
                moved += state * (2 if a else 1) + key * (before + n)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["model"].startswith("gpt2"):
        return {"rel": 3e-5, "max": 3e-4, "differ": 0.01}
    return {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------ the same results in 64 bits
def _chunks(n, size=256):
    return [(a, min(n, a + size)) for a in range(0, n, size)]


def _attend(q, k, v, seen, scale, mix=None, sink=None):
    """q [B, H, T, d], k and v [B, G, T, d], seen(i, j) -> mask; queries a few at a time."""
    B, H, T, _ = q.shape
    k, v = (x.repeat_interleave(H // x.shape[1], dim=1) for x in (k, v))
    out, j = torch.empty(B, H, T, v.shape[-1], dtype=q.dtype, device=q.device), torch.arange(T, device=q.device)
    for b in range(B):
        for i0, i1 in _chunks(T):
            score = q[b, :, i0:i1] @ k[b].transpose(1, 2) * scale
            if mix is not None:
                score = torch.einsum("ab,bij->aij", mix, score)
            score = score.masked_fill(~seen(torch.arange(i0, i1, device=q.device)[:, None], j[None, :]), -math.inf)
            if sink is not None:
                score = torch.cat([score, sink[:, None, None].expand(H, i1 - i0, 1)], 2)
            out[b, :, i0:i1] = score.softmax(-1)[:, :, :T] @ v[b]
    return out


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _gpt2_hidden(case, ids, weights):
    """Final hidden rows [B, T, c] and the output matrix; `weights` yields the tensors in order."""
    c, layers, heads = GPT2_SIZES[case["model"].split("-")[1]]
    narrow = case["mode"]

    def given():
        name, a = next(weights)
        a = a.double()
        if a.dim() == 2 and name.startswith("h."):
            a = a.t()  # [out, in]
        return (a, rounded(a)) if a.dim() == 2 and (name.startswith("h.") or name == "wte.weight") else (a, a)

    def rounded(a):
        if narrow == "bf16":
            return a.bfloat16().double()
        if narrow == "int8":  # one scale per row
            scale = (a.float().abs().amax(1, keepdim=True) / 127.0)
            x = a.float() / scale
            return (torch.sign(x) * torch.floor(x.abs() + 0.5)).clamp(-127, 127).double() * scale.double()
        return a

    def norm(x, w, b):
        return torch.nn.functional.layer_norm(x, (c,), w, b, 1e-5)

    (wte, head), (wpe, _) = given(), given()
    lookup = head if narrow == "bf16" else wte
    ln_f = given()[1], given()[1]
    B, T = ids.shape
    x = lookup[ids] + wpe[:T]
    for _ in range(layers):
        w = [given()[1] for _ in range(12)]
        q, k, v = (norm(x, w[0], w[1]) @ w[2].t() + w[3]).view(B, T, 3, heads, c // heads).permute(2, 0, 3, 1, 4)
        a = _attend(q, k, v, lambda i, j: j <= i, (c // heads) ** -0.5)
        x = x + a.transpose(1, 2).reshape(B, T, c) @ w[4].t() + w[5]
        x = x + torch.nn.functional.gelu(norm(x, w[6], w[7]) @ w[8].t() + w[9], approximate="tanh") @ w[10].t() + w[11]
    return norm(x, *ln_f), head


def _scan(step, B, H, dk, dv, T):
    state, out = torch.zeros(B, H, dk, dv, dtype=torch.float64, device="cuda"), []
    for t in range(T):
        state, read = step(state, t)
        out.append(torch.einsum("bhkv,bhk->bhv", state, read))
    return torch.stack(out, 1)


def _turned(x, dims, base, sign=1.0):
    """x [B, T, heads, d]: entry i of the first `dims` with entry i + dims / 2, by its position."""
    half = dims // 2
    angle = sign * torch.arange(x.shape[1], dtype=x.dtype, device=x.device)[:, None] * base ** (-2.0 * torch.arange(half, dtype=x.dtype, device=x.device) / dims)
    c, s, u, v = torch.cos(angle)[:, None], torch.sin(angle)[:, None], x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _mixer(kind, m, w, h, eps):
    """One layer's mixer on h [B, T, width]; `w` by the names behind the layer's prefix."""
    B, T, _ = h.shape

    def heads(x, n):
        return x.view(B, T, n, -1)

    def flat(x):
        return x.reshape(B, T, -1)

    if kind == "gla":
        H = m["heads"]
        q, k, v = heads(h @ w["q"].t(), H) / math.sqrt(m["dim"]), heads(h @ w["k"].t(), H), heads(h @ w["v"].t(), H)
        decay = heads(torch.sigmoid(h @ w["a1"].t() @ w["a2"].t() + w["a2.b"]), H) ** (1.0 / m["tau"])
        out = _scan(lambda s, t: (decay[:, t, :, :, None] * s + k[:, t, :, :, None] * v[:, t, :, None], q[:, t]), B, H, m["dim"], m["vdim"], T)
        gate = h @ w["g"].t()
        return (flat(_rms(out, eps) * w["norm"]) * gate * torch.sigmoid(gate)) @ w["o"].t()
    if kind == "left":
        size = m["mask"]["size"]
        q = _rms(heads(h @ w["q"].t(), m["heads"]), eps) * w["q.norm"]
        k = _rms(heads(h @ w["k"].t(), m["kv_heads"]), eps) * w["k.norm"]
        v = _rms(heads(h @ w["v"].t(), m["kv_heads"]), eps)
        a = _attend(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), lambda i, j: (j <= i) & (i // size == j // size), m["scale"])
        return flat(a.transpose(1, 2)) @ w["o"].t()
    if kind == "right":
        H, d = m["heads"], m["dim"]
        r, k, v = (heads(h @ w[n].t(), H) for n in "rkv")
        decay = heads(torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w["w1"].t()) @ w["w2"].t() + w["w0"])), H)
        unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        gone = heads(torch.sigmoid(h @ w["a"].t() + w["a.b"]), H) * unit

        def step(s, t):
            read = torch.einsum("bhk,bhkv->bhv", unit[:, t], s)
            return decay[:, t, :, :, None] * s - gone[:, t, :, :, None] * read[:, :, None] + k[:, t, :, :, None] * v[:, t, :, None], r[:, t]

        return (flat(_rms(_scan(step, B, H, d, d, T), eps)) * w["norm"] * torch.sigmoid(h @ w["g"].t())) @ w["o"].t()
    if kind == "parallel":
        under = lambda p: {n[len(p):]: a for n, a in w.items() if n.startswith(p)}  # noqa: E731
        return m["left_scale"] * _mixer("left", m["left"], under("left."), h, eps) + m["right_scale"] * _mixer("right", m["right"], under("right."), h, eps)
    if kind == "attention":
        dims, base, size, keep = m["rot"]["dims"], m["rot"]["base"], m["mask"]["size"], m["mask"]["keep_first"]
        q, k, v = (heads(h @ w[n].t() + w[n + ".b"], m[c]) for n, c in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
        q, k, v = (x.transpose(1, 2) for x in (_turned(q, dims, base), _turned(k, dims, base), _turned(v, m["vdim"], base)))
        a = _attend(q, k, v, lambda i, j: (j <= i) & ((i - j < size) | (j < keep)), m["scale"], w["talk"], w["sink"])
        return flat(_turned(a.transpose(1, 2), m["vdim"], base, -1.0)) @ w["o"].t()
    H = m["heads"]
    if kind == "latent_attention":
        latent = _rms(h @ w["dkv"].t(), eps) * w["dkv.norm"]
        q = heads(_rms(h @ w["dq"].t(), eps) * w["dq.norm"] @ w["uq"].t(), H)
        k, v = heads(latent @ w["uk"].t(), H), heads(latent @ w["uv"].t(), H)
        a = _attend(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), lambda i, j: j <= i, m["scale"]).transpose(1, 2)
        return flat(a * torch.sigmoid(h @ w["g"].t())[..., None]) @ w["o"].t()

    def conv(n):  # causal, per channel, the last tap on the current token
        x, taps = h @ w[n].t(), w[n + ".conv"]
        x = torch.nn.functional.pad(x, (0, 0, taps.shape[1] - 1, 0))
        x = sum(taps[:, i] * x[:, i:i + T] for i in range(taps.shape[1]))
        return x * torch.sigmoid(x)

    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q, k, v = unit(heads(conv("q"), H)) * m["dim"] ** -0.5, unit(heads(conv("k"), H)), heads(conv("v"), H)
    beta = torch.sigmoid(h @ w["b"].t())
    decay = torch.exp(-torch.exp(w["A_log"])[:, None] * heads(torch.nn.functional.softplus(h @ w["a1"].t() @ w["a2"].t() + w["dt_bias"]), H))

    def step(s, t):
        s = decay[:, t, :, :, None] * s
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhkv,bhk->bhv", s, k[:, t]))
        return s + k[:, t, :, :, None] * u[:, :, None], q[:, t]

    out = _rms(_scan(step, B, H, m["dim"], m["vdim"], T), eps) * w["norm"]
    return flat(out * heads(torch.sigmoid(h @ w["g1"].t() @ w["g2"].t()), H)) @ w["o"].t()


def _layered_hidden(case, ids):
    cfg = _layered_config(case["model"])
    eps, W, all_w = cfg["norm"]["eps"], cfg["width"], dict(_layered_weights(case["model"]))
    T = ids.shape[1]
    layer_norm = lambda x, n: torch.nn.functional.layer_norm(x, (W,), all_w[n].double(), all_w[n + ".b"].double(), eps)  # noqa: E731
    x = all_w["embed"].double()[ids]
    dirurax = cfg["architecture"] == "Dirurax"
    if dirurax:
        angle = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] / 10000.0 ** (2.0 * torch.arange(W // 2, dtype=torch.float64, device="cuda") / W)
        x = x + torch.stack([torch.sin(angle), torch.cos(angle)], -1).reshape(T, W)
    for i, layer in enumerate(cfg["layers"]):
        p = "l%d." % i
        w = {n[len(p) + 4:]: a.double() for n, a in all_w.items() if n.startswith(p + "mix.")}
        up, down = all_w[p + "mlp.up"].double(), all_w[p + "mlp.down"].double()
        if dirurax:
            x = x + layer_norm(_mixer(layer["type"], layer["mixer"], w, layer_norm(x, p + "norm1"), eps), p + "norm1b")
            x = x + layer_norm(torch.nn.functional.gelu(layer_norm(x, p + "norm2") @ up.t()) @ down.t(), p + "norm2b")
        else:
            h = _rms(x, eps) * all_w[p + "norm1"].double()
            a, b = torch.nn.functional.softplus(all_w[p + "mlp.act"].double())
            z = h @ up.t()
            neg = z.clamp(max=0.0)
            z = torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(neg) - neg)) + 0.5 * z
            x = x + _mixer(layer["type"], layer["mixer"], w, h, eps) + z @ down.t()
    if dirurax:
        return layer_norm(x, "final.norm"), all_w["embed"].double()
    return _rms(x, eps) * all_w["final.norm"].double(), all_w["head"].double()


@torch.no_grad()
def exact(case, seed):
    """Whole sequences at once, without a cache; shorter ones are filled up behind their end, where nothing looks."""
    ids, lens = _tokens(case, seed), _lengths(case)
    if case["path"] == "portions":
        plan, used = _portion_plan(case)
    else:
        used = [n + {"prefill": 0, "greedy": 1}.get(case["path"], case["steps"]) for n in lens]
    padded = np.zeros((len(ids), max(used)), np.int64)
    for i, n in enumerate(used):
        padded[i, :n] = ids[i][:n]
    padded = torch.from_numpy(padded).cuda()
    if case["model"].startswith("gpt2"):
        hidden, head = _gpt2_hidden(case, padded, _gpt2_weights(case["model"]))
    else:
        hidden, head = _layered_hidden(case, padded)
    logits = lambda at: torch.stack([hidden[i, j] for i, j in at]) @ head.t()  # noqa: E731
    if case["path"] == "portions":
        return [logits([(s, b - 1) for s, _, b in call]).cpu() for call in plan]
    out = {"logits": logits([(i, n - 1) for i, n in enumerate(used)]).cpu()}
    if case["path"] == "greedy":
        out["tokens"] = None
    elif case["path"] == "topk":
        steps = [logits([(i, n + t) for i, n in enumerate(lens)]).topk(TOP_K) for t in range(case["steps"])]
        out["top"] = torch.stack([s.values for s in steps]).cpu()
        if case["mode"] != "bf16" or case["model"].startswith("gpt2"):
            out["top_ids"] = None
    return out
