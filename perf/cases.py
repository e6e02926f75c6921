"""The engine's work as it is used: steps of `ModelRunner.step` with given tokens, over models that fit one GPU.

A case names a model, a type and one of three kinds of step.  *prefill*: whole prompts of `requests` requests, the longest of `tokens` tokens, the
others shorter in equal parts; the requests are opened before and closed after it.  *decode*: every one of `requests` requests brings one token on
`context` cached ones, replayed from a captured graph.  *mixed*: a prompt of `tokens` tokens beside decoding requests, a step of continuous batching
with chunked prefill.  The logits behind every prompt and every decoded token come back.

The models: Gemma-2B in full, and four-layer models of three further designs at the sizes that the benchmark names '2b' and '2k', whose mixers are
gated linear attention, retention, softmax attention with sinks, biases, windows or scaled turns, latent attention, the delta rule with a decay per head
or per key channel, and a state space.  Their feed-forwards are all dense: a routed layer sends a token whose scores nearly tie to another expert for
a difference in the last place, so that two correct programs may differ there without bound.
"""
from __future__ import annotations

import math

import torch

from wllm_b200.config import EngineConfig, resolve_architecture
from wllm_b200.engine import ComposedModel, StepEntry, build_runner

PAGE = 64              # tokens a cache page, as the benchmark has it
PORTION = 2048         # prompt tokens a step while a context is built
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# -- models -------------------------------------------------------------------------------------------------------------------------
def _pesanex() -> dict:
    heads, dim, vdim = 8, 128, 256
    linear = {"heads": heads, "dim": dim, "vdim": vdim, "tau": 16.0, "rank": 64}
    both = {"type": "parallel", "mlp": {"kind": "dense", "ff": 16384}, "mixer": {
        "left": {"heads": 8, "kv_heads": 1, "dim": 256, "vdim": 256, "scale": 256 ** -0.5, "rot": {"dims": 128, "base": 1e6}}, "right": linear}}
    retention = {"heads": heads, "dim": dim, "vdim": vdim, "rot": {"dims": dim, "base": 1e6},
                 "decay": [1.0 - 2.0 ** (-5 - 6.0 * i / (heads - 1)) for i in range(heads)]}
    return {"architecture": "Pesanex", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "layers": [
        {"type": "gla", "mlp": None, "mixer": linear}, both, {"type": "retention", "mlp": None, "mixer": retention}, both]}


def _gudarax() -> dict:
    dense = {"kind": "dense", "ff": 8192}
    attention = {"type": "attention", "mlp": dense, "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                                              "mask": {"size": 1024}, "v_mix": True}}
    latent = {"type": "latent_attention", "mlp": dense, "mixer": {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "q_rank": 768, "scale": 128 ** -0.5}}
    delta = {"type": "delta", "mlp": dense, "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4}}
    return {"architecture": "Gudarax", "vocab": 32000, "width": 2048, "max_positions": 16384, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "token_side": {"dim": 256}, "layers": [attention, latent, delta, attention]}


def _vifirax() -> dict:
    dense = {"kind": "dense", "ff": 6144}
    attention = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                 "rot": {"dims": 64, "base": 5e5, "scaling": {"factor": 8.0, "original": 4096, "fast": 24.0, "slow": 2.0}}}
    return {"architecture": "Vifirax", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "logit_scale": 0.5, "layers": [
        {"type": "mamba2", "mlp": dense, "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}},
        {"type": "channel_delta", "mlp": dense, "mixer": {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 128, "gate_rank": 128}},
        {"type": "attention", "mlp": dense, "mixer": attention}, {"type": "attention", "mlp": dense, "mixer": {**attention, "kv_from": 2}}]}


CONFIGS = {
    "gemma-2b": {"architectures": ["GemmaForCausalLM"], "vocab_size": 256000, "hidden_size": 2048, "intermediate_size": 16384, "num_hidden_layers": 18,
                 "num_attention_heads": 8, "num_key_value_heads": 1, "head_dim": 256, "rms_norm_eps": 1e-6, "rope_theta": 10000.0,
                 "max_position_embeddings": 8192},
    "pesanex-2b": _pesanex(), "gudarax-2k": _gudarax(), "vifirax-2k": _vifirax(),
}


def _config(model: str):
    raw = CONFIGS[model]
    arch = resolve_architecture(raw.get("architectures") or raw["architecture"])
    return arch, arch.config_class.from_dict(raw, where=model)


def _empty_model(case: dict) -> ComposedModel:
    arch, cfg = _config(case["model"])
    return ComposedModel(arch.make_plan(cfg), DTYPES[case["dtype"]])


def _weights(case: dict, seed: int, model: ComposedModel) -> dict:
    """Matrices N(0, 0.02) and gains near their neutral value; steps and decays as such models are initialised and stay: a head or channel forgets
    within a few tokens or within a thousand."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype, gemma = DTYPES[case["dtype"]], case["model"] == "gemma-2b"
    around_zero = ("norm1", "norm2", "final.norm") if case["model"] == "vifirax-2k" else ()       # gains that a norm adds to one

    def randn(shape, std):
        return torch.randn(shape, generator=g, device="cuda") * std

    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo
    out = {}
    for ps in model.param_specs():
        name, shape = ps.name, tuple(ps.shape)
        if gemma:
            t = randn(shape, 0.1 if ps.kind == "vector" else 0.02)
        elif name.endswith(".conv"):
            t = randn(shape, 0.4)
        elif name.endswith(".A_log"):
            t = torch.log(uniform(shape, 1.0, 16.0))
        elif name.endswith(".dt_bias"):
            step = torch.exp(uniform(shape, math.log(1e-3), math.log(1e-1)))
            t = step + torch.log(-torch.expm1(-step))
        elif name.endswith(".a2.b"):
            t = uniform(shape, 1.0, 5.0)
        elif name.endswith(".vmix"):
            t = uniform(shape, 0.3, 0.7)
        elif name.endswith((".q.b", ".k.b", ".v.b", ".o.b", ".conv.b", ".sink")):
            t = randn(shape, 0.2)
        elif ps.kind == "vector":
            t = randn(shape, 0.1) + (0.0 if name.endswith(around_zero) and around_zero else 1.0)
        else:
            t = randn(shape, 1.0 if name in ("embed", "side.embed") else 0.02)
        out[name] = t.to(dtype)
    return out


# -- cases --------------------------------------------------------------------------------------------------------------------------
def _case(name, model, kind, requests=1, tokens=0, context=0, dtype="bfloat16") -> dict:
    return {"name": name, "model": model, "dtype": dtype, "kind": kind, "requests": requests, "tokens": tokens, "context": context}


def listed() -> list:
    return [
        # one conversation, every token waited for
        _case("gemma decode 1 x 1024", "gemma-2b", "decode", 1, 0, 1024),
        # a small server with long contexts: weights and cached keys read for eight tokens
        _case("gemma decode 8 x 4096", "gemma-2b", "decode", 8, 0, 4096),
        # a busy server: the keys and values are as much as the weights, the products have 64 rows
        _case("gemma decode 64 x 1024", "gemma-2b", "decode", 64, 0, 1024),
        # short questions that arrive together, of odd lengths: the time to their first tokens
        _case("gemma prompts to 33", "gemma-2b", "prefill", 3, 33),
        # a document: the prompt length that the benchmark quotes
        _case("gemma prompt 2048", "gemma-2b", "prefill", 1, 2048),
        # continuous batching: a ragged portion of a prompt rides with decoded tokens
        _case("gemma 1531 beside 24", "gemma-2b", "mixed", 24, 1531, 1100),
        # the 32-bit path, which the equality checks and reference runs take
        _case("gemma float32 prompt 509", "gemma-2b", "prefill", 1, 509, 0, "float32"),
        # linear attention and retention beside softmax attention, whole prompt
        _case("pesanex prompt 2048", "pesanex-2b", "prefill", 1, 2048),
        # windowed, latent and delta-rule layers, prompts of odd lengths that arrive together
        _case("gudarax prompts to 1021", "gudarax-2k", "prefill", 3, 1021),
        # state space and delta rule with a decay per channel, whole prompt
        _case("vifirax prompt 2048", "vifirax-2k", "prefill", 1, 2048),
        # recurrent layers token by token: state read and written beside the weights
        _case("vifirax decode 8 x 2048", "vifirax-2k", "decode", 8, 0, 2048),
        _case("gudarax decode 32 x 1024", "gudarax-2k", "decode", 32, 0, 1024),
    ]


def _log_uniform(rng, lo, hi) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    model = rng.choice(["gemma-2b", "gemma-2b", "pesanex-2b", "gudarax-2k", "vifirax-2k"])
    kind = rng.choice(["prefill", "prefill", "decode", "decode", "mixed"])
    dtype = "float32" if model == "gemma-2b" and kind == "prefill" and rng.random() < 0.2 else "bfloat16"
    if kind == "prefill":
        requests = rng.choice([1, 1, 2, 3, 4])
        longest = 500 if dtype == "float32" else 2048
        case = _case("", model, kind, requests, _log_uniform(rng, requests, 2 * longest // (requests + 1)), 0, dtype)
    else:
        requests = _log_uniform(rng, 1, 64 if kind == "decode" else 48)
        top = min(4096, 65536 // requests)
        # the lower part of a power of two: the block tables that a graph was captured for hold the tokens still to come
        bottom = 256 << rng.randrange(int(math.log2(top // 256)) + 1)
        context = rng.randint(bottom, bottom + bottom // 4)
        case = _case("", model, kind, requests, _log_uniform(rng, 17, 2048) if kind == "mixed" else 0, context)
    del case["name"]
    return case


def _lengths(case: dict) -> list:
    """Prompt lengths of a prefill case: the longest and equal parts of it."""
    n, r = case["tokens"], case["requests"]
    return [max(1, n * (i + 1) // r) for i in range(r)]


def _tokens(case: dict, seed: int):
    """(prompts of the pass, contexts of the decoding requests, tokens that they are given step by step)."""
    g = torch.Generator().manual_seed(seed + 7)
    raw = CONFIGS[case["model"]]
    vocab = raw.get("vocab_size") or raw["vocab"]

    def some(n):
        return torch.randint(0, vocab, (n,), generator=g).tolist()
    if case["kind"] == "prefill":
        return [some(n) for n in _lengths(case)], [], []
    contexts = [some(case["context"]) for _ in range(case["requests"])]
    prompts = [some(case["tokens"])] if case["kind"] == "mixed" else []
    return prompts, contexts, [some(case["requests"]) for _ in range(64)]


def _widest(context: int) -> int:
    """Tokens that the block table of a captured decode step holds: the table is a power of two of pages wide, at least eight."""
    width = 8
    while width * PAGE < context + 2:
        width *= 2
    return width * PAGE


def prepare(case: dict, seed: int) -> dict:
    dtype = DTYPES[case["dtype"]]
    model = _empty_model(case)
    weights = _weights(case, seed, model)
    model.load(weights.__getitem__)
    model.config = _config(case["model"])[1]
    del weights
    prompts, contexts, stream = _tokens(case, seed)
    reach = _widest(case["context"]) if contexts else 0
    pages = len(contexts) * (reach // PAGE) + sum(-(-len(p) // PAGE) for p in prompts) + 1
    engine = EngineConfig(dtype=dtype, block_size=PAGE, max_num_seqs=len(contexts) + len(prompts), device="cuda:0")
    state = {"runner": build_runner(model, engine, num_pages=pages), "prompts": prompts, "contexts": contexts, "stream": stream, "reach": reach,
             "caches": [], "steps": 0, "serial": 0}
    if case["kind"] == "decode":
        state["runner"].enable_graphs()
    if contexts:
        _begin(state)
        if case["kind"] == "decode":
            run(state)                       # captures the decode step's graph
    return state


def _begin(state: dict) -> None:
    """The decoding requests, with their contexts read in portions."""
    runner = state["runner"]
    for rc in state["caches"]:
        runner.cache.close(rc)
    state["caches"] = [_open(state) for _ in state["contexts"]]
    todo = [(rc, list(c)) for rc, c in zip(state["caches"], state["contexts"])]
    while todo:
        room, entries, rest = PORTION, [], []
        for rc, tokens in todo:
            n = min(room, len(tokens))
            if n:
                entries.append(StepEntry(rc, tokens[:n], []))
                room -= n
            if tokens[n:]:
                rest.append((rc, tokens[n:]))
        runner.step(entries)
        todo = rest
    state["steps"] = 0


def _open(state: dict):
    state["serial"] += 1
    return state["runner"].cache.open(state["serial"])


@torch.inference_mode()
def run(state: dict):
    runner = state["runner"]
    if state["caches"] and state["caches"][0].num_tokens + 1 >= state["reach"]:
        _begin(state)                        # the conversations reached their end (after hundreds of passes): new ones begin
    new = [_open(state) for _ in state["prompts"]]
    entries = [StepEntry(rc, p, [len(p) - 1]) for rc, p in zip(new, state["prompts"])]
    if state["caches"]:
        tokens = state["stream"][state["steps"] % len(state["stream"])]
        entries += [StepEntry(rc, [t], [0]) for rc, t in zip(state["caches"], tokens)]
        state["steps"] += 1
    logits = runner.step(entries)
    for rc in new:
        runner.cache.close(rc)
    return logits


# -- what a pass cannot do without ----------------------------------------------------------------------------------------------------
def _mixers(case: dict):
    """([(query heads, key/value elements a cached token, score and value elements a head, window) of every softmax layer], state elements of all layers)."""
    raw, out, state = CONFIGS[case["model"]], [], 0
    if "num_hidden_layers" in raw:
        d = raw["head_dim"]
        return [(raw["num_attention_heads"], 2 * raw["num_key_value_heads"] * d, 2 * d, None)] * raw["num_hidden_layers"], 0
    for layer in raw["layers"]:
        for m in ([layer["mixer"]["left"], layer["mixer"]["right"]] if layer["type"] == "parallel" else [layer["mixer"]]):
            if "kv_rank" in m:
                out.append((m["heads"], m["kv_rank"], m["dim"] + m["vdim"], None))
            elif "scale" in m:
                own = 0 if m.get("kv_from") is not None else 1
                out.append((m["heads"], own * m["kv_heads"] * (m["dim"] + m["vdim"]), m["dim"] + m["vdim"], (m.get("mask") or {}).get("size")))
            else:
                state += m["heads"] * m.get("state", m.get("dim")) * m["vdim"]
    return out, state


def work(case: dict) -> dict:
    """Every weight, cached key and value and state read once, every new one written once; the products, scores and recurrences of every token."""
    item = 2 if case["dtype"] == "bfloat16" else 4
    model = _empty_model(case)
    matrices = table = 0
    for ps in model.param_specs():
        if ps.kind == "matrix":
            matrices += math.prod(ps.shape)
        elif ps.name in ("model.embed_tokens.weight", "head") or (ps.name == "embed" and case["model"] == "vifirax-2k"):
            table += math.prod(ps.shape)                      # the table that the logits are a product with
    vocab = model.plan.vocab_size
    prompts = _lengths(case) if case["kind"] == "prefill" else [case["tokens"]] if case["kind"] == "mixed" else []
    decoded = [case["context"]] * (case["requests"] if case["kind"] != "prefill" else 0)
    n, rows = sum(prompts) + len(decoded), len(prompts) + len(decoded)
    softmax, state = _mixers(case)
    flops = 2.0 * n * matrices + 2.0 * rows * table + 6.0 * n * state
    bytes_ = item * (matrices + table + n * model.plan.hidden_size) + 4.0 * rows * vocab + 4.0 * state * (len(prompts) + 2 * len(decoded))
    for heads, cached, width, window in softmax:
        seen = sum(min(p + 1, window or p + 1) for length in prompts for p in range(length))
        kept = sum(min(c + 1, window or c + 1) for c in decoded)
        flops += 2.0 * heads * width * (seen + kept)
        bytes_ += item * cached * (kept + n)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict) -> dict:
    """Measured against `exact`: 3.9e-6 in 32 bits; 0.005 to 0.013 in bfloat16, so that two programs whose roundings fall differently stand up to
    0.018 apart."""
    return {"rel": 1.6e-5} if case["dtype"] == "float32" else {"rel": 2.5e-2}


# -- the same in 64 bits, plainly -------------------------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    model = _empty_model(case)
    w = _weights(case, seed, model)
    prompts, contexts, stream = _tokens(case, seed)
    done = 2 if case["kind"] == "decode" else 1               # tokens given to a decoding request up to the end of the first pass
    sequences = prompts + [c + [stream[i][r] for i in range(done)] for r, c in enumerate(contexts)]
    products = 2.0 * sum(len(s) for s in sequences) * sum(math.prod(ps.shape) for ps in model.param_specs() if ps.kind == "matrix")
    if products > 2e14:                                       # (some ten seconds)
        return None
    forward = {"gemma-2b": _gemma_plain, "pesanex-2b": _pesanex_plain, "gudarax-2k": _gudarax_plain, "vifirax-2k": _vifirax_plain}[case["model"]]
    with torch.no_grad():
        rows = [forward(CONFIGS[case["model"]], _Doubles(w, case["dtype"]), torch.tensor(s, device="cuda")) for s in sequences]
    return torch.stack(rows)


class _Doubles:
    """The weights in 64 bits, each made when it is asked for."""

    def __init__(self, tensors: dict, dtype: str):
        self.tensors, self.rounded = tensors, dtype == "bfloat16"

    def __getitem__(self, name):
        return self.tensors[name].double()

    def rows(self, name, index):
        return self.tensors[name][index].double()


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, eps):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.log1p(torch.exp(-x.abs())) + x.clamp(min=0)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _turn(x, freq, factor=1.0):
    """x [n, heads, dim]: element i of a head with element i + len(freq), by position * freq[i]."""
    half = len(freq)
    a = torch.arange(x.shape[0], dtype=x.dtype, device=x.device)[:, None] * torch.tensor(freq, dtype=x.dtype, device=x.device)[None, :]
    c, s = (torch.cos(a) * factor)[:, None, :], (torch.sin(a) * factor)[:, None, :]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], dim=-1)


def _plain_freq(dims, base):
    return [base ** (-2.0 * i / dims) for i in range(dims // 2)]


def _attend(q, k, v, scale, window=None, slope=None, sink=None):
    """q [n, heads, dim] on k, v [n, kv heads, .]; `slope` [heads] times the distance off the scores; e^sink [heads] in the denominator."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    d = torch.arange(n, device=q.device)[:, None] - torch.arange(n, device=q.device)[None, :]
    hidden = d < 0 if window is None else (d < 0) | (d >= window)
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].T * scale
        if slope is not None:
            s = s - slope[h] * d
        s = s.masked_fill(hidden, float("-inf"))
        m = s.max(-1, keepdim=True).values if sink is None else s.max(-1, keepdim=True).values.clamp(min=float(sink[h]))
        e = torch.exp(s - m)
        z = e.sum(-1, keepdim=True) if sink is None else e.sum(-1, keepdim=True) + torch.exp(sink[h] - m)
        out.append(e / z @ v[:, h // (H // G)])
    return torch.stack(out, dim=1)


def _conv(x, taps, bias=None):
    n, T = x.shape[0], taps.shape[1]
    padded = torch.cat([x.new_zeros(T - 1, x.shape[1]), x])
    y = sum(padded[T - 1 - i:T - 1 - i + n] * taps[:, T - 1 - i] for i in range(T))
    return y if bias is None else y + bias


def _scan(q, k, v, decay, beta=None):
    """o_t = S^T q_t with S = decay_t S + k_t v_t^T, or with `beta` the delta rule's S += k (beta (v - S^T k))^T.  q, k, decay [n, heads, dim or 1]."""
    n, H, D = q.shape
    S, out = q.new_zeros(H, D, v.shape[2]), torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    for t in range(n):
        S = S * decay[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - (k[t][:, None, :] @ S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None, :])
        out[t] = (q[t][:, None, :] @ S)[:, 0]
    return out


def _gemma_plain(cfg, w, ids):
    H, G, D, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    n, freq = len(ids), _plain_freq(cfg["head_dim"], cfg["rope_theta"])
    # (the bfloat16 model holds the embedding's factor in bfloat16, as checkpoints of it were trained)
    factor = math.sqrt(cfg["hidden_size"])
    x = w.rows("model.embed_tokens.weight", ids) * (float(torch.tensor(factor).bfloat16()) if w.rounded else factor)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * (1 + w[p + "input_layernorm.weight"])
        q, k, v = ((h @ w[f"{p}self_attn.{c}_proj.weight"].T).view(n, -1, D) for c in "qkv")
        x = x + _attend(_turn(q, freq), _turn(k, freq), v, D ** -0.5).reshape(n, H * D) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, eps) * (1 + w[p + "post_attention_layernorm.weight"])
        x = x + (_gelu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return (_rms(x[-1:], eps) * (1 + w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T)[0]


def _pesanex_plain(cfg, w, ids):
    eps, n = cfg["norm"]["eps"], len(ids)

    def linear(h, p, m):
        H, D, V = m["heads"], m["dim"], m["vdim"]
        q, k, v = ((h @ w[p + c].T).view(n, H, -1) for c in "qkv")
        if "decay" in m:
            freq = _plain_freq(m["rot"]["dims"], m["rot"]["base"])
            decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device).expand(n, H)[:, :, None]
            o = _rms(_scan(_turn(q, freq), _turn(k, freq) * D ** -0.5, v, decay), eps)
        else:
            z = (h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "a2.b"]
            o = _rms(_scan(q * D ** -0.5, k, v, (torch.sigmoid(z) ** (1 / m["tau"])).view(n, H, D)), eps) * w[p + "norm"]
        return o.reshape(n, H * V) * _silu(h @ w[p + "g"].T) @ w[p + "o"].T

    def softmax(h, p, m):
        freq = _plain_freq(m["rot"]["dims"], m["rot"]["base"])
        q, k, v = ((h @ w[p + c].T).view(n, -1, m["dim"]) for c in "qkv")
        return _attend(_rms(_turn(q, freq), eps), _rms(_turn(k, freq), eps), v, m["scale"], sink=w[p + "sink"]).reshape(n, -1) @ w[p + "o"].T
    x = w.rows("embed", ids)
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h = _layer_norm(x, w[p + "norm1"], eps)
        if layer["type"] == "parallel":
            y = 0.5 * (_rms(softmax(h, p + "mix.left.", m["left"]), eps) * w[p + "mix.left.out"] +
                       _rms(linear(h, p + "mix.right.", m["right"]), eps) * w[p + "mix.right.out"])
        else:
            y = linear(h, p + "mix.", m)
        x = x + _layer_norm(y, w[p + "norm1b"], eps)
        if layer["mlp"]:
            h = _layer_norm(x, w[p + "norm2"], eps)
            y = (torch.relu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
            x = x + _layer_norm(y, w[p + "norm2b"], eps)
    return (_layer_norm(x[-1:], w["final.norm"], eps) @ w["head"].T)[0]


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _delta_inputs(h, w, p, m):
    n, G, H = len(h), m["kv_heads"], m["heads"]
    q, k, v = (_silu(_conv(h @ w[p + c].T, w[f"{p}{c}.conv"])) for c in "qkv")
    q, k = (_unit(t.view(n, G, m["dim"])).repeat_interleave(H // G, dim=1) for t in (q, k))
    return q * m["dim"] ** -0.5, k, v.view(n, H, m["vdim"]), torch.sigmoid(h @ w[p + "b"].T)


def _gudarax_plain(cfg, w, ids):
    eps, n, side = cfg["norm"]["eps"], len(ids), cfg["token_side"]["dim"]
    x, first = w.rows("embed", ids) * cfg["embedding"]["scale"] + w["pos"][:n], None
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        h = _rms(x, eps) * w[f"l{i}.norm1"]
        if layer["type"] == "attention":
            q, k = (_rms(h @ w[p + c].T + w[f"{p}{c}.b"], eps) * w[f"{p}{c}.norm"] for c in "qk")
            v = h @ w[p + "v"].T + w[p + "v.b"]
            v, first = (v, v) if first is None else ((1 - w[p + "vmix"]) * v + w[p + "vmix"] * first, first)
            slope = [2.0 ** (-8.0 * (a + 1) / m["heads"]) for a in range(m["heads"])]
            y = _attend(q.view(n, -1, m["dim"]), k.view(n, -1, m["dim"]), v.view(n, -1, m["vdim"]), m["scale"], m["mask"]["size"], slope)
            y = y.reshape(n, -1)
        elif layer["type"] == "latent_attention":
            q = (_rms(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T
            c = _rms(h @ w[p + "dkv"].T, eps) * w[p + "dkv.norm"]
            k, v = c @ w[p + "uk"].T, c @ w[p + "uv"].T
            y = _attend(q.view(n, -1, m["dim"]), k.view(n, -1, m["dim"]), v.view(n, -1, m["vdim"]), m["scale"]).reshape(n, -1)
            y = y * torch.sigmoid(h @ w[p + "g"].T)
        else:
            q, k, v, beta = _delta_inputs(h, w, p, m)
            decay = torch.exp(-torch.exp(w[p + "A_log"]) * _softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
            y = (_rms(_scan(q, k, v, decay[:, :, None], beta), eps) * w[p + "norm"]).reshape(n, -1) * _silu(h @ w[p + "g"].T)
        x = x + y @ w[p + "o"].T
        h, p = _rms(x, eps) * w[f"l{i}.norm2"], f"l{i}.mlp."
        x = x + (_silu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T
        own = w.rows("side.embed", ids)[:, i * side:(i + 1) * side]
        x = x + _rms((_gelu(x @ w[f"l{i}.side.gate"].T) * own) @ w[f"l{i}.side.proj"].T, eps) * w[f"l{i}.side.norm"]
    return (_rms(x[-1:], eps) * w["final.norm"] @ w["head"].T)[0]


def _stretched(rot):
    """(frequencies, factor on sines and cosines): pairs that turn often over the original context keep theirs, slow ones are divided by the factor."""
    dims, base, s = rot["dims"], rot["base"], rot["scaling"]

    def at(turns):
        return dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [f * (1 - r) + f / s["factor"] * r for f, r in zip(_plain_freq(dims, base), ramp)], 0.1 * math.log(s["factor"]) + 1.0


def _vifirax_plain(cfg, w, ids):
    eps, n, kept = cfg["norm"]["eps"], len(ids), {}
    x = w.rows("embed", ids)
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        if layer["type"] == "attention":
            freq, factor = _stretched(m["rot"])
            q = _turn((_rms(x @ w[p + "q"].T + w[p + "q.b"], eps) * w[p + "q.norm"]).view(n, -1, m["dim"]), freq, factor)
            if m.get("kv_from") is None:
                k = _turn((_rms(x @ w[p + "k"].T + w[p + "k.b"], eps) * w[p + "k.norm"]).view(n, -1, m["dim"]), freq, factor)
                kept[i] = k, (x @ w[p + "v"].T + w[p + "v.b"]).view(n, -1, m["vdim"])
            k, v = kept[m.get("kv_from") if m.get("kv_from") is not None else i]
            y = _attend(q, k, v, m["scale"], sink=torch.zeros(m["heads"], dtype=x.dtype, device=x.device))
            y = (y * torch.sigmoid(x @ w[p + "g"].T)[:, :, None]).reshape(n, -1) @ w[p + "o"].T + w[p + "o.b"]
        elif layer["type"] == "mamba2":
            H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            z, xbc, dt = torch.split(x @ w[p + "in"].T, [H * V, H * V + 2 * G * N, H], dim=-1)
            u, B, C = torch.split(_silu(_conv(xbc, w[p + "conv"], w[p + "conv.b"])), [H * V, G * N, G * N], dim=-1)
            B, C = (t.view(n, G, N).repeat_interleave(H // G, dim=1) for t in (B, C))
            dt, u = _softplus(dt + w[p + "dt_bias"]), u.view(n, H, V)
            y = _scan(C, B, u * dt[:, :, None], torch.exp(-torch.exp(w[p + "A_log"]) * dt)[:, :, None]) + w[p + "D"][:, None] * u
            y = _rms((y.reshape(n, -1) * _silu(z)).view(n, m["norm_groups"], -1), eps).reshape(n, -1) * w[p + "norm"] @ w[p + "o"].T
        else:
            q, k, v, beta = _delta_inputs(x, w, p, m)
            z = ((x @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"]).view(n, m["heads"], m["dim"])
            decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * _softplus(z))
            y = (_rms(_scan(q, k, v, decay, beta), eps) * w[p + "norm"]).reshape(n, -1)
            y = y * torch.sigmoid((x @ w[p + "g1"].T) @ w[p + "g2"].T) @ w[p + "o"].T
        x = x + _rms(y, eps) * (1 + w[f"l{i}.norm1"])
        p = f"l{i}.mlp."
        x = x + _rms((_silu(x @ w[p + "gate"].T) * (x @ w[p + "up"].T)) @ w[p + "down"].T, eps) * (1 + w[f"l{i}.norm2"])
    return (_rms(x[-1:], eps) * (1 + w["final.norm"]) @ w["embed"].T)[0] * cfg["logit_scale"]
