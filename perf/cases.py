"""What this package's speed is measured on: requests served through ``Engine.step``, the package's one step function.

A case is a model and a set of requests that arrive together.  One pass takes the requests from their token ids to the
logits of every step: slots are acquired, all prompts run in one step, then every sequence goes on one given token at a
time, then the slots are given back.  Short prompts with a few steps behind them are decoding (each step reads all
weights for a few tokens), long prompts with no step behind them are prompt processing; most requests are both.  The
decoded tokens are given and not sampled, so that the logits of two implementations can be compared step by step.

The models are those of this repository's benchmark, eight layers each: the dense decoder at Qwen3-8B layer sizes, a
small dense decoder, a dense decoder in float32, and one design for each kind of recurrence (decayed linear attention,
the gated delta rule, the state-space recurrence), which between them also have routed experts, latent attention, capped
scores, distance biases, learned sinks, windows that keep first tokens and keys that are values.

Weights are random: matrices N(0, 0.02), gains near one, the other vectors as the package's random-weights mode has them.
Where a model routes tokens to experts, its embedding rows hold two of a set of directions that the routers read, a
different pair for every token, so that routing is as decided as a trained router's and does not turn on rounding.
"""

import math

import numpy as np
import torch

from llmoxide_b200 import Engine, LoadOptions, read_config

LAYERS = 8
DEV = "cuda:0"

# ---- the models -------------------------------------------------------------------------------------------------


def _dense(dtype, **sizes):
    raw = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=LAYERS, rope_theta=1000000.0,
               rms_norm_eps=1e-6, max_position_embeddings=40960, use_sliding_window=False, sliding_window=None,
               torch_dtype=dtype, eos_token_id=0, tie_word_embeddings=False)
    raw.update(sizes)
    return raw


def _nested(architecture, layers):
    return dict(architecture=architecture, vocab=32768, width=2048, norm=dict(eps=1e-6), embedding=dict(scale=1.0),
                torch_dtype="bfloat16", layers=layers)


def _moe(**more):
    return dict(kind="moe", expert=dict(ff=1024), router=dict(experts=16, top=2, **more.pop("router", {})), **more)


def _tifapel():
    decay = [1.0 - 2.0 ** -(3 + 7 * h / 15) for h in range(16)]
    mlp = lambda: _moe(router=dict(scale=1.0, groups=dict(count=4, keep=2)))
    att = lambda: dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=1024, keep_first=4))
    out = []
    for i in range(LAYERS):
        if i % 4 == 0:
            out.append(dict(type="attention", mlp=mlp(), mixer=att()))
        elif i % 4 == 1:
            out.append(dict(type="lightning", mlp=mlp(), mixer=dict(heads=16, dim=128, vdim=128, decay=decay)))
        elif i % 4 == 2:
            out.append(dict(type="retention", mlp=mlp(), mixer=dict(heads=16, dim=128, vdim=128, decay=decay,
                                                                    rot=dict(dims=128, base=1000000.0))))
        else:
            out.append(dict(type="attention", mlp=mlp(), mixer=dict(att(), kv_from=i - 3)))
    return _nested("Tifapel", out)


def _soputar():
    mlp = lambda: dict(kind="dense", ff=2048, limit=7.0)
    att = lambda: dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, softcap=30.0,
                       q_temp=dict(coef=0.1, every=1024))
    delta = dict(heads=16, kv_heads=8, dim=128, vdim=128, conv=4)
    latent = dict(heads=16, dim=96, rot_dim=32, vdim=128, kv_rank=512, scale=128 ** -0.5, rot=dict(base=10000.0, dims=32))
    out = []
    for i in range(LAYERS):
        out.append((dict(type="attention", mlp=mlp(), mixer=att()), dict(type="delta", mlp=mlp(), mixer=dict(delta)),
                    dict(type="latent_attention", mlp=mlp(), mixer=dict(latent)),
                    dict(type="attention", mlp=mlp(), mixer=dict(att(), kv_from=i - 3)))[i % 4])
    return _nested("Soputar", out)


def _gebasun():
    mlp = lambda: _moe(shared=dict(ff=1024))
    ssm = lambda: dict(type="mamba2", mlp=mlp(), mixer=dict(heads=64, vdim=64, state=128, groups=2, conv=4, norm_groups=2))
    att = dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5)
    out = []
    for i in range(LAYERS):
        out.append((ssm(), dict(type="attention", mlp=mlp(), mixer=dict(att, mask=dict(size=1024), bias_max=2048, bias_rows=32)),
                    ssm(), dict(type="attention_2", mlp=mlp(), mixer=dict(att, mask=dict(size=1024, keep_first=4),
                                                                          rot=dict(dims=64, base=10000.0))))[i % 4])
    return _nested("Gebasun", out)


def _raw(model):
    if model == "dense_8b":             # Qwen3-8B layer sizes and vocabulary
        return _dense("bfloat16", hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                      intermediate_size=12288, vocab_size=151936)
    if model == "dense_small":          # head size 64, the head tied to the embedding
        return _dense("bfloat16", hidden_size=1024, num_attention_heads=16, num_key_value_heads=8, head_dim=64,
                      intermediate_size=1536, vocab_size=32768, tie_word_embeddings=True)
    if model == "dense_float32":        # a window of 1 024
        return _dense("float32", hidden_size=2048, num_attention_heads=16, num_key_value_heads=4, head_dim=128,
                      intermediate_size=2048, vocab_size=32768, use_sliding_window=True, sliding_window=1024,
                      max_window_layers=0)
    return {"tifapel": _tifapel, "soputar": _soputar, "gebasun": _gebasun}[model]()


MODELS = ("dense_8b", "dense_small", "dense_float32", "tifapel", "soputar", "gebasun")


def _width(raw):
    return raw.get("hidden_size") or raw["width"]


def _vocab(raw):
    return raw.get("vocab_size") or raw["vocab"]


def _tensors(raw):
    """(name, shape, mean, deviation) of every tensor of the model."""
    d, V = _width(raw), _vocab(raw)
    out = []
    mat = lambda name, *shape: out.append((name, shape, 0.0, 0.02))
    vec = lambda name, *shape, mean=1.0, dev=0.02: out.append((name, shape, mean, dev))
    if "hidden_size" in raw:
        H, G, D, f = (raw[k] for k in ("num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size"))
        out.append(("model.embed_tokens.weight", (V, d), 0.0, 0.02 if raw["tie_word_embeddings"] else 1.0))
        for i in range(LAYERS):
            p = f"model.layers.{i}."
            vec(p + "input_layernorm.weight", d)
            for r, n in (("q", H * D), ("k", G * D), ("v", G * D)):
                mat(f"{p}self_attn.{r}_proj.weight", n, d)
            mat(p + "self_attn.o_proj.weight", d, H * D)
            vec(p + "self_attn.q_norm.weight", D), vec(p + "self_attn.k_norm.weight", D)
            vec(p + "post_attention_layernorm.weight", d)
            mat(p + "mlp.gate_proj.weight", f, d), mat(p + "mlp.up_proj.weight", f, d), mat(p + "mlp.down_proj.weight", d, f)
        vec("model.norm.weight", d)
        if not raw["tie_word_embeddings"]:
            mat("lm_head.weight", V, d)
        return out
    post = raw["architecture"] == "Soputar"      # its norms sit behind the sublayers, weights stored as distances from one
    norm = (lambda name: vec(name, d, mean=0.0, dev=0.1)) if post else (lambda name: vec(name, d))
    out.append(("embed", (V, d), 0.0, 1.0))
    for i, layer in enumerate(raw["layers"]):
        p, m, kind, mlp = f"l{i}.", layer["mixer"], layer["type"], layer["mlp"]
        norm(p + "norm1")
        if raw["architecture"] != "Tifapel":
            norm(p + "norm2")
        H, D, Dv = m["heads"], m.get("dim"), m["vdim"]
        x = p + "mix."
        if kind in ("attention", "attention_2"):
            G, own = m["kv_heads"], m.get("kv_from") is None
            mat(x + "q", H * D, d), mat(x + "o", d, H * Dv)
            if own:
                mat(x + "k", G * D, d)
            if own and raw["architecture"] != "Gebasun":
                mat(x + "v", G * Dv, d)
            if post:
                vec(x + "q.norm", H * D)
                if own:
                    vec(x + "k.norm", G * D)
            if raw["architecture"] == "Gebasun":
                vec(x + "q.b", H * D, mean=0.0, dev=0.05), vec(x + "k.b", G * D, mean=0.0, dev=0.05)
                vec(x + "sink", H, mean=0.0, dev=1.0)
                if kind == "attention":
                    vec(x + "o.b", d, mean=0.0, dev=0.05), vec(x + "rel", m["bias_rows"], H, mean=0.0, dev=0.5)
                else:
                    mat(x + "g", H * D, d)
        elif kind in ("lightning", "retention"):
            for r, n in (("q", H * D), ("k", H * D), ("v", H * Dv), ("g", H * Dv)):
                mat(x + r, n, d)
            mat(x + "o", d, H * Dv)
            if kind == "lightning":
                vec(x + "norm", H * Dv)
        elif kind == "latent_attention":
            R, rank = m["rot_dim"], m["kv_rank"]
            mat(x + "q", H * (D + R), d), mat(x + "dkv", rank + R, d), vec(x + "dkv.norm", rank)
            mat(x + "uk", H * D, rank), mat(x + "uv", H * Dv, rank), vec(x + "sink", H, mean=0.0, dev=1.0)
            mat(x + "o", d, H * Dv)
        elif kind == "delta":
            G = m["kv_heads"]
            for r, n in (("q", G * D), ("k", G * D), ("v", H * Dv)):
                mat(x + r, n, d), vec(x + r + ".conv", n, m["conv"], mean=0.0, dev=0.5)
            mat(x + "b", H, d), mat(x + "a", H, d), mat(x + "g", H * Dv, d), mat(x + "o", d, H * Dv)
            vec(x + "A_log", H, mean=0.0, dev=0.5), vec(x + "dt_bias", H, mean=-3.0, dev=0.5), vec(x + "norm", Dv)
        else:                                                   # mamba2
            inner, channels = H * Dv, H * Dv + 2 * m["groups"] * m["state"]
            mat(x + "in", inner + channels + H, d), mat(x + "o", d, inner)
            vec(x + "conv", channels, m["conv"], mean=0.0, dev=0.5), vec(x + "conv.b", channels, mean=0.0, dev=0.05)
            vec(x + "dt_bias", H, mean=-2.0, dev=0.5), vec(x + "A_log", H, mean=0.0, dev=0.5), vec(x + "D", H)
            vec(x + "norm", inner)
        if mlp["kind"] == "dense":
            mat(p + "mlp.gate", mlp["ff"], d), mat(p + "mlp.up", mlp["ff"], d), mat(p + "mlp.down", d, mlp["ff"])
            continue
        f, E, gated = mlp["expert"]["ff"], mlp["router"]["experts"], raw["architecture"] != "Gebasun"
        mat(p + "mlp.router", E, d)
        if not gated:
            vec(p + "mlp.router.b", E, mean=0.0, dev=0.1)
        for e in [f"e{e}" for e in range(E)] + (["shared"] if mlp.get("shared") else []):
            if gated:
                mat(f"{p}mlp.{e}.gate", f, d)
            mat(f"{p}mlp.{e}.up", f, d), mat(f"{p}mlp.{e}.down", d, f)
    norm("final.norm")
    mat("head", V, d)
    return out


def _weights(raw, seed):
    """name -> tensor on the GPU, in the dtype that a checkpoint of this model holds."""
    dtype = {"bfloat16": torch.bfloat16, "float32": torch.float32}[raw["torch_dtype"]]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    w = {}
    for name, shape, mean, dev in _tensors(raw):
        w[name] = torch.empty(shape, dtype=dtype, device=DEV).normal_(mean, dev, generator=gen)
    routers = [n for n in w if n.endswith("mlp.router")]
    if routers:
        E, d = w[routers[0]].shape
        V = w["embed"].shape[0]
        dirs = torch.randn((E, d), generator=gen, device=DEV)
        dirs /= dirs.norm(dim=1, keepdim=True)
        first = torch.randint(0, E, (V,), generator=gen, device=DEV)
        second = (first + torch.randint(1, E, (V,), generator=gen, device=DEV)) % E
        w["embed"] = (w["embed"].float() + 25.0 * (dirs[first] + dirs[second])).to(dtype)
        for name in routers:
            w[name] = (0.2 * dirs[torch.randperm(E, generator=gen, device=DEV)]).to(dtype)
    return w


# ---- the cases ----------------------------------------------------------------------------------------------------


def _case(name, model, batch, shortest, longest, steps):
    c = dict(model=model, batch=batch, shortest=shortest, longest=longest, steps=steps)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a question to a small model on its own: every step is a few short kernels
        _case("small_one_request", "dense_small", 1, 23, 23, 16),
        # one user's chat with a large model: a short prompt, then token by token
        _case("one_request", "dense_8b", 1, 200, 200, 16),
        # a server with a few long conversations
        _case("few_long_requests", "dense_8b", 8, 1200, 2048, 16),
        # a server with many short requests
        _case("many_short_requests", "dense_8b", 64, 17, 250, 8),
        # a document scored or put into the cache: one prompt, nothing decoded
        _case("one_document", "dense_8b", 1, 2048, 2048, 0),
        # documents of unequal lengths together
        _case("unequal_documents", "dense_8b", 12, 64, 1999, 0),
        # the float32 mode: logits that do not depend on how requests are cut and batched
        _case("float32_requests", "dense_float32", 3, 130, 517, 8),
        # the other designs, as a server meets them: a few prompts of about a thousand tokens, some steps behind them
        _case("tifapel_requests", "tifapel", 4, 700, 1300, 8),
        _case("soputar_requests", "soputar", 4, 700, 1300, 8),
        _case("gebasun_requests", "gebasun", 4, 700, 1300, 8),
    ]


# most prompt tokens of a drawn case, so that none costs more than the largest listed one
_MOST = dict(dense_8b=12000, dense_small=16384, dense_float32=2500, tifapel=8192, soputar=8192, gebasun=8192)


def draw(rng):
    model = rng.choice(MODELS)
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    batch = spread(1, 64 if model != "dense_float32" else 16)
    most = max(20, min(4096, _MOST[model] // batch))
    longest = spread(16, most)
    shortest = rng.randint(max(1, longest // 8), longest)
    steps = rng.choice((0, 0, 1)) and rng.randint(0, 3) if longest * batch > 4000 else spread(1, 24)
    return _case(None, model, batch, shortest, longest, steps)


def _lengths(case):
    """Prompt lengths between the shortest and the longest, in no order; the last is the longest."""
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    return [hi if i == n - 1 else lo + int((hi - lo) * ((i * 0.6180339887) % 1.0)) for i in range(n)]


def _tokens(case, raw, seed):
    """Per sequence: the prompt's ids, then the ids it goes on with."""
    rng = np.random.default_rng(seed)
    return [rng.integers(0, _vocab(raw), n + case["steps"]).tolist() for n in _lengths(case)]


def prepare(case, seed):
    raw = _raw(case["model"])
    lengths = _lengths(case)
    rooms = [-(-(n + case["steps"]) // 64) * 64 for n in lengths]
    options = LoadOptions(dtype=raw["torch_dtype"], max_tokens=sum(rooms), max_batch=case["batch"], max_step_tokens=sum(lengths))
    engine = Engine(read_config(raw), _weights(raw, seed), options)
    tokens = _tokens(case, raw, seed)
    return dict(engine=engine, prompts=[t[:n] for t, n in zip(tokens, lengths)], rest=[t[n:] for t, n in zip(tokens, lengths)],
                steps=case["steps"])


def run(state):
    """The logits [sequences, vocabulary] behind the prompts and behind each further token."""
    engine = state["engine"]
    slots = [engine.acquire() for _ in state["prompts"]]
    out = [engine.step(list(zip(slots, state["prompts"])))]
    for i in range(state["steps"]):
        out.append(engine.step([(s, [t[i]]) for s, t in zip(slots, state["rest"])]))
    for s in slots:
        engine.release(s)
    return out


# ---- the work that a pass cannot do without -----------------------------------------------------------------------


def work(case):
    """Bytes: per step the weights that its tokens use (a routed expert when some token is expected to pick it), the
    embedding rows, the cached keys, values and states that are read, those that are written, and the logits.
    Operations: the products over the tokens' active weights, scores and weighted sums over the visible keys, the
    recurrences' state updates and reads."""
    raw = _raw(case["model"])
    size = 4 if raw["torch_dtype"] == "float32" else 2
    lengths, d, V = _lengths(case), _width(raw), _vocab(raw)
    dense = routed = 0
    for name, shape, _, _ in _tensors(raw):
        n = math.prod(shape)
        if ".mlp.e" in name and "expert" in str(raw["layers"][0]["mlp"]):
            routed += n
        elif "embed" not in name and name not in ("head", "lm_head.weight"):
            dense += n
    E, top = (16, 2) if routed else (1, 1)
    # per mixer: (cached values a token, visible keys at most, operations a visible key, state values, operations a token)
    mixers = []
    if "hidden_size" in raw:
        kv, hd = 2 * raw["num_key_value_heads"] * raw["head_dim"], raw["num_attention_heads"] * raw["head_dim"]
        mixers = [(kv, raw["sliding_window"] or 1 << 30, 4 * hd, 0, 0)] * LAYERS
    else:
        for layer in raw["layers"]:
            m, kind = layer["mixer"], layer["type"]
            H, Dv = m["heads"], m["vdim"]
            if kind in ("attention", "attention_2"):
                kv = m["kv_heads"] * (m["dim"] + (Dv if raw["architecture"] != "Gebasun" or kind == "attention_2" else 0))
                mixers.append((kv, (m.get("mask") or {}).get("size", 1 << 30), 2 * H * (m["dim"] + Dv), 0, 0))
            elif kind == "latent_attention":
                mixers.append((m["kv_rank"] + m["rot_dim"], 1 << 30, 2 * H * (m["dim"] + m["rot_dim"] + Dv), 0, 0))
            else:
                n = H * Dv * (m["state"] if kind == "mamba2" else m["dim"])
                mixers.append((0, 0, 0, n, (7 if kind == "delta" else 5) * n))
    total = flops = 0.0
    past = [0] * case["batch"]
    for step in range(case["steps"] + 1):
        new = lengths if step == 0 else [1] * case["batch"]
        T, rows = sum(new), case["batch"]
        total += size * (dense + routed * (1 - (1 - top / E) ** T) + V * d + T * d) + 4 * rows * V
        flops += 2.0 * (dense + routed * top / E) * T + 2.0 * V * d * rows
        for kv, window, per_key, state, per_token in mixers:
            for p, n in zip(past, new):
                total += size * kv * (min(p, window) + n) + 4 * state * (2 if p else 1)
                full = max(0, min(n, window - p))          # queries that see every earlier position
                seen = full * p + full * (full + 1) / 2 + (n - full) * min(window, p + n)
                flops += per_key * seen + per_token * n
        past = [p + n for p, n in zip(past, new)]
    return dict(bytes=total, flops=flops)


def tolerance(case):
    # bfloat16: weights and the activations between kernels are rounded to 8 bits, which eight layers of random weights
    # carry on to the logits: 0.003 to 0.01 off the 64-bit result, so up to 0.014 between two implementations, and six
    # deviations of that at the worst value.  float32: sums of a few thousand products in another order, 2e-6 off.
    if _raw(case["model"])["torch_dtype"] == "float32":
        return dict(rel=1e-5, max=1e-4)
    return dict(rel=0.03, max=0.3)


# ---- the same in 64 bits ------------------------------------------------------------------------------------------


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _angles(T, dims, base):
    freq = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEV) / dims)
    a = torch.arange(T, dtype=torch.float64, device=DEV)[:, None, None] * freq
    return torch.cos(a), torch.sin(a)


def _rotate(x, dims, base, neighbours=False):
    """x [T, heads, n]: pairs (i, i + dims/2), or (2i, 2i + 1), of the first ``dims`` turn with the position."""
    c, s = _angles(x.shape[0], dims, base)
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    out = x.clone()
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _attend(q, k, v, scale, window=None, keep=0, softcap=None, sink=None, bias=None):
    """q [T, H, D], k [T, G, D], v [T, G, Dv] -> [T, H * Dv]; ``bias`` [heads, distance], ``sink`` [heads]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None, :]
    hidden = j > i
    if window is not None:
        hidden = hidden | ((i - j >= window) & (j >= keep))
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        if softcap is not None:
            s = softcap * torch.tanh(s / softcap)
        if bias is not None:
            s = s + bias[h][(i - j).clamp_min(0)]
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, 1)[:, :T] @ v[:, h * G // H])
    return torch.cat(out, 1)


def _conv(u, taps, bias=0.0):
    padded = torch.cat([u.new_zeros(taps.shape[1] - 1, u.shape[1]), u])
    return bias + sum(padded[j : j + u.shape[0]] * taps[:, j] for j in range(taps.shape[1]))


def _decayed(q, k, v, log_decay):
    """o_t = sum over s <= t of exp(sum of log_decay over s+1..t) (q_t . k_s) v_s; per head, [T, D] each, log_decay [T]."""
    c = log_decay.cumsum(0)
    gap = (c[:, None] - c[None, :]).masked_fill(torch.ones(len(c), len(c), dtype=torch.bool, device=DEV).triu(1), -math.inf)
    return ((q @ k.T) * torch.exp(gap)) @ v


def _delta_rule(q, k, v, beta, g):
    """All heads at once, token by token: q, k [T, H, D], v [T, H, Dv], beta, g [T, H]."""
    S = q.new_zeros(q.shape[1], q.shape[2], v.shape[2])
    out = []
    for t in range(q.shape[0]):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
        out.append(torch.bmm(q[t, :, None], S)[:, 0])
    return torch.stack(out)


def _mixer(arch, layer, h, get, eps, kept, i):
    """One sequence through one layer's mixer: h [T, width], already normed where the design norms; ``get(name)`` in 64 bits."""
    m, kind, T = layer["mixer"], layer["type"], h.shape[0]
    lin = lambda name: h @ get("mix." + name).T
    H, D, Dv = m["heads"], m.get("dim"), m["vdim"]
    if kind in ("attention", "attention_2"):
        G, mask = m["kv_heads"], m.get("mask") or {}
        more = dict(window=mask.get("size"), keep=mask.get("keep_first", 0), softcap=m.get("softcap"))
        if arch == "Gebasun":
            q, k = (lin("q") + get("mix.q.b")).view(T, H, D), (lin("k") + get("mix.k.b")).view(T, G, D)
            v = k
            if kind == "attention_2":
                q, k = (_rotate(z, m["rot"]["dims"], m["rot"]["base"]) for z in (q, k))
                o = _attend(_unit(q, eps), _unit(k, eps), v, m["scale"], sink=get("mix.sink"), **more)
                return (o * torch.sigmoid(lin("g"))) @ get("mix.o").T
            rows, half, far = m["bias_rows"], m["bias_rows"] // 2, m["bias_max"]
            back = [n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(far / half) * (rows - half)))
                    for n in range(T)]
            bias = get("mix.rel")[torch.tensor(back, device=DEV)].T
            o = _attend(_unit(q, eps), _unit(k, eps), v, m["scale"], sink=get("mix.sink"), bias=bias, **more)
            return o @ get("mix.o").T + get("mix.o.b")
        q = lin("q")
        if arch == "Soputar":
            t = m["q_temp"]
            q = _unit(q, eps) * get("mix.q.norm")
            q = q * (1.0 + t["coef"] * torch.log(torch.floor((torch.arange(T, device=DEV).double() + 1) / t["every"]) + 1.0))[:, None]
        if m.get("kv_from") is None:
            k = lin("k")
            if arch == "Soputar":
                k = _unit(k, eps) * get("mix.k.norm")
            kept[i] = k.view(T, G, D), lin("v").view(T, G, Dv)
        k, v = kept[i if m.get("kv_from") is None else m["kv_from"]]
        return _attend(q.view(T, H, D), k, v, m["scale"], **more) @ get("mix.o").T
    if kind in ("lightning", "retention"):
        act = _silu if kind == "lightning" else (lambda z: z)
        q, k, v = (act(lin(r)).view(T, H, -1) for r in "qkv")
        if kind == "retention":
            q, k = (_rotate(z, m["rot"]["dims"], m["rot"]["base"]) for z in (q, k))
            k = k * D ** -0.5
        o = torch.stack([_decayed(q[:, x], k[:, x], v[:, x], torch.full((T,), math.log(m["decay"][x]), dtype=h.dtype, device=DEV))
                         for x in range(H)], 1)
        if kind == "retention":
            return (_unit(o, eps).reshape(T, -1) * _silu(lin("g"))) @ get("mix.o").T
        return (_unit(o.reshape(T, -1), eps) * get("mix.norm") * torch.sigmoid(lin("g"))) @ get("mix.o").T
    if kind == "latent_attention":
        R, rank, base = m["rot_dim"], m["kv_rank"], m["rot"]["base"]
        q, down = lin("q").view(T, H, D + R), lin("dkv")
        c = _unit(down[:, :rank], eps) * get("mix.dkv.norm")
        k_rot = _rotate(down[:, None, rank:], R, base, neighbours=True).expand(T, H, R)
        q = torch.cat([q[..., :D], _rotate(q[..., D:], R, base, neighbours=True)], -1)
        k = torch.cat([(c @ get("mix.uk").T).view(T, H, D), k_rot], -1)
        return _attend(q, k, (c @ get("mix.uv").T).view(T, H, Dv), m["scale"], sink=get("mix.sink")) @ get("mix.o").T
    if kind == "delta":
        G = m["kv_heads"]
        q, k, v = (_silu(_conv(lin(r), get(f"mix.{r}.conv"))).view(T, -1, D if r != "v" else Dv) for r in "qkv")
        q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        beta = torch.sigmoid(lin("b"))
        g = torch.exp(-torch.exp(get("mix.A_log")) * torch.nn.functional.softplus(lin("a") + get("mix.dt_bias"), threshold=1e9))
        o = _delta_rule(q.repeat_interleave(H // G, 1) * D ** -0.5, k.repeat_interleave(H // G, 1), v, beta, g)
        return (_unit(o, eps) * get("mix.norm") * _silu(lin("g")).view(T, H, Dv)).reshape(T, -1) @ get("mix.o").T
    N, G, inner = m["state"], m["groups"], H * Dv                                     # mamba2
    z, xbc, dt = lin("in").split([inner, inner + 2 * G * N, H], 1)
    x, B, C = _silu(_conv(xbc, get("mix.conv"), get("mix.conv.b"))).split([inner, G * N, G * N], 1)
    x, B, C = x.view(T, H, Dv), B.view(T, G, N), C.view(T, G, N)
    dt = torch.nn.functional.softplus(dt + get("mix.dt_bias"), threshold=1e9)
    y = torch.stack([_decayed(C[:, j * G // H], B[:, j * G // H] * dt[:, j, None], x[:, j], -torch.exp(get("mix.A_log")[j]) * dt[:, j])
                     + get("mix.D")[j] * x[:, j] for j in range(H)], 1).reshape(T, inner)
    parts = m["norm_groups"]
    return (_unit((y * _silu(z)).view(T, parts, -1), eps).reshape(T, inner) * get("mix.norm")) @ get("mix.o").T


def _feed_forward(arch, mlp, h, get):
    """h [tokens of all sequences, width]."""
    if mlp["kind"] == "dense":
        g = (h @ get("mlp.gate").T).clamp(max=mlp["limit"])
        u = (h @ get("mlp.up").T).clamp(-mlp["limit"], mlp["limit"])
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ get("mlp.down").T
    E, top = mlp["router"]["experts"], mlp["router"]["top"]
    z = h @ get("mlp.router").T
    if arch == "Gebasun":
        z, chosen = (z + get("mlp.router.b")).topk(top, 1)
        weight = torch.softmax(z, 1)
        expert = lambda e, x: torch.relu(x @ get(f"mlp.{e}.up").T) ** 2 @ get(f"mlp.{e}.down").T
    else:
        s = torch.sigmoid(z)
        groups = mlp["router"]["groups"]
        best = s.view(-1, groups["count"], E // groups["count"]).topk(2, 2).values.sum(2).topk(groups["keep"], 1).indices
        allowed = torch.zeros(len(h), groups["count"], dtype=torch.bool, device=DEV).scatter_(1, best, True)
        s = s.masked_fill(~allowed.repeat_interleave(E // groups["count"], 1), -1.0)
        weight, chosen = s.topk(top, 1)
        weight = weight / (weight.sum(1, keepdim=True) + 1e-20) * mlp["router"]["scale"]
        expert = lambda e, x: (_silu(x @ get(f"mlp.{e}.gate").T) * (x @ get(f"mlp.{e}.up").T)) @ get(f"mlp.{e}.down").T
    out = expert("shared", h) if mlp.get("shared") else torch.zeros_like(h)
    for e in range(E):
        rows, at = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            out.index_add_(0, rows, weight[rows, at, None] * expert(f"e{e}", h[rows]))
    return out


def exact(case, seed):
    raw = _raw(case["model"])
    w, seqs, lengths = _weights(raw, seed), _tokens(case, raw, seed), _lengths(case)
    sizes = [len(s) for s in seqs]
    get64 = lambda name: w[name].double()
    table = w["model.embed_tokens.weight" if "hidden_size" in raw else "embed"]
    x = table[torch.tensor([t for s in seqs for t in s], device=DEV)].double()           # all sequences, one after another
    each = lambda f, *packed: torch.cat([f(*parts) for parts in zip(*(p.split(sizes) for p in packed))])
    if "hidden_size" in raw:
        eps, D = raw["rms_norm_eps"], raw["head_dim"]
        for i in range(LAYERS):
            p = f"model.layers.{i}."
            h = _unit(x, eps) * get64(p + "input_layernorm.weight")
            q, k, v = ((h @ get64(f"{p}self_attn.{r}_proj.weight").T).view(len(h), -1, D) for r in "qkv")
            q, k = (_unit(z, eps) * get64(f"{p}self_attn.{r}_norm.weight") for z, r in ((q, "q"), (k, "k")))
            o = each(lambda a, b, c: _attend(_rotate(a, D, raw["rope_theta"]), _rotate(b, D, raw["rope_theta"]), c, D ** -0.5,
                                             window=raw["sliding_window"]), q, k, v)
            x = x + o @ get64(p + "self_attn.o_proj.weight").T
            h = _unit(x, eps) * get64(p + "post_attention_layernorm.weight")
            x = x + (_silu(h @ get64(p + "mlp.gate_proj.weight").T) * (h @ get64(p + "mlp.up_proj.weight").T)) @ \
                get64(p + "mlp.down_proj.weight").T
        norm, head = get64("model.norm.weight"), table if raw["tie_word_embeddings"] else w["lm_head.weight"]
    else:
        eps, arch = raw["norm"]["eps"], raw["architecture"]
        kept = [{} for _ in seqs]
        for i, layer in enumerate(raw["layers"]):
            cache = {}

            def get(name, i=i, cache=cache):
                if name.startswith("mlp."):
                    return get64(f"l{i}.{name}")
                if name not in cache:
                    cache[name] = get64(f"l{i}.{name}")
                return cache[name]

            mix = lambda h: torch.cat([_mixer(arch, layer, part, get, eps, keep, i) for part, keep in zip(h.split(sizes), kept)])
            if arch == "Soputar":
                x = x + _unit(mix(x), eps) * (1.0 + get("norm1"))
                x = x + _unit(_feed_forward(arch, layer["mlp"], x, get), eps) * (1.0 + get("norm2"))
            else:
                h = _unit(x, eps) * get("norm1")
                x = x + mix(h) + _feed_forward(arch, layer["mlp"], h if arch == "Tifapel" else _unit(x, eps) * get("norm2"), get)
        norm, head = get64("final.norm") + (1.0 if arch == "Soputar" else 0.0), w["head"]
    starts = np.cumsum([0] + sizes)[:-1]
    out = []
    for step in range(case["steps"] + 1):
        rows = torch.tensor([int(a) + n - 1 + step for a, n in zip(starts, lengths)], device=DEV)
        h = _unit(x[rows], eps) * norm
        out.append(torch.cat([h @ part.double().T for part in head.split(16384)], 1))
    return out
