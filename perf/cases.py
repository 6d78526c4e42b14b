"""What the engine's speed is judged by: steps of the kinds a user's program runs, through ``Engine.step``.

A case names a model, a number of decoding requests with the context that they have, and the prompts that arrive:

* decoding requests only: ``decode`` requests hold ``context`` positions each; a pass is one decode step, one token a
  request, and the requests grow by it (a request that is full is replaced by a new one with the same prompt);
* prompts only: a pass admits ``prompts`` requests of ``tokens`` tokens together, of unequal lengths, runs them as one
  step and closes them;
* both: the step a scheduler makes while requests decode and others arrive.

The layers have the sizes that ``bench.py`` measures, fewer of them (a layer's work does not depend on how many there
are) and a vocabulary cut in proportion.  Weights are random, drawn on the device; a router's are six times as large as
the rest, so that it prefers some experts clearly, as a trained one does, and a rounding seldom changes the outcome.
"""
from __future__ import annotations

import math
import zlib

import torch
import torch.nn.functional as F

from ferrox_b200 import Engine, StepEntry, resolve
from ferrox_b200.parts.base import Runtime
from ferrox_b200.parts.build import build_model
from ferrox_b200.weights.loader import WeightSource

PAGE = 64
CONTEXT = 4096          # the context limit of every engine
WARM = 2                # decode steps of a program that has been running: the first eager, the second captures its graph
VOCAB = 32768

# ---- models -----------------------------------------------------------------------------------------------------
_QWEN = dict(architectures=["Qwen2MoeForCausalLM"], head_dim=128, qkv_bias=True, vocab_size=VOCAB, rope_theta=1000000.0,
             rms_norm_eps=1e-6, tie_word_embeddings=False, max_position_embeddings=CONTEXT)


def _moe():
    """The layer sizes of the Qwen1.5-MoE-A2.7B shape."""
    return dict(_QWEN, num_hidden_layers=4, hidden_size=2048, num_attention_heads=16, num_key_value_heads=16, num_experts=60,
                num_experts_per_tok=4, moe_intermediate_size=1408, shared_expert_intermediate_size=5632,
                intermediate_size=5632, norm_topk_prob=False)


def _moe_wide():
    """The layer sizes of the Qwen2-57B-A14B shape."""
    return dict(_moe(), num_hidden_layers=2, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4,
                num_experts=64, num_experts_per_tok=8, moe_intermediate_size=2560, shared_expert_intermediate_size=20480,
                intermediate_size=20480)


def _dense():
    """A decoder without experts: heads of 128 on a quarter as many key heads."""
    return dict(_QWEN, num_hidden_layers=4, hidden_size=2048, num_attention_heads=16, num_key_value_heads=4, num_experts=0,
                intermediate_size=7808)


def _safepel():
    """Gated delta rule and windowed capped attention beside a decayed linear attention, in turn; heads of 128."""
    mlp = {"kind": "dense", "ff": 5632}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    par = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "mask": {"size": 1024},
                 "rot": {"dims": 64, "base": 1000000.0}, "scale": 128 ** -0.5, "softcap": 30.0},
        "right": {"heads": 16, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 8 * i / 15) for i in range(16)]},
        "left_scale": 1.0, "right_scale": 1.0}}
    return {"architecture": "Safepel", "vocab": VOCAB, "width": 2048, "norm": {"eps": 1e-6}, "logit_scale": 1.0,
            "max_positions": CONTEXT, "layers": [delta, par, delta, par]}


def _sesuzen():
    """Generalized delta rule (heads of 64) and windowed attention that keeps its first keys, in turn."""
    mlp = {"kind": "dense", "ff": 9344}
    delta = {"type": "general_delta", "mlp": mlp, "mixer": {"heads": 32, "dim": 64, "decay_rank": 64}}
    att = {"type": "attention", "mlp": mlp, "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128,
           "scale": 128 ** -0.5, "mask": {"size": 1024, "keep_first": 4}}}
    return {"architecture": "Sesuzen", "vocab": VOCAB, "width": 2048, "norm": {"eps": 1e-5}, "canon": {"taps": 4},
            "max_positions": CONTEXT, "logit_softcap": 30.0, "layers": [delta, att, delta, att]}


def _zanezen():
    """mLSTM, differential attention and latent attention with dense feed-forwards."""
    mlp = {"kind": "dense", "ff": 11264}
    rot = {"dims": 32, "base": 1000000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    mlstm = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": 16, "dim": 128, "vdim": 128, "gate_cap": 15.0}}
    att = {"type": "attention", "mlp": mlp, "mixer": {"heads": 16, "kv_heads": 4, "dim": 64, "vdim": 128,
           "scale": 64 ** -0.5, "diff": 0.5, "softcap": 30.0, "conv": 4, "rot": rot}}
    lat = {"type": "latent_attention", "mlp": mlp, "mixer": {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128,
           "rot": {"dims": 64, "base": 1000000.0}, "kv_rank": 512, "scale": 192 ** -0.5}}
    return {"architecture": "Zanezen", "vocab": VOCAB, "width": 2048, "norm": {"eps": 1e-6}, "max_positions": CONTEXT,
            "embedding": {"scale": 2048 ** 0.5}, "residual_mult": 0.5, "layers": [mlstm, att, att, lat]}


MODELS = {"moe": _moe, "moe-wide": _moe_wide, "dense": _dense, "safepel": _safepel, "sesuzen": _sesuzen,
          "zanezen": _zanezen}
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


# ---- cases ------------------------------------------------------------------------------------------------------
def _case(name, model, *, dtype="bf16", decode=0, context=0, prompts=0, tokens=0):
    return {"name": name, "model": model, "dtype": dtype, "decode": decode, "context": context, "prompts": prompts,
            "tokens": tokens}


def listed():
    return [
        # one user in a chat: the smallest call, a chain of short kernels
        _case("decode-1", "moe", decode=1, context=300),
        # the serving batch that bench.py reports first
        _case("decode-8", "moe", decode=8, context=2048),
        # a busy server
        _case("decode-64", "moe", decode=64, context=1000),
        # a long prompt of one user
        _case("prompt-2048", "moe", prompts=1, tokens=2048),
        # a short question arrives while others decode
        _case("mixed-7+53", "moe", decode=7, context=700, prompts=1, tokens=53),
        # a larger model, a full batch of prompts admitted together
        _case("wide-prompt-4096", "moe-wide", prompts=3, tokens=4096),
        # the true 32-bit engine, which checkpoints are checked with: a prompt of odd length, and its decoding (without
        # experts: two correct engines that differ in the last bit choose other ones now and then, and then their
        # results cannot be compared at the precision that this engine is for)
        _case("f32-prompt-517", "dense", dtype="f32", prompts=1, tokens=517),
        _case("f32-decode-4", "dense", dtype="f32", decode=4, context=700),
        # models that carry a state from token to token beside their attention: long prompts, one and several
        _case("safepel-prompt-2048", "safepel", prompts=1, tokens=2048),
        _case("sesuzen-prompt-3001", "sesuzen", prompts=3, tokens=3001),
        _case("zanezen-prompt-1531", "zanezen", prompts=1, tokens=1531),
        # and the decoding of such a model
        _case("zanezen-decode-16", "zanezen", decode=16, context=900),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    model = rng.choice(sorted(MODELS))
    kind = rng.choice(("decode", "prompt", "mixed"))
    f32 = model == "dense" and rng.random() < 0.5
    decode = context = prompts = tokens = 0
    if kind != "prompt":
        decode = _log(rng, 1, (8 if f32 else 64) if kind == "decode" else 16)
        context = _log(rng, 16, min(2048, 65536 // decode))
    if kind != "decode":
        tokens = _log(rng, 8, (600 if f32 else 3000) if kind == "prompt" else (200 if f32 else 500))
        prompts = rng.randint(1, max(1, min(4, int(math.sqrt(tokens)))))
    c = _case("", model, dtype="f32" if f32 else "bf16", decode=decode, context=context, prompts=prompts, tokens=tokens)
    del c["name"]
    return c


def _lengths(case):
    """Unequal lengths that add up to ``tokens``."""
    n, t = case["prompts"], case["tokens"]
    return [t * (i + 1) ** 2 // n ** 2 - t * i ** 2 // n ** 2 for i in range(n)]


# ---- weights and tokens, from the seed alone ----------------------------------------------------------------------
def _generator(seed, name):
    return torch.Generator("cuda").manual_seed(zlib.crc32(f"{seed}:{name}".encode()))


def _tensor(decl, seed, dtype):
    if decl.init == "ones":
        return torch.ones(decl.shape, dtype=dtype, device="cuda")
    name, std, mean = decl.name, 0.02, decl.mean
    if name.endswith(".mlp.gate.weight"):
        std = 0.12                                   # the router
    elif name == "model.embed_tokens.weight":
        std = 1.0                                    # a residual stream that layers add to, as in a deep model
    elif name.endswith(".conv"):
        std = 0.3
    elif name.endswith((".dt_bias", ".w0")):
        mean = -3.0                                  # decays near one, so that a state remembers
    elif name.endswith(".f.b"):
        mean = 3.0                                   # forget gates that start open
    x = torch.randn(decl.shape, generator=_generator(seed, name), device="cuda")
    return x.mul_(std).add_(mean).to(dtype)


class _Weights:
    """The tensors by name, as ``_engine`` loads them, in 64 bits."""

    def __init__(self, decls, seed, dtype):
        self.decls, self.seed, self.dtype = {d.name: d for d in decls}, seed, dtype

    def __getitem__(self, name):
        return _tensor(self.decls[name], self.seed, self.dtype).double()

    def __contains__(self, name):
        return name in self.decls


def _engine(case, seed, **cache):
    dtype = DTYPES[case["dtype"]]
    config, spec = resolve(MODELS[case["model"]]())
    model = build_model(spec)
    decls = {d.name: d for d in model.tensor_decls()}
    rt = Runtime(torch.device("cuda:0"), dtype)
    source = WeightSource(lambda n: _tensor(decls[n], seed, dtype), decls, rt.device, dtype, stored_dtype=lambda n: dtype)
    model.load(source, rt)
    return Engine(config, spec, model, page_size=PAGE, max_positions=CONTEXT, **cache)


def _token_lists(case, seed, tag, lengths):
    g = torch.Generator().manual_seed(zlib.crc32(f"{seed}:{tag}".encode()))
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in lengths]


class _State:
    pass


def _limit(case):
    """Positions that a decoding request may reach: its context and a long answer."""
    return min(CONTEXT, case["context"] + WARM + 2000)


def _admit(s):
    """Opens the decoding requests and brings their contexts into the cache."""
    s.slots = [s.engine.open_request() for _ in range(s.case["decode"])]
    s.length = s.case["context"]
    for slot, toks in zip(s.slots, s.answers):
        s.engine.step([StepEntry(slot, toks[:s.length])], check=False)


def _decoding(s):
    """The entries of one decode step of the requests that decode."""
    if s.length >= _limit(s.case):
        for slot in s.slots:
            s.engine.close_request(slot)
        _admit(s)
    entries = [StepEntry(slot, [toks[s.length]], want=[0]) for slot, toks in zip(s.slots, s.answers)]
    s.length += 1
    return entries


def prepare(case, seed):
    s = _State()
    s.case = case
    lengths = _lengths(case) if case["prompts"] else []
    pages = case["decode"] * (_limit(case) // PAGE + 1) + sum(n // PAGE + 1 for n in lengths) + 2
    s.engine = _engine(case, seed, n_pages=pages, max_slots=case["decode"] + case["prompts"])
    s.answers = _token_lists(case, seed, "answers", [_limit(case)] * case["decode"])
    s.prompts = _token_lists(case, seed, "prompts", lengths)
    if case["decode"]:
        _admit(s)
        for _ in range(WARM):
            s.engine.step(_decoding(s), check=False)
    return s


def run(s):
    eng = s.engine
    entries = _decoding(s) if s.case["decode"] else []
    new = [eng.open_request() for _ in s.prompts]
    entries += [StepEntry(slot, toks, want=[len(toks) - 1]) for slot, toks in zip(new, s.prompts)]
    logits = eng.step(entries, check=False)
    for slot in new:
        eng.close_request(slot)
    if s.case["decode"]:
        return {"logits": logits}
    # what the prompts leave in the cache: pages of keys and values, and states
    left = []
    for i in range(eng.spec.n_caches):
        c = eng.cache.layer_cache(i)
        for kept in (c.pages, c.states or {}):
            left += [kept[name] for name in sorted(kept)]
        if c.state is not None:
            left.append(c.state)
    return {"logits": logits, "cache": left}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    cfg = MODELS[case["model"]]()
    _, spec = resolve(cfg)
    size = 2 if case["dtype"] == "bf16" else 4
    lengths = _lengths(case) if case["prompts"] else []
    n_tokens, wanted = case["decode"] + sum(lengths), case["decode"] + len(lengths)
    weights = experts = head = 0
    for d in build_model(spec).tensor_decls():
        n = math.prod(d.shape)
        if d.name in (spec.embedding_name, spec.position_table):
            head += n if spec.head_name is None and d.name == spec.embedding_name else 0
        elif d.name == spec.head_name:
            head += n
        elif ".experts." in d.name:
            experts += n
        else:
            weights += n
    n_bytes, flops = weights * size, 2.0 * weights * n_tokens
    if experts:
        share = cfg["num_experts_per_tok"] / cfg["num_experts"]
        n_bytes += experts * size * (1.0 - (1.0 - share) ** n_tokens)
        flops += 2.0 * experts * share * n_tokens
    n_bytes += head * size + wanted * VOCAB * 4 + n_tokens * spec.hidden * size
    flops += 2.0 * head * wanted
    pairs = [(case["context"] + WARM + 1, 1)] * case["decode"] + [(n, n) for n in lengths]
    for layer in spec.layers:
        b, f = _mixer_work(layer.mixer, pairs, size)
        n_bytes, flops = n_bytes + b, flops + f
    return {"bytes": n_bytes, "flops": flops}


def _mixer_work(m, pairs, size):
    """(bytes, flops) of a mixer beside its products: keys and values or states read and written, scores and read-outs.
    ``pairs``: per request its length after the step and its tokens of the step."""
    if m.kind == "mixer_sum":
        parts = [_mixer_work(x, pairs, size) for x in m.mixers]
        return sum(p[0] for p in parts), sum(p[1] for p in parts)
    if m.kind == "input_conv":
        return _mixer_work(m.mixer, pairs, size)
    n_bytes = flops = 0.0
    window = getattr(m, "window", None)
    for length, new in pairs:
        if m.kind in ("gqa_attention", "differential_attention", "latent_attention"):
            first = length - new
            keys = sum(min(p + 1, window or CONTEXT) for p in range(first, length))
            maps = 2 if m.kind == "differential_attention" else 1
            if m.kind == "latent_attention":
                row, pair = m.kv_rank + m.rot_dim, m.head_dim + m.rot_dim + m.value_dim
            else:
                v = getattr(m, "value_dim", None) or m.head_dim
                row, pair = m.n_kv_heads * (maps * m.head_dim + v), maps * (m.head_dim + v)
            n_bytes += (min(length, (window or CONTEXT) + new) if first else new) * row * size
            flops += 2.0 * keys * m.n_heads * pair
        else:
            state = m.n_heads * m.head_dim * (getattr(m, "value_dim", None) or m.head_dim)
            n_bytes += 4.0 * state * (2 if length > new else 1)
            flops += 6.0 * new * state
    return n_bytes, flops


def tolerance(case):
    """Logits lie 0.3 to 1 per cent from the 64-bit ones in bfloat16 and 2e-6 in 32 bits (see :func:`exact`)."""
    return {"rel": 2.5e-2, "max": 0.3} if case["dtype"] == "bf16" else {"rel": 1e-5, "max": 1e-3}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _norm(x, eps, w, b=None):
    d = x - x.mean(-1, keepdim=True)
    y = _rms(d, eps) * w
    return y if b is None else y + b


def _conv(x, w):
    n, taps = x.shape[0], w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[j:j + n] * w[:, j] for j in range(taps))


def _angles(n, dims, base, scaling=None):
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device="cuda")
    mag = 1.0
    if scaling is not None:
        def pair_of(turns):
            return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

        lo = max(math.floor(pair_of(scaling["fast"])), 0)
        hi = min(math.ceil(pair_of(scaling["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0, 1).double()
        f = f / scaling["factor"] * ramp + f * (1.0 - ramp)
        mag = 0.1 * math.log(scaling["factor"]) + 1.0
    a = torch.arange(n, device="cuda", dtype=torch.float64)[:, None] * f.float().double()
    return torch.cos(a) * mag, torch.sin(a) * mag


def _turn(x, cs, adjacent=False):
    """x [n, heads, d]: pairs of the first elements turned by the position."""
    c, s = (t[:, None, :] for t in cs)
    dims = 2 * c.shape[-1]
    out = x.clone()
    i, j = (slice(0, dims, 2), slice(1, dims, 2)) if adjacent else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., i], x[..., j]
    out[..., i], out[..., j] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, window=None, keep=0, cap=None, sink=None):
    """q [n, H, d], k [n, G, d], v [n, G, e]; softmax over the visible keys, a head at a time."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    i, j = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None, :]
    hidden = j > i
    if window is not None:
        hidden |= (i - j >= window) & (j >= keep)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], dim=1)
        p = torch.softmax(s, -1)
        out.append(p[:, :n] @ v[:, h * G // H])
    return torch.stack(out, 1)


def _qwen_layer(cfg, W, l, h, seqs):
    p, eps, d = f"model.layers.{l}.", cfg["rms_norm_eps"], cfg["head_dim"]
    x = _rms(h, eps) * W[p + "input_layernorm.weight"]
    q, k, v = ((x @ W[f"{p}self_attn.{n}_proj.weight"].T + W[f"{p}self_attn.{n}_proj.bias"]).view(len(x), -1, d)
               for n in "qkv")
    o = []
    for a, b in seqs:
        cs = _angles(b - a, d, cfg["rope_theta"])
        o.append(_attend(_turn(q[a:b], cs), _turn(k[a:b], cs), v[a:b], d ** -0.5))
    h = h + torch.cat(o).flatten(1) @ W[p + "self_attn.o_proj.weight"].T
    x = _rms(h, eps) * W[p + "post_attention_layernorm.weight"]

    def unit(x, name):
        g, u, dn = (W[f"{p}mlp.{name}{n}_proj.weight"] for n in ("gate", "up", "down"))
        return (F.silu(x @ g.T) * (x @ u.T)) @ dn.T

    if not cfg["num_experts"]:
        return h + unit(x, "")
    weight, chosen = torch.softmax(x @ W[p + "mlp.gate.weight"].T, -1).topk(cfg["num_experts_per_tok"], -1)
    y = torch.sigmoid(x @ W[p + "mlp.shared_expert_gate.weight"].T) * unit(x, "shared_expert.")
    for e in range(cfg["num_experts"]):
        row, rank = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            y.index_add_(0, row, weight[row, rank, None] * unit(x[row], f"experts.{e}."))
    return h + y


def _safepel_delta(W, p, m, x, eps):
    n, H, G, D, V = len(x), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (F.silu(_conv(x @ W[p + t].T, W[p + t + ".conv"])) for t in "qkv")
    q, k, v = q.view(n, G, D), k.view(n, G, D), v.view(n, H, V)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(x @ W[p + "b"].T)
    g = torch.exp(-torch.exp(W[p + "A_log"]) * F.softplus(x @ W[p + "a"].T + W[p + "dt_bias"]))
    S, out = x.new_zeros(H, D, V), []
    for t in range(n):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    y = _rms(torch.stack(out), eps) * W[p + "norm"] * F.silu(x @ W[p + "g"].T).view(n, H, V)
    return y.flatten(1) @ W[p + "o"].T


def _safepel_parallel(W, p, m, x, eps):
    n, a, b = len(x), m["left"], m["right"]
    H, G, D = a["heads"], a["kv_heads"], a["dim"]
    q, k = (x @ W[p + "left.q"].T).view(n, H, D), (x @ W[p + "left.k"].T).view(n, G, D)
    cs = _angles(n, a["rot"]["dims"], a["rot"]["base"])
    o = _attend(_turn(q, cs, True), _turn(k, cs, True), k, a["scale"], a["mask"]["size"], cap=a["softcap"])
    left = o.flatten(1) @ W[p + "left.o"].T
    H, D, V = b["heads"], b["dim"], b["vdim"]
    q, k, v = (F.silu(x @ W[p + "right." + t].T).view(n, H, -1) for t in "qkv")
    d = torch.tensor(b["decay"], dtype=torch.float64, device="cuda")[:, None, None]
    S, out = x.new_zeros(H, D, V), []
    for t in range(n):
        S = d * S + k[t, :, :, None] * v[t, :, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    o = _rms(torch.stack(out).flatten(1), eps) * W[p + "right.norm"]
    right = (o * torch.sigmoid(x @ W[p + "right.g"].T)) @ W[p + "right.o"].T
    return m["left_scale"] * left + m["right_scale"] * right


def _safepel_layer(cfg, W, l, h, seqs):
    layer, p, eps = cfg["layers"][l], f"l{l}.", cfg["norm"]["eps"]
    mixer = _safepel_delta if layer["type"] == "delta" else _safepel_parallel
    x = _norm(h, eps, W[p + "norm1"])
    y = torch.cat([mixer(W, p + "mix.", layer["mixer"], x[a:b], eps) for a, b in seqs])
    h = h + _norm(y, eps, W[p + "norm1b"])
    x = _norm(h, eps, W[p + "norm2"])
    y = (torch.relu(x @ W[p + "mlp.gate"].T) * (x @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T
    return h + _norm(y, eps, W[p + "norm2b"])


def _sesuzen_delta(W, p, m, x, eps):
    n, H, D = len(x), m["heads"], m["dim"]
    r, k, v = ((x @ W[p + t].T).view(n, H, D) for t in "rkv")
    z = torch.tanh(x @ W[p + "w1"].T) @ W[p + "w2"].T + W[p + "w0"]
    w = torch.exp(-math.exp(-0.5) * torch.sigmoid(z)).view(n, H, D)
    a = torch.sigmoid(x @ W[p + "a"].T + W[p + "a.b"]).view(n, H, D)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S, out = x.new_zeros(H, D, D), []
    for t in range(n):
        S = (w[t, :, :, None] * S - (a[t] * u[t])[:, :, None] * torch.einsum("hi,hij->hj", u[t], S)[:, None, :]
             + k[t, :, :, None] * v[t, :, None, :])
        out.append(torch.einsum("hij,hi->hj", S, r[t]))
    y = _rms(torch.stack(out), eps).flatten(1) * W[p + "norm"] * torch.sigmoid(x @ W[p + "g"].T)
    return y @ W[p + "o"].T


def _sesuzen_attention(W, p, m, x, eps):
    n = len(x)
    q, k, v = ((x @ W[p + t].T + W[p + t + ".b"]).view(n, -1, m["dim"]) for t in "qkv")
    o = _attend(q, k, _rms(v, eps), m["scale"], m["mask"]["size"], m["mask"]["keep_first"]).flatten(1)
    return (o * torch.sigmoid(x @ W[p + "g"].T)) @ W[p + "o"].T


def _sesuzen_layer(cfg, W, l, h, seqs):
    layer, p, eps = cfg["layers"][l], f"l{l}.", cfg["norm"]["eps"]
    mixer = _sesuzen_delta if layer["type"] == "general_delta" else _sesuzen_attention
    x = _norm(h, eps, W[p + "norm1"], W[p + "norm1.b"])
    out = []
    for a, b in seqs:
        y = x[a:b] + _conv(x[a:b], W[p + "canon1"])
        out.append(mixer(W, p + "mix.", layer["mixer"], y, eps))
    h = h + torch.cat(out)
    x = _norm(h, eps, W[p + "norm2"], W[p + "norm2.b"])
    return h + torch.relu(x @ W[p + "mlp.up"].T) ** 2 @ W[p + "mlp.down"].T


def _zanezen_mlstm(W, p, m, x, eps):
    n, H, D, cap = len(x), m["heads"], m["dim"], m["gate_cap"]
    q, k, v = ((x @ W[p + t].T).view(n, H, -1) for t in "qkv")
    q = q * D ** -0.5
    gi = cap * torch.tanh((x @ W[p + "i"].T + W[p + "i.b"]) / cap)
    gf = F.logsigmoid(cap * torch.tanh((x @ W[p + "f"].T + W[p + "f.b"]) / cap))
    S, z, mx, out = x.new_zeros(H, D, m["vdim"]), x.new_zeros(H, D), x.new_zeros(H), []
    for t in range(n):
        new = torch.maximum(gf[t] + mx, gi[t])
        keep, take = torch.exp(gf[t] + mx - new), torch.exp(gi[t] - new)
        S = keep[:, None, None] * S + (take[:, None] * k[t])[:, :, None] * v[t, :, None, :]
        z, mx = keep[:, None] * z + take[:, None] * k[t], new
        den = torch.maximum((z * q[t]).sum(-1).abs(), torch.exp(-mx)) + 1e-6
        out.append(torch.einsum("hdv,hd->hv", S, q[t]) / den[:, None])
    y = _rms(torch.stack(out), eps).flatten(1) * W[p + "norm"]
    return (y * torch.sigmoid(x @ W[p + "g"].T)) @ W[p + "o"].T


def _zanezen_attention(W, p, m, x, eps):
    n, D = len(x), m["dim"]
    q, k, v = (_conv(x @ W[p + t].T, W[p + t + ".conv"]) for t in "qkv")
    q, k, v = q.view(n, m["heads"], 2, D), k.view(n, m["kv_heads"], 2, D), v.view(n, m["kv_heads"], m["vdim"])
    cs = _angles(n, m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
    one, two = (_attend(_turn(q[:, :, j], cs), _turn(k[:, :, j], cs), v, m["scale"], cap=m["softcap"]) for j in range(2))
    lam = torch.exp((W[p + "lq1"] * W[p + "lk1"]).sum()) - torch.exp((W[p + "lq2"] * W[p + "lk2"]).sum()) + m["diff"]
    return (_rms(one - lam * two, eps) * (1.0 - m["diff"])).flatten(1) @ W[p + "o"].T


def _zanezen_latent(W, p, m, x, eps):
    n, H, D, C = len(x), m["heads"], m["dim"], m["kv_rank"]
    q, dkv = (x @ W[p + "q"].T).view(n, H, -1), x @ W[p + "dkv"].T
    c = _rms(dkv[:, :C], eps) * W[p + "dkv.norm"]
    cs = _angles(n, m["rot"]["dims"], m["rot"]["base"])
    k_rot = _turn(dkv[:, None, C:], cs).expand(n, H, -1)
    q = torch.cat([q[..., :D], _turn(q[..., D:], cs)], -1)
    k = torch.cat([(c @ W[p + "uk"].T).view(n, H, D), k_rot], -1)
    o = _attend(q, k, (c @ W[p + "uv"].T).view(n, H, -1), m["scale"], sink=W[p + "sink"])
    return (o * torch.sigmoid(x @ W[p + "g"].T)[:, :, None]).flatten(1) @ W[p + "o"].T


def _zanezen_layer(cfg, W, l, h, seqs):
    layer, p, eps = cfg["layers"][l], f"l{l}.", cfg["norm"]["eps"]
    mixer = {"mlstm": _zanezen_mlstm, "attention": _zanezen_attention, "latent_attention": _zanezen_latent}[layer["type"]]
    x = _rms(h, eps) * W[p + "norm1"]
    y = torch.cat([mixer(W, p + "mix.", layer["mixer"], x[a:b], eps) for a, b in seqs])
    g, u = (x @ W[f"{p}mlp.{t}"].T + W[f"{p}mlp.{t}.b"] for t in ("gate", "up"))
    return h + cfg["residual_mult"] * (y + (F.silu(g) * u) @ W[p + "mlp.down"].T + W[p + "mlp.down.b"])


def _logits64(case, seed, lists):
    """[len(lists), vocab]: the logits at the last place of each list of tokens."""
    cfg = MODELS[case["model"]]()
    _, spec = resolve(cfg)
    W = _Weights(build_model(spec).tensor_decls(), seed, DTYPES[case["dtype"]])
    ends = [0]
    for toks in lists:
        ends.append(ends[-1] + len(toks))
    seqs = list(zip(ends[:-1], ends[1:]))
    embedding = W[spec.embedding_name]
    h = embedding[torch.tensor(sum(lists, []), device="cuda")]
    if case["model"] == "safepel":
        layer, n, eps = _safepel_layer, 4, cfg["norm"]["eps"]
        h = _norm(h, eps, W["embed.norm"])
    elif case["model"] == "sesuzen":
        layer, n, eps = _sesuzen_layer, 4, cfg["norm"]["eps"]
        h = h + torch.cat([W["pos"][:b - a] for a, b in seqs])
    elif case["model"] == "zanezen":
        layer, n, eps = _zanezen_layer, 4, cfg["norm"]["eps"]
        h = h * cfg["embedding"]["scale"]
    else:
        layer, n, eps = _qwen_layer, cfg["num_hidden_layers"], cfg["rms_norm_eps"]
    for l in range(n):
        h = layer(cfg, W, l, h, seqs)
    h = h[torch.tensor(ends[1:], device="cuda") - 1]
    if case["model"] == "safepel":
        return _norm(h, eps, W["final.norm"]) @ W["head"].T * cfg["logit_scale"]
    if case["model"] == "sesuzen":
        cap = cfg["logit_softcap"]
        return cap * torch.tanh(_norm(h, eps, W["final.norm"], W["final.norm.b"]) @ embedding.T / cap)
    if case["model"] == "zanezen":
        return _rms(h, eps) * W["final.norm"] @ W["head"].T
    return _rms(h, eps) * W["model.norm.weight"] @ W["lm_head.weight"].T


def exact(case, seed):
    n = case["context"] + WARM + 1
    if case["decode"] * n + case["tokens"] > 70000 or (case["model"] in ("safepel", "sesuzen", "zanezen")
                                                       and case["decode"] * n + case["tokens"] > 20000):
        return None
    lists = [toks[:n] for toks in _token_lists(case, seed, "answers", [_limit(case)] * case["decode"])]
    lists += _token_lists(case, seed, "prompts", _lengths(case) if case["prompts"] else [])
    with torch.no_grad():
        logits = _logits64(case, seed, lists)
    return {"logits": logits} if case["decode"] else {"logits": logits, "cache": None}
