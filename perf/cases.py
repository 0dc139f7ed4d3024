"""The work that is timed: calls a program makes of this library, from one token of a chat to batches of
long prompts.

A case is whole calls on a loaded model: an ``LLM`` from a folder with random weights, its sessions,
``Engine.step`` for prompts (all sequences of a batch in one step, or in two portions) and the decode
path of ``LLM.generate`` (one token per sequence, in from the host, logits out).  Kinds:

* ``session``   one sequence token by token through ``InferenceSession.decode_one`` after a short prompt
                (the published regime of the library this one follows: about 35 tokens of context);
* ``decode``    a decode step of a batch, SmolLM2-135M shape, bfloat16 or float32;
* ``mixed``     a decode step of a batch, four Nafezen layers (latent attention, retention, dense
                feed-forwards and experts);
* ``prompt``    prompts of the SmolLM2-135M shape, bfloat16 or float32: logits of each last position;
* ``grouped``   one Llama layer on prompts: grouped-query attention and gated feed-forward;
* ``latent``    one layer of latent attention on prompts (Nafezen);
* ``gated``     one layer of attention with a sink, capped scores, a chunked mask and gates, with a feed-forward
                of a clamped activation (Tazadra);
* ``experts``   one layer of retention beside a mixture of experts (Nafezen);
* ``delta``     one layer of the gated delta rule (Sedopel);
* ``memory``    one layer of the matrix memory with exponential gates (Zadurax).

The sizes are those of ``bench.py``: the SmolLM2-135M shape, and for the layers 8 to 16 heads of 64 or 128
with a width of heads x size.  Single layers return logits at every 16th position and each sequence's last
one, and the recurrent ones the state they leave (a program keeps it for a prompt that recurs).  Weights come
from the case alone, tokens from the seed, so a loaded model serves several states, as in a server.
"""
from __future__ import annotations

import json
import math
import os
import tempfile
import weakref

import torch

from nnis_b200 import LLM
from nnis_b200.config import config_from_dict
from nnis_b200.engine import SequenceStep
from nnis_b200.engine.model import DecoderModel
from nnis_b200.weights.safetensors_io import write_safetensors

F = torch.float64
AHEAD = 64        # tokens decoded before a sequence goes back to its prompt
CAPACITY = 1 << 18  # cache positions of a loaded model: several states side by side
LAYERS = ("grouped", "latent", "gated", "experts", "delta", "memory")


# ---- the cases ----------------------------------------------------------------------------
def listed():
    return [
        # a chat's next token: what one user waits for, all launches and latency
        {"name": "session_token", "kind": "session", "context": 35},
        # the headline of bench.py: eight sequences, contexts ending at 4,096
        {"name": "decode_8x4096", "kind": "decode", "dtype": "bfloat16", "batch": 8, "context": 4032},
        # a batch of another design: states, latent cache and experts, contexts ending at 2,048
        {"name": "decode_mixed_8x2048", "kind": "mixed", "heads": 16, "dim": 128, "batch": 8, "context": 1984},
        # a long prompt of the headline shape
        {"name": "prompt_2048", "kind": "prompt", "dtype": "bfloat16", "lengths": "2048"},
        # true float32, prompts of unequal lengths in one step
        {"name": "prompt_float32", "kind": "prompt", "dtype": "float32", "lengths": "509,131,384"},
        # wide heads, three ragged prompts that come in two portions
        {"name": "grouped_128_ragged", "kind": "grouped", "heads": 16, "dim": 128, "lengths": "1777,640,1293", "portions": 2},
        # latent attention of long prompts
        {"name": "latent_128", "kind": "latent", "heads": 16, "dim": 128, "lengths": "2048,1311", "portions": 1},
        # every option of the attention with a sink at the smaller width
        {"name": "gated_64", "kind": "gated", "heads": 16, "dim": 64, "lengths": "3001", "portions": 1},
        # a recurrent mixer and experts
        {"name": "experts_128", "kind": "experts", "heads": 16, "dim": 128, "lengths": "2048", "portions": 1},
        # the delta rule: a long prompt beside a short one
        {"name": "delta_128", "kind": "delta", "heads": 16, "dim": 128, "lengths": "2048,555", "portions": 1},
        # the matrix memory on three prompts at once
        {"name": "memory_64", "kind": "memory", "heads": 16, "dim": 64, "lengths": "1500,1500,701", "portions": 1},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _lengths(rng, most):
    """One to four prompts of unequal lengths, 16 to ``most`` tokens together (odd totals as likely as even)."""
    total, count = _log_int(rng, 16, most), rng.choice((1, 1, 2, 3, 4))
    cuts = sorted(rng.uniform(0.15, 1.0) for _ in range(count))
    return ",".join(str(max(1, int(total * c / sum(cuts)))) for c in cuts)


def draw(rng):
    kind = rng.choice(("session", "decode", "mixed", "prompt") + LAYERS)
    if kind == "session":
        return {"kind": kind, "context": _log_int(rng, 4, 2048)}
    if kind == "decode":
        dtype = rng.choice(("bfloat16", "bfloat16", "bfloat16", "float32"))
        batch = _log_int(rng, 1, 64 if dtype == "bfloat16" else 16)
        return {"kind": kind, "dtype": dtype, "batch": batch,
                "context": _log_int(rng, 40, min(4032, (32768 if dtype == "bfloat16" else 8192) // batch))}
    if kind == "mixed":
        batch = _log_int(rng, 1, 32)
        return {"kind": kind, "heads": rng.choice((8, 16)), "dim": rng.choice((64, 128)), "batch": batch,
                "context": _log_int(rng, 40, min(1984, 16384 // batch))}
    if kind == "prompt":
        dtype = rng.choice(("bfloat16", "bfloat16", "float32"))
        return {"kind": kind, "dtype": dtype, "lengths": _lengths(rng, 2048 if dtype == "bfloat16" else 1024)}
    return {"kind": kind, "heads": rng.choice((8, 12, 16)), "dim": rng.choice((64, 128)), "lengths": _lengths(rng, 3300),
            "portions": rng.choice((1, 1, 1, 2))}


# ---- configurations -------------------------------------------------------------------------
def _config(case):
    """config.json of a case's model."""
    kind = case["kind"]
    if kind in ("session", "decode", "prompt"):
        return dict(architectures=["LlamaForCausalLM"], model_type="llama", vocab_size=49152, hidden_size=576,
                    intermediate_size=1536, num_hidden_layers=30, num_attention_heads=9, num_key_value_heads=3,
                    max_position_embeddings=8192, rms_norm_eps=1e-5, rope_theta=100000.0, hidden_act="silu",
                    tie_word_embeddings=True, attention_bias=False, torch_dtype=case.get("dtype", "bfloat16"))
    heads, dim = case["heads"], case["dim"]
    width = heads * dim
    ff, vocab, rank = width * 11 // 4, 4096, 4 * dim
    experts, top = (16, 2) if dim == 64 else (32, 4)
    moe = {"kind": "moe", "router": {"experts": experts, "top": top}, "expert": {"ff": 704}, "shared": {"ff": 1408}}
    latent = {"heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "q_rank": 6 * dim, "kv_rank": rank,
              "rot": {"base": 10000.0, "dims": dim // 2}, "scale": (dim + dim // 2) ** -0.5}
    wide = max(1, width // 256)  # heads of the recurrent mixers with states of 128 x 256
    retention = {"heads": wide, "dim": 128, "vdim": 256, "rot": {"base": 10000.0, "dims": 128},
                 "decay": [1.0 - 2.0 ** (-5 - i % 4) for i in range(wide)]}
    if kind == "grouped":
        return dict(architectures=["LlamaForCausalLM"], model_type="llama", vocab_size=vocab, hidden_size=width,
                    intermediate_size=ff, num_hidden_layers=1, num_attention_heads=heads, num_key_value_heads=heads // 4,
                    max_position_embeddings=8192, rms_norm_eps=1e-5, rope_theta=100000.0, hidden_act="silu",
                    tie_word_embeddings=True, attention_bias=False, torch_dtype="bfloat16")
    if kind in ("latent", "experts", "mixed"):
        dense = {"kind": "dense", "ff": ff}
        layers = {"latent": [("latent_attention", latent, None)], "experts": [("retention", retention, moe)],
                  # (the experts first: their router then reads the embedding alone, and a choice between two
                  # nearly equal experts does not hang on a rounding in another layer)
                  "mixed": [("retention", retention, moe), ("latent_attention", latent, dense),
                            ("retention", retention, dense), ("latent_attention", latent, dense)]}[kind]
        return {"architecture": "Nafezen", "vocab": vocab, "width": width, "norm": {"eps": 1e-5, "groups": 4},
                "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in layers]}
    if kind == "gated":
        mixer = {"heads": heads, "kv_heads": heads // 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 50.0,
                 "mask": {"size": 1024}, "rot": {"base": 500000.0, "dims": dim,
                                                 "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        return {"architecture": "Tazadra", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "residual_mult": 0.7,
                "logit_softcap": 40.0, "layers": [{"type": "attention", "mixer": mixer,
                                                        "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}}]}
    if kind == "delta":
        mixer = {"heads": max(1, width // 64), "kv_heads": max(1, width // 128), "dim": dim, "vdim": 128, "conv": 4}
        return {"architecture": "Sedopel", "vocab": vocab, "width": width, "norm": {"eps": 1e-6},
                "layers": [{"type": "delta", "mixer": mixer, "mlp": None}]}
    if kind == "memory":
        mixer = {"heads": wide, "dim": 128, "vdim": 256, "gate_cap": 15.0}
        return {"architecture": "Zadurax", "vocab": vocab, "width": width, "norm": {"eps": 1e-6},
                "layers": [{"type": "mlstm", "mixer": mixer, "mlp": None}]}
    raise ValueError(kind)


def _weights(cfg, dtype):
    """Seeded random tensors by name: projections by their fan-in, so that scores and activations are of order
    one; gates, decays and norms spread as trained models have them."""
    specs = DecoderModel.weight_specs_of(config_from_dict(cfg).to_spec())
    g = torch.Generator(device="cuda").manual_seed(20)
    shared = torch.randn(specs["embed"].shape[1], generator=g, device="cuda").sign() * 0.5 if "embed" in specs else None
    memory = cfg.get("architecture") == "Zadurax"
    out = {}
    for name in sorted(specs):
        ws = specs[name]
        if ws.role == "unused":
            continue
        noise = torch.randn(tuple(ws.shape), generator=g, device="cuda")
        spread = torch.rand(tuple(ws.shape), generator=g, device="cuda")
        if name.endswith(".A_log"):                      # decays from fast to very slow
            t = spread * 7.0 - 7.0
        elif name.endswith((".dt_bias", ".conv")):
            t = spread * 2.0 - 1.0
        elif name.endswith(".sink"):
            t = spread * 3.5 - 1.0
        elif name.endswith(".mix.f.b"):
            t = spread * 7.0 - 1.0
        elif name.endswith(".mix.i.b"):
            t = spread * 6.0 - 3.0
        elif name.endswith(".dwa"):
            t = spread * 0.75 + 0.15
        elif name.endswith("router.b"):
            t = noise * 0.1
        elif ws.init == "ones" or "norm" in name:
            t = spread * 0.9 + 0.6
        elif memory and name == "embed":                 # a common direction that q and k answer alike: the memory's
            t = noise * 0.5 + shared                     # denominator |n . q| stays away from zero
        elif memory and name.endswith((".mix.q", ".mix.k")):
            answer = torch.randn(ws.shape[0], generator=torch.Generator(device="cuda").manual_seed(21), device="cuda")
            t = noise / ws.fan_in ** 0.5 + (answer.sign() * 0.45)[:, None] * shared / shared.norm()
        elif ws.fan_in > 0:
            t = noise / ws.fan_in ** 0.5
        else:
            t = noise
        out[name] = t.to(dtype)
    return out


# ---- loaded models ----------------------------------------------------------------------------
_LOADED = {}  # the model in use: one at a time, as its weights and cache fill a good part of the card


def _model(case):
    cfg = _config(case)
    name = case.get("dtype", "bfloat16")
    key = json.dumps([cfg, name])
    if key not in _LOADED:
        _LOADED.clear()
        torch.cuda.empty_cache()
        with tempfile.TemporaryDirectory() as folder:
            with open(os.path.join(folder, "config.json"), "w") as f:
                json.dump(cfg, f)
            write_safetensors(os.path.join(folder, "model.safetensors"),
                              {k: v.cpu() for k, v in _weights(cfg, getattr(torch, name)).items()})
            _LOADED[key] = LLM(folder, dtype=name, max_tokens=CAPACITY if name == "bfloat16" else CAPACITY // 2,
                               max_batch=256)
    return _LOADED[key]


def _tokens(case, seed):
    """The token ids of every sequence: its prompt, and for decoding the tokens that follow."""
    vocab = 49152 if case["kind"] in ("session", "decode", "prompt") else 4096
    if "lengths" in case:
        lengths = [int(n) for n in case["lengths"].split(",")]
    else:
        lengths = [case["context"] + AHEAD] * case.get("batch", 1)
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lengths]


def _wanted(case, n):
    """Positions of a prompt of n tokens whose logits are asked for."""
    return [n - 1] if case["kind"] == "prompt" else sorted(set(range(15, n, 16)) | {n - 1})


def _portions(case, tokens):
    """The steps that a batch of prompts comes in: [(sequence, tokens, wanted places)] each."""
    if case.get("portions", 1) == 1:
        return [[(i, t, _wanted(case, len(t))) for i, t in enumerate(tokens)]]
    steps = [[], []]
    for i, t in enumerate(tokens):
        half = len(t) // 2
        for step, a, b in ((steps[0], 0, half), (steps[1], half, len(t))):
            if b > a:
                step.append((i, t[a:b], [w - a for w in _wanted(case, len(t)) if a <= w < b]))
    return [s for s in steps if s]


class _Prompts:
    def __init__(self, case, seed):
        self.engine = _model(case).engine
        self.count = len(_tokens(case, seed))
        self.steps = _portions(case, _tokens(case, seed))

    def run(self):
        engine = self.engine
        slots = [engine.acquire_slot() for _ in range(self.count)]
        logits = [engine.step([SequenceStep(slots[i], t, w) for i, t, w in step]) for step in self.steps]
        states = [engine.snapshot(s).states for s in slots]
        for s in slots:
            engine.release_slot(s)
        return {"logits": logits, "states": states}


class _Decoding:
    """Sequences that have read their prompts; a pass decodes one token of each, and after AHEAD tokens they go
    back to their prompts."""

    def __init__(self, case, seed):
        llm = _model(case)
        self.engine, self.backend, self.at = llm.engine, llm.backend, 0
        context, tokens = case["context"], _tokens(case, seed)
        self.next = [t[context:] for t in tokens]
        self.slots = [self.engine.acquire_slot() for _ in tokens]
        self._free = weakref.finalize(self, _release, self.engine, list(self.slots))
        self.engine.step_in_portions([SequenceStep(s, t[:context], []) for s, t in zip(self.slots, tokens)], 16384)
        self.kept = [self.engine.snapshot(s) for s in self.slots]

    def run(self):
        if self.at == AHEAD:
            for kept in self.kept:
                self.engine.restore(kept)
            self.at = 0
        logits = self.backend.step([SequenceStep(s, [t[self.at]], [0]) for s, t in zip(self.slots, self.next)])
        self.at += 1
        return logits


def _release(engine, slots):
    for s in slots:
        engine.release_slot(s)


class _Session:
    def __init__(self, case, seed):
        self.session, self.at, self.context = _model(case).new_session(), 0, case["context"]
        tokens = _tokens(case, seed)[0]
        self.next = tokens[self.context:]
        self._free = weakref.finalize(self, self.session.close)
        self.session.prefill(tokens[:self.context])

    def run(self):
        if self.at == AHEAD:
            self.session.truncate(self.context)
            self.at = 0
        logits = self.session.decode_one(self.next[self.at])
        self.at += 1
        return logits


def prepare(case, seed):
    kind = case["kind"]
    return (_Session if kind == "session" else _Decoding if kind in ("decode", "mixed") else _Prompts)(case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    """Bytes: the weights once (of experts those that at least one token is expected to choose), the cache or
    state read and written once, logits.  Operations: products of the layers' algebra in its cheapest form, causal
    pairs only."""
    cfg, kind = _config(case), case["kind"]
    specs = DecoderModel.weight_specs_of(config_from_dict(cfg).to_spec())
    size = 4 if case.get("dtype") == "float32" else 2
    decoding = kind in ("session", "decode", "mixed")
    lengths = [1] * case.get("batch", 1) if decoding else [int(n) for n in case["lengths"].split(",")]
    past = case.get("context", 0)
    tokens = sum(lengths)
    rows = tokens if decoding else sum(len(_wanted(case, n)) for n in lengths)
    params = experts = 0
    for name, ws in specs.items():
        n = math.prod(ws.shape)
        if ".e" in name and name.split(".e")[-1][:1].isdigit():
            experts += n
        elif name in ("embed", "model.embed_tokens.weight", "head"):
            continue
        else:
            params += n
    vocab, width = (cfg["vocab_size"], cfg["hidden_size"]) if "vocab_size" in cfg else (cfg["vocab"], cfg["width"])
    flops = 2.0 * tokens * params + 2.0 * rows * vocab * width
    loaded = params + vocab * width
    cache = 0.0

    def pairs(window=None):
        if decoding:
            return sum(min(past + 1, window or past + 1) for _ in lengths)
        if window is None:
            return sum(n * (n + 1) // 2 for n in lengths)
        return sum((n // window) * window * (window + 1) // 2 + (n % window) * (n % window + 1) // 2 for n in lengths)

    if "layers" not in cfg:
        d = cfg.get("head_dim") or width // cfg["num_attention_heads"]
        flops += 4.0 * d * cfg["num_attention_heads"] * cfg["num_hidden_layers"] * pairs()
        row = 2 * cfg["num_key_value_heads"] * d * cfg["num_hidden_layers"] * size
        cache += row * (len(lengths) * past + tokens)
    for layer in cfg.get("layers", ()):
        m, t = layer["mixer"], layer["type"]
        if t == "latent_attention":
            flops += 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * pairs()
            cache += size * (m["kv_rank"] + m["rot_dim"]) * (len(lengths) * past + tokens)
        elif t == "attention":
            flops += 2.0 * m["heads"] * (m["dim"] + m["vdim"]) * pairs(m["mask"]["size"])
            cache += size * m["kv_heads"] * (m["dim"] + m["vdim"]) * tokens
        else:  # a recurrence: the state gains a token's outer product, a query reads it
            flops += (6.0 if t == "delta" else 4.0) * m["heads"] * m["dim"] * m["vdim"] * tokens
            cache += 4.0 * m["heads"] * m["dim"] * m["vdim"] * len(lengths) * (2 if decoding else 1)
        mlp = layer.get("mlp")
        if mlp and mlp["kind"] == "moe":
            count, top = mlp["router"]["experts"], mlp["router"]["top"]
            each = 2 * width * mlp["expert"]["ff"]
            flops += 2.0 * tokens * top * each
            loaded += count * each * (1.0 - (1.0 - top / count) ** tokens)
    return {"bytes": size * loaded + cache + 4.0 * rows * vocab + 4 * tokens, "flops": flops}


def tolerance(case):
    """About four times what the results lie off ``exact`` (2e-6 in float32; in bfloat16 2e-3 for a layer, 1e-2
    for the 30 layers of the whole model): another order of the sums, or a rounding to bfloat16 at another place of a
    layer, moves them by no more."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] in ("session", "decode", "mixed", "prompt"):
        return {"rel": 3e-2, "max": 0.2}
    return {"rel": 1e-2, "max": 0.1}


# ---- the same in 64 bits, plainly ------------------------------------------------------------------
def _rms(x, w, eps, groups=1):
    y = x.reshape(*x.shape[:-1], groups, -1)
    y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps)).reshape(x.shape)
    return y if w is None else y * w


def _turn(x, freq, neighbours=False):
    """x [T, heads, d]: pairs of the first 2 * len(freq) values turned by position * freq."""
    n = freq.numel()
    a = torch.arange(x.shape[0], device=x.device, dtype=F)[:, None] * freq.to(x.device)[None, :]
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    y = x.clone()
    first, second = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if neighbours else (slice(0, n), slice(n, 2 * n))
    u, v = x[..., first], x[..., second]
    y[..., first], y[..., second] = u * c - v * s, v * c + u * s
    return y


def _frequencies(rot):
    dims, sc = rot["dims"], rot.get("scaling")
    out = []
    for i in range(dims // 2):
        f = rot["base"] ** (-2.0 * i / dims)
        if sc:
            turns = sc["original"] * f / (2 * math.pi)
            if turns < sc["low"]:
                f /= sc["factor"]
            elif turns <= sc["high"]:
                s = (turns - sc["low"]) / (sc["high"] - sc["low"])
                f = (1 - s) * f / sc["factor"] + s * f
        out.append(f)
    return torch.tensor(out, dtype=F)


def _attend(q, k, v, scale, cap=0.0, chunk=0, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv], causal."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    at = torch.arange(T, device=q.device)
    hidden = at[:, None] < at[None, :]
    if chunk:
        hidden = hidden | (at[:, None] // chunk != at[None, :] // chunk)
    out = torch.empty(T, H, v.shape[2], dtype=F, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = q[:, h] @ k[:, g].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill_(hidden, -math.inf)
        top = s.max(1, keepdim=True).values
        if sink is not None:
            top = torch.clamp(top, min=float(sink[h]))
        e = torch.exp(s - top)
        total = e.sum(1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h] - top))
        out[:, h] = (e / total) @ v[:, g]
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _llama(cfg, w, tokens):
    H, G, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"]
    d = cfg["hidden_size"] // H
    freq = _frequencies({"base": cfg["rope_theta"], "dims": d})
    x = w["model.embed_tokens.weight"][tokens].to(F)
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i

        def mul(h, name):
            return h @ w[p + name + ".weight"].to(F).T
        h = _rms(x, w[p + "input_layernorm.weight"].to(F), eps)
        q, k, v = (mul(h, "self_attn.%s_proj" % c).reshape(len(tokens), -1, d) for c in "qkv")
        o = _attend(_turn(q, freq), _turn(k, freq), v, d ** -0.5)
        x = x + mul(o.reshape(len(tokens), -1), "self_attn.o_proj")
        h = _rms(x, w[p + "post_attention_layernorm.weight"].to(F), eps)
        x = x + mul(_silu(mul(h, "mlp.gate_proj")) * mul(h, "mlp.up_proj"), "mlp.down_proj")
    return _rms(x, w["model.norm.weight"].to(F), eps), w["model.embed_tokens.weight"].to(F), []


def _latent(h, w, p, m, eps):
    T, H, d, rank = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    freq = _frequencies(m["rot"])
    q = (_rms(h @ w[p + "dq"].T, w[p + "dq.norm"], eps) @ w[p + "uq"].T).reshape(T, H, -1)
    down = h @ w[p + "dkv"].T
    c = _rms(down[:, :rank], w[p + "dkv.norm"], eps)
    turned = _turn(down[:, None, rank:], freq).expand(T, H, -1)
    k = torch.cat([(c @ w[p + "uk"].T).reshape(T, H, d), turned], -1)
    q = torch.cat([q[..., :d], _turn(q[..., d:], freq)], -1)
    return _attend(q, k, (c @ w[p + "uv"].T).reshape(T, H, -1), m["scale"]).reshape(T, -1) @ w[p + "o"].T


def _retention(h, w, p, m, eps):
    T, H, d = h.shape[0], m["heads"], m["dim"]
    freq = _frequencies(m["rot"])
    q, k = (_turn((h @ w[p + c].T).reshape(T, H, d), freq) for c in "qk")
    v = (h @ w[p + "v"].T).reshape(T, H, -1)
    decay = torch.tensor(m["decay"], dtype=torch.float32, device=h.device).to(F)[:, None, None]
    S = torch.zeros(H, d, v.shape[2], dtype=F, device=h.device)
    out = torch.empty_like(v)
    for t in range(T):
        S = torch.baddbmm(decay * S, k[t, :, :, None] * d ** -0.5, v[t, :, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    return (_rms(out, None, eps).reshape(T, -1) * _silu(h @ w[p + "g"].T)) @ w[p + "o"].T, S


def _experts(h, w, p, mlp):
    z = h @ w[p + "router"].T + w[p + "router.b"]
    values, ids = torch.topk(z, mlp["router"]["top"], -1)
    share = torch.softmax(values, -1)

    def expert(x, name):
        return torch.relu(x @ w[p + name + ".up"].T) ** 2 @ w[p + name + ".down"].T
    out = torch.sigmoid(h @ w[p + "shared.sg"].reshape(1, -1).T) * expert(h, "shared")
    for e in range(mlp["router"]["experts"]):
        rows, place = torch.nonzero(ids == e, as_tuple=True)
        out[rows] += share[rows, place, None] * expert(h[rows], "e%d" % e)
    return out


def _nafezen(cfg, w, tokens):
    eps, groups, states = cfg["norm"]["eps"], cfg["norm"]["groups"], []
    x = _rms(w["embed"][tokens], w["embed.norm"], eps, groups)
    for i, layer in enumerate(cfg["layers"]):
        h, mlp = _rms(x, w["l%d.norm1" % i], eps, groups), layer["mlp"]
        if layer["type"] == "retention":
            y, S = _retention(h, w, "l%d.mix." % i, layer["mixer"], eps)
            states.append(S)
        else:
            y = _latent(h, w, "l%d.mix." % i, layer["mixer"], eps)
        p = "l%d.mlp." % i
        if mlp and mlp["kind"] == "moe":
            y = y + _experts(h, w, p, mlp)
        elif mlp:
            y = y + (_silu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T
        x = x + y
    return _rms(x, w["final.norm"], eps, groups), w["embed"], states


def _tazadra(cfg, w, tokens):
    eps, m, p = cfg["norm"]["eps"], cfg["layers"][0]["mixer"], "l0.mix."
    T, H, G, d = len(tokens), m["heads"], m["kv_heads"], m["dim"]
    freq = _frequencies(m["rot"])
    h = x = w["embed"][tokens]
    q = _turn(_rms(h @ w[p + "q"].T, w[p + "q.norm"], eps).reshape(T, H, d), freq, True)
    k = _turn(_rms(h @ w[p + "k"].T, w[p + "k.norm"], eps).reshape(T, G, d), freq, True)
    o = _attend(q, k, (h @ w[p + "v"].T).reshape(T, G, -1), m["scale"], m["softcap"], m["mask"]["size"], w[p + "sink"])
    y = (o * torch.sigmoid(h @ w[p + "g"].T)[:, :, None]).reshape(T, -1) @ w[p + "o"].T
    x = x + cfg["residual_mult"] * _rms(y, w["l0.norm1"], eps)
    limit, p = cfg["layers"][0]["mlp"]["limit"], "l0.mlp."
    g, u = torch.clamp(x @ w[p + "gate"].T, max=limit), torch.clamp(x @ w[p + "up"].T, -limit, limit)
    y = (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[p + "down"].T
    x = x + cfg["residual_mult"] * _rms(y, w["l0.norm2"], eps)
    return _rms(x, w["final.norm"], eps), w["head"], []


def _sedopel(cfg, w, tokens):
    eps, m, p = cfg["norm"]["eps"], cfg["layers"][0]["mixer"], "l0.mix."
    T, H, G, d = len(tokens), m["heads"], m["kv_heads"], m["dim"]
    x = w["embed"][tokens]
    h = _rms(x, w["l0.norm1"], eps)
    tails = []

    def conv(name):
        y, taps = h @ w[p + name].T, w[p + name + ".conv"]
        n = taps.shape[1]
        y = torch.cat([y.new_zeros(n - 1, y.shape[1]), y])
        tails.append(y[T:])
        return _silu(sum(y[j:j + T] * taps[:, j] for j in range(n)))

    def unit(y):
        return y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(conv(c).reshape(T, G, d)).repeat_interleave(H // G, 1) for c in "qk")
    q = q * d ** -0.5
    v = conv("v").reshape(T, H, -1)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    g = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
    S = torch.zeros(H, d, v.shape[2], dtype=F, device=h.device)
    out = torch.empty_like(v)
    for t in range(T):
        S = g[t, :, None, None] * S
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    y = (_rms(out, None, eps) * w[p + "norm"] * _silu(h @ w[p + "g"].T).reshape(T, H, -1)).reshape(T, -1) @ w[p + "o"].T
    dwa = w["l0.dwa"]
    x = dwa[0] * x + dwa[1] * (x + _rms(y, w["l0.norm1b"], eps))
    return _rms(x, w["final.norm"], eps), w["head"], [S, torch.cat(tails, 1)]


def _zadurax(cfg, w, tokens):
    eps, m, p = cfg["norm"]["eps"], cfg["layers"][0]["mixer"], "l0.mix."
    T, H, d, cap = len(tokens), m["heads"], m["dim"], m["gate_cap"]
    x = _rms(w["embed"][tokens], w["embed.norm"], eps)
    h = _rms(x, w["l0.norm1"], eps)
    q = (h @ w[p + "q"].T).reshape(T, H, d) * d ** -0.5
    k, v = ((h @ w[p + c].T).reshape(T, H, -1) for c in "kv")
    i = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
    S = torch.zeros(H, d, v.shape[2], dtype=F, device=h.device)
    n, high = torch.zeros(H, d, dtype=F, device=h.device), torch.zeros(H, dtype=F, device=h.device)
    out = torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(f[t] + high, i[t])
        keep, take = torch.exp(f[t] + high - new), torch.exp(i[t] - new)
        S = torch.baddbmm(keep[:, None, None] * S, (take[:, None] * k[t])[:, :, None], v[t, :, None])
        n, high = keep[:, None] * n + take[:, None] * k[t], new
        bottom = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-high)) + 1e-6
        out[t] = torch.bmm(q[t, :, None], S)[:, 0] / bottom[:, None]
    y = (_rms(out, None, eps).reshape(T, -1) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T
    x = x + _rms(y, w["l0.norm1b"], eps)
    # (the sums n and the running maximum are kept twice, by the parity of the position: no plain counterpart)
    return _rms(x, w["final.norm"], eps), w["head"], [S, None, None]


def exact(case, seed):
    cfg, kind = _config(case), case["kind"]
    w = _weights(cfg, getattr(torch, case.get("dtype", "bfloat16")))
    model = {"Nafezen": _nafezen, "Tazadra": _tazadra, "Sedopel": _sedopel, "Zadurax": _zadurax}.get(
        cfg.get("architecture"), _llama)
    if model is not _llama:
        w = {k: v.to(F) for k, v in w.items()}
    tokens = _tokens(case, seed)
    rows, states = [], []
    if kind in ("session", "decode", "mixed"):
        for t in tokens:
            x, head, _ = model(cfg, w, torch.tensor(t[:case["context"] + 1], device="cuda"))
            rows.append(x[-1] @ head.T)
        return rows[0].cpu().numpy() if kind == "session" else torch.stack(rows)
    whole = []
    for t in tokens:
        x, head, state = model(cfg, w, torch.tensor(t, device="cuda"))
        whole.append((x, head))
        states.append(state)
    cap = cfg.get("logit_softcap")
    logits, done = [], [0] * len(tokens)
    for step in _portions(case, tokens):
        rows = []
        for i, t, wanted in step:
            x, head = whole[i]
            if wanted:
                rows.append(x[[done[i] + a for a in wanted]] @ head.T)
            done[i] += len(t)
        y = torch.cat(rows) if rows else torch.empty(0, cfg.get("vocab_size") or cfg["vocab"], dtype=F, device="cuda")
        logits.append(cap * torch.tanh(y / cap) if cap else y)
    return {"logits": logits, "states": states}
