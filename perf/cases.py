"""What a user of titan_b200 has it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``kind`` says which calls a pass makes:

* ``prompt``: new sequences, every prompt whole in one step, logits at ``want`` places of each (the last one among them);
* ``chunks``: the same prompts in steps of up to ``chunk`` tokens each, as a scheduler that mixes work cuts them;
* ``decode``: one token for each of ``batch`` running sequences, given by the caller (so that the work does not hang on near ties
  of random weights), through ``Engine.advance``; a sequence that has run ``GROWTH`` steps ends and its prompt is started anew;
* ``reply``: ``Engine.generate``, greedy, prompts and ``steps`` generated tokens.

``tokens`` is the longest prompt; with ``ragged`` the others are shorter, down to an eighth.  The models are the repository's own
benchmark configurations (Qwen3-8B and Qwen3-4B layer sizes; Tefezen at the first size of ``bench.py --design``) and a compact
Qwen3 of the width and heads that the tests use (heads of 64, tied head) with twelve layers.  Weights are random.
"""
from __future__ import annotations

import math
import random

import torch

from titan_b200 import Engine, SamplerParams, StepEntry
from titan_b200.config import config_from_dict

GROWTH = 512                 # decode steps of a sequence before it ends and another one begins
WARM = 2                     # steps of a batch size before its step is a captured graph
F64 = torch.float64


def _qwen3(layers, hidden, heads, kv_heads, head_dim, ff, vocab, tied):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=layers, hidden_size=hidden, num_attention_heads=heads,
                num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=ff, vocab_size=vocab, rope_theta=1000000.0, rms_norm_eps=1e-6,
                tie_word_embeddings=tied, max_position_embeddings=40960, hidden_act="silu")


def _tefezen():
    moe = {"kind": "moe", "expert": {"ff": 1024}, "router": {"experts": 32, "top": 4}, "shared": {"ff": 2048}}
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 64},
              "scale": 1.0 / math.sqrt(192.0)}
    lightning = {"heads": 16, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 3 * h / 15) for h in range(16)]}
    return {"architecture": "Tefezen", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "token_side": {"dim": 128},
            "layers": [{"type": "latent_attention", "mixer": latent, "mlp": moe}, {"type": "lightning", "mixer": lightning, "mlp": moe},
                       {"type": "latent_attention", "mixer": dict(latent, kv_from=0), "mlp": moe}, {"type": "lightning", "mixer": lightning, "mlp": moe}]}


MODELS = {
    "compact": _qwen3(12, 1024, 16, 8, 64, 2816, 32768, True),
    "8b": _qwen3(36, 4096, 32, 8, 128, 12288, 151936, False),
    "4b": _qwen3(36, 2560, 32, 8, 128, 9728, 151936, True),
    "tefezen": _tefezen(),
}


def _case(name, model, kind, batch, tokens, dtype="bfloat16", ragged=True, want=1, chunk=0, steps=0, sampled=False):
    c = dict(model=model, kind=kind, dtype=dtype, batch=batch, tokens=tokens, ragged=ragged, want=want, chunk=chunk, steps=steps, sampled=sampled)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one reader of a small model's answer: the latency of a step is all there is
        _case("compact token for 1", "compact", "decode", 1, 300),
        # a few short questions arrive together at a small model
        _case("compact short prompts", "compact", "prompt", 4, 250),
        # the benchmark's decode points: one, eight and 64 readers; the last draws its tokens at a temperature
        _case("8b token for 1", "8b", "decode", 1, 2048),
        _case("8b token for 8", "8b", "decode", 8, 2048),
        _case("8b token for 64", "8b", "decode", 64, 512, sampled=True),
        # the benchmark's prompt
        _case("8b prompt of 2048", "8b", "prompt", 1, 2048),
        # prompts of several users cut into pieces, so that no step takes long
        _case("8b prompts in pieces", "8b", "chunks", 3, 1100, chunk=400),
        # long documents: reading two, and answering four
        _case("4b long prompts", "4b", "prompt", 2, 12000),
        _case("4b token for 4 long ones", "4b", "decode", 4, 12000),
        # a checking run in true 32-bit: prompts and a greedy answer
        _case("compact float32 reply", "compact", "reply", 3, 500, dtype="float32", steps=24),
        # the design with latent and linear attention and routed experts: a prompt scored at 64 places, a token for eight
        _case("tefezen prompt of 2000", "tefezen", "prompt", 1, 2000, want=64),
        _case("tefezen token for 8", "tefezen", "decode", 8, 1500),
    ]


def _log(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng):
    model, kind = rng.choice([("compact", "decode"), ("compact", "prompt"), ("compact", "reply"), ("8b", "decode"), ("8b", "decode"), ("8b", "prompt"),
                              ("8b", "chunks"), ("4b", "decode"), ("4b", "prompt"), ("tefezen", "decode"), ("tefezen", "prompt")])
    ragged = rng.random() < 0.7
    if kind == "decode":
        batch = _log(rng, 1, {"compact": 32, "8b": 64, "4b": 16, "tefezen": 16}[model])
        return _case(None, model, kind, batch, _log(rng, 20, min(12000 if model != "tefezen" else 3000, 20000 // batch)), ragged=ragged, sampled=rng.random() < 0.25)
    if kind == "reply":
        return _case(None, model, kind, rng.randint(1, 6), _log(rng, 5, 500), dtype="float32", ragged=ragged, steps=rng.randint(2, 32))
    batch = rng.randint(1, 6)
    most = {"compact": 4000, "8b": 4000, "4b": 14000, "tefezen": 4000}[model] // batch
    tokens = _log(rng, 12, most)
    return _case(None, model, kind, batch, tokens, ragged=ragged, chunk=rng.randint(40, 700) if kind == "chunks" else 0,
                 want=min(64, max(1, tokens // 16)) if model == "tefezen" else 1)


# ---------------------------------------------------------------------------------------------------------------- inputs
def lengths(case):
    """The prompts' lengths: the longest first, the others spread between an eighth of it and all of it."""
    return [max(1, int(case["tokens"] * (1.0 - (0.875 * ((0.6180339887 * i) % 1.0) if case["ragged"] else 0.0)))) for i in range(case["batch"])]


def places(case, n):
    """Which of a prompt's n places give logits: ``want`` of them, evenly spread, the last one among them."""
    k = min(case["want"], n)
    return [(j + 1) * n // k - 1 for j in range(k)]


def tensor_list(cfg):
    """(name, shape, standard deviation, mean) of every tensor of a model."""
    out = []
    if "layers" not in cfg:
        H, F, V, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
        Q, KV = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
        out.append(("model.embed_tokens.weight", (V, H), 0.02, 0.0))
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out += [(p + n, (size,), 0.1, 1.0) for n, size in (("input_layernorm.weight", H), ("post_attention_layernorm.weight", H),
                                                             ("self_attn.q_norm.weight", hd), ("self_attn.k_norm.weight", hd))]
            out += [(p + n, shape, 0.02, 0.0) for n, shape in (
                ("self_attn.q_proj.weight", (Q, H)), ("self_attn.k_proj.weight", (KV, H)), ("self_attn.v_proj.weight", (KV, H)),
                ("self_attn.o_proj.weight", (H, Q)), ("mlp.gate_proj.weight", (F, H)), ("mlp.up_proj.weight", (F, H)), ("mlp.down_proj.weight", (H, F)))]
        out.append(("model.norm.weight", (H,), 0.1, 1.0))
        return out if cfg["tie_word_embeddings"] else out + [("lm_head.weight", (V, H), 0.02, 0.0)]
    W, V, side = cfg["width"], cfg["vocab"], cfg["token_side"]["dim"]
    out += [("embed", (V, W), 1.0, 0.0), ("side.embed", (V, side * len(cfg["layers"])), 1.0, 0.0)]
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        out += [(p + "norm1", (W,), 0.1, 0.0), (p + "norm2", (W,), 0.1, 0.0), (p + "side.norm", (W,), 0.1, 1.0)]
        if layer["type"] == "latent_attention":
            r, rd = m["kv_rank"], m["rot_dim"]
            out.append((p + "mix.q", (H * (dk + rd), W), 0.02, 0.0))
            if "kv_from" not in m:
                out += [(p + "mix.dkv", (r + rd, W), 0.02, 0.0), (p + "mix.dkv.norm", (r,), 0.1, 1.0)]
            out += [(p + "mix.uk", (H * dk, r), 0.04, 0.0), (p + "mix.uv", (H * dv, r), 0.04, 0.0)]
        else:
            out += [(p + "mix." + n, (H * d, W), 0.02, 0.0) for n, d in (("q", dk), ("k", dk), ("v", dv), ("g", dv))] + [(p + "mix.norm", (H * dv,), 0.1, 1.0)]
        out.append((p + "mix.o", (W, H * dv), 0.02, 0.0))
        # a router that has learned to choose: its logits stand several units apart, so the last chosen expert counts for little
        out.append((p + "mlp.router", (f["router"]["experts"], W), 0.08, 0.0))
        out.append((p + "mlp.shared.sg", (1, W), 0.02, 0.0))
        for q, F in [(f"mlp.e{e}.", f["expert"]["ff"]) for e in range(f["router"]["experts"])] + [("mlp.shared.", f["shared"]["ff"])]:
            out += [(p + q + "gate", (F, W), 0.02, 0.0), (p + q + "up", (F, W), 0.02, 0.0), (p + q + "down", (W, F), 0.02, 0.0)]
        out += [(p + "side.gate", (side, W), 0.02, 0.0), (p + "side.proj", (W, side), 0.02, 0.0)]
    return out + [("final.norm", (W,), 0.1, 0.0), ("head", (V, W), 0.02, 0.0)]


class Weights:
    """A checkpoint's bfloat16 tensors, each made from (seed, its place in the list) when it is asked for."""

    def __init__(self, cfg, seed):
        self.where = {name: (i, shape, std, mean) for i, (name, shape, std, mean) in enumerate(tensor_list(cfg))}
        self.seed, self.generator = int(seed), torch.Generator(device="cuda")

    def __getitem__(self, name):
        i, shape, std, mean = self.where[name]
        self.generator.manual_seed((self.seed * 1000003 + i) & 0x7fffffffffffffff)
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(mean, std, generator=self.generator)

    def wide(self, name):
        return self[name].to(F64)


def vocab_of(case):
    cfg = MODELS[case["model"]]
    return cfg["vocab"] if "layers" in cfg else cfg["vocab_size"]


def prompts_of(case, seed):
    rng, V = random.Random(int(seed) * 7919 + 1), vocab_of(case)
    return [rng.choices(range(V), k=n) for n in lengths(case)]


def forced_of(case, seed):
    """The tokens that a decode case feeds: row i for step i of a sequence's life."""
    rng, V = random.Random(int(seed) * 7919 + 2), vocab_of(case)
    return [rng.choices(range(V), k=case["batch"]) for _ in range(WARM + GROWTH)]


class State:
    def __init__(self, case, seed):
        cfg = MODELS[case["model"]]
        self.case, self.prompts = case, prompts_of(case, seed)
        more = {"decode": WARM + GROWTH, "reply": case["steps"]}.get(case["kind"], 0)
        room = sum(-(-(len(p) + more) // 64) * 64 for p in self.prompts)
        weights = Weights(cfg, seed)
        self.engine = Engine.from_tensors(config_from_dict(cfg), {name: weights[name] for name in weights.where}, case["dtype"], max_tokens=room,
                                          max_context=min(room, max(8192, case["tokens"] + more)), max_slots=case["batch"], max_batch=case["batch"])
        p = SamplerParams(0.7, 0.95, 0, 1.0, 3) if case["sampled"] else SamplerParams.greedy()
        self.params, self.slots, self.at = [p] * case["batch"], [], 0
        if case["kind"] == "decode":
            self.forced = forced_of(case, seed)
            self.begin()
            for _ in range(WARM):
                self.next()

    def begin(self):
        for s in self.slots:
            self.engine.finish(s)
        self.slots, _ = self.engine.start(self.prompts, self.params, list(range(len(self.prompts))))
        self.at = 0

    def next(self):
        if self.at == len(self.forced):
            self.begin()
        self.engine.advance(self.slots, self.forced[self.at])
        self.at += 1
        return self.engine.last_logits


def prepare(case, seed):
    return State(case, seed)


def run(state):
    case, engine = state.case, state.engine
    if case["kind"] == "decode":
        return {"logits": state.next()}
    if case["kind"] == "reply":
        results = engine.generate(state.prompts, max_tokens=case["steps"], params=SamplerParams.greedy(), stop_tokens=())
        return {"tokens": torch.tensor([r.tokens for r in results]), "logits": engine.last_logits}
    slots = [engine.alloc_slot() for _ in state.prompts]
    try:
        if case["kind"] == "prompt":
            return {"logits": engine.step([StepEntry(s, p, places(case, len(p))) for s, p in zip(slots, state.prompts)])}
        done, found = [0] * len(slots), [None] * len(slots)
        while True:
            entries, last = [], []
            for i, p in enumerate(state.prompts):
                piece = p[done[i]:done[i] + case["chunk"]]
                if piece:
                    done[i] += len(piece)
                    if done[i] == len(p):
                        last.append(i)
                    entries.append(StepEntry(slots[i], piece, [len(piece) - 1] if done[i] == len(p) else []))
            if not entries:
                return {"logits": torch.cat(found)}
            logits = engine.step(entries)
            for row, i in enumerate(last):
                found[i] = logits[row:row + 1]
    finally:
        for s in slots:
            engine.free_slot(s)


# ---------------------------------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(spans, window=None):
    """(query, key) pairs of causal attention for tokens start .. stop - 1 of each sequence, at most ``window`` keys a query."""
    total = 0
    for start, stop in spans:
        full = stop if window is None else max(start, min(stop, window))       # queries below it see all keys before them
        total += (full * (full + 1) - start * (start + 1)) // 2 + (stop - full) * (window or 0)
    return total


def _qwen3_step(cfg, size, spans, rows):
    L, H, F, V, hd = (cfg[k] for k in ("num_hidden_layers", "hidden_size", "intermediate_size", "vocab_size", "head_dim"))
    Q, KV = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
    tokens, layer = sum(z - a for a, z in spans), H * (Q + 2 * KV) + Q * H + 3 * H * F
    cached = sum(z for _, z in spans) * 2 * KV * L                             # every key and value read or written once
    return {"bytes": (L * layer + H * V + tokens * H + cached) * size + 4 * rows * V,
            "flops": 2 * tokens * L * layer + 4 * Q * L * _pairs(spans) + 2 * rows * H * V}


def _tefezen_step(cfg, size, spans, rows):
    W, V, tokens = cfg["width"], cfg["vocab"], sum(z - a for a, z in spans)
    elements, flops, states = W * V + tokens * W, 2 * rows * W * V, 0
    for layer in cfg["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        E, top, F, S = f["router"]["experts"], f["router"]["top"], f["expert"]["ff"], f["shared"]["ff"]
        if layer["type"] == "latent_attention":
            r, rd, window = m["kv_rank"], m["rot_dim"], m["mask"]["size"]
            mats = W * H * (dk + rd) + (0 if "kv_from" in m else W * (r + rd)) + H * (dk + dv) * r + H * dv * W
            elements += (r + rd) * sum(z - max(0, a - window) for a, z in spans)
            flops += 2 * H * (dk + rd + dv) * _pairs(spans, window)
        else:
            mats = W * H * (2 * dk + 3 * dv)
            states += 2 * H * dk * dv * len(spans)                             # read and written
            flops += 4 * tokens * H * dk * dv
        mats += 3 * W * S + W * (E + 1) + 2 * W * cfg["token_side"]["dim"]
        hit = E * (1.0 - (1.0 - top / E) ** tokens)                            # experts that some token chose
        elements += mats + hit * 3 * W * F
        flops += 2 * tokens * (mats + top * 3 * W * F)
    return {"bytes": elements * size + 4 * states + 4 * rows * V, "flops": flops}


def work(case):
    cfg, n, B = MODELS[case["model"]], lengths(case), case["batch"]
    step, size = _tefezen_step if "layers" in cfg else _qwen3_step, 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "decode":
        steps = [([(k, k + 1) for k in n], B)]
    elif case["kind"] == "prompt":
        steps = [([(0, k) for k in n], sum(len(places(case, k)) for k in n))]
    elif case["kind"] == "reply":
        steps = [([(0, k) for k in n], B)] + [([(k + i, k + i + 1) for k in n], B) for i in range(case["steps"] - 1)]
    else:
        c = case["chunk"]
        steps = [([(a, min(a + c, k)) for k in n if a < k], sum(1 for k in n if a < k <= a + c)) for a in range(0, max(n), c)]
    total = [step(cfg, size, spans, rows) for spans, rows in steps]
    return {k: float(sum(t[k] for t in total)) for k in ("bytes", "flops")}


def tolerance(case):
    # Measured against 64 bits: 4e-6 in float32; 1e-2 (four layers) to 3.7e-2 (36 layers) in bfloat16, where two runs on the same inputs
    # are up to 1.5e-2 apart (partial sums of a decode product add up in no fixed order).
    if case["dtype"] == "float32":
        return {"rel": 1.6e-5, "max": 4e-4, "differ": 0.0}
    return {"rel": 0.03, "max": 0.5}


# ---------------------------------------------------------------------------------------------------------------- the same in 64 bits, plainly
def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window):
    """Causal attention of one sequence: q [T, heads, d], k [T, kv heads, d], v [T, kv heads, dv]; heads of a group are neighbours."""
    T, heads, group = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    out = torch.empty((T, heads, v.shape[2]), dtype=F64, device=q.device)
    place = torch.arange(T, device=q.device)
    for a in range(0, T, 1024):
        z = min(T, a + 1024)
        low = max(0, a - window + 1) if window else 0
        away = place[a:z, None] - place[None, low:z]
        hidden = (away < 0) | (away >= window) if window else away < 0
        for g in range(k.shape[1]):
            mine = slice(g * group, (g + 1) * group)
            s = torch.einsum("ihd,jd->hij", q[a:z, mine], k[low:z, g]) * scale
            out[a:z, mine] = torch.einsum("hij,jd->ihd", torch.softmax(s.masked_fill_(hidden, -math.inf), -1), v[low:z, g])
    return out.reshape(T, -1)


def _turn(x, place, base, adjacent):
    """Rotary positions over the last axis of x [T, heads, d]: halves paired, or neighbours."""
    d = x.shape[-1]
    angle = place.to(F64)[:, None, None] * torch.as_tensor(base, dtype=F64, device=x.device) ** (-2.0 * torch.arange(d // 2, dtype=F64, device=x.device) / d)
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = (x[..., 0::2], x[..., 1::2]) if adjacent else (x[..., :d // 2], x[..., d // 2:])
    turned = (a * c - b * s, b * c + a * s)
    return torch.stack(turned, -1).flatten(-2) if adjacent else torch.cat(turned, -1)


def _silu(z):
    return z * torch.sigmoid(z)


def _gated(x, w, p, names=("gate", "up", "down")):
    return (_silu(x @ w.wide(p + names[0]).t()) * (x @ w.wide(p + names[1]).t())) @ w.wide(p + names[2]).t()


def _qwen3_rows(cfg, w, tokens, bounds, place):
    H, KH, hd, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    x = w["model.embed_tokens.weight"][tokens].to(F64)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _unit(x, eps) * w.wide(p + "input_layernorm.weight")
        q, k, v = ((h @ w.wide(f"{p}self_attn.{n}_proj.weight").t()).view(len(tokens), -1, hd) for n in "qkv")
        q = _turn(_unit(q, eps) * w.wide(p + "self_attn.q_norm.weight"), place, cfg["rope_theta"], False)
        k = _turn(_unit(k, eps) * w.wide(p + "self_attn.k_norm.weight"), place, cfg["rope_theta"], False)
        o = torch.cat([_attend(q[a:z], k[a:z], v[a:z], hd ** -0.5, 0) for a, z in bounds])
        x = x + o @ w.wide(p + "self_attn.o_proj.weight").t()
        h = _unit(x, eps) * w.wide(p + "post_attention_layernorm.weight")
        x = x + _gated(h, w, p + "mlp.", ("gate_proj.weight", "up_proj.weight", "down_proj.weight"))
    head = w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
    return lambda rows: (_unit(x[rows], eps) * w.wide("model.norm.weight")) @ head.to(F64).t()


def _linear_attention(q, k, v, decay):
    """o_t = sum over s <= t of decay^(t - s) (q_t . k_s) v_s, a head at a time, blocks of tokens with the state between them."""
    T, heads, dk = q.shape
    out = torch.empty((T, heads, v.shape[2]), dtype=F64, device=q.device)
    i = torch.arange(256, dtype=F64, device=q.device)
    for h in range(heads):
        S, d = torch.zeros((dk, v.shape[2]), dtype=F64, device=q.device), torch.as_tensor(decay[h], dtype=F64, device=q.device)
        inside = torch.where(i[:, None] >= i[None, :], d ** (i[:, None] - i[None, :]).clamp_min(0), 0.0)
        for a in range(0, T, 256):
            Q, K, U = q[a:a + 256, h], k[a:a + 256, h], v[a:a + 256, h]
            n = Q.shape[0]
            out[a:a + n, h] = ((Q @ K.t()) * inside[:n, :n]) @ U + (d ** (i[:n, None] + 1)) * (Q @ S)
            S = d ** n * S + (K * d ** (n - 1 - i[:n, None])).t() @ U
    return out.reshape(T, -1)


def _tefezen_rows(cfg, w, tokens, bounds, place):
    eps, side, n = cfg["norm"]["eps"], cfg["token_side"]["dim"], len(tokens)
    x, kept = w["embed"][tokens].to(F64) * cfg["embedding"]["scale"], {}
    table = w["side.embed"][tokens].to(F64)
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        H, dk, dv, mix = m["heads"], m["dim"], m["vdim"], f"l{i}.mix."
        if layer["type"] == "latent_attention":
            r, rd, owner = m["kv_rank"], m["rot_dim"], m.get("kv_from", i)
            if owner == i:
                both = x @ w.wide(mix + "dkv").t()
                kept[i] = _unit(both[:, :r], eps) * w.wide(mix + "dkv.norm"), _turn(both[:, None, r:], place, m["rot"]["base"], True)
            c, shared = kept[owner]
            q = (x @ w.wide(mix + "q").t()).view(n, H, dk + rd)
            q = torch.cat([q[..., :dk], _turn(q[..., dk:], place, m["rot"]["base"], True)], -1)
            k = torch.cat([(c @ w.wide(mix + "uk").t()).view(n, H, dk), shared.expand(n, H, rd)], -1)
            v = (c @ w.wide(mix + "uv").t()).view(n, H, dv)
            y = torch.cat([_attend(q[a:z], k[a:z], v[a:z], m["scale"], m["mask"]["size"]) for a, z in bounds])
        else:
            q, k, v = (_silu(x @ w.wide(mix + t).t()).view(n, H, -1) for t in "qkv")
            y = torch.cat([_linear_attention(q[a:z], k[a:z], v[a:z], m["decay"]) for a, z in bounds])
            y = _unit(y, eps) * w.wide(mix + "norm") * torch.sigmoid(x @ w.wide(mix + "g").t())
        x = x + _unit(y @ w.wide(mix + "o").t(), eps) * (1.0 + w.wide(p + "norm1"))
        top = torch.topk(x @ w.wide(p + "mlp.router").t(), f["router"]["top"], -1)
        share = torch.softmax(top.values, -1)
        y = torch.sigmoid(x @ w.wide(p + "mlp.shared.sg").t()) * _gated(x, w, p + "mlp.shared.")
        for e in range(f["router"]["experts"]):
            row, col = torch.nonzero(top.indices == e, as_tuple=True)
            if len(row):
                y.index_add_(0, row, share[row, col, None] * _gated(x[row], w, f"{p}mlp.e{e}."))
        x = x + _unit(y, eps) * (1.0 + w.wide(p + "norm2"))
        z = x @ w.wide(p + "side.gate").t()
        z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3))) * table[:, i * side:(i + 1) * side]
        x = x + _unit(z @ w.wide(p + "side.proj").t(), eps) * w.wide(p + "side.norm")
    return lambda rows: (_unit(x[rows], eps) * (1.0 + w.wide("final.norm"))) @ w.wide("head").t()


def _logits(case, w, sequences, wanted):
    """Logits in 64 bits at the ``wanted`` places of each of the ``sequences``."""
    tokens = torch.tensor([t for s in sequences for t in s], device="cuda")
    ends = [0]
    for s in sequences:
        ends.append(ends[-1] + len(s))
    bounds = list(zip(ends, ends[1:]))
    place = torch.cat([torch.arange(len(s), device="cuda") for s in sequences])
    rows = torch.tensor([a + j for (a, _), js in zip(bounds, wanted) for j in js], device="cuda")
    cfg = MODELS[case["model"]]
    return (_tefezen_rows if "layers" in cfg else _qwen3_rows)(cfg, w, tokens, bounds, place)(rows)


@torch.no_grad()
def exact(case, seed):
    w, sequences = Weights(MODELS[case["model"]], seed), prompts_of(case, seed)
    if case["kind"] == "decode":
        forced = forced_of(case, seed)
        sequences = [p + [forced[i][b] for i in range(WARM + 1)] for b, p in enumerate(sequences)]
    elif case["kind"] == "reply":
        found = [[] for _ in sequences]
        for _ in range(case["steps"]):
            logits = _logits(case, w, sequences, [[len(s) - 1] for s in sequences])
            for i, t in enumerate(logits.argmax(-1).tolist()):
                found[i].append(t)
                sequences[i] = sequences[i] + [t]
        return {"tokens": torch.tensor(found), "logits": logits}
    return {"logits": _logits(case, w, sequences, [places(case, len(s)) if case["kind"] == "prompt" else [len(s) - 1] for s in sequences])}
