"""What is measured: the work that a program has this library do through its step function, from one sequence's next
token to a batch of long prompts.

A case names a model, a data type, a kind of step and the sequences that take part:

  prompt   new sequences with their whole prompts in one step (a request arrives, or a batch of them)
  turn     sequences that hold `shortest`..`longest` tokens go on by `new` tokens each (the next question of a chat)
  decode   `steps` single-token steps, one after another, of sequences that hold that many tokens

The sequences' lengths are spread evenly over the logarithm between `shortest` and `longest`.  Every pass returns the
logits that a sampler would read.  Turns and decode steps leave the sequences as long as they found them, so that a pass
can follow on a pass.

Models: Gemma-2 at its 2B layer sizes (26 layers, width 2,304), and two of the layer-by-layer designs at eight layers of
width 2,048: Nuvivik (latent attention with windows and sinks, grouped queries with a soft-cap, dense and routed
feed-forwards) and Vagonex (decay-rule and delta-rule matrix states, chunked attention, dense feed-forwards).  Weights
are random, scaled so that activations keep the size that trained ones have.
"""
from __future__ import annotations

import math
import random

import torch

from hos_b200.engine.runner import Runner
from hos_b200.registry import config_from_dict

VOCAB_ROWS = 512                # rows of the head that `exact` multiplies at a time
EXACT_TOKENS = 40_000           # above this many tokens a pass in 64 bits takes longer than is worth waiting for

# ---- models ---------------------------------------------------------------------------------------------------
GEMMA = dict(architectures=["Gemma2ForCausalLM"], model_type="gemma2", num_hidden_layers=26, hidden_size=2304,
             num_attention_heads=8, num_key_value_heads=4, head_dim=256, intermediate_size=9216, vocab_size=256000,
             rope_theta=10000.0, sliding_window=4096, max_position_embeddings=8192, query_pre_attn_scalar=256,
             attn_logit_softcapping=50.0, final_logit_softcapping=30.0, rms_norm_eps=1e-6, tie_word_embeddings=True)


def _nuvivik():
    dense = {"kind": "dense", "ff": 8192}
    moe = {"kind": "moe", "expert": {"ff": 2304}, "router": {"experts": 16, "top": 2, "groups": {"count": 4, "keep": 2}}}
    lat = {"type": "latent_attention",
           "mixer": {"heads": 16, "dim": 64, "rot_dim": 64, "vdim": 128, "q_rank": 768, "kv_rank": 512, "scale": 128 ** -0.5,
                     "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 64}}}
    att = {"type": "attention",
           "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                     "mask": {"size": 1024},
                     "rot": {"base": 500000.0, "dims": 64,
                             "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
    return {"architecture": "Nuvivik", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6},
            "embedding": {"scale": 2048 ** 0.5}, "logit_scale": 1.0, "logit_softcap": 30.0,
            "layers": [dict(lat, mlp=dense), dict(att, mlp=moe), dict(lat, mlp=dense), dict(lat, mlp=moe)] * 2}


def _vagonex():
    mlp = {"kind": "dense", "ff": 8192}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 2048},
                     "rot": {"base": 10000.0, "dims": 64,
                             "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    dec = {"type": "lightning", "mlp": mlp,
           "mixer": {"heads": 16, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 5 * i / 15) for i in range(16)]}}
    dlt = {"type": "delta", "mlp": mlp, "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    return {"architecture": "Vagonex", "vocab": 32000, "width": 2048, "postln_alpha": 2.0, "norm": {"eps": 1e-6},
            "embedding": {"scale": 2048 ** 0.5}, "layers": [dec, dlt, att, dlt] * 2}


def _raw(model):
    return {"gemma2-2b": lambda: GEMMA, "nuvivik": _nuvivik, "vagonex": _vagonex}[model]()


# ---- the cases ------------------------------------------------------------------------------------------------
def _case(model, kind, n, shortest, longest, new=0, steps=0, dtype="bfloat16", name=None):
    c = {"model": model, "dtype": dtype, "kind": kind, "n": n, "shortest": shortest, "longest": longest, "new": new,
         "steps": steps}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one person chatting: one sequence of some hundred tokens, its next tokens one by one
        _case("gemma2-2b", "decode", 1, 517, 517, steps=8, name="gemma-decode-1"),
        # eight long documents at the end of the context: the benchmark's headline step
        _case("gemma2-2b", "decode", 8, 8184, 8184, steps=8, name="gemma-decode-8-long"),
        # a busy service: 64 sequences of all lengths
        _case("gemma2-2b", "decode", 64, 64, 2036, steps=8, name="gemma-decode-64-ragged"),
        # a short question: latency until the first token
        _case("gemma2-2b", "prompt", 1, 97, 97, name="gemma-prompt-97"),
        # the benchmark's prompt
        _case("gemma2-2b", "prompt", 1, 2048, 2048, name="gemma-prompt-2048"),
        # a batch of requests of all lengths in one step
        _case("gemma2-2b", "prompt", 16, 64, 2048, name="gemma-prompts-16-ragged"),
        # the next turn of a chat, with a pasted page, on top of some thousand tokens
        _case("gemma2-2b", "turn", 1, 2901, 2901, new=739, name="gemma-turn-739"),
        # true 32-bit arithmetic: a trace that another implementation is compared with
        _case("gemma2-2b", "prompt", 1, 121, 121, dtype="float32", name="gemma-float32-prompt-121"),
        # the layer-by-layer designs: a long prompt, and a small batch's next tokens
        _case("nuvivik", "prompt", 1, 2048, 2048, name="nuvivik-prompt-2048"),
        _case("nuvivik", "decode", 8, 300, 1999, steps=8, name="nuvivik-decode-8"),
        _case("vagonex", "prompt", 1, 2048, 2048, name="vagonex-prompt-2048"),
        _case("vagonex", "decode", 24, 150, 1777, steps=8, name="vagonex-decode-24"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["gemma2-2b", "gemma2-2b", "gemma2-2b", "nuvivik", "vagonex"])
    gemma = model == "gemma2-2b"
    if gemma and rng.random() < 0.15:
        return _case(model, "prompt", 1, *(2 * [_log(rng, 2, 121)]), dtype="float32")
    kind = rng.choice(["prompt", "turn", "decode", "decode"])
    if kind == "prompt":
        n = _log(rng, 1, 16)
        longest = _log(rng, 16, min(4000, (8000 if gemma else 4096) // n))
        return _case(model, kind, n, max(1, int(longest * rng.uniform(0.05, 1.0))), longest)
    if kind == "turn":
        n = _log(rng, 1, 4)
        longest = _log(rng, 32, 5500)
        return _case(model, kind, n, max(1, int(longest * rng.uniform(0.2, 1.0))), longest, new=_log(rng, 2, 2000 // n))
    n = _log(rng, 1, 64)
    longest = _log(rng, 32, min(8184, 65000 // n))
    return _case(model, kind, n, max(1, int(longest * rng.uniform(0.05, 1.0))), longest, steps=8)


def _lengths(case):
    """The sequences' lengths: a prompt's own, or what a sequence holds before the step."""
    n, lo, hi = case["n"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    out = [int(round(lo * (hi / lo) ** (i / (n - 1)))) for i in range(n)]
    random.Random(n).shuffle(out)
    return out


# ---- inputs ---------------------------------------------------------------------------------------------------
def _weight_list(model):
    """(name, shape, mean, deviation) of every tensor of the checkpoint."""
    out = []

    def mat(name, rows, cols, gain=1.0):
        out.append((name, (rows, cols), 0.0, gain * cols ** -0.5))

    def vec(name, n, mean, std):
        out.append((name, (n,), mean, std))

    raw = _raw(model)
    if model == "gemma2-2b":
        d, hd, ff = raw["hidden_size"], raw["head_dim"], raw["intermediate_size"]
        q, kv = raw["num_attention_heads"] * hd, raw["num_key_value_heads"] * hd
        out.append(("model.embed_tokens.weight", (raw["vocab_size"], d), 0.0, 0.02))
        for i in range(raw["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for name, mean in (("input", 0.0), ("post_attention", -0.7), ("pre_feedforward", 0.0), ("post_feedforward", -0.7)):
                vec(p + name + "_layernorm.weight", d, mean, 0.1)
            mat(p + "self_attn.q_proj.weight", q, d, 1.5)
            mat(p + "self_attn.k_proj.weight", kv, d, 1.5)
            mat(p + "self_attn.v_proj.weight", kv, d)
            mat(p + "self_attn.o_proj.weight", d, q)
            mat(p + "mlp.gate_proj.weight", ff, d)
            mat(p + "mlp.up_proj.weight", ff, d)
            mat(p + "mlp.down_proj.weight", d, ff)
        vec("model.norm.weight", d, 0.0, 0.1)
        return out
    d, post = raw["width"], model == "vagonex"
    out.append(("embed", (raw["vocab"], d), 0.0, 0.02))
    for i, layer in enumerate(raw["layers"]):
        m, p, mlp = layer["mixer"], f"l{i}.mix.", layer["mlp"]
        kind, H = layer["type"], m["heads"]
        if kind == "latent_attention":
            mat(p + "dq", m["q_rank"], d)
            vec(p + "dq.norm", m["q_rank"], 1.0, 0.1)
            mat(p + "uq", H * (m["dim"] + m["rot_dim"]), m["q_rank"], 1.5)
            mat(p + "dkv", m["kv_rank"] + m["rot_dim"], d)
            vec(p + "dkv.norm", m["kv_rank"], 1.0, 0.1)
            mat(p + "uk", H * m["dim"], m["kv_rank"], 1.5)
            mat(p + "uv", H * m["vdim"], m["kv_rank"])
            vec(p + "sink", H, 0.0, 1.0)
        elif kind == "attention":
            G = m["kv_heads"]
            for name, rows in (("q", H * m["dim"]), ("k", G * m["dim"]), ("v", G * m["vdim"])):
                mat(p + name, rows, d, 1.5 if name != "v" else 1.0)
                vec(p + name + ".b", rows, 0.0, 0.1)
            if post:
                vec(p + "q.norm", m["dim"], 1.0, 0.1)
                vec(p + "k.norm", m["dim"], 1.0, 0.1)
                vec(p + "sink", H, 0.0, 1.0)
                mat(p + "g", H, d)
        else:
            keys = (m["kv_heads"] if kind == "delta" else H) * m["dim"]
            for name, rows in (("q", keys), ("k", keys), ("v", H * m["vdim"])):
                mat(p + name, rows, d)
                if kind == "delta":
                    mat(p + name + ".conv", rows, m["conv"])
            mat(p + "g", H * m["vdim"], d)
            if kind == "delta":
                mat(p + "a", H, d)
                mat(p + "b", H, d)
                vec(p + "A_log", H, 0.0, 0.5)
                vec(p + "dt_bias", H, -3.0, 1.0)
            vec(p + "norm", m["vdim"] if kind == "delta" else H * m["vdim"], 1.0, 0.1)
        mat(p + "o", d, H * m["vdim"])
        q = f"l{i}.mlp."
        if mlp["kind"] == "dense":
            if post:
                mat(q + "gate", mlp["ff"], d)
            mat(q + "up", mlp["ff"], d)
            mat(q + "down", d, mlp["ff"])
        else:
            mat(q + "router", mlp["router"]["experts"], d, 0.1)
            for e in range(mlp["router"]["experts"]):
                mat(f"{q}e{e}.up", mlp["expert"]["ff"], d)
                mat(f"{q}e{e}.down", d, mlp["expert"]["ff"])
        for norm in ("norm1", "norm2"):
            vec(f"l{i}.{norm}", d, 1.0 if post else 0.3, 0.1 if post else 0.03)
    vec("final.norm", d, 1.0, 0.1)
    if not post:
        out.append(("head", (raw["vocab"], d), 0.0, 0.02))
    return out


class _Weights:
    """A checkpoint of random numbers, made on the GPU as it is read: the same ones for the same seed and name."""

    def __init__(self, model, seed, dtype=torch.bfloat16):
        self.model, self.seed, self.dtype = model, seed, dtype
        self.at = {name: (i, shape, mean, std) for i, (name, shape, mean, std) in enumerate(_weight_list(model))}

    def names(self):
        return list(self.at)

    def info(self, name):
        return self.dtype, self.at[name][1]

    def _normal(self, name):
        i, shape, mean, std = self.at[name]
        g = torch.Generator(device="cuda").manual_seed(self.seed * 4099 + i)
        return torch.empty(shape, dtype=self.dtype, device="cuda").normal_(mean, std, generator=g)

    def read(self, name):
        t = self._normal(name)
        if self.model == "nuvivik" and name == "embed":
            # A trained router knows its tokens: every token leans to two experts of each routed layer, so that which
            # experts it uses does not hang on the last bit of a sum.
            g = torch.Generator(device="cuda").manual_seed(self.seed * 4099 + 4098)
            for other in (x for x in self.at if x.endswith("router")):
                rows = self._normal(other).float()
                pick = torch.rand((t.shape[0], rows.shape[0]), generator=g, device="cuda").topk(2).indices
                t += (0.2 * (14.0 * rows[pick[:, 0]] + 11.0 * rows[pick[:, 1]])).to(t.dtype)
        return t

    def close(self):
        pass


def _tokens(case, seed):
    """For every sequence the tokens that it holds, or that its prompt is, and the ones that the step brings after them."""
    vocab = GEMMA["vocab_size"] if case["model"] == "gemma2-2b" else 32000
    rng = random.Random(seed * 7919 + 13)
    more = {"prompt": 0, "turn": case["new"], "decode": case["steps"]}[case["kind"]]
    return [([rng.randrange(vocab) for _ in range(n)], [rng.randrange(vocab) for _ in range(more)]) for n in _lengths(case)]


def prepare(case, seed):
    config = config_from_dict(_raw(case["model"]))
    seqs = _tokens(case, seed)
    room = sum((len(a) + len(b) + 63) // 64 * 64 for a, b in seqs)
    kept = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    runner = Runner(config, _Weights(case["model"], seed, kept), dtype=case["dtype"], max_tokens=room, max_seq_len=8192)
    state = {"kind": case["kind"], "runner": runner, "held": [len(a) for a, _ in seqs]}
    if case["kind"] == "prompt":
        return dict(state, prompts=[a for a, _ in seqs])
    slots = runner.admit(len(seqs))
    at = 0
    while at < len(seqs):                      # the sequences' first tokens, some thousand at a time
        end, total = at, 0
        while end < len(seqs) and (end == at or total + len(seqs[end][0]) <= 8192):
            total += len(seqs[end][0])
            end += 1
        runner.step(slots[at:end], [a for a, _ in seqs[at:end]])
        at = end
    return dict(state, slots=slots, new=[b for _, b in seqs])


def run(state):
    runner, kind = state["runner"], state["kind"]
    if kind == "prompt":
        slots = runner.admit(len(state["prompts"]))
        logits = runner.step(slots, state["prompts"])
        for s in slots:
            runner.release(s)
        return logits
    slots, new = state["slots"], state["new"]
    if kind == "turn":
        out = runner.step(slots, new)
    else:
        out = [runner.step(slots, [[t[i]] for t in new]) for i in range(len(new[0]))]
    runner.write_records(slots, pos=state["held"])
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------------
def _pairs(start, new, window):
    """Keys that `new` tokens after `start` others see together, within a window."""
    if not window:
        return new * start + new * (new + 1) // 2
    full = max(0, min(new, start + new - window))              # the last tokens, which see a whole window
    part = new - full
    return part * start + part * (part + 1) // 2 + full * window


def work(case):
    raw, wide = _raw(case["model"]), 4 if case["dtype"] == "float32" else 2
    gemma = case["model"] == "gemma2-2b"
    d = raw["hidden_size"] if gemma else raw["width"]
    lengths, n = _lengths(case), case["n"]
    if case["kind"] == "prompt":
        passes = [[(0, x) for x in lengths]]
    elif case["kind"] == "turn":
        passes = [[(x, case["new"]) for x in lengths]]
    else:
        passes = [[(x + i, 1) for x in lengths] for i in range(case["steps"])]
    sizes = {name: math.prod(shape) for name, shape, _, _ in _weight_list(case["model"])}
    head = raw["vocab_size"] * d if gemma else raw["vocab"] * d
    dense = sum(s for name, s in sizes.items() if "embed" not in name and name != "head" and ".mlp.e" not in name)
    total = flops = 0.0
    for steps in passes:
        tokens = sum(k for _, k in steps)
        total += (dense + head + tokens * d) * wide + n * head // d * 4
        flops += 2.0 * tokens * dense + 2.0 * n * head

        def attend(query, key, value, kv, window):
            """Numbers per query and key, per key and value row of a position, of one layer."""
            nonlocal total, flops
            for start, new in steps:
                seen = min(start + new, window + new - 1) if window else start + new
                total += seen * kv * wide + (new * kv * wide if start else 0)
                flops += 2.0 * _pairs(start, new, window) * query * (key + value)

        if gemma:
            hd, kv = raw["head_dim"], raw["num_key_value_heads"]
            for i in range(raw["num_hidden_layers"]):
                attend(raw["num_attention_heads"], hd, hd, 2 * kv * hd, raw["sliding_window"] if i % 2 == 0 else 0)
            continue
        for layer in raw["layers"]:
            m, mlp = layer["mixer"], layer["mlp"]
            if layer["type"] == "latent_attention":
                # the expanded form's arithmetic; the cache holds one latent row per position
                attend(m["heads"], m["dim"] + m["rot_dim"], m["vdim"], m["kv_rank"] + m["rot_dim"], m["mask"]["size"])
            elif layer["type"] == "attention":
                kv = m["kv_heads"] * (m["dim"] + m["vdim"])
                attend(m["heads"], m["dim"], m["vdim"], kv, m["mask"]["size"])
            else:
                cells = m["heads"] * m["dim"] * m["vdim"]
                total += n * cells * 4 * 2
                flops += tokens * cells * (4.0 if layer["type"] == "lightning" else 6.0)
            if mlp["kind"] == "moe":
                one = 2 * mlp["expert"]["ff"] * d
                top = mlp["router"]["top"]
                total += min(mlp["router"]["experts"], tokens * top) * one * wide
                flops += 2.0 * tokens * top * one
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """The logits stand this far from the same weights and tokens in 64 bits, measured: 9e-6 in 32-bit arithmetic (the
    angles of the rotary positions are 32-bit too), 0.017 for 26 layers and 0.006 for eight in bfloat16.  Two correct
    implementations differ by up to the sum of theirs."""
    if case["dtype"] == "float32":
        return {"rel": 3e-5}
    return {"rel": 0.03 if case["model"] == "gemma2-2b" else 0.02}


# ---- the same in 64 bits --------------------------------------------------------------------------------------
F = torch.float64


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _cap(x, c):
    return c * torch.tanh(x / c) if c else x


def _turned(x, pos, freqs, factor=1.0, pairs=False):
    """Rotary positions on the first 2 x len(freqs) numbers of x [T, heads, n]; pairs (i, i + half), or neighbours."""
    a = pos.to(F)[:, None] * torch.tensor(freqs, dtype=F, device=x.device)
    c, s = (a.cos() * factor)[:, None], (a.sin() * factor)[:, None]
    half = len(freqs)
    left, right = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if pairs else (slice(0, half), slice(half, 2 * half))
    u, v, out = x[..., left], x[..., right], x.clone()
    out[..., left], out[..., right] = u * c - v * s, v * c + u * s
    return out


def _freqs(rot):
    base, dims, sc = rot["base"], rot["dims"], rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if sc and "low" in sc:                     # by bands of wavelengths
        out = []
        for x in f:
            turns = sc["original"] * x / (2.0 * math.pi)
            s = min(1.0, max(0.0, (turns - sc["low"]) / (sc["high"] - sc["low"])))
            out.append(x * s + x / sc["factor"] * (1.0 - s))
        return out, 1.0
    if sc:                                     # by a ramp over the pairs
        def at(turns):
            return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = [min(1.0, max(0.0, (i - lo) / max(hi - lo, 0.001))) for i in range(len(f))]
        return [x / sc["factor"] * r + x * (1.0 - r) for x, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1.0
    return f, 1.0


def _attend(q, k, v, scale, cap=0.0, window=0, chunk=0, sink=None):
    """q [T, H, n], k and v [T, G, ...]: causal attention of one sequence."""
    T, H, group = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F, device=q.device)
    for lo in range(0, T, 1024):
        hi = min(T, lo + 1024)
        first = max(0, lo + 1 - window) if window else lo // chunk * chunk if chunk else 0
        i, j = torch.arange(lo, hi, device=q.device)[:, None], torch.arange(first, hi, device=q.device)[None]
        hidden = j > i
        if window:
            hidden |= i - j >= window
        if chunk:
            hidden |= j < i // chunk * chunk
        for h in range(H):
            s = _cap(q[lo:hi, h] @ k[first:hi, h // group].T * scale, cap).masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(hi - lo, 1)], 1)
            p = s.softmax(1)
            out[lo:hi, h] = p[:, : hi - first] @ v[first:hi, h // group]
    return out


class _Exact:
    """The forward pass of whole sequences, side by side as rows, in 64 bits."""

    def __init__(self, case, seed):
        self.raw = _raw(case["model"])
        self.source = _Weights(case["model"], seed, torch.float32 if case["dtype"] == "float32" else torch.bfloat16)

    def w(self, name):
        return self.source.read(name).to(F)

    def product(self, x, name):
        return x @ self.w(name).T

    def each(self, fn, *rows):
        """`fn` of every sequence's rows and positions."""
        return torch.cat([fn(pos, *(r[lo:hi] for r in rows)) for (lo, hi), pos in zip(self.spans, self.pos)])

    def padded(self, x):
        out = torch.zeros((len(self.spans), self.longest) + x.shape[1:], dtype=F, device=x.device)
        for i, (lo, hi) in enumerate(self.spans):
            out[i, : hi - lo] = x[lo:hi]
        return out

    def logits(self, seqs, rows):
        """`rows[i]`: the places of sequence i whose logits are wanted; [sequences x places, vocab]."""
        at = 0
        self.spans = []
        for s in seqs:
            self.spans.append((at, at + len(s)))
            at += len(s)
        self.pos = [torch.arange(len(s), device="cuda") for s in seqs]
        self.longest = max(len(s) for s in seqs)
        picked = torch.tensor([lo + j for (lo, _), r in zip(self.spans, rows) for j in r], device="cuda")
        tokens = torch.tensor([t for s in seqs for t in s], device="cuda")
        gemma = "hidden_size" in self.raw
        h, head = (self.gemma if gemma else self.layered)(tokens, picked)
        table = self.source.read(head)
        out = torch.cat([h @ table[i:i + VOCAB_ROWS].to(F).T for i in range(0, table.shape[0], VOCAB_ROWS)], 1)
        return _cap(out, self.raw["final_logit_softcapping"] if gemma else self.raw.get("logit_softcap", 0.0))

    def gemma(self, tokens, picked):
        z = self.raw
        eps, hd = z["rms_norm_eps"], z["head_dim"]
        freqs = [z["rope_theta"] ** (-2.0 * i / hd) for i in range(hd // 2)]

        def norm(x, name):
            return _rms(x, eps) * (1.0 + self.w(name))

        x = self.source.read("model.embed_tokens.weight")[tokens].to(F) * z["hidden_size"] ** 0.5
        for i in range(z["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = norm(x, p + "input_layernorm.weight")
            q, k, v = (self.product(h, f"{p}self_attn.{n}_proj.weight").view(len(h), -1, hd) for n in "qkv")
            a = self.each(lambda pos, q, k, v: _attend(_turned(q, pos, freqs), _turned(k, pos, freqs), v,
                                                       z["query_pre_attn_scalar"] ** -0.5, z["attn_logit_softcapping"],
                                                       z["sliding_window"] if i % 2 == 0 else 0), q, k, v)
            a = self.product(a.flatten(1), p + "self_attn.o_proj.weight")
            x = x + norm(a, p + "post_attention_layernorm.weight")
            h = norm(x, p + "pre_feedforward_layernorm.weight")
            f = _gelu(self.product(h, p + "mlp.gate_proj.weight")) * self.product(h, p + "mlp.up_proj.weight")
            x = x + norm(self.product(f, p + "mlp.down_proj.weight"), p + "post_feedforward_layernorm.weight")
        return norm(x[picked], "model.norm.weight"), "model.embed_tokens.weight"

    def layered(self, tokens, picked):
        z = self.raw
        self.eps, post = z["norm"]["eps"], "postln_alpha" in z
        x = self.source.read("embed")[tokens].to(F) * z["embedding"]["scale"]
        for i, layer in enumerate(z["layers"]):
            for part, norm in (("mix", "norm1"), ("mlp", "norm2")):
                m = layer["mixer"] if part == "mix" else layer["mlp"]
                kind = layer["type"] if part == "mix" else m["kind"]
                y = getattr(self, kind)(m, f"l{i}.{part}.", x)
                w = self.w(f"l{i}.{norm}")
                x = _rms(z["postln_alpha"] * x + y, self.eps) * w if post else x + _rms(y, self.eps) * w
        return _rms(x[picked], self.eps) * self.w("final.norm"), "embed" if post else "head"

    def latent_attention(self, m, p, x):
        H, d, r, rank, n = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], len(x)
        freqs, _ = _freqs(m["rot"])
        q = self.product(_rms(self.product(x, p + "dq"), self.eps) * self.w(p + "dq.norm"), p + "uq").view(n, H, d + r)
        down = self.product(x, p + "dkv")
        c = _rms(down[:, :rank], self.eps) * self.w(p + "dkv.norm")
        k, v = self.product(c, p + "uk").view(n, H, d), self.product(c, p + "uv").view(n, H, m["vdim"])
        sink = self.w(p + "sink")

        def one(pos, q, k, v, kr):
            q = torch.cat([q[..., :d], _turned(q[..., d:], pos, freqs)], -1)
            k = torch.cat([k, _turned(kr[:, None], pos, freqs).expand(-1, H, -1)], -1)
            return _attend(q, k, v, m["scale"], window=m["mask"]["size"], sink=sink)
        return self.product(self.each(one, q, k, v, down[:, rank:]).flatten(1), p + "o")

    def attention(self, m, p, x):
        n, post = len(x), "postln_alpha" in self.raw
        freqs, factor = _freqs(m["rot"])
        q, k, v = (self.product(x, p + a) + self.w(p + a + ".b") for a in "qkv")
        q, k = q.view(n, -1, m["dim"]), k.view(n, -1, m["dim"])
        if post:                               # norms with weights before the rotation, a chunk, a sink, a gate
            q, k = _rms(q, self.eps) * self.w(p + "q.norm"), _rms(k, self.eps) * self.w(p + "k.norm")
            sink = self.w(p + "sink")

            def one(pos, q, k, v):
                q, k = (_turned(a, pos, freqs, factor, pairs=True) for a in (q, k))
                return _attend(q, k, v, m["scale"], chunk=m["mask"]["size"], sink=sink)
        else:                                  # norms without weights after it, a window, a soft-cap

            def one(pos, q, k, v):
                q, k = (_rms(_turned(a, pos, freqs), self.eps) for a in (q, k))
                return _attend(q, k, v, m["scale"], m["softcap"], m["mask"]["size"])
        a = self.each(one, q, k, v.view(n, -1, m["vdim"]))
        if post:
            a = a * torch.sigmoid(self.product(x, p + "g"))[..., None]
        return self.product(a.flatten(1), p + "o")

    def scan(self, q, k, v, decay, beta=None):
        """S <- decay S + k u^T with u = v, or beta (v - (decay S)^T k); the read-outs S^T q.  Rows [n, H, ...]."""
        q, k, v, decay = (self.padded(a) for a in (q, k, v, decay))
        beta = self.padded(beta) if beta is not None else None
        S = torch.zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3], dtype=F, device=q.device)
        out = torch.empty_like(v)
        for t in range(q.shape[1]):
            S *= decay[:, t, :, None, None]
            u = v[:, t]
            if beta is not None:
                u = beta[:, t, :, None] * (u - (k[:, t, :, None] @ S)[:, :, 0])
            S += k[:, t, :, :, None] * u[:, :, None]
            out[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        return torch.cat([out[i, : hi - lo] for i, (lo, hi) in enumerate(self.spans)])

    def lightning(self, m, p, x):
        n, H = len(x), m["heads"]
        q, k, v = (_silu(self.product(x, p + a)).view(n, H, -1) for a in "qkv")
        o = self.scan(q, k, v, torch.tensor(m["decay"], dtype=F, device=x.device).expand(n, H))
        y = _rms(o.flatten(1), self.eps) * self.w(p + "norm") * torch.sigmoid(self.product(x, p + "g"))
        return self.product(y, p + "o")

    def delta(self, m, p, x):
        n, H, G = len(x), m["heads"], m["kv_heads"]

        def conv(a):
            taps = self.w(p + a + ".conv")

            def one(pos, y):
                z = torch.cat([y.new_zeros(taps.shape[1] - 1, y.shape[1]), y])
                return sum(taps[:, j] * z[j:j + len(y)] for j in range(taps.shape[1]))
            return _silu(self.each(one, self.product(x, p + a)))

        q, k, v = conv("q").view(n, G, -1), conv("k").view(n, G, -1), conv("v").view(n, H, -1)
        q, k = (a * torch.rsqrt((a * a).sum(-1, keepdim=True) + 1e-6) for a in (q, k))
        q, k = (a.repeat_interleave(H // G, 1) for a in (q * m["dim"] ** -0.5, k))
        dt = torch.nn.functional.softplus(self.product(x, p + "a") + self.w(p + "dt_bias"))
        o = self.scan(q, k, v, torch.exp(-torch.exp(self.w(p + "A_log")) * dt), torch.sigmoid(self.product(x, p + "b")))
        y = _rms(o, self.eps) * self.w(p + "norm") * _silu(self.product(x, p + "g")).view(n, H, -1)
        return self.product(y.flatten(1), p + "o")

    def dense(self, m, p, x):
        if "postln_alpha" in self.raw:
            return self.product(_gelu(self.product(x, p + "gate")) * self.product(x, p + "up"), p + "down")
        return self.product(_gelu(self.product(x, p + "up")), p + "down")

    def moe(self, m, p, x):
        r = m["router"]
        s = torch.sigmoid(self.product(x, p + "router"))
        count, keep = r["groups"]["count"], r["groups"]["keep"]
        by_group = s.view(len(x), count, -1)
        best = by_group.topk(2, -1).values.sum(-1).topk(keep, -1).indices
        closed = torch.ones(len(x), count, dtype=torch.bool, device=x.device).scatter_(1, best, False)
        value, chosen = by_group.masked_fill(closed[..., None], -1.0).flatten(1).topk(r["top"], -1)
        out = torch.zeros_like(x)
        for e in range(r["experts"]):
            rows, place = (chosen == e).nonzero(as_tuple=True)
            y = self.product(torch.relu(self.product(x[rows], f"{p}e{e}.up")) ** 2, f"{p}e{e}.down")
            out.index_add_(0, rows, y * value[rows, place][:, None])
        return out


def exact(case, seed):
    seqs = _tokens(case, seed)
    if sum(len(a) + len(b) for a, b in seqs) > EXACT_TOKENS:
        return None
    held, model = [len(a) for a, _ in seqs], _Exact(case, seed)
    places = [[n + i for i in range(case["steps"])] if case["kind"] == "decode" else [len(a) + len(b) - 1]
              for n, (a, b) in zip(held, seqs)]
    out = model.logits([a + b for a, b in seqs], places)
    if case["kind"] != "decode":
        return out
    out = out.view(case["n"], case["steps"], -1)
    return [out[:, i].contiguous() for i in range(case["steps"])]
