"""Cases that stand for what programs have this library do: its layers alone, through the parts' public interface
(``make_part``, ``bind``, ``forward`` on a ``StepContext``), and whole requests through ``CausalLM.step``.

A case is a dict of plain values with a ``kind``:

* ``requests``   a batch of prompts of unequal lengths and then single tokens, on a Falcon-shaped model: what ``generate``
                 does, with the tokens given. Results: the logits after the prompts and after every token.
* ``memory``     the same on a Pogezen model (matrix memories, attentions with mixed heads, short filters, float32 stream):
                 many small kernels a step.
* ``attention``  one windowed or full attention layer with what the designs put around the softmax, on prompts.
* ``latent``     one latent-attention layer on prompts.
* ``experts``    one routed mixture of experts, from a decoding step's few tokens to a long prompt's thousands.
* ``delta``, ``gla``, ``mlstm``, ``rglru``   one recurrent layer each on prompts.
* ``block``      one sequential block (norms, attention, dense feed-forward) of a float32 model.

Widths, head counts and expert sizes are those that the benchmark of this repository runs (its sizes "s" and "m") and
Falcon's; prompts have odd lengths as prompts do.
"""
from __future__ import annotations

import math

import torch

import pytorch_transformers_b200 as ptb
from pytorch_transformers_b200 import kernels as K
from pytorch_transformers_b200.engine.batch import StepContext
from pytorch_transformers_b200.parts.base import make_part, resolve

DEV = "cuda"
F64 = torch.float64
EPS = 1e-6
FALCON_EPS = 1e-5


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # Falcon-7B's layers (two of them: all layers are alike) serving eight requests: prompts of a page or two of text,
        # then decoding in replayed graphs, where the step reads all weights for eight tokens
        dict(name="falcon requests", kind="requests", dtype="bfloat16", hidden=4544, heads=71, kv_heads=1, head_dim=64,
             ffn=18176, layers=2, vocab=65024, batch=8, prompt=1024, steps=40),
        # a small batch on a small model of many small kernels: latency and launches are what a step costs
        dict(name="memory requests", kind="memory", dtype="bfloat16", width=2048, heads=16, kv_heads=4, ffn=8192, window=1024,
             keep=4, vocab=32000, batch=4, prompt=200, steps=40),
        # a windowed attention that keeps the first tokens, rotates half a head and adds one to the denominator: one long prompt
        dict(name="window attention", kind="attention", dtype="bfloat16", hidden=2048, heads=16, kv_heads=4, dim=128,
             window=1024, keep=4, cap=0.0, sink="one", gate="none", norm=True, rot=64, temp=False, tokens=2048, seqs=1),
        # a full attention with capped scores, a query temperature and a gate per entry: a few prompts at once, ragged
        dict(name="capped attention", kind="attention", dtype="bfloat16", hidden=2048, heads=16, kv_heads=4, dim=128,
             window=0, keep=0, cap=30.0, sink="none", gate="entry", norm=False, rot=0, temp=True, tokens=3001, seqs=3),
        # keys and values through a low-rank latent, unfolded for a prompt
        dict(name="latent attention", kind="latent", dtype="bfloat16", hidden=2048, heads=16, dim=96, rot=32, vdim=128,
             rank=512, q_rank=0, gate="head", wide=True, tokens=2048, seqs=1),
        # 64 experts of which a token uses 6: a prompt, and a decoding step of eight sequences, which reads most experts
        dict(name="experts prompt", kind="experts", dtype="bfloat16", hidden=2048, inner=1408, experts=64, top=6, groups=8,
             keep=4, expert="gated_silu", tokens=2048),
        dict(name="experts step", kind="experts", dtype="bfloat16", hidden=2048, inner=1408, experts=64, top=6, groups=8,
             keep=4, expert="gated_silu", tokens=8),
        # the recurrent layers on prompts: states of 128 x 128 a head, in chunks
        dict(name="delta rule", kind="delta", dtype="bfloat16", hidden=2048, heads=16, kv_heads=16, dim=128, taps=4, rank=64,
             decay="channel", tokens=2048, seqs=1),
        dict(name="gated linear", kind="gla", dtype="bfloat16", hidden=2048, heads=16, dim=128, rank=64, tau=16.0, tokens=2900,
             seqs=2),
        dict(name="matrix memory", kind="mlstm", dtype="bfloat16", hidden=2048, heads=16, dim=128, cap=15.0, tokens=2048, seqs=1),
        dict(name="gated recurrence", kind="rglru", dtype="bfloat16", hidden=2048, width=2560, blocks=16, taps=4, tokens=2048,
             seqs=1),
        # a checkpoint run in true 32 bits
        dict(name="float32 block", kind="block", dtype="float32", hidden=1024, heads=16, head_dim=64, ffn=4096, tokens=700,
             seqs=2),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["requests", "memory", "attention", "attention", "latent", "experts", "experts", "delta", "gla", "mlstm",
                       "rglru", "block"])
    tokens, seqs = _log(rng, 130, 3500), rng.choice([1, 1, 2, 3, 5])
    c = dict(kind=kind, dtype="bfloat16")
    heads, dim = rng.choice([8, 12, 16, 32]), rng.choice([64, 128, 128])
    kv = rng.choice([g for g in (1, 2, 4, 8) if heads % g == 0])
    hidden = rng.choice([1024, 1536, 2048, 4096])
    if kind == "requests":
        heads = rng.choice([16, 32, 48, 71])
        c.update(hidden=64 * heads, heads=heads, kv_heads=1, head_dim=64, ffn=256 * heads, layers=rng.choice([1, 2]),
                 vocab=rng.choice([32000, 65024]), batch=_log(rng, 1, 12), prompt=_log(rng, 20, 900), steps=rng.choice([16, 24, 40]))
        return c
    if kind == "memory":
        heads = rng.choice([8, 16])
        c.update(width=128 * heads, heads=heads, kv_heads=4, ffn=512 * heads, window=rng.choice([64, 500, 1024]), keep=rng.choice([0, 4]),
                 vocab=32000, batch=_log(rng, 1, 8), prompt=_log(rng, 20, 400), steps=rng.choice([16, 24, 40]))
        return c
    if kind == "attention":
        c.update(hidden=hidden, heads=heads, kv_heads=kv, dim=dim, tokens=tokens, seqs=seqs)
        if rng.random() < 0.5:
            keep = rng.choice([0, 4, 70])
            c.update(window=rng.choice([100, 512, 1024, 2000]), keep=keep, cap=rng.choice([0.0, 30.0]), sink=rng.choice(["one", "learned"]),
                     gate="none", norm=True, rot=dim // 2, temp=False)
        else:
            c.update(window=0, keep=0, cap=rng.choice([0.0, 30.0]), sink="none", gate=rng.choice(["entry", "head"]), norm=False,
                     rot=0, temp=rng.choice([True, False]))
        return c
    if kind == "latent":
        c.update(hidden=hidden, heads=heads, dim=rng.choice([96, 128]), rot=rng.choice([32, 64]), vdim=128, rank=512,
                 q_rank=rng.choice([0, 768]), gate=rng.choice(["head", "entry"]), wide=rng.choice([True, False]), tokens=tokens, seqs=seqs)
        if c["dim"] + c["rot"] not in (128, 192):
            c["rot"] = 128 - c["dim"] if c["dim"] == 96 else 64
        return c
    if kind == "experts":
        c.update(hidden=rng.choice([1024, 2048]), inner=rng.choice([704, 1000, 1408]), experts=rng.choice([16, 64]), top=rng.choice([2, 6]),
                 groups=rng.choice([1, 8]), expert=rng.choice(["gated_silu", "clamped_glu", "plain"]), tokens=_log(rng, 1, 3500))
        c["keep"] = 1 if c["groups"] == 1 else 4
        return c
    if kind == "block":
        heads = rng.choice([8, 16, 24])
        c.update(dtype="float32", hidden=64 * heads, heads=heads, head_dim=64, ffn=256 * heads, tokens=_log(rng, 20, 900), seqs=seqs)
        return c
    heads, dim = rng.choice([8, 16]), rng.choice([64, 128])
    tokens = max(tokens, 260 * seqs)
    c.update(hidden=rng.choice([1024, 2048]), heads=heads, dim=dim, tokens=tokens, seqs=seqs)
    if kind == "delta":
        c.update(kv_heads=heads // rng.choice([1, 2]), taps=4, rank=64, decay=rng.choice(["channel", "head"]))
    elif kind == "gla":
        c.update(rank=64, tau=16.0)
    elif kind == "mlstm":
        c.update(cap=15.0)
    else:
        c = dict(kind=kind, dtype="bfloat16", hidden=c["hidden"], width=rng.choice([1280, 2560, 3840]), blocks=rng.choice([10, 16]), taps=4,
                 tokens=tokens, seqs=seqs)
        c["width"] = c["width"] // c["blocks"] * c["blocks"]
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _lengths(tokens, seqs):
    """Unequal lengths that sum to ``tokens``: sequence i has about (i + 1) shares."""
    shares = seqs * (seqs + 1) // 2
    out = [max(1, tokens * (i + 1) // shares) for i in range(seqs)]
    out[-1] = tokens - sum(out[:-1])
    return out


def _prompt_lengths(c):
    """A batch of prompts around the case's length, each another."""
    return [max(2, c["prompt"] - 37 * i % max(1, c["prompt"] // 2)) for i in range(c["batch"])]


class _Draws:
    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed * 7919 + 11)

    def normal(self, shape, std, mean=0.0, dtype=torch.float32):
        t = torch.empty(shape, dtype=dtype, device=DEV)
        return t.normal_(mean, std, generator=self.gen)

    def ids(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.gen, device=DEV).tolist()


def _dtype(c):
    return getattr(torch, c["dtype"])


def _layer_tensors(c, seed):
    """({logical name: tensor}, x): a layer's weights as a checkpoint would hold them, and its normed input rows."""
    d, dt, kind, h = _Draws(seed), _dtype(c), c["kind"], c["hidden"]
    w = {}

    def mat(name, *shape, std=None):
        w[name] = d.normal(shape, std or shape[-1] ** -0.5, dtype=dt)

    def vec(name, *shape, std=0.02, mean=0.0):
        w[name] = d.normal(shape, std, mean)

    if kind == "attention":
        H, G, dim = c["heads"], c["kv_heads"], c["dim"]
        mat("q", H * dim, h), mat("k", G * dim, h), mat("v", G * dim, h), mat("o", h, H * dim)
        if c["norm"]:
            vec("q_norm", dim, std=0.1, mean=1.0), vec("k_norm", dim, std=0.1, mean=1.0)
        if c["sink"] == "learned":
            vec("sink", H, std=1.0)
        if c["gate"] != "none":
            mat("g", H * dim if c["gate"] == "entry" else H, h)
    elif kind == "latent":
        H, qd = c["heads"], c["dim"] + c["rot"]
        if c["q_rank"]:
            mat("dq", c["q_rank"], h), vec("dq_norm", c["q_rank"], mean=1.0), mat("uq", H * qd, c["q_rank"])
        else:
            mat("q", H * qd, h)
        mat("uk", H * c["dim"], c["rank"]), mat("uv", H * c["vdim"], c["rank"])
        mat("g", H if c["gate"] == "head" else H * c["vdim"], h), mat("o", h, H * c["vdim"])
        mat("dkv", c["rank"] + c["rot"], h), vec("dkv_norm", c["rank"], mean=1.0)
    elif kind == "experts":
        vec("router", c["experts"], h), vec("correction", c["experts"], std=0.01)
        for e in range(c["experts"]):
            if c["expert"] != "plain":
                mat(f"e{e}.gate", c["inner"], h)
            mat(f"e{e}.up", c["inner"], h), mat(f"e{e}.down", h, c["inner"])
    elif kind == "delta":
        H, G, dim, r = c["heads"], c["kv_heads"], c["dim"], c["rank"]
        mat("q", G * dim, h), mat("k", G * dim, h), mat("v", H * dim, h), mat("b", H, h)
        vec("q_conv", G * dim, c["taps"], std=0.4), vec("k_conv", G * dim, c["taps"], std=0.4), vec("v_conv", H * dim, c["taps"], std=0.4)
        vec("a_log", H, std=0.5), vec("norm", dim, std=0.1, mean=1.0), mat("o", h, H * dim)
        if c["decay"] == "channel":
            mat("a1", r, h), mat("a2", H * dim, r, std=0.2), vec("dt_bias", H * dim, std=1.0, mean=-3.0)
            mat("g1", r, h), mat("g2", H * dim, r, std=0.2)
        else:
            mat("a", H, h), vec("dt_bias", H, std=1.0, mean=-3.0), mat("g", H * dim, h)
    elif kind == "gla":
        H, dim, r = c["heads"], c["dim"], c["rank"]
        mat("q", H * dim, h), mat("k", H * dim, h), mat("v", H * dim, h), mat("g", H * dim, h), mat("o", h, H * dim)
        vec("norm", dim, std=0.1, mean=1.0)
        mat("a1", r, h), mat("a2", H * dim, r, std=0.2), vec("a2_b", H * dim, std=2.0, mean=1.0)
    elif kind == "mlstm":
        H, dim = c["heads"], c["dim"]
        mat("q", H * dim, h), mat("k", H * dim, h), mat("v", H * dim, h), mat("g", H * dim, h), mat("o", h, H * dim)
        vec("norm", H * dim, std=0.1, mean=1.0)
        mat("i", H, h), vec("i_b", H, std=1.0), mat("f", H, h), vec("f_b", H, std=1.0, mean=2.0)
    elif kind == "rglru":
        R, B = c["width"], c["blocks"]
        mat("y", R, h), vec("y_b", R), mat("x", R, h), vec("x_b", R), vec("conv", R, c["taps"], std=0.3), vec("conv_b", R)
        mat("ra", B, R // B, R // B), vec("ra_b", B, R // B), mat("ri", B, R // B, R // B), vec("ri_b", B, R // B)
        vec("lam", R, std=1.0, mean=-3.0), mat("o", h, R)
    elif kind == "block":
        f, hd = c["ffn"], c["head_dim"]
        for n in ("n1", "n2"):
            vec(n + ".weight", h, mean=1.0), vec(n + ".bias", h)
        mat("qkv.weight", 3 * c["heads"] * hd, h), mat("out.weight", h, c["heads"] * hd)
        mat("up.weight", f, h), mat("down.weight", h, f)
    return w, d.normal((c["tokens"], h), 1.0, dtype=dt)


def _layer_spec(c):
    kind, h = c["kind"], c["hidden"]
    if kind == "attention":
        pos = {"position": ptb.PartSpec("position", "rotary", {"head_dim": c["dim"], "theta": 10000.0, "rotary_dim": c["rot"], "factor": 8.0})}
        return ptb.PartSpec("mixer", "sink_attention", dict(
            hidden=h, heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"], vdim=c["dim"], scale=c["dim"] ** -0.5, eps=EPS,
            window=c["window"], keep_first=c["keep"], softcap=c["cap"], qk_norm=c["norm"], norm_first=c["norm"],
            sink=c["sink"] == "learned", sink_value=0.0 if c["sink"] == "one" else None, gate=c["gate"] != "none",
            gate_wide=c["gate"] == "entry", q_temp=(0.1, 512) if c["temp"] else None), children=pos if c["rot"] else {})
    if kind == "latent":
        return ptb.PartSpec("mixer", "latent_attention", dict(
            hidden=h, heads=c["heads"], dim=c["dim"], rot_dim=c["rot"], vdim=c["vdim"], q_rank=c["q_rank"] or None, kv_rank=c["rank"],
            scale=(c["dim"] + c["rot"]) ** -0.5, eps=EPS, gate=c["gate"], wide_weights=c["wide"], wide_out=True),
            children={"position": ptb.PartSpec("position", "rotary", {"head_dim": c["rot"], "theta": 10000.0, "interleaved": True})})
    if kind == "experts":
        return ptb.PartSpec("feed_forward", "routed_experts", dict(
            hidden=h, inner=c["inner"], experts=c["experts"], top=c["top"], groups=c["groups"], keep=c["keep"], scale=1.5, expert=c["expert"],
            limit=7.0 if c["expert"] == "clamped_glu" else 0.0))
    if kind == "delta":
        return ptb.PartSpec("mixer", "delta_rule", dict(
            hidden=h, heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"], vdim=c["dim"], taps=c["taps"], eps=EPS, decay=c["decay"],
            gate="low_rank" if c["decay"] == "channel" else "full", gate_act="sigmoid" if c["decay"] == "channel" else "silu"))
    if kind == "gla":
        return ptb.PartSpec("mixer", "gla", dict(hidden=h, heads=c["heads"], dim=c["dim"], vdim=c["dim"], tau=c["tau"], eps=EPS))
    if kind == "mlstm":
        return ptb.PartSpec("mixer", "mlstm", dict(hidden=h, heads=c["heads"], dim=c["dim"], vdim=c["dim"], gate_cap=c["cap"], eps=EPS))
    if kind == "rglru":
        return ptb.PartSpec("mixer", "rglru", dict(hidden=h, width=c["width"], blocks=c["blocks"], taps=c["taps"]))
    norm = dict(size=h, eps=FALCON_EPS, bias=True)
    return ptb.PartSpec("block", "sequential", children={
        "norm_mixer": ptb.PartSpec("norm", "layernorm", norm), "norm_ff": ptb.PartSpec("norm", "layernorm", norm),
        "mixer": ptb.PartSpec("mixer", "attention", dict(hidden=h, heads=c["heads"], kv_heads=c["heads"], head_dim=c["head_dim"]),
                              children={"position": ptb.PartSpec("position", "rotary", {"head_dim": c["head_dim"], "theta": 10000.0})}),
        "feed_forward": ptb.PartSpec("feed_forward", "dense", dict(hidden=h, inner=c["ffn"], activation="gelu"))})


def _falcon_tensors(c, seed):
    d, dt, h = _Draws(seed), _dtype(c), c["hidden"]
    w = {"transformer.word_embeddings.weight": d.normal((c["vocab"], h), 0.02, dtype=dt)}
    for i in range(c["layers"]):
        p = f"transformer.h.{i}."
        w[p + "input_layernorm.weight"], w[p + "input_layernorm.bias"] = d.normal((h,), 0.02, 1.0), d.normal((h,), 0.02)
        w[p + "self_attention.query_key_value.weight"] = d.normal(((c["heads"] + 2) * c["head_dim"], h), 0.02, dtype=dt)
        w[p + "self_attention.dense.weight"] = d.normal((h, h), 0.02, dtype=dt)
        w[p + "mlp.dense_h_to_4h.weight"] = d.normal((c["ffn"], h), 0.02, dtype=dt)
        w[p + "mlp.dense_4h_to_h.weight"] = d.normal((h, c["ffn"]), 0.02, dtype=dt)
    w["transformer.ln_f.weight"], w["transformer.ln_f.bias"] = d.normal((h,), 0.02, 1.0), d.normal((h,), 0.02)
    lengths = _prompt_lengths(c)
    return w, [d.ids(n + c["steps"], c["vocab"]) for n in lengths], lengths


def _memory_config(c):
    mem = {"heads": c["heads"], "dim": 128, "vdim": 128, "gate_cap": 15.0}
    att = {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
           "mask": {"size": c["window"], "keep_first": c["keep"]},
           "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 2048, "fast": 32.0, "slow": 1.0}}, "v_mix": True}
    mlp = {"kind": "dense", "ff": c["ffn"]}
    return {"architecture": "Pogezen", "vocab": c["vocab"], "width": c["width"], "norm": {"eps": EPS}, "embedding": {"scale": 1.0},
            "canon": {"taps": 4}, "layers": [{"type": t, "mixer": dict(m), "mlp": mlp} for t, m in (("mlstm", mem), ("attention", att)) * 2]}


def _memory_tensors(c, seed):
    d, dt, W, H, G, F = _Draws(seed), _dtype(c), c["width"], c["heads"], c["kv_heads"], c["ffn"]
    w = {"embed": d.normal((c["vocab"], W), 1.0, dtype=dt)}

    def dyt(name):
        w[name], w[name + ".b"], w[name + ".alpha"] = d.normal((W,), 0.1, 1.0), d.normal((W,), 0.02), d.normal((), 0.05, 0.6)

    def mat(name, n, k):
        w[name] = d.normal((n, k), k ** -0.5, dtype=dt)

    for i in range(4):
        p = f"l{i}."
        dyt(p + "norm1"), dyt(p + "norm2")
        w[p + "canon1"] = d.normal((W, 4), 0.3)
        q = p + "mix."
        if i % 2 == 0:
            for n in ("q", "k", "v", "g", "o"):
                mat(q + n, H * 128, W) if n != "o" else mat(q + n, W, H * 128)
            w[q + "norm"] = d.normal((H * 128,), 0.1, 1.0)
            mat(q + "i", H, W), mat(q + "f", H, W)
            w[q + "i.b"], w[q + "f.b"] = d.normal((H,), 1.0), d.normal((H,), 1.0, 2.0)
        else:
            mat(q + "q", H * 128, W), mat(q + "k", G * 128, W), mat(q + "v", G * 128, W), mat(q + "o", W, H * 128)
            for n, size in (("q", H * 128), ("k", G * 128), ("v", G * 128), ("o", W)):
                w[q + n + ".b"] = d.normal((size,), 0.1)
            w[q + "talk"], w[q + "vmix"] = d.normal((H, H), 0.25) + torch.eye(H, device=DEV), d.normal((), 0.1, 0.5)
        mat(p + "mlp.up", F, W), mat(p + "mlp.down", W, F)
    dyt("final.norm")
    lengths = _prompt_lengths(c)
    return w, [d.ids(n + c["steps"], c["vocab"]) for n in lengths], lengths


# ------------------------------------------------------------------------------------------------ the path
def prepare(case, seed):
    c = case
    if c["kind"] in ("requests", "memory"):
        if c["kind"] == "requests":
            w, ids, lengths = _falcon_tensors(c, seed)
            cfg = ptb.FalconConfig.from_dict(dict(
                vocab_size=c["vocab"], hidden_size=c["hidden"], num_hidden_layers=c["layers"], num_attention_heads=c["heads"],
                multi_query=True, parallel_attn=True, new_decoder_architecture=False, bias=False, alibi=False, rope_theta=10000.0,
                layer_norm_epsilon=FALCON_EPS, max_position_embeddings=2048, tie_word_embeddings=True, activation="gelu",
                ffn_hidden_size=c["ffn"]))
            spec = ptb.models.falcon_spec(cfg)
        else:
            w, ids, lengths = _memory_tensors(c, seed)
            cfg = ptb.PogezenConfig.from_dict(_memory_config(c))
            spec = ptb.models.pogezen_spec(cfg)
        model = ptb.CausalLM(spec, cfg, device=DEV, dtype=_dtype(c))
        model.bind(w)
        rounded = sum((n + c["steps"] + 63) // 64 * 64 for n in lengths)
        cache = model.new_cache(rounded, max_slots=c["batch"])
        return {"case": c, "model": model, "cache": cache, "ids": ids, "lengths": lengths}
    w, x = _layer_tensors(c, seed)
    build = ptb.BuildContext(device=torch.device(DEV), dtype=_dtype(c), kernels=K)
    part = make_part(build, _layer_spec(c))
    if c["kind"] == "block":
        for name, prefix in (("norm_mixer", "n1."), ("norm_ff", "n2.")):
            part.children[name].bind({n: w[prefix + n] for n in ("weight", "bias")})
        part.children["mixer"].bind({n: w[n] for n in ("qkv.weight", "out.weight")})
        part.children["feed_forward"].bind({n: w[n] for n in ("up.weight", "down.weight")})
    else:
        part.bind(w)
    state = {"case": c, "part": part, "x": x}
    if c["kind"] == "experts":
        return state
    mixer = part.children["mixer"] if c["kind"] == "block" else part
    lengths = _lengths(c["tokens"], c["seqs"])
    cache = ptb.Cache([(0, mixer.cache_need(), mixer.state_need())], sum((n + 63) // 64 * 64 for n in lengths), _dtype(c), DEV,
                      max_slots=c["seqs"])
    slots = [cache.open() for _ in lengths]
    planner = mixer.planner()
    planners = list(planner) if isinstance(planner, (list, tuple)) else [planner]
    state["cache"] = cache
    state["ctx"] = StepContext(cache, slots, [[0] * n for n in lengths], 1, [[] for _ in lengths], planners)
    return state


def run(state):
    c = state["case"]
    if c["kind"] in ("requests", "memory"):
        model, cache, ids, lengths = state["model"], state["cache"], state["ids"], state["lengths"]
        slots = [cache.open() for _ in ids]
        out = [model.step(cache, slots, [t[:n] for t, n in zip(ids, lengths)], want="last")]
        for s in range(c["steps"] - 1):
            out.append(model.step(cache, slots, [[t[n + s]] for t, n in zip(ids, lengths)], want="last"))
        cache.close_all()
        return out
    if c["kind"] == "experts":
        return state["part"].forward(state["x"], None)
    cache, ctx = state["cache"], state["ctx"]
    ctx.begin_forward()
    if cache.state_width:
        cache.state.zero_()         # new sequences begin, as a slot's opening has it
    out = {"y": resolve(K, state["part"].forward(state["x"], ctx, ptb.ScheduleEntry(0, 0)))}
    if c["kind"] == "attention":
        out["keys"], out["values"], _ = cache.entry_storage(0)
    elif c["kind"] == "latent":
        out["rows"] = cache.entry_storage(0)[0]
    elif cache.state_width:
        out["state"] = cache.state
    return out


# ------------------------------------------------------------------------------------------------ work and tolerance
def _pairs(n, window, keep):
    """(query, key) pairs that a sequence of n tokens has inside the mask."""
    if window <= 0 or window >= n:
        return n * (n + 1) // 2
    return window * (window + 1) // 2 + (n - window) * window + sum(min(keep, i + 1 - window) for i in range(window, n))


def work(case):
    c = case
    if c["kind"] == "requests":
        h, L, hd = c["hidden"], c["layers"], c["head_dim"]
        layer = (c["heads"] + 2) * hd * h + h * h + 2 * h * c["ffn"]
        lengths, steps = _prompt_lengths(c), c["steps"]
        new = sum(lengths) + (steps - 1) * c["batch"]
        cached = sum(n * (steps - 1) + steps * (steps - 1) // 2 for n in lengths)
        weights = 2 * (L * layer + c["vocab"] * h)
        pairs = sum(_pairs(n, 0, 0) for n in lengths) + cached
        return {"bytes": steps * (weights + 4 * c["batch"] * c["vocab"]) + L * cached * 4 * hd,
                "flops": 2.0 * new * L * layer + 2.0 * steps * c["batch"] * c["vocab"] * h + 4.0 * L * c["heads"] * hd * pairs}
    if c["kind"] == "memory":
        W, H, G, F = c["width"], c["heads"], c["kv_heads"], c["ffn"]
        mem, att = 5 * H * 128 * W + 2 * H * W, 2 * (H + G) * 128 * W
        layers = 2 * mem + 2 * att + 8 * W * F
        lengths, steps = _prompt_lengths(c), c["steps"]
        new = sum(lengths) + (steps - 1) * c["batch"]
        state = 2 * 4 * H * 128 * 128 * c["batch"]
        return {"bytes": steps * (2 * (layers + c["vocab"] * W) + 4 * c["batch"] * c["vocab"]) + (steps - 1) * 2 * state,
                "flops": 2.0 * new * layers + 2.0 * steps * c["batch"] * c["vocab"] * W + 2 * 6.0 * new * H * 128 * 128
                + 2 * 2.0 * H * (128 + G * 128) * sum(_pairs(n, c["window"], c["keep"]) for n in lengths)}
    e, t, h = (4 if c["dtype"] == "float32" else 2), c["tokens"], c["hidden"]
    if c["kind"] == "experts":
        mats = 2 if c["expert"] == "plain" else 3
        used = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** t)      # distinct experts under even routing
        return {"bytes": e * (used * mats * h * c["inner"] + 2 * t * h) + 4 * c["experts"] * h,
                "flops": 2.0 * t * (c["top"] * mats * h * c["inner"] + c["experts"] * h)}
    if c["kind"] == "block":
        a = c["heads"] * c["head_dim"]
        mats = 4 * a * h + 2 * h * c["ffn"]
        return {"bytes": e * (mats + 2 * t * h),
                "flops": 2.0 * t * mats + 4.0 * a * sum(_pairs(n, 0, 0) for n in _lengths(t, c["seqs"]))}
    if c["kind"] == "attention":
        H, G, d = c["heads"], c["kv_heads"], c["dim"]
        gate = {"none": 0, "head": H, "entry": H * d}[c["gate"]]
        mats = (2 * H * d + 2 * G * d + gate) * h
        pairs = sum(_pairs(n, c["window"], c["keep"]) for n in _lengths(t, c["seqs"]))
        return {"bytes": e * (mats + 2 * t * h + 2 * t * G * d), "flops": 2.0 * t * mats + 4.0 * H * d * pairs}
    if c["kind"] == "latent":
        H, qd, r = c["heads"], c["dim"] + c["rot"], c["rank"]
        q = c["q_rank"] * (h + H * qd) if c["q_rank"] else H * qd * h
        gate = H if c["gate"] == "head" else H * c["vdim"]
        mats = q + (gate + r + c["rot"] + H * c["vdim"]) * h + H * (c["dim"] + c["vdim"]) * r
        pairs = sum(_pairs(n, 0, 0) for n in _lengths(t, c["seqs"]))
        return {"bytes": e * (mats + t * (h + r + c["rot"])) + 4 * t * h, "flops": 2.0 * t * mats + 2.0 * H * (qd + c["vdim"]) * pairs}
    if c["kind"] == "rglru":
        R = c["width"]
        mats = 3 * R * h + 2 * R * R // c["blocks"]
        return {"bytes": e * (mats + 2 * t * h) + 4 * R * c["taps"] * c["seqs"], "flops": 2.0 * t * mats + 12.0 * t * R}
    H, d = c["heads"], c["dim"]
    G = c.get("kv_heads", H)
    mats = (2 * G * d + 3 * H * d + 2 * H) * h      # q, k; v, gate, output; the gates' rows
    if c["kind"] == "gla" or c.get("decay") == "channel":
        mats += c["rank"] * (h + H * d)
    return {"bytes": e * (mats + 2 * t * h) + 4 * H * d * d * c["seqs"], "flops": 2.0 * t * (mats + 3 * H * d * d)}


def tolerance(case):
    """Four times what the path shows against 64 bits. Whole requests (0.005): bfloat16 roundings travel through the layers.
    Experts (0.0017): the rounding of the inner values and of the result. Mixers (0.002 to 0.0045): projections, heads and
    result are rounded. float32 (3e-7): sums of up to 4,096 products, whose order alone moves them by as much."""
    kind = case["kind"]
    if kind == "block":
        return {"rel": 2e-6, "max": 4e-5}
    if kind in ("requests", "memory"):
        return {"rel": 0.02, "max": 0.3}
    return {"rel": 0.007, "max": 0.2} if kind == "experts" else {"rel": 0.016, "max": 0.3}


# ------------------------------------------------------------------------------------------------ in 64 bits
def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _layernorm(x, g, b):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + FALCON_EPS) * g + b


def _gelu(x):
    return 0.5 * x * (1 + torch.erf(x / math.sqrt(2.0)))


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, freq, mult=1.0, interleaved=False):
    """x [tokens, heads, dim]: the first 2 len(freq) entries of a head turn by position * freq."""
    n = len(freq)
    a = torch.arange(x.shape[0], dtype=F64, device=DEV)[:, None] * freq
    c, s = (torch.cos(a) * mult)[:, None, :], (torch.sin(a) * mult)[:, None, :]
    y = x.clone()
    if interleaved:
        u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        y[..., 0:2 * n:2], y[..., 1:2 * n:2] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., :n], x[..., n:2 * n]
        y[..., :n], y[..., n:2 * n] = u * c - v * s, v * c + u * s
    return y


def _frequencies(dims, base=10000.0):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEV) / dims)


def _visible(T, window, keep):
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None, :]
    return (j <= i) & (((i - j) < window) | (j < keep)) if window > 0 else j <= i


def _attend(q, k, v, scale, seen, cap=0.0, sink=None):
    """[T, H, d] queries on [T, G, .] keys and values, a head at a time; ``sink`` [H] joins the denominators."""
    H, G = q.shape[1], k.shape[1]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T) * scale
        if cap > 0:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, -math.inf)
        top = s.max(-1, keepdim=True).values
        if sink is not None:
            top = top.clamp_min(float(sink[h]))
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0.0)
        out.append((e / total) @ v[:, h // (H // G)])
    return torch.stack(out, 1)


def _pages(rows_of, heads, width, lengths):
    """The cache's pages of 64 positions [pages, heads, 64, width] in the order in which the sequences took them."""
    pool = []
    for rows, n in zip(rows_of, lengths):
        pages = (n + 63) // 64
        t = torch.zeros((pages * 64, heads, width), dtype=F64, device=DEV)
        t[:n] = rows
        pool.append(t.view(pages, 64, heads, width).transpose(1, 2))
    return torch.cat(pool).contiguous()


def _exact_attention(c, w, x, lengths):
    H, G, d = c["heads"], c["kv_heads"], c["dim"]
    ys, ks, vs, at = [], [], [], 0
    for T in lengths:
        h, at = x[at:at + T], at + T
        q, k, v = (h @ w["q"].T).view(T, H, d), (h @ w["k"].T).view(T, G, d), (h @ w["v"].T).view(T, G, d)
        if c["norm"]:
            q, k = _rms(q) * w["q_norm"], _rms(k) * w["k_norm"]
        if c["rot"]:
            f = _frequencies(c["rot"]) / 8.0
            q, k = _rotate(q, f), _rotate(k, f)
        if c["temp"]:
            p = torch.arange(T, device=DEV)
            q = q * (1 + 0.1 * torch.log((p + 1).div(512, rounding_mode="floor").to(F64) + 1))[:, None, None]
        sink = {"one": torch.zeros(H, dtype=F64, device=DEV), "learned": w.get("sink"), "none": None}[c["sink"]]
        o = _attend(q, k, v, d ** -0.5, _visible(T, c["window"], c["keep"]), c["cap"], sink)
        if c["gate"] == "head":
            o = o * torch.sigmoid(h @ w["g"].T)[:, :, None]
        o = o.reshape(T, H * d)
        if c["gate"] == "entry":
            o = o * torch.sigmoid(h @ w["g"].T)
        ys.append(o @ w["o"].T), ks.append(k), vs.append(v)
    return {"y": torch.cat(ys), "keys": _pages(ks, G, d, lengths), "values": _pages(vs, G, d, lengths)}


def _exact_latent(c, w, x, lengths):
    H, d, rd, vd, r = c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"]
    f, ys, rows, at = _frequencies(rd), [], [], 0
    for T in lengths:
        h, at = x[at:at + T], at + T
        q = (_rms(h @ w["dq"].T) * w["dq_norm"]) @ w["uq"].T if c["q_rank"] else h @ w["q"].T
        q = q.view(T, H, d + rd)
        q = torch.cat([q[..., :d], _rotate(q[..., d:], f, interleaved=True)], -1)
        down = h @ w["dkv"].T
        lat, kr = _rms(down[:, :r]) * w["dkv_norm"], _rotate(down[:, None, r:], f, interleaved=True)
        k = torch.cat([(lat @ w["uk"].T).view(T, H, d), kr.expand(T, H, rd)], -1)
        o = _attend(q, k, (lat @ w["uv"].T).view(T, H, vd), (d + rd) ** -0.5, _visible(T, 0, 0))
        g = torch.sigmoid(h @ w["g"].T)
        o = (o * (g[:, :, None] if c["gate"] == "head" else g.view(T, H, vd))).reshape(T, H * vd)
        ys.append(o @ w["o"].T), rows.append(torch.cat([lat[:, None], kr], -1))
    return {"y": torch.cat(ys), "rows": _pages(rows, 1, r + rd, lengths)}


def _exact_experts(c, w, x):
    s = torch.softmax(x @ w["router"].T, -1)
    choice = s + w["correction"]
    groups = choice.view(len(x), c["groups"], -1)
    kept = torch.zeros(groups.shape[:2], dtype=torch.bool, device=DEV)
    kept.scatter_(1, groups.max(-1).values.topk(c["keep"], -1).indices, True)
    chosen = groups.masked_fill(~kept[:, :, None], -math.inf).view_as(choice).topk(c["top"], -1).indices
    weight = torch.zeros_like(s).scatter_(1, chosen, s.gather(1, chosen) * 1.5)
    y = torch.zeros_like(x)
    for e in range(c["experts"]):
        rows = (weight[:, e] > 0).nonzero()[:, 0]
        h = x[rows]
        up = h @ w[f"e{e}.up"].to(F64).T
        if c["expert"] == "plain":
            a = _gelu(up)
        else:
            g = h @ w[f"e{e}.gate"].to(F64).T
            if c["expert"] == "clamped_glu":
                g, up = g.clamp(max=7.0), up.clamp(-7.0, 7.0)
                a = g * torch.sigmoid(1.702 * g) * (up + 1)
            else:
                a = _silu(g) * up
        y[rows] += weight[rows, e:e + 1] * (a @ w[f"e{e}.down"].to(F64).T)
    return y


def _filtered(x, taps):
    n, y = taps.shape[1], torch.zeros_like(x)
    for j in range(n):
        y[n - 1 - j:] += taps[:, j] * x[:x.shape[0] - (n - 1 - j)]
    return y


def _exact_delta(c, w, x, lengths):
    H, G, d = c["heads"], c["kv_heads"], c["dim"]
    owner = torch.arange(H, device=DEV) // (H // G)
    ys, at = [], 0
    for T in lengths:
        h, at = x[at:at + T], at + T
        q, k = (_silu(_filtered(h @ w[n].T, w[n + "_conv"])).view(T, G, d) for n in ("q", "k"))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = q[:, owner] * d ** -0.5, k[:, owner]
        v = _silu(_filtered(h @ w["v"].T, w["v_conv"])).view(T, H, d)
        beta = torch.sigmoid(h @ w["b"].T)
        if c["decay"] == "channel":
            z = torch.nn.functional.softplus((h @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(T, H, d)
            g, gate = torch.exp(-torch.exp(w["a_log"])[:, None] * z), torch.sigmoid((h @ w["g1"].T) @ w["g2"].T)
        else:
            z = torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"])
            g, gate = torch.exp(-torch.exp(w["a_log"]) * z)[:, :, None].expand(T, H, d), _silu(h @ w["g"].T)
        S, o = torch.zeros((H, d, d), dtype=F64, device=DEV), torch.empty((T, H, d), dtype=F64, device=DEV)
        for t in range(T):
            S = g[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None]
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        ys.append(((_rms(o) * w["norm"]).view(T, H * d) * gate) @ w["o"].T)
    return {"y": torch.cat(ys), "state": None}


def _exact_gla(c, w, x, lengths):
    H, d = c["heads"], c["dim"]
    ys, states, at = [], [], 0
    for T in lengths:
        h, at = x[at:at + T], at + T
        q, k, v = ((h @ w[n].T).view(T, H, d) for n in ("q", "k", "v"))
        z = (h @ w["a1"].T) @ w["a2"].T + w["a2_b"]
        a = torch.exp(torch.nn.functional.logsigmoid(z) / c["tau"]).view(T, H, d)
        S, o = torch.zeros((H, d, d), dtype=F64, device=DEV), torch.empty((T, H, d), dtype=F64, device=DEV)
        for t in range(T):
            S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
            o[t] = torch.bmm(q[t][:, None], S)[:, 0] * d ** -0.5
        ys.append(((_rms(o) * w["norm"]).view(T, H * d) * _silu(h @ w["g"].T)) @ w["o"].T)
        states.append(S.reshape(-1))
    return {"y": torch.cat(ys), "state": torch.stack(states)}


def _memory_walk(q, k, v, i, f):
    T, H, d = q.shape
    S, n = torch.zeros((H, d, v.shape[-1]), dtype=F64, device=DEV), torch.zeros((H, d), dtype=F64, device=DEV)
    m, o = torch.zeros(H, dtype=F64, device=DEV), torch.empty(v.shape, dtype=F64, device=DEV)
    for t in range(T):
        top = torch.maximum(f[t] + m, i[t])
        a, b = torch.exp(f[t] + m - top)[:, None], torch.exp(i[t] - top)[:, None]
        S = a[:, :, None] * S + (b * k[t])[:, :, None] * v[t][:, None]
        n, m = a * n + b * k[t], top
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        o[t] = torch.bmm(q[t][:, None], S)[:, 0] / den[:, None]
    return o


def _memory_layer(h, w, H, d, cap):
    """The matrix memory up to its gated heads; ``w(name)`` gives a tensor."""
    T = h.shape[0]
    q, k, v = ((h @ w(n).T).view(T, H, d) for n in ("q", "k", "v"))
    i = cap * torch.tanh((h @ w("i").T + w("i_b")) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w("f").T + w("f_b")) / cap))
    o = _rms(_memory_walk(q * d ** -0.5, k, v, i, f)).reshape(T, H * d)
    return (o * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _exact_mlstm(c, w, x, lengths):
    ys, at = [], 0
    for T in lengths:
        ys.append(_memory_layer(x[at:at + T], lambda n: w[n], c["heads"], c["dim"], c["cap"]))
        at += T
    return {"y": torch.cat(ys), "state": None}


def _exact_rglru(c, w, x, lengths):
    R, B = c["width"], c["blocks"]
    ys, at = [], 0
    for T in lengths:
        h, at = x[at:at + T], at + T
        y = torch.nn.functional.gelu(h @ w["y"].T + w["y_b"], approximate="tanh")
        u = _filtered(h @ w["x"].T + w["x_b"], w["conv"]) + w["conv_b"]
        ub = u.view(T, B, R // B)
        r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, w[n]) + w[n + "_b"]).reshape(T, R) for n in ("ra", "ri"))
        log_a = -8.0 * r * torch.nn.functional.softplus(w["lam"])
        a, drive = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
        S, o = torch.zeros(R, dtype=F64, device=DEV), torch.empty((T, R), dtype=F64, device=DEV)
        for t in range(T):
            S = a[t] * S + drive[t]
            o[t] = S
        ys.append((o * y) @ w["o"].T)
    return {"y": torch.cat(ys), "state": None}


def _exact_block(c, w, x, lengths):
    H, d = c["heads"], c["head_dim"]
    ys, at = [], 0
    for T in lengths:
        r, at = x[at:at + T], at + T
        # the fused projection's rows are grouped per head as query, key, value
        qkv = (_layernorm(r, w["n1.weight"], w["n1.bias"]) @ w["qkv.weight"].T).view(T, H, 3, d)
        f = _frequencies(d)
        o = _attend(_rotate(qkv[:, :, 0], f), _rotate(qkv[:, :, 1], f), qkv[:, :, 2], d ** -0.5, _visible(T, 0, 0))
        r = r + o.reshape(T, H * d) @ w["out.weight"].T
        ys.append(r + _gelu(_layernorm(r, w["n2.weight"], w["n2.bias"]) @ w["up.weight"].T) @ w["down.weight"].T)
    return {"y": torch.cat(ys)}


def _exact_requests(c, seed):
    w, ids, lengths = _falcon_tensors(c, seed)
    w = {n: t.to(F64) for n, t in w.items()}
    H, d, f, per_seq = c["heads"], c["head_dim"], _frequencies(c["head_dim"]), []
    for seq, n in zip(ids, lengths):
        T = n + c["steps"] - 1
        x = w["transformer.word_embeddings.weight"][torch.tensor(seq[:T], device=DEV)]
        for i in range(c["layers"]):
            p = f"transformer.h.{i}."
            h = _layernorm(x, w[p + "input_layernorm.weight"], w[p + "input_layernorm.bias"])
            qkv = (h @ w[p + "self_attention.query_key_value.weight"].T).view(T, H + 2, d)
            o = _attend(_rotate(qkv[:, :H], f), _rotate(qkv[:, H:H + 1], f), qkv[:, H + 1:], d ** -0.5, _visible(T, 0, 0))
            x = x + o.reshape(T, H * d) @ w[p + "self_attention.dense.weight"].T + \
                _gelu(h @ w[p + "mlp.dense_h_to_4h.weight"].T) @ w[p + "mlp.dense_4h_to_h.weight"].T
        rows = _layernorm(x[n - 1:], w["transformer.ln_f.weight"], w["transformer.ln_f.bias"])
        per_seq.append(rows @ w["transformer.word_embeddings.weight"].T)
    return [torch.stack([p[s] for p in per_seq]) for s in range(c["steps"])]


def _exact_memory(c, seed):
    w, ids, lengths = _memory_tensors(c, seed)
    w = {n: t.to(F64) for n, t in w.items()}
    H, G, d, per_seq = c["heads"], c["kv_heads"], 128, []
    dims, base, factor, orig = 64, 10000.0, 8.0, 2048
    idx, freq = torch.arange(dims // 2, dtype=F64, device=DEV), _frequencies(dims)
    where = lambda turns: dims * math.log(orig / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(where(32.0)), 0), min(math.ceil(where(1.0)), dims - 1)
    ramp = ((idx - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    freq, mult = freq / factor * ramp + freq * (1 - ramp), 0.1 * math.log(factor) + 1.0

    def dyt(x, name):
        return torch.tanh(w[name + ".alpha"] * x) * w[name] + w[name + ".b"]

    for seq, n in zip(ids, lengths):
        T = n + c["steps"] - 1
        x, first = w["embed"][torch.tensor(seq[:T], device=DEV)], None
        for i in range(4):
            p, q = f"l{i}.", f"l{i}.mix."
            h = dyt(x, p + "norm1")
            h = h + _filtered(h, w[p + "canon1"])
            if i % 2 == 0:
                x = x + _memory_layer(h, lambda m: w[q + m.replace("_", ".")], H, d, 15.0)
            else:
                Q, Kx, V = ((h @ w[q + m].T + w[q + m + ".b"]).view(T, g, d) for m, g in (("q", H), ("k", G), ("v", G)))
                Q, Kx = _rms(_rotate(Q, freq, mult)), _rms(_rotate(Kx, freq, mult))
                if first is None:
                    first = V
                else:
                    V = (1 - w[q + "vmix"]) * V + w[q + "vmix"] * first
                s = torch.einsum("ihd,jhd->hij", Q, Kx.repeat_interleave(H // G, 1)) * d ** -0.5
                s = torch.softmax(s.masked_fill(~_visible(T, c["window"], c["keep"]), -math.inf), -1)
                o = torch.einsum("hij,jhv->ihv", torch.einsum("hg,gij->hij", w[q + "talk"], s), V.repeat_interleave(H // G, 1))
                x = x + o.reshape(T, H * d) @ w[q + "o"].T + w[q + "o.b"]
            x = x + torch.relu(dyt(x, p + "norm2") @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T
        per_seq.append(dyt(x[n - 1:], "final.norm") @ w["embed"].T)
    return [torch.stack([p[s] for p in per_seq]) for s in range(c["steps"])]


def exact(case, seed):
    c = case
    if c["kind"] == "requests":
        return _exact_requests(c, seed)
    if c["kind"] == "memory":
        return _exact_memory(c, seed)
    w, x = _layer_tensors(c, seed)
    x = x.to(F64)
    if c["kind"] == "experts":
        return _exact_experts(c, {n: t.to(F64) if n in ("router", "correction") else t for n, t in w.items()}, x)
    w = {n: t.to(F64) for n, t in w.items()}
    by_kind = {"attention": _exact_attention, "latent": _exact_latent, "delta": _exact_delta, "gla": _exact_gla, "mlstm": _exact_mlstm,
               "rglru": _exact_rglru, "block": _exact_block}
    return by_kind[c["kind"]](c, w, x, _lengths(c["tokens"], c["seqs"]))
