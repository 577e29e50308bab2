"""The work that this framework is used for, as measurable cases.

Two cases are whole calls of the engine at the sizes of Qwen2.5-1.5B in bfloat16: a decoding step of eight requests (a
replayed graph) and a prompt of 2,048 tokens.  The others are single parts of a layer, built from the registries the way a
model is built and called the way a block calls them: float32 attention and float32 feed-forward (the true 32-bit path), the
attention through a latent while decoding, the four recurrent mixers over prompt portions (Mamba-2, linear attention with a
constant decay, with a decay per channel, the gated linear recurrence) and routed experts in both kinds of step.

A part gives a step of few rows as partial sums; `run` adds those up, as whoever calls a part by itself has to.
"""
import math

import numpy as np
import torch

from beglin_b200 import Engine, Entry, load_config
from beglin_b200.cache.manager import CacheManager
from beglin_b200.engine.batch import StepBatch
from beglin_b200.parts import registry
from beglin_b200.parts.context import BuildContext
from beglin_b200.parts.spec import (AttentionSpec, DecayAttentionSpec, GatedLinearAttentionSpec, LatentAttentionSpec,
                                    Mamba2Spec, PositionSpec, RGLRUSpec, RoutedExpertsSpec, SharedExpertSpec, SwiGLUSpec)
from beglin_b200.weights import TensorDict

PAGE = 64
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}
ROPE_THETA, LATENT_THETA = 1000000.0, 10000.0


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # decoding, the steady state of a server with few users: eight requests near the end of a 4,096-token context
        {"name": "decode_1.5b", "kind": "model_decode", "dtype": "bfloat16", "width": 1536, "layers": 28, "heads": 12,
         "kv_heads": 2, "ff": 8960, "vocab": 151936, "batch": 8, "held": 4090},
        # a prompt as it comes in, whole, logits wanted at a few places
        {"name": "prompt_1.5b", "kind": "model_prompt", "dtype": "bfloat16", "width": 1536, "layers": 28, "heads": 12,
         "kv_heads": 2, "ff": 8960, "vocab": 151936, "tokens": 2048},
        # the 32-bit path (exact comparisons, evaluation): attention of a portion behind 1,536 held positions, beside a
        # short portion and a decoding request
        {"name": "attention_f32", "kind": "attention", "dtype": "float32", "width": 1536, "heads": 12, "kv_heads": 2,
         "dim": 128, "lens": "512,37,1", "held": "1536,200,3000"},
        # the same path's feed-forward over a portion, and over a decoding step
        {"name": "mlp_f32_portion", "kind": "mlp", "dtype": "float32", "width": 1536, "ff": 8960, "tokens": 550},
        {"name": "mlp_f32_decode", "kind": "mlp", "dtype": "float32", "width": 1536, "ff": 8960, "tokens": 8},
        # attention through a latent, decoding many requests at a long context (bound by the cache)
        {"name": "latent_decode", "kind": "latent", "dtype": "bfloat16", "width": 4096, "heads": 32, "dim": 64, "rot": 64,
         "vdim": 128, "q_rank": 2048, "kv_rank": 512, "batch": 64, "held": 4000},
        # recurrent mixers over a prompt portion: the layer that such a model has most of
        {"name": "mamba2_prompt", "kind": "mamba2", "dtype": "bfloat16", "width": 1536, "heads": 24, "vdim": 128, "state": 128,
         "groups": 1, "conv": 4, "lens": "2048"},
        {"name": "decay_prompt", "kind": "decay", "dtype": "bfloat16", "width": 1536, "heads": 12, "dim": 128, "vdim": 128,
         "lens": "2048"},
        {"name": "gla_prompt", "kind": "gla", "dtype": "bfloat16", "width": 4096, "heads": 32, "dim": 128, "vdim": 128,
         "write": "key", "rank": 16, "lens": "1500,500,48"},
        {"name": "rglru_prompt", "kind": "rglru", "dtype": "bfloat16", "width": 4096, "blocks": 16, "conv": 4, "lens": "2048"},
        # routed experts: a prompt portion (plain experts), and a decoding step (gated experts, identity experts, a shared one)
        {"name": "experts_prompt", "kind": "experts", "dtype": "bfloat16", "width": 1536, "ff": 3072, "experts": 8, "top": 2,
         "shared": 0, "identity": 0, "tokens": 2048},
        {"name": "experts_decode", "kind": "experts", "dtype": "bfloat16", "width": 1536, "ff": 1024, "experts": 8, "top": 2,
         "shared": 2048, "identity": 2, "tokens": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _portions(rng, lo, hi):
    """One portion of a prompt, or (one time in three) several side by side."""
    total = _log(rng, lo, hi)
    if rng.random() < 0.67 or total < 4 * lo:
        return str(total)
    a = rng.randint(total // 3, 2 * total // 3)
    return ",".join(str(n) for n in (a, total - a - lo, lo))


def draw(rng):
    kind = rng.choice(["model_decode", "model_prompt", "attention", "attention", "mlp", "mlp", "latent", "latent", "mamba2",
                       "mamba2", "decay", "decay", "gla", "gla", "rglru", "rglru", "experts", "experts"])
    width = 128 * rng.randint(6, 32)
    if kind in ("model_decode", "model_prompt"):
        kv = rng.choice([1, 2, 4])
        heads = kv * rng.randint(2, 7)
        c = {"kind": kind, "dtype": "bfloat16", "width": 64 * heads * rng.choice([1, 2]), "layers": rng.randint(2, 8), "heads": heads,
             "kv_heads": kv, "ff": 64 * rng.randint(32, 140), "vocab": 64 * rng.randint(100, 1000)}
        if kind == "model_decode":
            c.update(batch=_log(rng, 1, 64), held=_log(rng, 64, 6000))
        else:
            c.update(tokens=_log(rng, 16, 4000))
        return c
    if kind == "attention":
        kv = rng.choice([1, 2, 3, 4])
        a, b = _log(rng, 16, 700), _log(rng, 1, 64)
        return {"kind": kind, "dtype": "float32", "width": width, "heads": kv * rng.randint(1, 8), "kv_heads": kv,
                "dim": rng.choice([64, 80, 128]), "lens": "%d,%d" % (a, b), "held": "%d,%d" % (_log(rng, 1, 1500), _log(rng, 1, 3000))}
    if kind == "mlp":
        return {"kind": kind, "dtype": "float32", "width": width, "ff": 32 * rng.randint(32, 300), "tokens": _log(rng, 1, 700)}
    if kind == "latent":
        batch = _log(rng, 4, 96)
        return {"kind": kind, "dtype": "bfloat16", "width": width, "heads": rng.choice([8, 12, 16, 20, 32]), "dim": 64, "rot": rng.choice([32, 64]),
                "vdim": rng.choice([64, 128]), "q_rank": width // 2, "kv_rank": 64 * rng.randint(4, 8), "batch": batch,
                "held": min(_log(rng, 128, 9000), 270000 // batch)}
    if kind == "mamba2":
        groups = rng.choice([1, 1, 2])
        return {"kind": kind, "dtype": "bfloat16", "width": width, "heads": groups * rng.randint(4, 16), "vdim": rng.choice([64, 128]),
                "state": rng.choice([64, 128]), "groups": groups, "conv": 4, "lens": _portions(rng, 48, 2500)}
    if kind in ("decay", "gla"):
        c = {"kind": kind, "dtype": "bfloat16", "width": width, "heads": rng.randint(4, 32), "dim": rng.choice([64, 96, 128]),
             "vdim": rng.choice([64, 128]), "lens": _portions(rng, 48, 2500)}
        if kind == "gla":
            c.update(write=rng.choice(["forget", "key"]), rank=rng.choice([8, 16]))
        return c
    if kind == "rglru":
        return {"kind": kind, "dtype": "bfloat16", "width": 256 * rng.randint(3, 16), "blocks": rng.choice([4, 8, 16]), "conv": 4,
                "lens": _portions(rng, 64, 3000)}
    shared = rng.choice([0, 1])
    return {"kind": kind, "dtype": "bfloat16", "width": width, "ff": 64 * rng.randint(8, 48), "experts": rng.choice([4, 8, 16]), "top": 2,
            "shared": 64 * rng.randint(8, 40) if shared else 0, "identity": rng.choice([0, 2]) if shared else 0,
            "tokens": _log(rng, 2, 2500)}


# ------------------------------------------------------------------------------------------------ inputs, from the seed alone
def _ints(text):
    return [int(v) for v in str(text).split(",")]


class _Draws:
    def __init__(self, seed, dtype):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))
        self.dtype = dtype

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=self.g)
        return t.to(dtype or self.dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=None):
        t = torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=self.g)
        return t.to(dtype or self.dtype)

    def matrix(self, n_out, n_in):
        return self.normal(n_out, n_in, std=n_in ** -0.5)

    def scale(self, n):
        return self.normal(n, std=0.02, mean=1.0)


def _rows(c):
    """(new rows, held positions) of each request of the step."""
    if c["kind"] == "attention":
        return _ints(c["lens"]), _ints(c["held"])
    if c["kind"] == "latent":
        return [1] * c["batch"], [max(1, c["held"] - 17 * i) for i in range(c["batch"])]
    if "lens" in c:
        lens = _ints(c["lens"])
        return lens, [0] * len(lens)
    return [c["tokens"]], [0]


def _decays(heads):
    """Decays of linear attention, from 7/8 for the first head to 1 - 2^-8 for the last."""
    return tuple(1.0 - 2.0 ** (-3.0 - 5.0 * i / max(1, heads - 1)) for i in range(heads))


def _inputs(c, seed):
    """Weights by the part's own names, the normed rows h [T, width], and what the requests hold already."""
    d = _Draws(seed, DTYPES[c["dtype"]])
    W, kind, w, held = c["width"], c["kind"], {}, None
    lens, past = _rows(c)
    if kind == "attention":
        H, kv, hd = c["heads"], c["kv_heads"], c["dim"]
        for name, n in (("q", H * hd), ("k", kv * hd), ("v", kv * hd)):
            w[name + "_proj.weight"], w[name + "_proj.bias"] = d.matrix(n, W), d.normal(n, std=0.1)
        w["o_proj.weight"] = d.matrix(W, H * hd)
        held = [d.normal(2, kv, n, hd) for n in past]
    elif kind == "mlp":
        w = {"gate_proj.weight": d.matrix(c["ff"], W), "up_proj.weight": d.matrix(c["ff"], W), "down_proj.weight": d.matrix(W, c["ff"])}
    elif kind == "latent":
        H, qr, kr, rot = c["heads"], c["q_rank"], c["kv_rank"], c["rot"]
        w = {"q_down.weight": d.matrix(qr, W), "q_down.norm": d.scale(qr), "q_up.weight": d.matrix(H * (c["dim"] + rot), qr),
             "k_up.weight": d.matrix(H * c["dim"], kr), "v_up.weight": d.matrix(H * c["vdim"], kr),
             "o_proj.weight": d.matrix(W, H * c["vdim"]), "kv_down.weight": d.matrix(kr + rot, W), "kv_down.norm": d.scale(kr),
             "gate.weight": d.matrix(H, W)}
        held = [d.normal(n, kr + rot) for n in past]
    elif kind == "mamba2":
        inner, ch, H = c["heads"] * c["vdim"], c["heads"] * c["vdim"] + 2 * c["groups"] * c["state"], c["heads"]
        step = torch.exp(d.uniform(H, lo=math.log(1e-3), hi=math.log(0.1), dtype=torch.float32))
        w = {"in_proj.weight": d.matrix(inner + ch + H, W), "conv.weight": d.normal(ch, c["conv"], std=0.5), "conv.bias": d.normal(ch, std=0.1),
             "dt_bias": (step + torch.log(-torch.expm1(-step))).to(d.dtype), "A_log": torch.log(d.uniform(H, lo=1.0, hi=16.0, dtype=torch.float32)).to(d.dtype),
             "D": d.scale(H), "norm.weight": d.scale(inner), "o_proj.weight": d.matrix(W, inner)}
    elif kind in ("decay", "gla"):
        qd, vd = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        w = {"q_proj.weight": d.matrix(qd, W), "v_proj.weight": d.matrix(vd, W), "o_proj.weight": d.matrix(W, vd)}
        if kind == "decay":
            w.update({"k_proj.weight": d.matrix(qd, W), "g_proj.weight": d.matrix(vd, W), "norm.weight": d.scale(vd)})
        elif c["write"] == "forget":
            w.update({"f_proj.weight": d.matrix(qd, W), "f_proj.bias": d.normal(qd), "lower": d.uniform(qd, hi=0.9), "norm.weight": d.scale(c["vdim"])})
        else:
            w.update({"k_proj.weight": d.matrix(qd, W), "decay_in.weight": d.matrix(c["rank"], W), "decay_out.weight": d.matrix(qd, c["rank"]),
                      "decay_out.bias": d.normal(qd), "g_proj.weight": d.matrix(vd, W), "norm.weight": d.scale(c["vdim"])})
    elif kind == "rglru":
        B, bs = c["blocks"], W // c["blocks"]
        w = {"y_proj.weight": d.matrix(W, W), "y_proj.bias": d.normal(W, std=0.1), "x_proj.weight": d.matrix(W, W), "x_proj.bias": d.normal(W, std=0.1),
             "conv.weight": d.normal(W, c["conv"], std=0.5), "conv.bias": d.normal(W, std=0.1),
             "gate_r.weight": d.normal(B, bs, bs, std=bs ** -0.5), "gate_r.bias": d.normal(B, bs, std=0.1),
             "gate_i.weight": d.normal(B, bs, bs, std=bs ** -0.5), "gate_i.bias": d.normal(B, bs, std=0.1),
             # softplus(lam) such that a channel's decay at half-open gates lies between 0.9 and 0.999
             "lam": torch.log(torch.expm1(-torch.log(d.uniform(W, lo=0.9, hi=0.999, dtype=torch.float32)) / 4.0)).to(d.dtype),
             "o_proj.weight": d.matrix(W, W)}
    elif kind == "experts":
        out, ff = c["experts"] + c["identity"], c["ff"]
        w["router.weight"] = d.matrix(out, W)
        if c["shared"]:
            w["router.bias"] = d.normal(out, std=0.02)
        for e in range(c["experts"]):
            if c["shared"]:
                w[f"experts.{e}.gate.weight"] = d.matrix(ff, W)
            w[f"experts.{e}.up.weight"], w[f"experts.{e}.down.weight"] = d.matrix(ff, W), d.matrix(W, ff)
        if c["shared"]:
            w.update({"shared.gate.weight": d.matrix(c["shared"], W), "shared.up.weight": d.matrix(c["shared"], W),
                      "shared.down.weight": d.matrix(W, c["shared"]), "shared.scale.weight": d.matrix(1, W)})
    return w, d.normal(sum(lens), W), held


def _spec(c):
    W, kind = c["width"], c["kind"]
    if kind == "attention":
        return AttentionSpec(hidden=W, n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["dim"], qkv_bias=True,
                             position=PositionSpec(rotary_dim=c["dim"], theta=ROPE_THETA))
    if kind == "mlp":
        return SwiGLUSpec(hidden=W, intermediate=c["ff"])
    if kind == "latent":
        return LatentAttentionSpec(hidden=W, n_heads=c["heads"], dim=c["dim"], rot_dim=c["rot"], vdim=c["vdim"], q_rank=c["q_rank"],
                                   kv_rank=c["kv_rank"], scale=(c["dim"] + c["rot"]) ** -0.5, eps=1e-5,
                                   position=PositionSpec(rotary_dim=c["rot"], theta=LATENT_THETA, pairing="interleaved"))
    if kind == "mamba2":
        return Mamba2Spec(hidden=W, n_heads=c["heads"], vdim=c["vdim"], state=c["state"], groups=c["groups"], conv=c["conv"], norm_groups=1, eps=1e-5)
    if kind == "decay":
        return DecayAttentionSpec(hidden=W, n_heads=c["heads"], dim=c["dim"], vdim=c["vdim"], decay=_decays(c["heads"]), eps=1e-5)
    if kind == "gla":
        key = c["write"] == "key"
        return GatedLinearAttentionSpec(hidden=W, n_heads=c["heads"], dim=c["dim"], vdim=c["vdim"], eps=1e-6, write=c["write"], query_silu=not key,
                                        query_scale=c["dim"] ** -0.5 if key else 1.0, decay_rank=c["rank"] if key else 0,
                                        decay_power=1.0 / 16.0 if key else 1.0, gated=key)
    if kind == "rglru":
        return RGLRUSpec(hidden=W, width=W, blocks=c["blocks"], conv=c["conv"])
    if c["shared"]:
        return RoutedExpertsSpec(hidden=W, intermediate=c["ff"], experts=c["experts"], top=c["top"], activation="glu_clamped", limit=7.0,
                                 router_activation="softmax", choice_bias=True, route_scale=2.5, identity=c["identity"], scale_input=False,
                                 shared=SharedExpertSpec(intermediate=c["shared"], limit=7.0))
    return RoutedExpertsSpec(hidden=W, intermediate=c["ff"], experts=c["experts"], top=c["top"])


def _qwen2_config(c):
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": c["layers"], "hidden_size": c["width"],
            "num_attention_heads": c["heads"], "num_key_value_heads": c["kv_heads"], "intermediate_size": c["ff"], "vocab_size": c["vocab"],
            "rope_theta": ROPE_THETA, "rms_norm_eps": 1e-6, "tie_word_embeddings": True, "use_sliding_window": False, "hidden_act": "silu",
            "max_position_embeddings": 32768}


def _qwen2_inputs(c, seed):
    d = _Draws(seed, torch.bfloat16)
    W, hd, kv = c["width"], c["width"] // c["heads"], c["kv_heads"]
    # the residual sum grows by half over all layers, as it does in trained models: its start is not drowned by the first layers
    part = (2 * c["layers"]) ** -0.5
    w = {"model.embed_tokens.weight": d.normal(c["vocab"], W), "model.norm.weight": d.scale(W)}
    for i in range(c["layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = d.scale(W), d.scale(W)
        for name, n in (("q", c["heads"] * hd), ("k", kv * hd), ("v", kv * hd)):
            w[p + f"self_attn.{name}_proj.weight"], w[p + f"self_attn.{name}_proj.bias"] = d.matrix(n, W), d.normal(n, std=0.1)
        w[p + "self_attn.o_proj.weight"] = d.normal(W, c["heads"] * hd, std=part * (c["heads"] * hd) ** -0.5)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = d.matrix(c["ff"], W), d.matrix(c["ff"], W)
        w[p + "mlp.down_proj.weight"] = d.normal(W, c["ff"], std=part * c["ff"] ** -0.5)
    n = c["batch"] if c["kind"] == "model_decode" else c["tokens"]
    ids = torch.randint(0, c["vocab"], (n,), device="cuda", generator=d.g).tolist()
    # what the requests hold: keys and values of every layer [layers, requests, 2, kv heads, positions, features]
    held = d.normal(c["layers"], n, 2, kv, c["held"], hd) if c["kind"] == "model_decode" else None
    return w, ids, held


def _wanted(c):
    """Up to sixteen places of a prompt whose logits are wanted, the last among them."""
    T = c["tokens"]
    return sorted({T - 1 - i * max(1, T // 16) for i in range(min(16, T))})


# ------------------------------------------------------------------------------------------------ what a program keeps
def _fill(pool, table, values):
    """Puts what a request holds, [2, kv heads, positions, features] or [positions, width], into its pages."""
    rows = values.shape[-2]
    pages = -(-rows // PAGE)
    room = torch.zeros(values.shape[:-2] + (pages * PAGE, values.shape[-1]), dtype=values.dtype, device=values.device)
    room[..., :rows, :] = values
    room = room.view(values.shape[:-2] + (pages, PAGE, values.shape[-1]))
    pool[table[:pages].long()] = room.movedim(-3, 0)


class _Part:
    """A part with its weights, its cache, the step's batch and the rows it reads."""

    def __init__(self, c, seed):
        spec, dtype = _spec(c), DTYPES[c["dtype"]]
        w, self.h, held = _inputs(c, seed)
        family = "feed_forward" if c["kind"] in ("mlp", "experts") else "mixer"
        cls = registry.part_class(family, spec.kind)
        ctx = BuildContext(device="cuda:0", compute_dtype=dtype, page_size=PAGE)
        self.part = cls(spec, w, ctx)
        need = None
        if family == "mixer":
            need = cls.cache_need(spec, ctx) if getattr(cls, "cache_need_takes_context", False) else cls.cache_need(spec)
        lens, past = _rows(c)
        pages = sum(-(-(n + p) // PAGE) for n, p in zip(lens, past))
        cache = CacheManager([need], PAGE, pages, len(lens), max(n + p for n, p in zip(lens, past)) + PAGE)
        cache.allocate(ctx.device, ctx.cache_dtype)
        for i in range(len(lens)):
            cache.add_request(i)
        plan = [(i, n + p) for i, (n, p) in enumerate(zip(lens, past))]
        cache.reserve(plan)
        self.batch = StepBatch([Entry(i, np.zeros(n, dtype=np.int64)) for i, n in enumerate(lens)], past, ctx.device, cache)
        cache.commit(plan)
        self.view = cache.view(0, self.batch) if need is not None else None
        self.takes_cache = family == "mixer"
        if hasattr(self.view, "pool"):
            self.view.pool.zero_()
            for i, values in enumerate(held):
                _fill(self.view.pool, self.view.block_table[i], values)

    def run(self):
        y = self.part.forward(self.h, self.batch, self.view) if self.takes_cache else self.part.forward(self.h, self.batch)
        if y.dim() == 3:
            y = y.sum(0)
        if self.view is None:
            return {"y": y}
        return {"y": y, "cache": self.view.pool if hasattr(self.view, "pool") else self.view.state}


class _Model:
    def __init__(self, c, seed):
        w, self.ids, held = _qwen2_inputs(c, seed)
        arch, cfg = load_config(_qwen2_config(c))
        decode = c["kind"] == "model_decode"
        per = (c["held"] + PAGE if decode else c["tokens"]) // PAGE + 1
        n = c["batch"] if decode else 1
        self.eng = Engine(arch.build_spec(cfg), TensorDict(w), config=cfg, dtype=c["dtype"], device="cuda:0", max_tokens=n * per * PAGE,
                          page_size=PAGE, max_requests=n, max_context=per * PAGE)
        self.want = None if decode else _wanted(c)
        if decode:
            cache = self.eng.cache
            self.rids = list(range(n))
            self.back = [(r, c["held"]) for r in self.rids]
            for r in self.rids:
                cache.add_request(r)
            cache.reserve(self.back)
            cache.commit(self.back)
            group = cache.kv_groups[0]
            tables = torch.from_numpy(cache.block_table(0, self.rids)).cuda()
            for layer in range(c["layers"]):
                for r in self.rids:
                    _fill(group.device_pool[layer], tables[r], held[layer, r])

    def run(self):
        if self.want is not None:
            return {"logits": self.eng.step([("p", self.ids, self.want)], end=["p"])}
        # one token per request; then the requests go back to the length they had, as for a program that scores several
        # continuations of the same contexts
        self.eng.decode(self.rids, self.ids, read_back=False)
        self.eng.cache.commit(self.back)
        return {"logits": self.eng.decode_graph(len(self.rids)).logits[:len(self.rids)]}


def prepare(case, seed):
    return _Model(case, seed) if case["kind"].startswith("model") else _Part(case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c, W, kind = case, case["width"], case["kind"]
    e = 4 if c["dtype"] == "float32" else 2
    if kind in ("model_decode", "model_prompt"):
        hd, kv, H = W // c["heads"], c["kv_heads"], c["heads"]
        layer = W * (H + 2 * kv) * hd + W * H * hd + 3 * W * c["ff"]
        if kind == "model_decode":
            keys = c["batch"] * (c["held"] + 1)
            return {"bytes": 2 * (c["layers"] * layer + c["vocab"] * W + c["layers"] * keys * 2 * kv * hd) + 4 * c["batch"] * c["vocab"],
                    "flops": 2 * c["batch"] * (c["layers"] * layer + c["vocab"] * W) + 4 * c["layers"] * keys * H * hd}
        T, places = c["tokens"], len(_wanted(c))
        return {"bytes": 2 * (c["layers"] * layer + c["vocab"] * W + c["layers"] * T * 2 * kv * hd) + 4 * places * c["vocab"],
                "flops": 2 * T * c["layers"] * layer + 2 * places * c["vocab"] * W + 4 * c["layers"] * H * hd * T * (T + 1) // 2}
    lens, past = _rows(c)
    T, R = sum(lens), len(lens)
    rows_io = 2 * T * W * e
    if kind == "attention":
        H, kv, hd = c["heads"], c["kv_heads"], c["dim"]
        weights = W * (2 * H + 2 * kv) * hd
        pairs = sum(n * p + n * (n + 1) // 2 for n, p in zip(lens, past))
        keys = sum(n + p for n, p in zip(lens, past))
        return {"bytes": e * (weights + 2 * keys * kv * hd) + rows_io, "flops": 2 * T * weights + 4 * pairs * H * hd}
    if kind == "mlp":
        return {"bytes": e * 3 * W * c["ff"] + rows_io, "flops": 6 * T * W * c["ff"]}
    if kind == "latent":
        H, kr, rot = c["heads"], c["kv_rank"], c["rot"]
        weights = W * (c["q_rank"] + kr + rot + H) + c["q_rank"] * H * (c["dim"] + rot) + H * kr * (c["dim"] + c["vdim"]) + W * H * c["vdim"]
        keys = sum(n + p for n, p in zip(lens, past))
        return {"bytes": e * (weights + keys * (kr + rot)) + rows_io, "flops": 2 * T * weights + 2 * keys * H * (2 * kr + rot)}
    if kind == "mamba2":
        inner = c["heads"] * c["vdim"]
        ch = inner + 2 * c["groups"] * c["state"]
        weights, state = W * (2 * inner + ch - inner + c["heads"]) + W * inner, c["heads"] * c["vdim"] * c["state"]
        return {"bytes": e * weights + rows_io + 8 * R * state, "flops": 2 * T * weights + 6 * T * state + 2 * T * ch * c["conv"]}
    if kind in ("decay", "gla"):
        qd, vd = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        gate = vd if kind == "decay" or c["write"] == "key" else 0
        low = c["rank"] * (W + qd) if kind == "gla" and c["write"] == "key" else 0
        weights, state = W * (2 * qd + 2 * vd + gate) + low, c["heads"] * c["dim"] * c["vdim"]
        return {"bytes": e * weights + rows_io + 8 * R * state, "flops": 2 * T * weights + 5 * T * state}
    if kind == "rglru":
        weights = 3 * W * W + 2 * W * (W // c["blocks"])
        return {"bytes": e * weights + rows_io + 8 * R * W * c["conv"], "flops": 2 * T * weights + 2 * T * W * c["conv"]}
    mats = 3 if c["shared"] else 2
    used = min(c["experts"], T * c["top"])
    return {"bytes": e * (used * mats * W * c["ff"] + 3 * W * c["shared"]) + T * W * (e + 4) + 4 * W * (c["experts"] + c["identity"]),
            "flops": 2 * T * (c["top"] * mats * W * c["ff"] + 3 * W * c["shared"] + W * (c["experts"] + c["identity"]))}


def tolerance(case):
    """float32 parts: sums of some thousand products in 32 bits, in another order.  bfloat16 parts: a few roundings of rows to
    eight bits between the products.  Whole models: the same through all layers."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"].startswith("model"):
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.012, "max": 0.2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _angles(pos, dims, theta):
    """Angles as the checkpoints were run with them: frequencies and their products with the position are 32-bit numbers."""
    expo = -(np.float32(2.0) * np.arange(dims // 2, dtype=np.float32)) / np.float32(dims)
    inv = np.power(np.float64(np.float32(theta)), expo.astype(np.float64)).astype(np.float32)
    return (pos.float()[:, None] * torch.from_numpy(inv).cuda()[None, :]).double()


def _turn(x, ang, halves):
    """x [..., T, features] turned in pairs (i, i + n/2) or (2i, 2i + 1)."""
    cos, sin = torch.cos(ang), torch.sin(ang)
    if halves:
        a, b = x.chunk(2, dim=-1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * cos - b * sin, b * cos + a * sin], dim=-1).flatten(-2)


def _attend(q, k, v, first, scale):
    """q [H, n, d] at positions first .. first + n - 1, k and v [kv, n + first, d] -> [n, H d]."""
    H, n, hd = q.shape
    g = H // k.shape[0]
    out = []
    see = torch.arange(k.shape[1], device="cuda")[None, :] <= torch.arange(first, first + n, device="cuda")[:, None]
    for h in range(H):
        s = (q[h] @ k[h // g].T) * scale
        out.append(torch.softmax(s.masked_fill(~see, -math.inf), dim=-1) @ v[h // g])
    return torch.stack(out, dim=1).reshape(n, H * hd)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _exact_qwen2(c, seed):
    w, ids, held = _qwen2_inputs(c, seed)
    W, H, kv = c["width"], c["heads"], c["kv_heads"]
    hd = W // H
    decode = c["kind"] == "model_decode"
    x = w["model.embed_tokens.weight"][torch.tensor(ids, device="cuda")].double()
    n = len(ids)
    pos = torch.full((n,), c["held"], device="cuda") if decode else torch.arange(n, device="cuda")
    ang = _angles(pos, hd, ROPE_THETA)
    for i in range(c["layers"]):
        p = {k[len(f"model.layers.{i}."):]: t.double() for k, t in w.items() if k.startswith(f"model.layers.{i}.")}
        h = _rms(x, p["input_layernorm.weight"], 1e-6)
        q, k, v = ((h @ p[f"self_attn.{m}_proj.weight"].T + p[f"self_attn.{m}_proj.bias"]).view(n, -1, hd).transpose(0, 1) for m in "qkv")
        q, k = _turn(q, ang, True), _turn(k, ang, True)
        if decode:
            a = torch.cat([_attend(q[:, r:r + 1], torch.cat([held[i, r, 0].double(), k[:, r:r + 1]], dim=1),
                                   torch.cat([held[i, r, 1].double(), v[:, r:r + 1]], dim=1), c["held"], hd ** -0.5) for r in range(n)])
        else:
            a = _attend(q, k, v, 0, hd ** -0.5)
        x = x + a @ p["self_attn.o_proj.weight"].T
        h = _rms(x, p["post_attention_layernorm.weight"], 1e-6)
        x = x + (_silu(h @ p["mlp.gate_proj.weight"].T) * (h @ p["mlp.up_proj.weight"].T)) @ p["mlp.down_proj.weight"].T
    if not decode:
        x = x[torch.tensor(_wanted(c), device="cuda")]
    return {"logits": _rms(x, w["model.norm.weight"].double(), 1e-6) @ w["model.embed_tokens.weight"].double().T}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind.startswith("model"):
        return _exact_qwen2(c, seed)
    w, h, held = _inputs(c, seed)
    w, h = {k: t.double() for k, t in w.items()}, h.double()
    lens, past = _rows(c)
    if kind == "mlp":
        return {"y": (_silu(h @ w["gate_proj.weight"].T) * (h @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T}
    if kind == "experts":
        return {"y": _exact_experts(c, w, h)}
    f = {"attention": _exact_attention, "latent": _exact_latent, "mamba2": _exact_mamba2, "decay": _exact_decay, "gla": _exact_gla,
         "rglru": _exact_rglru}[kind]
    ys, row = [], 0
    for i, (n, p) in enumerate(zip(lens, past)):
        ys.append(f(c, w, h[row:row + n], None if held is None else held[i].double(), p))
        row += n
    return {"y": torch.cat(ys), "cache": None}


def _exact_attention(c, w, h, held, first):
    n, hd = h.shape[0], c["dim"]
    ang = _angles(torch.arange(first, first + n, device="cuda"), hd, ROPE_THETA)
    q, k, v = ((h @ w[m + "_proj.weight"].T + w[m + "_proj.bias"]).view(n, -1, hd).transpose(0, 1) for m in "qkv")
    q, k = _turn(q, ang, True), _turn(k, ang, True)
    a = _attend(q, torch.cat([held[0], k], dim=1), torch.cat([held[1], v], dim=1), first, hd ** -0.5)
    return a @ w["o_proj.weight"].T


def _exact_latent(c, w, h, held, first):
    H, kr, dim = c["heads"], c["kv_rank"], c["dim"]
    ang = _angles(torch.arange(first, first + 1, device="cuda"), c["rot"], LATENT_THETA)
    q = (_rms(h @ w["q_down.weight"].T, w["q_down.norm"], 1e-5) @ w["q_up.weight"].T).view(H, -1)
    row = h @ w["kv_down.weight"].T
    rows = torch.cat([held, torch.cat([_rms(row[:, :kr], w["kv_down.norm"], 1e-5), _turn(row[:, kr:], ang, False)], dim=1)])
    lat = torch.einsum("hd,hdk->hk", q[:, :dim], w["k_up.weight"].view(H, dim, kr))
    s = (lat @ rows[:, :kr].T + _turn(q[:, None, dim:], ang, False)[:, 0] @ rows[:, kr:].T) * (dim + c["rot"]) ** -0.5
    o = torch.softmax(s, dim=-1) @ rows[:, :kr]
    o = torch.einsum("hk,hvk->hv", o, w["v_up.weight"].view(H, c["vdim"], kr)) * torch.sigmoid(h @ w["gate.weight"].T).view(H, 1)
    return o.reshape(1, -1) @ w["o_proj.weight"].T


def _convolved(x, weight, bias):
    """A causal convolution per channel of rows that begin a request; the last tap meets the row itself."""
    taps = weight.shape[1]
    x = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=x.dtype, device=x.device), x])
    return sum(x[j:j + x.shape[0] - taps + 1] * weight[:, j] for j in range(taps)) + bias


def _exact_mamba2(c, w, h, held, first):
    n, H, P, N, G = h.shape[0], c["heads"], c["vdim"], c["state"], c["groups"]
    z, xbc, dt = (h @ w["in_proj.weight"].T).split([H * P, H * P + 2 * G * N, H], dim=1)
    x, B, C = _silu(_convolved(xbc, w["conv.weight"], w["conv.bias"])).split([H * P, G * N, G * N], dim=1)
    x, B, C = x.reshape(n, H, P), B.reshape(n, G, N).repeat_interleave(H // G, 1), C.reshape(n, G, N).repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])
    a = torch.exp(-torch.exp(w["A_log"]) * dt)
    S, ys = torch.zeros(H, P, N, dtype=h.dtype, device=h.device), []
    for t in range(n):
        S = S * a[t, :, None, None] + (dt[t, :, None] * x[t])[:, :, None] * B[t][:, None, :]
        ys.append((S @ C[t][:, :, None])[:, :, 0])
    y = (torch.stack(ys) + w["D"][:, None] * x).reshape(n, H * P)
    return _rms(y * _silu(z), w["norm.weight"], 1e-5) @ w["o_proj.weight"].T


def _walk(a, k, v, q):
    """S <- diag(a_t) S + k_t v_t^T, o_t = S^T q_t for rows [n, heads, features]."""
    S, out = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=k.dtype, device=k.device), []
    for t in range(k.shape[0]):
        S = S * a[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
        out.append((q[t][:, None, :] @ S)[:, 0])
    return torch.stack(out)


def _exact_decay(c, w, h, held, first):
    n, H = h.shape[0], c["heads"]
    q, k, v = (_silu(h @ w[m + "_proj.weight"].T).view(n, H, -1) for m in "qkv")
    a = torch.tensor(_decays(H), dtype=torch.float32, device="cuda").double()[None, :, None].expand(n, H, 1)
    y = _rms(_walk(a, k, v, q).reshape(n, -1), w["norm.weight"], 1e-5)
    return (y * torch.sigmoid(h @ w["g_proj.weight"].T)) @ w["o_proj.weight"].T


def _exact_gla(c, w, h, held, first):
    n, H = h.shape[0], c["heads"]
    q, v = ((h @ w[m + "_proj.weight"].T).view(n, H, -1) for m in "qv")
    if c["write"] == "forget":
        a = w["lower"] + (1.0 - w["lower"]) * torch.sigmoid(h @ w["f_proj.weight"].T + w["f_proj.bias"])
        a, q = a.view(n, H, -1), _silu(q)
        k = 1.0 - a
    else:
        z = (h @ w["decay_in.weight"].T) @ w["decay_out.weight"].T + w["decay_out.bias"]
        a, q, k = (torch.sigmoid(z) ** (1.0 / 16.0)).view(n, H, -1), q * c["dim"] ** -0.5, (h @ w["k_proj.weight"].T).view(n, H, -1)
    y = _rms(_walk(a, k, v, q), w["norm.weight"], 1e-6).reshape(n, -1)
    if c["write"] == "key":
        y = y * _silu(h @ w["g_proj.weight"].T)
    return y @ w["o_proj.weight"].T


def _exact_rglru(c, w, h, held, first):
    n, W, B = h.shape[0], c["width"], c["blocks"]
    y = _gelu(h @ w["y_proj.weight"].T + w["y_proj.bias"])
    u = _convolved(h @ w["x_proj.weight"].T + w["x_proj.bias"], w["conv.weight"], w["conv.bias"])
    r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(n, B, -1), w[f"gate_{m}.weight"]) + w[f"gate_{m}.bias"]).reshape(n, W) for m in "ri")
    log_a = -8.0 * r * torch.nn.functional.softplus(w["lam"])
    a, b = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * i * u
    S, out = torch.zeros(W, dtype=h.dtype, device=h.device), []
    for t in range(n):
        S = a[t] * S + b[t]
        out.append(S)
    return (torch.stack(out) * y) @ w["o_proj.weight"].T


def _exact_experts(c, w, h):
    def expert(name, x, gated):
        up = x @ w[name + "up.weight"].T
        if gated:
            g = torch.clamp(x @ w[name + "gate.weight"].T, max=7.0)
            up = g * torch.sigmoid(1.702 * g) * (torch.clamp(up, -7.0, 7.0) + 1.0)
        else:
            up = torch.relu(up) ** 2
        return up @ w[name + "down.weight"].T

    logits = h @ w["router.weight"].T
    gated = c["shared"] > 0
    scores = torch.softmax(logits, dim=-1) if gated else torch.sigmoid(logits)
    chosen = torch.topk(scores + w["router.bias"] if gated else logits, c["top"], dim=-1).indices
    y = torch.zeros_like(h)
    for e in range(c["experts"] + c["identity"]):
        rows = (chosen == e).any(-1).nonzero()[:, 0]
        if rows.numel() == 0:
            continue
        s = scores[rows, e][:, None]
        if not gated:
            y[rows] += expert(f"experts.{e}.", h[rows] * s, False)
        elif e >= c["experts"]:
            y[rows] += 2.5 * s * h[rows]
        else:
            y[rows] += 2.5 * s * expert(f"experts.{e}.", h[rows], True)
    if gated:
        y = y + torch.sigmoid(h @ w["shared.scale.weight"].T) * expert("shared.", h, True)
    return y
