"""The work whose time is watched: steps of the seven designs through ``GpuRuntime.step``.

A case is one call of the step function: the prompts of a batch (``"pass": "prompt"``; slots are taken and given
back around the step, as a server does for a request) or one more token for every sequence of a batch
(``"pass": "decode"``).  Logits at the last position of every sequence come back.  Weights are seeded random
values, N(0, 0.02) for matrices; token ids are uniform.  Sizes: Gemma-2 2B whole, and of the other designs the
layers that ``bench.py`` sets side by side (eight of them; four of Tarorax, whose differences of two averages
over nearly equal weights magnify every rounding), with dense feed-forwards where an expert is chosen by a
score (a rounding of that score chooses another expert, and outputs could not be compared); Teselix, whose
experts are looked up by token, has its experts.

``exact`` is the designs' arithmetic in 64 bits in plain torch.
"""
import hashlib
import math

import torch

VOCAB = 32000

# ---------------------------------------------------------------------------------------------- the cases

GEMMA = {"model": "gemma2", "width": 2304, "layers": 26, "dtype": "bfloat16"}


def _other(name, model, what, batch, tokens, ragged=False, width=2304):
    return {"name": name, "model": model, "width": width, "layers": 4 if model == "tarorax" else 8, "dtype": "bfloat16", "pass": what, "batch": batch,
            "tokens": tokens, "ragged": ragged}


def listed():
    return [
        # one conversation: the smallest step of the flagship, where launches and hand-overs count
        dict(GEMMA, **{"name": "gemma2 decode b1", "pass": "decode", "batch": 1, "tokens": 700, "ragged": False}),
        # the headline workload: eight sequences behind 2,048-token prompts
        dict(GEMMA, **{"name": "gemma2 decode b8", "pass": "decode", "batch": 8, "tokens": 2048, "ragged": False}),
        # a full server: 64 sequences of unequal lengths
        dict(GEMMA, **{"name": "gemma2 decode b64 ragged", "pass": "decode", "batch": 64, "tokens": 2048, "ragged": True}),
        # a question of a few words: time to the first token is launches
        dict(GEMMA, **{"name": "gemma2 prompt 37", "pass": "prompt", "batch": 1, "tokens": 37, "ragged": False}),
        # a document: the products' rate counts
        dict(GEMMA, **{"name": "gemma2 prompt 2048", "pass": "prompt", "batch": 1, "tokens": 2048, "ragged": False}),
        # the 32-bit path, as it is used to check a model
        dict(GEMMA, **{"name": "gemma2 f32 prompt 301", "dtype": "float32", "pass": "prompt", "batch": 1, "tokens": 301, "ragged": False}),
        # the other designs: a document, a batch of unequal prompts, a prompt of odd length, and single tokens
        _other("fiferax prompt 2048", "fiferax", "prompt", 1, 2048),
        _other("zatasun prompts ragged", "zatasun", "prompt", 4, 1023, ragged=True),
        _other("teselix prompt 999", "teselix", "prompt", 1, 999),
        _other("banitar decode b8", "banitar", "decode", 8, 2048),
        _other("tarorax decode b16 ragged", "tarorax", "decode", 16, 1500, ragged=True),
        _other("retudra decode b1", "retudra", "decode", 1, 500, width=1024),
    ]


def draw(rng):
    model = rng.choice(["gemma2", "gemma2", "gemma2", "fiferax", "zatasun", "teselix", "banitar", "tarorax", "retudra"])
    what = rng.choice(["prompt", "decode"])
    dtype = "float32" if rng.random() < 0.1 else "bfloat16"
    batch = int(round(2 ** rng.uniform(0, 6 if what == "decode" and model == "gemma2" else 4)))
    most = 300 if dtype == "float32" else 3000 if model == "gemma2" else 2048
    if what == "decode":
        batch = min(batch, 8) if dtype == "float32" else batch
        most = min(2048 if dtype == "bfloat16" else 300, 40000 // batch)
    else:
        most = max(2, most // batch)
    tokens = max(1, min(most, int(round(math.exp(rng.uniform(math.log(4), math.log(most + 1)))))))
    width = 2304 if model == "gemma2" else rng.choice([1024, 2304, 4096] if dtype == "bfloat16" else [1024])
    return {"model": model, "width": width, "layers": {"gemma2": 26, "tarorax": 4}.get(model, 8), "dtype": dtype, "pass": what,
            "batch": batch, "tokens": tokens, "ragged": bool(batch > 1 and rng.random() < 0.6)}


def _lengths(case):
    """Tokens of every sequence: all equal, or from the longest down over the logarithm of the range."""
    n, b = case["tokens"], case["batch"]
    if not case["ragged"]:
        return [n] * b
    return [n] + [max(1, int(n ** ((i * 0.6180339887498949) % 1.0 * 0.7 + 0.3))) for i in range(1, b)]


# ---------------------------------------------------------------------------------------------- configurations

_SIZES = {
    1024: dict(heads=16, kv=4, dim=64, vdim=64, lat=32, rot=32, kv_rank=96, q_rank=256, rank=64, window=1024, near=512, keep=16, ff=4096,
               diff_heads=8, diff_kv=2, diff_vdim=128, blocks=8, experts=16, top=2, expert_ff=1024, side=64),
    2304: dict(heads=18, kv=6, dim=128, vdim=128, lat=64, rot=64, kv_rank=192, q_rank=768, rank=96, window=4096, near=1024, keep=64, ff=9216,
               diff_heads=9, diff_kv=3, diff_vdim=256, blocks=9, experts=16, top=2, expert_ff=2304, side=128),
    4096: dict(heads=32, kv=8, dim=128, vdim=128, lat=64, rot=64, kv_rank=512, q_rank=1536, rank=128, window=4096, near=1024, keep=64, ff=14336,
               diff_heads=16, diff_kv=4, diff_vdim=256, blocks=16, experts=32, top=4, expert_ff=2048, side=128),
}


def _config(case):
    W, n = case["width"], case["layers"]
    if case["model"] == "gemma2":
        return {"architectures": ["Gemma2ForCausalLM"], "model_type": "gemma2", "num_hidden_layers": n, "hidden_size": 2304,
                "num_attention_heads": 8, "num_key_value_heads": 4, "head_dim": 256, "intermediate_size": 9216, "vocab_size": 256000,
                "rope_theta": 10000.0, "sliding_window": 4096, "query_pre_attn_scalar": 256, "attn_logit_softcapping": 50.0,
                "final_logit_softcapping": 30.0, "max_position_embeddings": 8192, "rms_norm_eps": 1e-6,
                "hidden_activation": "gelu_pytorch_tanh", "tie_word_embeddings": True, "torch_dtype": "bfloat16"}
    z = _SIZES[W]
    H, d, dv = z["heads"], z["dim"], z["vdim"]
    decay = [1.0 - 2.0 ** (-5 - 4 * h / (H - 1)) for h in range(H)]
    rot = {"base": 10000.0, "dims": d}
    attn = {"heads": H, "kv_heads": z["kv"], "dim": d, "vdim": dv, "scale": d ** -0.5}
    lat = {"heads": H, "dim": z["lat"], "rot_dim": z["rot"], "vdim": dv, "kv_rank": z["kv_rank"],
           "scale": (z["lat"] + z["rot"]) ** -0.5, "rot": {"base": 10000.0, "dims": z["rot"]}}
    dense = {"kind": "dense", "ff": z["ff"]}
    top = {"vocab": VOCAB, "width": W, "norm": {"eps": 1e-6}}

    def layers(order):
        return [{"type": t, "mixer": m, "mlp": f} for t, m, f in (order[i % len(order)] for i in range(n))]

    if case["model"] == "fiferax":
        delta = {"heads": H, "dim": d, "rank": 64}
        hd = 256 if W == 2304 else d
        par = {"left": {"heads": W // hd, "kv_heads": 3 if W == 2304 else z["kv"], "dim": hd, "vdim": hd, "mask": {"size": z["window"]},
                        "rot": {"base": 10000.0, "dims": hd}, "scale": hd ** -0.5}, "left_scale": 1.0,
               "right": {"heads": H, "dim": d, "vdim": dv, "decay": decay}, "right_scale": 1.0}
        return dict(top, architecture="Fiferax", embedding={"scale": 1.0}, layers=layers(
            [("general_delta", delta, None), ("parallel", par, dense), ("general_delta", delta, None), ("mingru", {"width": W}, dense)]))
    if case["model"] == "banitar":
        a = dict(attn, mask={"size": z["window"]}, rot=dict(rot, scaling={"factor": 4.0, "original": 4096, "fast": 16.0, "slow": 2.0}))
        return dict(top, architecture="Banitar", embedding={"scale": 1.0}, loop={"start": 2, "stop": 4, "times": 2},
                    layers=layers([("attention", a, dense), ("latent_attention", dict(lat, mask={"size": z["window"]}), dense)]))
    if case["model"] == "zatasun":
        left = dict(attn, rot={"base": 500000.0, "dims": d, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})
        mix = {"left": left, "left_scale": 1.0, "right": {"width": W, "blocks": z["blocks"], "conv": 4}, "right_scale": 1.0}
        return dict(top, architecture="Zatasun", logit_scale=1.0, layers=layers([("parallel", mix, dense)]))
    if case["model"] == "tarorax":
        gla = {"heads": H, "dim": d, "vdim": dv, "tau": 8.0, "rank": z["rank"]}
        att = {"heads": z["diff_heads"], "kv_heads": z["diff_kv"], "dim": d, "vdim": z["diff_vdim"], "conv": 4, "diff": 0.5,
               "q_temp": {"coef": 0.3, "every": 128}, "scale": d ** -0.5, "softcap": 30.0}
        return dict(top, architecture="Tarorax", streams=4,
                    layers=layers([("gla", gla, dense), ("gla", gla, dense), ("attention", att, dense), ("gla", gla, dense)]))
    if case["model"] == "teselix":
        ret = {"heads": H, "dim": d, "vdim": dv, "rot": rot, "decay": decay}
        la = dict(lat, q_rank=z["q_rank"], rot=dict(lat["rot"], scaling={"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}))
        moe = {"kind": "moe", "expert": {"ff": z["expert_ff"], "limit": 7.0}, "router": {"experts": z["experts"], "top": z["top"]},
               "shared": {"ff": z["expert_ff"], "limit": 7.0}}
        return dict(top, architecture="Teselix", postln_alpha=2.0, layers=layers([("retention", ret, moe), ("latent_attention", la, moe)]))
    assert case["model"] == "retudra"
    delta = {"heads": H, "kv_heads": H, "dim": d, "vdim": dv, "conv": 4, "rank": z["rank"]}
    a = dict(attn, rot={"base": 10000.0, "dims": d // 2}, mask={"size": z["near"], "keep_first": z["keep"]})
    return dict(top, architecture="Retudra", residual_mult=0.7, logit_softcap=30.0, token_side={"dim": z["side"]},
                layers=layers([("channel_delta", delta, dense), ("attention", a, dense), ("channel_delta", delta, dense),
                               ("latent_attention", lat, dense)]))


# ---------------------------------------------------------------------------------------------- weights

_MATRIX, _NORM, _GAIN, _BLEND = (0.0, 0.02), (0.0, 0.1), (1.0, 0.1), (0.5, 0.1)


def _tensors(cfg):
    """name -> (shape, (mean, deviation)) of a configuration's weights; ("table", below) for rows of distinct integers,
    "mixing" for a matrix near the identity, "share" for factors of a mean."""
    out = {}

    def put(name, *shape, how=_MATRIX):
        out[name] = (tuple(shape), how)

    if "hidden_size" in cfg:
        W, hd, F = cfg["hidden_size"], cfg["head_dim"], cfg["intermediate_size"]
        nq, nkv = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
        put("model.embed_tokens.weight", cfg["vocab_size"], W)
        put("model.norm.weight", W, how=_NORM)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for n in ("input_layernorm", "post_attention_layernorm", "pre_feedforward_layernorm", "post_feedforward_layernorm"):
                put(p + n + ".weight", W, how=_NORM)
            for n, rows in (("q", nq), ("k", nkv), ("v", nkv)):
                put(p + f"self_attn.{n}_proj.weight", rows, W)
            put(p + "self_attn.o_proj.weight", W, nq)
            put(p + "mlp.gate_proj.weight", F, W)
            put(p + "mlp.up_proj.weight", F, W)
            put(p + "mlp.down_proj.weight", W, F)
        return out
    W, arch = cfg["width"], cfg["architecture"]
    put("embed", cfg["vocab"], W)

    def gated(p, ff):
        put(p + "gate", ff, W), put(p + "up", ff, W), put(p + "down", W, ff)

    def norm(name, how=_NORM, bias=False, alpha=False):
        put(name, W, how=how)
        if bias:
            put(name + ".b", W, how=_NORM)
        if alpha:
            put(name + ".alpha", how=_GAIN)

    def attention(p, m, whole=None, biases=False):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        put(p + "q", H * d, W), put(p + "k", G * d, W), put(p + "o", W, H * dv)
        if arch != "Fiferax":
            put(p + "v", G * dv, W)
        if whole is not None:
            put(p + "q.norm", H * d if whole else d, how=_NORM), put(p + "k.norm", G * d if whole else d, how=_NORM)
        if biases:
            put(p + "q.b", H * d, how=_NORM), put(p + "k.b", G * d, how=_NORM), put(p + "v.b", G * dv, how=_NORM)

    def latent(p, m):
        H, d, r, dv, c = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        if m.get("q_rank"):
            put(p + "dq", m["q_rank"], W), put(p + "dq.norm", m["q_rank"], how=_GAIN), put(p + "uq", H * (d + r), m["q_rank"])
        else:
            put(p + "q", H * (d + r), W)
        put(p + "dkv", c + r, W), put(p + "dkv.norm", c, how=_NORM)
        put(p + "uk", H * d, c), put(p + "uv", H * dv, c), put(p + "o", W, H * dv)

    for i, layer in enumerate(cfg["layers"]):
        p, m, f, t = f"l{i}.", layer["mixer"], layer["mlp"], layer["type"]
        x = p + "mix."
        if arch == "Fiferax":
            norm(p + "norm1")
            if t == "general_delta":
                n = m["heads"] * m["dim"]
                for k in "rkvga":
                    put(x + k, n, W)
                put(x + "a.b", n, how=_NORM), put(x + "w1", m["rank"], W), put(x + "w2", n, m["rank"]), put(x + "w0", n, how=_NORM)
                put(x + "norm", n, how=_NORM), put(x + "o", W, n)
            elif t == "parallel":
                attention(x + "left.", m["left"], whole=False)
                n = m["right"]["heads"] * m["right"]["dim"]
                for k in "qkvg":
                    put(x + "right." + k, n, W)
                put(x + "right.norm", n, how=_NORM), put(x + "right.o", W, n)
            else:
                for k in "zxgo":
                    put(x + k, W, W)
                put(x + "z.b", W, how=_NORM), put(x + "x.b", W, how=_NORM)
            if f:
                norm(p + "norm2"), gated(p + "mlp.", f["ff"])
        elif arch == "Banitar":
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                norm(p + n, how=_GAIN, bias=True, alpha=True)
            if t == "attention":
                attention(x, m, biases=True)
                put(x + "g", m["heads"], W)
            else:
                latent(x, m)
                put(x + "sink", m["heads"], how=_NORM)
            gated(p + "mlp.", f["ff"])
        elif arch == "Zatasun":
            L, R = m["left"], m["right"]
            attention(x + "left.", L, whole=True)
            put(x + "left.sink", L["heads"], how=_NORM)
            n, b = R["width"], R["blocks"]
            for k in "yx":
                put(x + "right." + k, n, W), put(x + f"right.{k}.b", n, how=_NORM)
            put(x + "right.conv", n, R["conv"], how=_GAIN), put(x + "right.conv.b", n, how=_NORM)
            for k in ("ra", "ri"):
                put(x + "right." + k, b, n // b, n // b), put(x + f"right.{k}.b", b, n // b, how=_NORM)
            put(x + "right.lam", n, how=_GAIN), put(x + "right.o", W, n)
            norm(p + "norm1"), norm(p + "norm2"), gated(p + "mlp.", f["ff"])
        elif arch == "Tarorax":
            S = cfg["streams"]
            for k in "12":
                norm(p + "norm" + k), put(p + "ls" + k, W, how=_GAIN)
                put(p + f"hc{k}.in", S, how="share"), put(p + f"hc{k}.mix", S, S, how="mixing"), put(p + f"hc{k}.out", S, how=_GAIN)
            if t == "gla":
                n, nv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
                put(x + "q", n, W), put(x + "k", n, W), put(x + "v", nv, W), put(x + "g", nv, W), put(x + "o", W, nv)
                put(x + "a1", m["rank"], W), put(x + "a2", n, m["rank"]), put(x + "a2.b", n, how=_NORM), put(x + "norm", m["vdim"], how=_GAIN)
            else:
                H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
                for k, n in (("q", 2 * H * d), ("k", 2 * G * d), ("v", G * dv)):
                    put(x + k, n, W), put(x + k + ".b", n, how=_NORM), put(x + k + ".conv", n, m["conv"], how=_GAIN)
                put(x + "g", H * dv, W), put(x + "o", W, H * dv), put(x + "o.b", W, how=_NORM)
                for k in ("lq1", "lk1", "lq2", "lk2"):
                    put(x + k, d, how=_NORM)
            gated(p + "mlp.", f["ff"])
        elif arch == "Teselix":
            norm(p + "norm1", _GAIN, bias=True), norm(p + "norm2", _GAIN, bias=True), put(p + "shift", W, how=_BLEND)
            for k in "12":
                put(p + "rg" + k, W, W), put(p + f"rg{k}.b", W, how=_NORM)
            if t == "retention":
                n, nv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
                put(x + "q", n, W), put(x + "k", n, W), put(x + "v", nv, W), put(x + "g", nv, W), put(x + "o", W, nv)
            else:
                latent(x, m)
                put(x + "g", m["heads"], W), put(x + "sink", m["heads"], how=_NORM)
            E = f["router"]["experts"]
            put(p + "mlp.table", cfg["vocab"], f["router"]["top"], how=("table", E))
            for e in range(E):
                gated(f"{p}mlp.e{e}.", f["expert"]["ff"])
            gated(p + "mlp.shared.", f["shared"]["ff"])
        else:
            norm(p + "norm1", _GAIN, bias=True), norm(p + "norm2", _GAIN, bias=True), norm(p + "side.norm", _GAIN)
            side = cfg["token_side"]["dim"]
            put(p + "side.gate", side, W), put(p + "side.proj", W, side)
            if t == "channel_delta":
                n, nv = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
                for k, c in (("q", n), ("k", n), ("v", nv)):
                    put(x + k, c, W), put(x + k + ".conv", c, m["conv"], how=_GAIN)
                put(x + "b", m["heads"], W), put(x + "a1", m["rank"], W), put(x + "a2", m["heads"] * m["dim"], m["rank"])
                put(x + "dt_bias", m["heads"] * m["dim"], how=_NORM), put(x + "A_log", m["heads"], how=_NORM)
                put(x + "g1", m["rank"], W), put(x + "g2", nv, m["rank"]), put(x + "norm", m["vdim"], how=_GAIN), put(x + "o", W, nv)
            elif t == "attention":
                attention(x, m, whole=True)
            else:
                latent(x, m)
                put(x + "g", m["heads"] * m["vdim"], W)
            gated(p + "mlp.", f["ff"])
    if arch == "Banitar":
        put("loop.in", W, 2 * W), put("loop.step", cfg["loop"]["times"], W, how=_NORM)
    if arch == "Zatasun":
        norm("embed.norm")
    if arch == "Retudra":
        put("side.embed", cfg["vocab"], len(cfg["layers"]) * cfg["token_side"]["dim"])
    how = _GAIN if arch in ("Banitar", "Teselix", "Retudra") else _NORM
    norm("final.norm", how, bias=arch in ("Banitar", "Teselix", "Retudra"), alpha=arch == "Banitar")
    if arch in ("Fiferax", "Banitar", "Retudra"):
        put("head", cfg["vocab"], W)
    return out


class _Weights:
    """The tensors of a case by name, each made on the GPU from (seed, name) when it is asked for."""

    def __init__(self, case, cfg, seed):
        self.what = _tensors(cfg)
        self.seed = seed
        self.dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16

    def describe(self):
        return f"seeded weights ({self.seed})"

    def names(self):
        return list(self.what)

    def info(self, name):
        shape, how = self.what[name]
        return (torch.int32 if how[0] == "table" else self.dtype), shape

    def read(self, name, device=None):
        shape, how = self.what[name]
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int.from_bytes(hashlib.sha256(f"{self.seed}:{name}".encode()).digest()[:7], "little"))
        if how[0] == "table":
            return torch.rand(shape[0], how[1], generator=gen, device="cuda").argsort(dim=1)[:, :shape[1]].to(torch.int32)
        mean, dev = how if isinstance(how, tuple) else (1.0 if how == "share" else 0.0, 0.1)
        t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, dev, generator=gen)
        if how == "mixing":
            t += torch.eye(shape[0], device="cuda")
        elif how == "share":
            t /= shape[0]
        return t.to(self.dtype)

    def __getitem__(self, name):
        """The stored values, in 64 bits (``exact``)."""
        return self.read(name).to(torch.float64 if self.what[name][1][0] != "table" else torch.int64)


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


_ROOM = 2048      # single tokens a decode state has room for before it starts over from its prompts


def _room(case):
    return _ROOM if case["batch"] <= 16 else 512


def _tokens(case, cfg, seed):
    """The prompts, and for single tokens the ``_room`` tokens that follow each."""
    gen = torch.Generator()
    gen.manual_seed(seed * 7 + 3)
    more = _room(case) if case["pass"] == "decode" else 0
    return [torch.randint(0, _vocab(cfg), (n + more,), generator=gen).tolist() for n in _lengths(case)]


# ---------------------------------------------------------------------------------------------- one pass

def _start(state):
    """Prompts into fresh slots (at most 16,384 tokens a step), and the first single token, with which the step function
    captures the decode step's graph."""
    from airframe_b200.engine import StepEntry
    rt = state["rt"]
    rt.reset()
    state["slots"] = [rt.engine.take_slot() for _ in state["lens"]]
    entries, held = [], 0
    for s, n, t in zip(state["slots"], state["lens"], state["tokens"]):
        if entries and held + n > 16384:
            rt.step(entries)
            entries, held = [], 0
        entries.append(StepEntry(s, t[:n], []))
        held += n
    rt.step(entries)
    state["done"] = 0
    run(state)


def prepare(case, seed):
    from airframe_b200.config import config_from_dict
    from airframe_b200.engine import Engine, GpuRuntime, Model
    from airframe_b200.weights import load_weights
    cfg = _config(case)
    config = config_from_dict(cfg)
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    model = Model(config.model_spec(), dtype, "cuda:0")
    model.load(load_weights(_Weights(case, cfg, seed), model.weight_decls(), dtype, torch.device("cuda:0")))
    lens = _lengths(case)
    room = _room(case) if case["pass"] == "decode" else 0
    engine = Engine(model, max_tokens=sum((n + room + 63) // 64 * 64 for n in lens), max_context=8192, max_sequences=len(lens))
    state = {"rt": GpuRuntime(config, model, engine), "lens": lens, "tokens": _tokens(case, cfg, seed), "pass": case["pass"], "room": room}
    if case["pass"] == "decode":
        _start(state)
    return state


def run(state):
    from airframe_b200.engine import StepEntry
    rt = state["rt"]
    if state["pass"] == "prompt":
        slots = [rt.engine.take_slot() for _ in state["lens"]]
        logits = rt.step([StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, state["tokens"])])
        for s in slots:
            rt.engine.free_slot(s)
        return logits
    if state["done"] == state["room"]:
        _start(state)
    k = state["done"]
    state["done"] = k + 1
    return rt.step([StepEntry(s, [t[n + k]], [0]) for s, n, t in zip(state["slots"], state["lens"], state["tokens"])])


# ---------------------------------------------------------------------------------------------- what a pass cannot do without

def _mixers(cfg):
    """(type, mixer) of every run of a layer, branches apart."""
    if "hidden_size" in cfg:
        m = {"heads": cfg["num_attention_heads"], "kv_heads": cfg["num_key_value_heads"], "dim": cfg["head_dim"], "vdim": cfg["head_dim"]}
        return [("attention", dict(m, mask={"size": cfg["sliding_window"]}) if i % 2 == 0 else m) for i in range(cfg["num_hidden_layers"])]
    out = []
    for i in _order(cfg):
        t, m = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"]
        if t == "parallel":
            out += [("attention", m["left"]), ("scan", m["right"]) if "heads" in m["right"] else ("vector", m["right"])]
        else:
            out.append((t, m))
    return out


def _order(cfg):
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return list(range(n))
    return list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def work(case):
    cfg = _config(case)
    size = 4 if case["dtype"] == "float32" else 2
    lens = _lengths(case)
    rows = sum(lens) if case["pass"] == "prompt" else len(lens)
    tied = "head" not in _tensors(cfg)
    times = {}
    for i in (_order(cfg) if "layers" in cfg else []):
        times[i] = times.get(i, 0) + 1
    bytes_, flops = 0.0, 0.0
    for name, (shape, how) in _tensors(cfg).items():
        n = math.prod(shape)
        if name in ("embed", "model.embed_tokens.weight", "head"):
            if name == "head" or tied:
                bytes_ += n * size
                flops += 2.0 * n * len(lens)
            continue
        if name == "side.embed" or name.endswith("table"):
            continue
        share = 1.0                                # of the tokens that use it
        if ".mlp.e" in name:
            f = cfg["layers"][0]["mlp"]["router"]
            share = f["top"] / f["experts"]
        used = 1.0 - (1.0 - share) ** rows if share < 1.0 else 1.0
        again = times.get(int(name[1:name.index(".")]), 1) if name[0] == "l" and name[1].isdigit() else 2 if name == "loop.in" else 1
        bytes_ += n * size * used
        if len(shape) >= 2 and "conv" not in name and "hc" not in name and name != "loop.step":
            flops += 2.0 * n * share * rows * again
    for t, m in _mixers(cfg):
        for n in lens:
            if t in ("attention", "latent_attention"):
                size_of = (m.get("mask") or {}).get("size") or 1 << 30
                maps = 2 if "diff" in m else 1
                dk = m["dim"] + m.get("rot_dim", 0)
                if case["pass"] == "prompt":
                    w = min(n, size_of)
                    seen = w * (w + 1) / 2 + (n - w) * w
                else:
                    seen = min(n + 2, size_of)
                    row = m["kv_rank"] + m["rot_dim"] if "kv_rank" in m else m["kv_heads"] * (maps * m["dim"] + m["vdim"])
                    bytes_ += seen * row * size
                flops += 2.0 * seen * maps * m["heads"] * (dk + m["vdim"])
            else:
                heads = m.get("heads", 1)
                cell = m["dim"] * m.get("vdim", m["dim"]) if "dim" in m else m["width"]
                steps = n if case["pass"] == "prompt" else 1
                flops += (4.0 if t in ("gla", "retention", "scan") else 6.0) * steps * heads * cell
                if case["pass"] == "decode":
                    bytes_ += 8.0 * heads * cell       # the state, in 32 bits, read and written
    bytes_ += 4.0 * len(lens) * _vocab(cfg)            # the logits
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # 32-bit: sums of up to 9,216 products in another order, through the layers; bfloat16: every matrix product rounds its
    # inputs to 8 bits, and a path that rounds the same values elsewhere ends up about that far away
    return {"rel": 2e-5, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.3}


# ---------------------------------------------------------------------------------------------- the same in 64 bits

def _rms(x, eps, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _layer_norm(x, w, b, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu(z):
    return z * torch.sigmoid(z)


def _frequencies(rot):
    """Angles a position, and the factor on cosines and sines: plain, stretched by a ramp over the dimensions, or by
    wavelength."""
    base, dims, s = float(rot["base"]), rot["dims"], rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    mag = 1.0
    if s and "fast" in s:
        lo, hi = (dims * math.log(s["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base)) for t in (s["fast"], s["slow"]))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f = [a / s["factor"] * r + a * (1.0 - r) for a, r in zip(f, ramp)]
        mag = 0.1 * math.log(s["factor"]) + 1.0
    elif s:
        for i, a in enumerate(f):
            share = (s["original"] * a / (2.0 * math.pi) - s["low"]) / (s["high"] - s["low"])
            share = min(max(share, 0.0), 1.0)
            f[i] = (1.0 - share) * a / s["factor"] + share * a
    return torch.tensor(f, dtype=torch.float64, device="cuda"), mag


def _rotate(x, rot, neighbours=False):
    """x [T, heads, d] at positions 0 .. T - 1."""
    f, mag = _frequencies(rot)
    n = f.numel()
    ang = torch.arange(x.shape[0], dtype=torch.float64, device="cuda")[:, None, None] * f
    c, s = ang.cos() * mag, ang.sin() * mag
    if neighbours:
        a, b = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        turned = torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)
    else:
        a, b = x[..., :n], x[..., n:2 * n]
        turned = torch.cat([a * c - b * s, b * c + a * s], dim=-1)
    return torch.cat([turned, x[..., 2 * n:]], dim=-1)


def _attend(q, k, v, scale, cap=None, size=None, chunk=False, keep=0, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    hidden = j > i
    if size is not None:
        hidden = hidden | (i // size != j // size) if chunk else hidden | ((i - j >= size) & (j >= keep))
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], dim=1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[:, h * G // H])
    return torch.stack(out, dim=1)


def _delta(W, x, m, eps, h):
    """The generalized delta rule (Fiferax)."""
    T, H, d = h.shape[0], m["heads"], m["dim"]
    r, k, v = ((h @ W[x + n].T).view(T, H, d) for n in "rkv")
    w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ W[x + "w1"].T) @ W[x + "w2"].T + W[x + "w0"])).view(T, H, d)
    a = torch.sigmoid(h @ W[x + "a"].T + W[x + "a.b"]).view(T, H, d)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S, out = torch.zeros(H, d, d, dtype=h.dtype, device="cuda"), []
    for t in range(T):
        S = w[t, :, :, None] * S - (a[t] * u[t])[:, :, None] * (u[t, :, None] @ S) + k[t, :, :, None] * v[t, :, None]
        out.append((r[t, :, None] @ S)[:, 0])
    o = _rms(torch.stack(out), eps).reshape(T, H * d) * W[x + "norm"] * torch.sigmoid(h @ W[x + "g"].T)
    return o @ W[x + "o"].T


def _decayed(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q; decay [T or 1, H, dk or 1]."""
    S, out = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=q.dtype, device="cuda"), []
    for t in range(q.shape[0]):
        S = decay[t if decay.shape[0] > 1 else 0][:, :, None] * S + k[t, :, :, None] * v[t, :, None]
        out.append((q[t, :, None] @ S)[:, 0])
    return torch.stack(out)


def _latent(W, x, m, eps, h, neighbours=False, sink=False, gate=None):
    T, H, d, r, dv, c = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    q = (_rms(h @ W[x + "dq"].T, eps, W[x + "dq.norm"]) @ W[x + "uq"].T if m.get("q_rank") else h @ W[x + "q"].T).view(T, H, d + r)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"], neighbours)], -1)
    down = h @ W[x + "dkv"].T
    lat = _rms(down[:, :c], eps, W[x + "dkv.norm"])
    shared = _rotate(down[:, None, c:], m["rot"], neighbours).expand(T, H, r)
    k = torch.cat([(lat @ W[x + "uk"].T).view(T, H, d), shared], -1)
    o = _attend(q, k, (lat @ W[x + "uv"].T).view(T, H, dv), m["scale"], size=(m.get("mask") or {}).get("size"), sink=W[x + "sink"] if sink else None)
    if gate == "head":
        o = o * torch.sigmoid(h @ W[x + "g"].T)[..., None]
    o = o.reshape(T, H * dv)
    if gate == "value":
        o = o * torch.sigmoid(h @ W[x + "g"].T)
    return o @ W[x + "o"].T


def _gated(W, p, h, act):
    return (act(h @ W[p + "gate"].T) * (h @ W[p + "up"].T)) @ W[p + "down"].T


def _conv(x, w):
    taps = w.shape[1]
    pad = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=x.dtype, device="cuda"), x])
    return sum(pad[j:j + x.shape[0]] * w[:, j] for j in range(taps))


def _gemma2(W, cfg, ids):
    eps, H, G, d = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    table, T = W["model.embed_tokens.weight"], len(ids)
    x = table[ids] * math.sqrt(cfg["hidden_size"])
    rot = {"base": cfg["rope_theta"], "dims": d}

    def norm(y, name):
        return _rms(y, eps, 1.0 + W[name + ".weight"])

    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm")
        q, k, v = ((h @ W[p + f"self_attn.{n}_proj.weight"].T).view(T, -1, d) for n in "qkv")
        o = _attend(_rotate(q, rot), _rotate(k, rot), v, cfg["query_pre_attn_scalar"] ** -0.5, cap=cfg["attn_logit_softcapping"],
                    size=cfg["sliding_window"] if i % 2 == 0 else None)
        x = x + norm(o.reshape(T, H * d) @ W[p + "self_attn.o_proj.weight"].T, p + "post_attention_layernorm")
        h = norm(x, p + "pre_feedforward_layernorm")
        f = (_gelu(h @ W[p + "mlp.gate_proj.weight"].T) * (h @ W[p + "mlp.up_proj.weight"].T)) @ W[p + "mlp.down_proj.weight"].T
        x = x + norm(f, p + "post_feedforward_layernorm")
    cap = cfg["final_logit_softcapping"]
    return cap * torch.tanh((norm(x[-1], "model.norm") @ table.T) / cap)


def _fiferax(W, cfg, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = W["embed"][ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        h = _rms(x, eps, W[f"l{i}.norm1"])
        if layer["type"] == "general_delta":
            y = _delta(W, p, m, eps, h)
        elif layer["type"] == "parallel":
            L, R = m["left"], m["right"]
            q, k = ((h @ W[p + "left." + n].T).view(T, -1, L["dim"]) for n in "qk")
            o = _attend(_rotate(_rms(q, eps, W[p + "left.q.norm"]), L["rot"]), _rotate(_rms(k, eps, W[p + "left.k.norm"]), L["rot"]), k,
                        L["scale"], size=L["mask"]["size"])
            y = m["left_scale"] * (o.reshape(T, -1) @ W[p + "left.o"].T)
            q, k, v = (_silu(h @ W[p + "right." + n].T).view(T, R["heads"], -1) for n in "qkv")
            o = _decayed(q, k, v, torch.tensor(R["decay"], dtype=h.dtype, device="cuda")[None, :, None])
            o = _rms(o.reshape(T, -1), eps, W[p + "right.norm"]) * torch.sigmoid(h @ W[p + "right.g"].T)
            y = y + m["right_scale"] * (o @ W[p + "right.o"].T)
        else:
            z = torch.sigmoid(h @ W[p + "z"].T + W[p + "z.b"])
            u = h @ W[p + "x"].T + W[p + "x.b"]
            c = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            S, out = torch.zeros_like(z[0]), []
            for t in range(T):
                S = (1.0 - z[t]) * S + z[t] * c[t]
                out.append(S)
            y = (torch.stack(out) * _silu(h @ W[p + "g"].T)) @ W[p + "o"].T
        x = x + y
        if layer["mlp"]:
            x = x + _gated(W, f"l{i}.mlp.", _rms(x, eps, W[f"l{i}.norm2"]), _gelu)
    return _rms(x[-1], eps, W["final.norm"]) @ W["head"].T


def _banitar(W, cfg, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x0 = x = W["embed"][ids] * cfg["embedding"]["scale"]
    entered = 0

    def norm(y, name):
        return torch.tanh(W[name + ".alpha"] * y) * W[name] + W[name + ".b"]

    for i in _order(cfg):
        if i == cfg["loop"]["start"]:
            x = torch.cat([x, x0], -1) @ W["loop.in"].T + W["loop.step"][entered]
            entered += 1
        p, m = f"l{i}.mix.", cfg["layers"][i]["mixer"]
        h = norm(x, f"l{i}.norm1")
        if cfg["layers"][i]["type"] == "attention":
            q, k, v = ((h @ W[p + n].T + W[p + n + ".b"]).view(T, -1, m["dim"]) for n in "qkv")
            q, k = (_rms(_rotate(y, m["rot"], True), eps) for y in (q, k))
            o = _attend(q, k, v, m["scale"], size=m["mask"]["size"], chunk=True) * torch.sigmoid(h @ W[p + "g"].T)[..., None]
            y = o.reshape(T, -1) @ W[p + "o"].T
        else:
            y = _latent(W, p, m, eps, h, sink=True)
        x = x + norm(y, f"l{i}.norm1b")
        x = x + norm(_gated(W, f"l{i}.mlp.", norm(x, f"l{i}.norm2"), _silu), f"l{i}.norm2b")
    return norm(x[-1], "final.norm") @ W["head"].T


def _zatasun(W, cfg, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = _rms(W["embed"][ids], eps, W["embed.norm"])
    for i, layer in enumerate(cfg["layers"]):
        p, L, R = f"l{i}.mix.left.", layer["mixer"]["left"], layer["mixer"]["right"]
        q = _rms(x @ W[p + "q"].T, eps, W[p + "q.norm"]).view(T, -1, L["dim"])
        k = _rms(x @ W[p + "k"].T, eps, W[p + "k.norm"]).view(T, -1, L["dim"])
        v = (x @ W[p + "v"].T).view(T, -1, L["vdim"])
        o = _attend(_rotate(q, L["rot"]), _rotate(k, L["rot"]), v, L["scale"], sink=W[p + "sink"])
        y = layer["mixer"]["left_scale"] * (o.reshape(T, -1) @ W[p + "o"].T)
        p, n, b = f"l{i}.mix.right.", R["width"], R["blocks"]
        u = _conv(x @ W[p + "x"].T + W[p + "x.b"], W[p + "conv"]) + W[p + "conv.b"]
        r, g = (torch.sigmoid(torch.einsum("boi,tbi->tbo", W[p + k], u.view(T, b, n // b)) + W[p + k + ".b"]).reshape(T, n) for k in ("ra", "ri"))
        a = torch.exp(-8.0 * r * torch.nn.functional.softplus(W[p + "lam"]))
        add = torch.sqrt(1.0 - a * a) * g * u
        S, out = torch.zeros_like(u[0]), []
        for t in range(T):
            S = a[t] * S + add[t]
            out.append(S)
        y = y + layer["mixer"]["right_scale"] * ((torch.stack(out) * _gelu(x @ W[p + "y"].T + W[p + "y.b"])) @ W[p + "o"].T)
        x = x + _rms(y, eps, W[f"l{i}.norm1"])
        x = x + _rms(_gated(W, f"l{i}.mlp.", x, _silu), eps, W[f"l{i}.norm2"])
    return (_rms(x[-1], eps, W["final.norm"]) @ W["embed"].T) * cfg["logit_scale"]


def _tarorax(W, cfg, ids):
    eps, T, n = cfg["norm"]["eps"], len(ids), cfg["streams"]
    X = W["embed"][ids].expand(n, T, -1)
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        for k in "12":
            h = _rms(torch.einsum("s,stw->tw", W[f"l{i}.hc{k}.in"], X), eps, 1.0 + W[f"l{i}.norm{k}"])
            if k == "2":
                y = _gated(W, f"l{i}.mlp.", h, _gelu)
            elif layer["type"] == "gla":
                H, d, dv = m["heads"], m["dim"], m["vdim"]
                z = (h @ W[p + "a1"].T) @ W[p + "a2"].T + W[p + "a2.b"]
                decay = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(T, H, d)
                o = _decayed((h @ W[p + "q"].T).view(T, H, d) * d ** -0.5, (h @ W[p + "k"].T).view(T, H, d), (h @ W[p + "v"].T).view(T, H, dv), decay)
                y = ((_rms(o, eps) * W[p + "norm"]).reshape(T, -1) * _silu(h @ W[p + "g"].T)) @ W[p + "o"].T
            else:
                H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
                q, kk, v = (_conv(h @ W[p + j].T + W[p + j + ".b"], W[p + j + ".conv"]) for j in "qkv")
                temp = torch.tensor([1.0 + m["q_temp"]["coef"] * math.log((t + 1) // m["q_temp"]["every"] + 1) for t in range(T)], dtype=h.dtype, device="cuda")
                q, kk, v = (q * temp[:, None]).view(T, H, 2, d), kk.view(T, G, 2, d), v.view(T, G, dv)
                lam = math.exp((W[p + "lq1"] * W[p + "lk1"]).sum()) - math.exp((W[p + "lq2"] * W[p + "lk2"]).sum()) + m["diff"]
                a, b = (_attend(q[:, :, j], kk[:, :, j], v, m["scale"], cap=m["softcap"]) for j in (0, 1))
                y = (_rms(a - lam * b, eps) * (1.0 - m["diff"])).reshape(T, -1) * torch.sigmoid(h @ W[p + "g"].T)
                y = y @ W[p + "o"].T + W[p + "o.b"]
            y = y * W[f"l{i}.ls{k}"]
            X = torch.einsum("st,srw->trw", W[f"l{i}.hc{k}.mix"], X) + W[f"l{i}.hc{k}.out"][:, None, None] * y
    return _rms(X.sum(0)[-1], eps, 1.0 + W["final.norm"]) @ W["embed"].T


def _teselix(W, cfg, ids):
    eps, alpha, T = cfg["norm"]["eps"], cfg["postln_alpha"], len(ids)
    x = W["embed"][ids]

    def clamped(p, h, limit):
        g, u = (h @ W[p + "gate"].T).clamp(max=limit), (h @ W[p + "up"].T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W[p + "down"].T

    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        h = x + (torch.cat([torch.zeros_like(x[:1]), x[:-1]]) - x) * W[f"l{i}.shift"]
        if layer["type"] == "retention":
            H, d = m["heads"], m["dim"]
            q, k = (_rotate((h @ W[p + n].T).view(T, H, d), m["rot"]) for n in "qk")
            o = _decayed(q, k * d ** -0.5, (h @ W[p + "v"].T).view(T, H, -1), torch.tensor(m["decay"], dtype=h.dtype, device="cuda")[None, :, None])
            y = (_rms(o, eps).reshape(T, -1) * _silu(h @ W[p + "g"].T)) @ W[p + "o"].T
        else:
            y = _latent(W, p, m, eps, h, neighbours=True, sink=True, gate="head")
        y = y * torch.sigmoid(x @ W[f"l{i}.rg1"].T + W[f"l{i}.rg1.b"])
        x = _layer_norm(alpha * x + y, W[f"l{i}.norm1"], W[f"l{i}.norm1.b"], eps)
        p, limit = f"l{i}.mlp.", f["expert"]["limit"]
        y = clamped(p + "shared.", x, limit)
        chosen = W[p + "table"][ids]
        for e in range(f["router"]["experts"]):
            rows = (chosen == e).any(1).nonzero()[:, 0]
            y[rows] += clamped(f"{p}e{e}.", x[rows], limit) / f["router"]["top"]
        y = y * torch.sigmoid(x @ W[f"l{i}.rg2"].T + W[f"l{i}.rg2.b"])
        x = _layer_norm(alpha * x + y, W[f"l{i}.norm2"], W[f"l{i}.norm2.b"], eps)
    return _layer_norm(x[-1], W["final.norm"], W["final.norm.b"], eps) @ W["embed"].T


def _retudra(W, cfg, ids):
    eps, mult, T, side = cfg["norm"]["eps"], cfg["residual_mult"], len(ids), cfg["token_side"]["dim"]
    x = W["embed"][ids]
    own = W["side.embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        if layer["type"] == "channel_delta":
            H, d, dv = m["heads"], m["dim"], m["vdim"]
            q, k, v = (_silu(_conv(x @ W[p + n].T, W[p + n + ".conv"])).view(T, H, -1) for n in "qkv")
            q, k = (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (q, k))
            q = q * d ** -0.5
            beta = torch.sigmoid(x @ W[p + "b"].T)
            z = (x @ W[p + "a1"].T) @ W[p + "a2"].T + W[p + "dt_bias"]
            g = torch.exp(-torch.exp(W[p + "A_log"])[None, :, None] * torch.nn.functional.softplus(z).view(T, H, d))
            S, out = torch.zeros(H, d, dv, dtype=x.dtype, device="cuda"), []
            for t in range(T):
                S = g[t, :, :, None] * S
                u = beta[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
                S = S + k[t, :, :, None] * u[:, None]
                out.append((q[t, :, None] @ S)[:, 0])
            o = (_rms(torch.stack(out), eps) * W[p + "norm"]).reshape(T, -1)
            y = (o * torch.sigmoid((x @ W[p + "g1"].T) @ W[p + "g2"].T)) @ W[p + "o"].T
        elif layer["type"] == "attention":
            q = _rms(x @ W[p + "q"].T, eps, W[p + "q.norm"]).view(T, -1, m["dim"])
            k = _rms(x @ W[p + "k"].T, eps, W[p + "k.norm"]).view(T, -1, m["dim"])
            v = (x @ W[p + "v"].T).view(T, -1, m["vdim"])
            y = _attend(_rotate(q, m["rot"]), _rotate(k, m["rot"]), v, m["scale"], size=m["mask"]["size"], keep=m["mask"]["keep_first"])
            y = y.reshape(T, -1) @ W[p + "o"].T
        else:
            y = _latent(W, p, m, eps, x, gate="value")
        x = x + mult * _layer_norm(y, W[f"l{i}.norm1"], W[f"l{i}.norm1.b"], eps)
        x = x + mult * _layer_norm(_gated(W, f"l{i}.mlp.", x, _silu), W[f"l{i}.norm2"], W[f"l{i}.norm2.b"], eps)
        y = (_gelu(x @ W[f"l{i}.side.gate"].T) * own[:, i * side:(i + 1) * side]) @ W[f"l{i}.side.proj"].T
        x = x + mult * _rms(y, eps, W[f"l{i}.side.norm"])
    z = _layer_norm(x[-1], W["final.norm"], W["final.norm.b"], eps) @ W["head"].T
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


_EXACT = {"gemma2": _gemma2, "fiferax": _fiferax, "banitar": _banitar, "zatasun": _zatasun, "tarorax": _tarorax, "teselix": _teselix,
          "retudra": _retudra}


def exact(case, seed):
    if sum(_lengths(case)) > 18000:
        return None                                    # minutes in 64 bits
    cfg = _config(case)
    W = _Weights(case, cfg, seed)
    more = 2 if case["pass"] == "decode" else 0        # the token prepare() runs, and the first that run() does
    return torch.stack([_EXACT[case["model"]](W, cfg, torch.tensor(t[:n + more], device="cuda"))
                        for n, t in zip(_lengths(case), _tokens(case, cfg, seed))])
