"""The workloads this library is timed on: whole requests through the engine's step function, as
`Engine.generate` and the replay tool issue them.

A pass opens a slot for every prompt of a batch, feeds the prompts in one step, feeds `new` more
tokens to every sequence one step at a time, and closes the slots; it returns the logits that
every step returns. In bfloat16 the tokens after the prompts are given (a replay: rounding
cannot send two runs down different paths); in float32 they are the greedy choices of the run.

Models have random weights at sizes this repository's benchmark and tests use. `exact` is the same
pass in 64 bits: one function for each mechanism of the seven designs, whole sequences at a time.
"""

from __future__ import annotations

import math
import zlib

import numpy as np
import torch

import semantic_aware_adaptive_kv_cache_precision_b200 as sakv
from semantic_aware_adaptive_kv_cache_precision_b200 import sampling
from semantic_aware_adaptive_kv_cache_precision_b200.engine.model import DecoderModel

BLOCK = 64              # the cache counts a sequence's positions in blocks of this many


# -- the models ------------------------------------------------------------------------

def _qwen2(layers, hidden, heads, kv_heads, ff, vocab, tied, positions=32768, theta=1e6, eps=1e-6):
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2",
            "num_hidden_layers": layers, "hidden_size": hidden, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "intermediate_size": ff, "vocab_size": vocab,
            "max_position_embeddings": positions, "rope_theta": theta, "rms_norm_eps": eps,
            "tie_word_embeddings": tied, "hidden_act": "silu", "torch_dtype": "bfloat16",
            "use_sliding_window": False, "eos_token_id": vocab - 1}


QWEN2 = {
    "tiny_a": _qwen2(2, 64, 4, 2, 176, 512, True, 128, 1e4),
    "tiny_b": _qwen2(3, 192, 6, 1, 352, 1000, False, 256, 1e6, 1e-5),
    "1.5b": _qwen2(28, 1536, 12, 2, 8960, 151936, True),
    "7b": _qwen2(28, 3584, 28, 4, 18944, 152064, False),
}


def _tebonex(big):
    w, h = (2048, 16) if big else (1024, 8)
    mlp = {"kind": "dense", "ff": 4 * w}
    delta = {"type": "general_delta", "mlp": mlp,
             "mixer": {"heads": w // 64, "dim": 64, "decay_rank": 64}}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                     "mask": {"size": w // 2}}}
    return {"architecture": "Tebonex", "vocab": 32768, "width": w, "streams": 2,
            "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6}, "initializer_range": 0.02,
            "layers": [delta, delta, att] * 2}


def _venanex(big, routed=True):
    """`routed` False: as many experts as a token chooses, so every token goes to all of them."""
    w, h, q_rank = (2048, 16, 768) if big else (1024, 8, 384)
    experts, top, shared = (32, 4, 4096) if big else (16, 2, 2048)
    experts = experts if routed else top
    mlp = {"kind": "moe", "router": {"experts": experts, "top": top},
           "expert": {"ff": 1024, "limit": 7.0}, "shared": {"ff": shared, "limit": 7.0}}
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512,
                        "q_rank": q_rank, "scale": 192 ** -0.5,
                        "rot": {"base": 10000.0, "dims": 64,
                                "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0,
                                            "slow": 1.0}}}}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": h // 2, "kv_heads": h // 4, "dim": 128, "vdim": 256,
                     "scale": 128 ** -0.5, "diff": 0.3, "mask": {"size": w}}}
    return {"architecture": "Venanex", "vocab": 32768, "width": w, "norm": {"eps": 1e-6},
            "initializer_range": 0.02, "layers": [latent, latent, att] * 2,
            "loop": {"start": 0, "stop": 3, "times": 1}}


def _zodirax(big):
    w, h = (2048, 16) if big else (1024, 8)
    f = 2 * h
    mlp = {"kind": "dense", "ff": 4 * w}
    scan = {"type": "mamba1", "mlp": mlp,
            "mixer": {"inner": 2 * w, "state": 16, "dt_rank": w // 16, "conv": 4}}
    left = {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
            "mask": {"size": w // 2, "keep_first": 4},
            "rot": {"base": 10000.0, "dims": 64,
                    "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    right = {"heads": f, "dim": 64, "vdim": 64, "decay": [1.0 - 2.0 ** -(2 + 8 * i / f) for i in range(f)]}
    both = {"type": "parallel", "mlp": mlp,
            "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}}
    return {"architecture": "Zodirax", "vocab": 32768, "width": w, "embedding": {"scale": 1.0},
            "norm": {"eps": 1e-6}, "initializer_range": 0.02, "layers": [scan, scan, both] * 2}


def _gesuvik(big):
    w, h = (2048, 16) if big else (1024, 8)
    experts, identity, top, shared = (32, 4, 4, 4096) if big else (16, 2, 2, 2048)
    mlp = {"kind": "moe", "router": {"experts": experts, "identity": identity, "top": top},
           "expert": {"ff": 1024, "limit": 7.0}, "shared": {"ff": shared, "limit": 7.0}}
    mixers = {
        "retention": {"heads": h, "dim": 128, "vdim": 128,
                      "decay": [1.0 - 2.0 ** -(5 + 6 * i / h) for i in range(h)],
                      "rot": {"base": 1000000.0, "dims": 128}},
        "latent_attention": {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512,
                             "scale": 192 ** -0.5, "mask": {"size": w},
                             "rot": {"base": 10000.0, "dims": 64}},
        "attention": {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                      "mask": {"size": w},
                      "rot": {"base": 1000000.0, "dims": 64,
                              "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0,
                                          "slow": 1.0}}}}
    layers = [{"type": kind, "mixer": mixers[kind], "mlp": mlp} for kind in list(mixers) * 2]
    layers[4]["weights_of"] = 1
    return {"architecture": "Gesuvik", "vocab": 32768, "width": w, "norm": {"eps": 1e-6},
            "logit_scale": 1.0, "logit_softcap": 30.0, "initializer_range": 0.02, "layers": layers}


def _felovik(big, dense=False):
    w, h = (2048, 16) if big else (1024, 8)
    experts, top, groups, keep = (32, 4, 8, 4) if big else (16, 2, 4, 2)
    mixer = {"left": {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                      "q_temp": {"coef": 0.1, "every": 1024}},
             "right": {"heads": w // 32, "vdim": 64, "state": 128, "groups": 1, "conv": 4,
                       "norm_groups": 1}}
    ff = {"kind": "dense", "ff": 4 * w, "limit": 7.0}
    moe = {"kind": "moe", "expert": {"ff": 1024},
           "router": {"experts": experts, "top": top, "groups": {"count": groups, "keep": keep}}}
    return {"architecture": "Felovik", "vocab": 32768, "width": w, "max_positions": 16384,
            "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6}, "postln_alpha": 2.0,
            "initializer_range": 0.02,
            "layers": [{"type": "parallel", "mixer": mixer, "mlp": ff if dense or i % 3 == 0 else moe}
                       for i in range(6)]}


def _gozolix(big, dense=False):
    w, h = (2048, 16) if big else (1024, 8)
    experts, top, groups, keep, shared = (32, 4, 8, 4, 2048) if big else (16, 2, 4, 2, 1024)
    d = 128 if big else 64
    delta = {"heads": 16, "kv_heads": 8, "dim": d, "vdim": d, "conv": 4}
    own = {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
           "softcap": 50.0, "q_temp": {"coef": 0.1, "every": 1024}}
    ff = {"kind": "dense", "ff": 4 * w}
    moe = {"kind": "moe", "expert": {"ff": 1024}, "shared": {"ff": shared},
           "router": {"experts": experts, "top": top, "scale": 2.5,
                      "groups": {"count": groups, "keep": keep}}}
    layers = []
    for i in range(6):
        m = ff if dense or i % 3 == 0 else moe
        layers.append({"type": "delta", "mixer": delta, "mlp": m} if i % 3 < 2 else
                      {"type": "attention", "mixer": own if i < 3 else dict(own, kv_from=2), "mlp": m})
    return {"architecture": "Gozolix", "vocab": 32768, "width": w, "norm": {"eps": 1e-6},
            "initializer_range": 0.02, "layers": layers,
            "embedding": {"scale": 1.0, "bigram": {"buckets": 32749, "mul_prev": 17, "mul_cur": 3}}}


DESIGNS = {"tebonex": _tebonex, "venanex": _venanex, "zodirax": _zodirax, "gesuvik": _gesuvik,
           "felovik": _felovik, "gozolix": _gozolix,
           "venanex_all": lambda big: _venanex(big, False),
           "felovik_dense": lambda big: _felovik(big, True),
           "gozolix_dense": lambda big: _gozolix(big, True)}


def model_of(case) -> dict:
    """The config.json of the case's model."""
    if case["design"] == "qwen2":
        return QWEN2[case["size"]]
    return DESIGNS[case["design"]](case["size"] == "2k")


# -- the cases -------------------------------------------------------------------------

def _case(design, size, batch, longest, new, *, shortest=None, dtype="bfloat16", **more):
    return {**more, "design": design, "size": size, "dtype": dtype, "batch": batch,
            "longest": longest, "shortest": longest if shortest is None else shortest, "new": new}


def listed():
    return [
        # the smallest call: a few short prompts in true 32-bit, as a check of a checkpoint runs
        _case("qwen2", "tiny_b", 4, 64, 16, shortest=1, dtype="float32", name="tiny_float32_greedy"),
        # one user and an ordinary prompt: latency of the first token and of every later one
        _case("qwen2", "1.5b", 1, 2048, 32, name="1.5b_one_user"),
        # a small batch of conversations of unequal lengths
        _case("qwen2", "1.5b", 8, 2048, 32, shortest=256, name="1.5b_batch_8"),
        # a full batch of short requests
        _case("qwen2", "1.5b", 64, 512, 16, shortest=33, name="1.5b_batch_64"),
        # a long document and a short answer
        _case("qwen2", "1.5b", 1, 16384, 16, name="1.5b_long_document"),
        # a larger model, unequal prompts
        _case("qwen2", "7b", 8, 2048, 8, shortest=256, name="7b_batch_8"),
        # the other designs: prompts and answers in the proportions in which they are served
        _case("tebonex", "2k", 1, 2048, 16, name="tebonex_one_user"),
        # (bfloat16 with experts: where one choice of an expert more or less changes a row's logits
        # by a third, as in Venanex and Gozolix with random weights, rounding alone sends two
        # right runs apart; those two run with every expert chosen and without experts)
        _case("venanex_all", "1k", 8, 700, 24, shortest=90, name="venanex_batch_8"),
        _case("zodirax", "2k", 4, 1500, 16, shortest=200, name="zodirax_batch_4"),
        _case("gesuvik", "2k", 1, 3001, 8, name="gesuvik_one_user"),
        _case("felovik", "1k", 16, 500, 32, shortest=17, name="felovik_batch_16"),
        _case("gozolix_dense", "2k", 2, 2048, 16, shortest=1111, name="gozolix_two_users"),
    ]


#: most prompt tokens of a drawn case, all sequences together, by model
ROOM = {"tiny_a": 256, "tiny_b": 512, "1.5b": 12000, "7b": 6000, "1k": 8000, "2k": 6000}


def draw(rng):
    def spread(low, high):                       # over the logarithm of the range
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.random()
    if kind < 0.15:                              # 32-bit: short requests, small and real widths
        design, size = rng.choice([("qwen2", "tiny_a"), ("qwen2", "tiny_b"), ("qwen2", "1.5b"),
                                   ("tebonex", "1k"), ("gozolix", "1k"), ("venanex", "1k")])
        batch, longest = rng.randint(1, 4), spread(4, 96)
        return _case(design, size, batch, longest, rng.randint(1, 16), dtype="float32",
                     shortest=max(1, longest // rng.choice([1, 2, 7])))
    if kind < 0.5:
        design, size = "qwen2", rng.choice(["1.5b", "1.5b", "1.5b", "7b"])
    else:
        design = rng.choice(sorted(d for d in DESIGNS if d not in ("venanex", "gozolix")))
        size = rng.choice(["1k", "2k"])
    batch = spread(1, 64)
    longest = spread(16, min(4096, ROOM[size] // batch)) if batch < ROOM[size] // 16 else 16
    return _case(design, size, batch, longest, rng.randint(1, 32),
                 shortest=max(1, longest // rng.choice([1, 1, 2, 5])))


class _State:
    pass


def _tokens(case, seed):
    """(prompts, the tokens after them [new, batch]) on the host, int32."""
    rng = np.random.default_rng([int(seed), 7])
    vocab = model_of(case).get("vocab") or model_of(case)["vocab_size"]
    sizes = np.linspace(case["shortest"], case["longest"], case["batch"]).round().astype(int) \
        if case["batch"] > 1 else [case["longest"]]
    prompts = [rng.integers(0, vocab, int(n)).astype(np.int32) for n in sizes]
    return prompts, rng.integers(0, vocab, (case["new"], case["batch"])).astype(np.int32)


def prepare(case, seed):
    s = _State()
    prompts, after = _tokens(case, seed)
    room = sum(-(-(len(p) + case["new"]) // BLOCK) * BLOCK for p in prompts)
    s.engine = sakv.Engine(config=dict(model_of(case)), dtype=case["dtype"], random_seed=int(seed),
                           max_batch=case["batch"], max_tokens=room,
                           max_step_tokens=16384).load_weights()
    s.prompts = prompts
    s.after = [torch.from_numpy(row).cuda() for row in after]
    s.greedy = case["dtype"] == "float32"
    s.new = case["new"]
    return s


GREEDY = sampling.SamplingParams()


def run(s):
    engine = s.engine
    slots = engine.open(len(s.prompts))
    try:
        logits, tokens = [engine.step(slots, s.prompts)], []
        for i in range(s.new):
            if s.greedy:
                tokens.append(sampling.choose(logits[-1], GREEDY))
                logits.append(engine.step(slots, device_tokens=tokens[-1]))
            else:
                logits.append(engine.step(slots, device_tokens=s.after[i]))
    finally:
        engine.close(slots)
    out = {"first": logits[0], "later": torch.cat(logits[1:])}
    if s.greedy:
        out["tokens"] = torch.cat(tokens)
    return out


# -- what a pass cannot do without -----------------------------------------------------

def _mixers(config):
    """For every layer call: [(heads, key size, value size, window, bytes a cached position)] of
    its attentions and [(state numbers, operations a token)] of its recurrences."""
    if "num_hidden_layers" in config:
        h, g = config["num_attention_heads"], config["num_key_value_heads"]
        d = config["hidden_size"] // h
        return [([(h, d, d, None, 4 * g * d)], [])] * config["num_hidden_layers"]

    def one(kind, m):
        size = (m.get("mask") or {}).get("size")
        if kind == "latent_attention":      # against the cached latent, or a head's own keys: the
            return [(m["heads"], m["dim"] + m["rot_dim"], m["vdim"], size,      # fewer operations
                     2 * (m["kv_rank"] + m["rot_dim"]))], []
        if kind == "attention":
            maps = 2 if "diff" in m else 1
            return [(m["heads"] * maps, m["dim"], m["vdim"], size,
                     2 * m["kv_heads"] * (maps * m["dim"] + m["vdim"]))], []
        if kind == "mamba1":
            return [], [(m["inner"] * m["state"], 6 * m["inner"] * m["state"])]
        if kind == "dual":
            n = m["heads"] * m["vdim"] * m["state"]
            return [], [(n, 6 * n)]
        n = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
        return [], [(n, (7 if kind in ("delta", "general_delta") else 5) * n)]

    out = []
    for layer in config["layers"]:
        if layer["type"] == "parallel":
            a, _ = one("attention", layer["mixer"]["left"])
            _, r = one("dual" if "state" in layer["mixer"]["right"] else "fading", layer["mixer"]["right"])
            out.append((a, r))
        else:
            out.append(one(layer["type"], layer["mixer"]))
    return out


def work(case):
    config = model_of(case)
    width = 2 if case["dtype"] == "bfloat16" else 4
    prompts, _ = _tokens(case, 0)
    lens, B, new = [len(p) for p in prompts], case["batch"], case["new"]
    T = sum(lens)
    decls = DecoderModel.tensor_decls_of(sakv.config_from_dict(dict(config)).model_spec())
    numel = {d.name: math.prod(d.shape) for d in decls}
    top, experts = 1, 1
    for layer in config.get("layers", []):
        if (layer.get("mlp") or {}).get("kind") == "moe":
            top, experts = layer["mlp"]["router"]["top"], layer["mlp"]["router"]["experts"]
    embed = "model.embed_tokens.weight" if "num_hidden_layers" in config else "embed"
    head = next((n for n in numel if n in ("lm_head.weight", "head")), embed)
    routed = sum(n for name, n in numel.items() if ".mlp.e" in name)
    tables = sum(n for name, n in numel.items() if name in (embed, "pos", "bigram")) \
        - (numel[embed] if head == embed else 0)
    dense = sum(numel.values()) - routed - tables              # the head among them
    if "weights_of" in str(config):
        again = sum(n for name, n in numel.items() if name.startswith("l1.") and ".mlp.e" not in name)
        routed_again = sum(n for name, n in numel.items() if name.startswith("l1.mlp.e"))
    else:
        again = routed_again = 0
    steps = [(T, lens, [0] * B)] + [(B, [1] * B, [n + i for n in lens]) for i in range(new)]
    nbytes = flops = 0.0
    for tokens, counts, held in steps:
        share = min(1.0, tokens * top / experts)
        nbytes += width * (dense + share * routed + tokens * config.get("width", config.get("hidden_size", 0)))
        flops += 2.0 * tokens * (dense - numel[head] + again + (routed + routed_again) * top / experts) \
            + 2.0 * B * numel[head]
        nbytes += 4.0 * B * numel[head] / (config.get("width") or config["hidden_size"])   # the logits
        for attentions, recurrences in _mixers(config):
            for heads, dk, dv, window, row in attentions:
                w = window or (1 << 60)
                for c, h0 in zip(counts, held):
                    if h0 + c <= w:
                        seen = c * h0 + c * (c + 1) / 2
                    else:
                        seen = sum(min(h0 + j + 1, w) for j in range(c))
                    flops += 2.0 * heads * (dk + dv) * seen
                    nbytes += (min(h0, w) + c) * row * width / 2
            for state, ops in recurrences:
                flops += float(ops) * tokens
                nbytes += 4.0 * state * B * (1 if held[0] == 0 else 2)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}
    # the same sequences one by one instead of as a batch: 0.003 to 0.011 at 6 and 28 layers, 0.020
    # at the widths of the 7b model
    return {"rel": 0.03, "max": 0.5}


# -- the same in 64 bits ---------------------------------------------------------------

class _Weights:
    """The tensors of a model with random weights, by name: the values the engine's seeded mode
    puts on the device (a generator a tensor, numbers rounded to bfloat16), as 64-bit numbers."""

    def __init__(self, seed, std):
        self.seed, self.std, self.made = int(seed), std, {}
        self.gen = torch.Generator(device="cuda")

    def __call__(self, name, *shape, init="normal", span=None, keep=True):
        if name in self.made:
            return self.made[name]
        self.gen.manual_seed((self.seed << 32) ^ zlib.crc32(name.encode()))
        if init == "uniform":
            t = torch.rand(shape, generator=self.gen, device="cuda", dtype=torch.float32)
            t = (t * (span[1] - span[0]) + span[0]).to(torch.bfloat16).double()
        else:
            t = torch.empty(math.prod(shape), dtype=torch.float64, device="cuda")
            for begin in range(0, t.numel(), 1 << 26):
                part = t[begin:begin + (1 << 26)]
                noise = torch.randn(part.shape, generator=self.gen, device="cuda") * self.std
                if init == "ones":
                    noise += 1.0
                elif init == "eye":
                    noise = (noise.view(shape) + torch.eye(*shape, device="cuda")).reshape(-1)
                part.copy_(noise.to(torch.bfloat16))
            t = t.view(shape)
        if keep:
            self.made[name] = t
        return t


def _rms(x, w, eps):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _layer_norm(x, w, eps):
    y = x - x.mean(-1, keepdim=True)
    return y * torch.rsqrt((y * y).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _frequencies(rot):
    """Angles a position of a rotation's pairs and the factor on cos and sin; wavelengths may be
    stretched in bands (low, high) or along a ramp over the pairs (fast, slow)."""
    dims, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    size = 1.0
    if sc and "low" in sc:
        for i, v in enumerate(f):
            turns = sc["original"] * v / (2 * math.pi)          # original / wavelength
            s = min(max((turns - sc["low"]) / (sc["high"] - sc["low"]), 0.0), 1.0)
            f[i] = (1 - s) * v / sc["factor"] + s * v
    elif sc:
        pair = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
        for i, v in enumerate(f):
            r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            f[i] = v / sc["factor"] * r + v * (1 - r)
        size = 0.1 * math.log(sc["factor"]) + 1.0
    return torch.tensor(f, dtype=torch.float64, device="cuda"), size


def _turn(x, pos, rot, neighbours=False):
    """x [T, heads, D]: the first `dims` numbers of each head turned by their position's angles,
    pairs (i, i + dims / 2) or, with `neighbours`, (2i, 2i + 1)."""
    f, size = _frequencies(rot)
    a = pos.double()[:, None] * f
    cos, sin = (a.cos() * size)[:, None], (a.sin() * size)[:, None]
    d = rot["dims"]
    out = x.clone()
    at = (slice(0, d, 2), slice(1, d, 2)) if neighbours else (slice(0, d // 2), slice(d // 2, d))
    u, v = x[..., at[0]], x[..., at[1]]
    out[..., at[0]], out[..., at[1]] = u * cos - v * sin, v * cos + u * sin
    return out


class _Batch:
    """The sequences of a pass side by side: tokens in a row, `spans` of them."""

    def __init__(self, seqs):
        self.spans, at = [], 0
        for s in seqs:
            self.spans.append((at, at + len(s)))
            at += len(s)
        self.ids = torch.from_numpy(np.concatenate(seqs).astype(np.int64)).cuda()
        self.pos = torch.cat([torch.arange(b - a, device="cuda") for a, b in self.spans])
        longest = max(b - a for a, b in self.spans)
        self.place = torch.full((len(seqs), longest), -1, dtype=torch.long, device="cuda")
        for i, (a, b) in enumerate(self.spans):
            self.place[i, :b - a] = torch.arange(a, b, device="cuda")

    def before(self, x, back, first=0.0):
        """Rows moved `back` tokens later, `first` where a sequence has none."""
        y = torch.roll(x, back, 0)
        y[self.pos < back] = first
        return y

    def conv(self, x, w, b=None):
        taps = w.shape[1]
        y = sum(self.before(x, taps - 1 - j) * w[:, j] if j < taps - 1 else x * w[:, j]
                for j in range(taps))
        return _silu(y if b is None else y + b)

    def walk(self, step, state, width):
        """step(state, rows, alive) -> (state, out) token by token over all sequences."""
        out = torch.empty((len(self.pos),) + width, dtype=torch.float64, device="cuda")
        for t in range(self.place.shape[1]):
            rows = self.place[:, t].clamp_min(0)
            state, y = step(state, rows)
            alive = self.place[:, t] >= 0
            out[rows[alive]] = y[alive]
        return out

    def attention(self, q, k, v, scale, *, window=None, keep=0, sink=None, cap=None, lose=None):
        """q [T, H, D], k [T, G, D], v [T, G, Dv]; lose(head, distance): what a score loses."""
        H, G = q.shape[1], k.shape[1]
        out = torch.empty((q.shape[0], H, v.shape[2]), dtype=torch.float64, device="cuda")
        for a, b in self.spans:
            for h in range(H):
                kk, vv = k[a:b, h // (H // G)], v[a:b, h // (H // G)]
                for c in range(a, b, 4096):
                    e = min(b, c + 4096)
                    s = q[c:e, h] @ kk[:e - a].T * scale
                    if cap is not None:
                        s = cap * torch.tanh(s / cap)
                    i = torch.arange(c - a, e - a, device="cuda")[:, None]
                    j = torch.arange(e - a, device="cuda")[None]
                    if lose is not None:
                        s = s - lose(h, (i - j).clamp_min(0).double())
                    seen = j <= i
                    if window:
                        seen &= (i - j < window) | (j < keep)
                    s.masked_fill_(~seen, -math.inf)
                    top = s.amax(-1, keepdim=True)
                    if sink is not None:
                        top = top.clamp_min(float(sink[h]))
                    p = torch.exp(s - top)
                    total = p.sum(-1, keepdim=True)
                    if sink is not None:
                        total = total + torch.exp(sink[h] - top)
                    out[c:e, h] = (p @ vv[:e - a]) / total
        return out


def _qwen2_exact(c, w, b):
    H, A, G, I = (c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"],
                  c["intermediate_size"])
    d, eps, n = H // A, c["rms_norm_eps"], len(b.ids)
    rot = {"dims": d, "base": c["rope_theta"]}
    embed = w("model.embed_tokens.weight", c["vocab_size"], H)
    x = embed[b.ids]
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        m = lambda name, *s, **k: w(p + name, *s, keep=False, **k)
        h = _rms(x, m("input_layernorm.weight", H, init="ones"), eps)
        q, k, v = ((h @ m(f"self_attn.{t}_proj.weight", r * d, H).T
                    + m(f"self_attn.{t}_proj.bias", r * d)).view(n, r, d)
                   for t, r in (("q", A), ("k", G), ("v", G)))
        o = b.attention(_turn(q, b.pos, rot), _turn(k, b.pos, rot), v, d ** -0.5)
        x = x + o.reshape(n, A * d) @ m("self_attn.o_proj.weight", H, A * d).T
        h = _rms(x, m("post_attention_layernorm.weight", H, init="ones"), eps)
        for a in range(0, n, 4096):
            g = _silu(h[a:a + 4096] @ m("mlp.gate_proj.weight", I, H).T)
            g *= h[a:a + 4096] @ m("mlp.up_proj.weight", I, H).T
            x[a:a + 4096] += g @ m("mlp.down_proj.weight", H, I).T
    head = embed if c["tie_word_embeddings"] else w("lm_head.weight", c["vocab_size"], H)
    return x, lambda y: _rms(y, w("model.norm.weight", H, init="ones"), eps) @ head.T


def _tebonex_exact(c, w, b):
    W, eps, n, S = c["width"], c["norm"]["eps"], len(b.ids), c["streams"]
    xs = torch.stack([w("embed", c["vocab"], W)[b.ids] * c["embedding"]["scale"]] * S)
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        for part in (1, 2):
            hc = f"{p}hc{part}."
            h = torch.einsum("s,snw->nw", w(hc + "in", S, init="uniform", span=(0.2, 0.8)), xs)
            h = _rms(h, w(f"{p}norm{part}", W, init="ones"), eps)
            if part == 2:
                ff = layer["mlp"]["ff"]
                y = _gelu(h @ w(p + "mlp.up", ff, W).T) @ w(p + "mlp.down", W, ff).T
            else:
                h = h + (b.before(h, 1) - h) * w(p + "shift", W, init="uniform", span=(0.0, 0.8))
                y = (_general_delta if layer["type"] == "general_delta" else _log_distance)(
                    h, w, p + "mix.", m, W, eps, b)
            xs = torch.einsum("st,snw->tnw", w(hc + "mix", S, S, init="eye"), xs) \
                + w(hc + "out", S, init="ones")[:, None, None] * y
    return xs.sum(0), lambda y: _rms(y, w("final.norm", W, init="ones"), eps) @ w("head", c["vocab"], W).T


def _general_delta(h, w, p, m, W, eps, b):
    n, H, D, R = h.shape[0], m["heads"], m["dim"], m["decay_rank"]
    r, k, v = ((h @ w(p + t, H * D, W).T).view(n, H, D) for t in "rkv")
    low = torch.tanh(h @ w(p + "w1", R, W).T) @ w(p + "w2", H * D, R).T
    f = torch.exp(-math.exp(-0.5) * torch.sigmoid(
        low + w(p + "w0", H * D, init="uniform", span=(-6.0, 0.0)))).view(n, H, D)
    a = torch.sigmoid(h @ w(p + "a", H * D, W).T + w(p + "a.b", H * D)).view(n, H, D)
    unit = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = a * unit

    def step(S, t):
        along = torch.einsum("bhk,bhkv->bhv", unit[t], S)
        S = f[t][..., None] * S - au[t][..., None] * along[:, :, None] + k[t][..., None] * v[t][:, :, None]
        return S, torch.einsum("bhkv,bhk->bhv", S, r[t])

    o = b.walk(step, h.new_zeros(len(b.spans), H, D, D), (H, D))
    o = _rms(o, None, eps).reshape(n, H * D) * w(p + "norm", H * D, init="ones")
    return (o * torch.sigmoid(h @ w(p + "g", H * D, W).T)) @ w(p + "o", W, H * D).T


def _log_distance(h, w, p, m, W, eps, b):
    n, H, G, D, Dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = ((h @ w(p + t, r * d, W).T + w(p + t + ".b", r * d)).view(n, r, d)
               for t, r, d in (("q", H, D), ("k", G, D), ("v", G, Dv)))
    slope = w(p + "r1", H, init="uniform", span=(0.0, 2.0))
    rate = w(p + "r2", H, init="uniform", span=(0.1, 0.5))
    o = b.attention(q, k, v, m["scale"], window=m["mask"]["size"],
                    lose=lambda a, dist: slope[a] * torch.log1p(rate[a] * dist))
    o = o * torch.sigmoid(h @ w(p + "g", H, W).T)[..., None]
    return o.reshape(n, H * Dv) @ w(p + "o", W, H * Dv).T + w(p + "o.b", W)


def _clamped(g, u, limit):
    g, u = g.clamp_max(limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _gated(h, w, p, W, ff, limit=None):
    g, u = h @ w(p + "gate", ff, W).T, h @ w(p + "up", ff, W).T
    return (_silu(g) * u if limit is None else _clamped(g, u, limit)) @ w(p + "down", W, ff).T


def _routed(h, w, p, W, mlp, score, *, scale_input=False):
    """Routed experts: score(logits) are the weights; groups of experts, a correction for the
    choice and experts that return their input where the router has them."""
    r, ff, limit = mlp["router"], mlp["expert"]["ff"], mlp["expert"].get("limit")
    total = r["experts"] + r.get("identity", 0)
    s = score(h @ w(p + "router", total, W).T)
    choice = s + w(p + "correction", total) if "identity" in r else s
    groups = r.get("groups")
    if groups:
        part = s.view(len(s), groups["count"], -1)
        best = part.topk(2, -1).values.sum(-1) if "scale" in r else part.amax(-1)
        open_ = torch.zeros_like(best, dtype=torch.bool).scatter_(
            1, best.topk(groups["keep"], -1).indices, True)
        choice = s.masked_fill(~open_.repeat_interleave(total // groups["count"], 1), -math.inf)
    chosen = choice.topk(r["top"], -1).indices
    weight = s.gather(1, chosen)
    if groups:
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20) * r.get("scale", 1.0)
    out = torch.zeros_like(h)
    for e in range(total):
        rows, place = torch.nonzero(chosen == e, as_tuple=True)
        if len(rows):
            x, f = h[rows], weight[rows, place][:, None]
            if e >= r["experts"]:
                y = f * x
            elif scale_input:
                y = _gated(f * x, w, f"{p}e{e}.", W, ff, limit)
            else:
                y = f * _gated(x, w, f"{p}e{e}.", W, ff, limit)
            out.index_add_(0, rows, y)
    return out


def _latent(h, w, p, m, W, eps, b, neighbours):
    n, H, D, R, Dv, C = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    if m.get("q_rank"):
        low = _rms(h @ w(p + "dq", m["q_rank"], W).T, w(p + "dq.norm", m["q_rank"], init="ones"), eps)
        q = low @ w(p + "uq", H * (D + R), m["q_rank"]).T
    else:
        q = h @ w(p + "q", H * (D + R), W).T
    q = q.view(n, H, D + R)
    q = torch.cat([q[..., :D], _turn(q[..., D:], b.pos, m["rot"], neighbours)], -1)
    down = h @ w(p + "dkv", C + R, W).T
    lat = _rms(down[:, :C], w(p + "dkv.norm", C, init="ones"), eps)
    shared = _turn(down[:, None, C:], b.pos, m["rot"], neighbours).expand(n, H, R)
    k = torch.cat([(lat @ w(p + "uk", H * D, C).T).view(n, H, D), shared], -1)
    v = (lat @ w(p + "uv", H * Dv, C).T).view(n, H, Dv)
    if not neighbours:
        return b.attention(q, k, v, m["scale"]).reshape(n, H * Dv) @ w(p + "o", W, H * Dv).T
    o = b.attention(q, k, v, m["scale"], window=m["mask"]["size"], sink=w(p + "sink", H))
    o = o * torch.sigmoid(h @ w(p + "g", H, W).T)[..., None]
    return o.reshape(n, H * Dv) @ w(p + "o", W, H * Dv).T


def _differential(h, w, p, m, W, eps, b):
    n, H, G, D, Dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q = (h @ w(p + "q", H * 2 * D, W).T).view(n, H, 2, D)
    k = (h @ w(p + "k", G * 2 * D, W).T).view(n, G, 2, D)
    v = (h @ w(p + "v", G * Dv, W).T).view(n, G, Dv)
    lam = (torch.exp((w(p + "lq1", D) * w(p + "lk1", D)).sum())
           - torch.exp((w(p + "lq2", D) * w(p + "lk2", D)).sum()) + m["diff"])
    size, o = m["mask"]["size"], []
    for j in (0, 1):       # chunks of positions: sequences of their own
        whole, cut = b.spans, [(s, min(s + size, e)) for a, e in b.spans for s in range(a, e, size)]
        b.spans = cut
        o.append(b.attention(q[:, :, j], k[:, :, j], v, m["scale"]))
        b.spans = whole
    o = _rms(o[0] - lam * o[1], None, eps).reshape(n, H * Dv) * (1.0 - m["diff"])
    return (o * torch.sigmoid(h @ w(p + "g", H * Dv, W).T)) @ w(p + "o", W, H * Dv).T


def _venanex_exact(c, w, b):
    W, eps, n = c["width"], c["norm"]["eps"], len(b.ids)
    embed = w("embed", c["vocab"], W)
    x0 = embed[b.ids]
    x = x0
    for i, layer in enumerate(c["layers"]):       # the loop runs once
        p, mlp = f"l{i}.", layer["mlp"]
        if i == c["loop"]["start"]:
            x = torch.cat([x, x0], -1) @ w("loop.in", W, 2 * W).T
        h = _layer_norm(x, w(p + "norm1", W, init="ones"), eps)
        y = _latent(h, w, p + "mix.", layer["mixer"], W, eps, b, False) \
            if layer["type"] == "latent_attention" else _differential(h, w, p + "mix.", layer["mixer"], W, eps, b)
        x = x + _layer_norm(y, w(p + "norm1b", W, init="ones"), eps)
        h = _layer_norm(x, w(p + "norm2", W, init="ones"), eps)
        q = p + "mlp."
        y = _routed(h, w, q, W, mlp, torch.sigmoid, scale_input=True) \
            + _gated(h, w, q + "shared.", W, mlp["shared"]["ff"], mlp["shared"]["limit"]) \
            * torch.sigmoid(h @ w(q + "shared.sg", 1, W).T)
        x = x + _layer_norm(y, w(p + "norm2b", W, init="ones"), eps)
    return x, lambda y: _layer_norm(y, w("final.norm", W, init="ones"), eps) @ embed.T


def _selective_scan(h, w, p, m, W, b):
    n, E, N, R = h.shape[0], m["inner"], m["state"], m["dt_rank"]
    xz = h @ w(p + "in", 2 * E, W).T
    x = b.conv(xz[:, :E], w(p + "conv", E, m["conv"]), w(p + "conv.b", E))
    low = x @ w(p + "x", R + 2 * N, E).T
    dt = torch.nn.functional.softplus(
        low[:, :R] @ w(p + "dt", E, R).T + w(p + "dt.b", E, init="uniform", span=(-4.0, -1.0)))
    A = -torch.exp(w(p + "A_log", E, N, init="uniform", span=(-3.0, 1.0)))
    B, C = low[:, R:R + N], low[:, R + N:]
    u = dt * x

    def step(S, t):
        S = torch.exp(dt[t][..., None] * A) * S + u[t][..., None] * B[t][:, None]
        return S, torch.einsum("ben,bn->be", S, C[t])

    y = b.walk(step, h.new_zeros(len(b.spans), E, N), (E,)) + w(p + "D", E, init="ones") * x
    return (y * _silu(xz[:, E:])) @ w(p + "o", W, E).T


def _fading(q, k, v, decay, b):
    f = torch.tensor(decay, dtype=torch.float64, device="cuda")[None, :, None, None]

    def step(S, t):
        S = f * S + k[t][..., None] * v[t][:, :, None]
        return S, torch.einsum("bhkv,bhk->bhv", S, q[t])

    H, D, Dv = q.shape[1], q.shape[2], v.shape[2]
    return b.walk(step, q.new_zeros(len(b.spans), H, D, Dv), (H, Dv))


def _zodirax_exact(c, w, b):
    W, eps, n = c["width"], c["norm"]["eps"], len(b.ids)
    embed = w("embed", c["vocab"], W)
    x = embed[b.ids] * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        if layer["type"] == "mamba1":
            y = _selective_scan(x, w, p + "mix.", m, W, b)
        else:
            l, q = m["left"], p + "mix.left."
            H, G, D, Dv = l["heads"], l["kv_heads"], l["dim"], l["vdim"]
            qq = _rms(x @ w(q + "q", H * D, W).T + w(q + "q.b", H * D), w(q + "q.norm", H * D, init="ones"), eps)
            kk = _rms(x @ w(q + "k", G * D, W).T + w(q + "k.b", G * D), w(q + "k.norm", G * D, init="ones"), eps)
            vv = (x @ w(q + "v", G * Dv, W).T + w(q + "v.b", G * Dv)).view(n, G, Dv)
            o = b.attention(_turn(qq.view(n, H, D), b.pos, l["rot"]), _turn(kk.view(n, G, D), b.pos, l["rot"]),
                            vv, l["scale"], window=l["mask"]["size"], keep=l["mask"]["keep_first"],
                            sink=w(q + "sink", H))
            y = o.reshape(n, H * Dv) @ w(q + "o", W, H * Dv).T * m["left_scale"]
            r, q = m["right"], p + "mix.right."
            H, D, Dv = r["heads"], r["dim"], r["vdim"]
            qq, kk, vv = (_silu(x @ w(q + t, H * d, W).T).view(n, H, d)
                          for t, d in (("q", D), ("k", D), ("v", Dv)))
            o = _fading(qq, kk, vv, r["decay"], b).reshape(n, H * Dv)
            o = _rms(o, w(q + "norm", H * Dv, init="ones"), eps) * torch.sigmoid(x @ w(q + "g", H * Dv, W).T)
            y = y + o @ w(q + "o", W, H * Dv).T * m["right_scale"]
        x = x + _rms(y, 1.0 + w(p + "norm1", W), eps)
        y = _gated(x, w, p + "mlp.", W, layer["mlp"]["ff"])
        x = x + _rms(y, 1.0 + w(p + "norm2", W), eps)
    return x, lambda y: _rms(y, 1.0 + w("final.norm", W), eps) @ embed.T


def _gesuvik_exact(c, w, b):
    W, eps, n = c["width"], c["norm"]["eps"], len(b.ids)
    x = w("embed", c["vocab"], W)[b.ids]
    for i, layer in enumerate(c["layers"]):
        p, m, mlp = f"l{layer.get('weights_of', i)}.", layer["mixer"], layer["mlp"]
        q = p + "mix."
        h = _rms(x, w(p + "norm1", W, init="ones"), eps)
        if layer["type"] == "latent_attention":
            y = _latent(h, w, q, m, W, eps, b, True)
        elif layer["type"] == "retention":
            H, D, Dv = m["heads"], m["dim"], m["vdim"]
            qq, kk, vv = ((h @ w(q + t, H * d, W).T).view(n, H, d) for t, d in (("q", D), ("k", D), ("v", Dv)))
            o = _fading(_turn(qq, b.pos, m["rot"]), _turn(kk, b.pos, m["rot"]) * D ** -0.5, vv, m["decay"], b)
            o = _rms(o, None, eps).reshape(n, H * Dv) * _silu(h @ w(q + "g", H * Dv, W).T)
            y = o @ w(q + "o", W, H * Dv).T
        else:
            H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            qq = _rms(h @ w(q + "q", H * D, W).T, w(q + "q.norm", H * D, init="ones"), eps).view(n, H, D)
            kk = _rms(h @ w(q + "k", G * D, W).T, w(q + "k.norm", G * D, init="ones"), eps).view(n, G, D)
            o = b.attention(_turn(qq, b.pos, m["rot"]), _turn(kk, b.pos, m["rot"]),
                            (h @ w(q + "v", G * Dv, W).T).view(n, G, Dv), m["scale"],
                            window=m["mask"]["size"], sink=w(q + "sink", H))
            y = o.reshape(n, H * Dv) @ w(q + "o", W, H * Dv).T
        x = x + y
        h = _rms(x, w(p + "norm2", W, init="ones"), eps)
        x = x + _routed(h, w, p + "mlp.", W, mlp, lambda z: torch.softmax(z, -1)) \
            + _gated(h, w, p + "mlp.shared.", W, mlp["shared"]["ff"], mlp["shared"]["limit"])

    def head(y):
        z = _rms(y, w("final.norm", W, init="ones"), eps) @ w("head", c["vocab"], W).T * c["logit_scale"]
        return c["logit_softcap"] * torch.tanh(z / c["logit_softcap"])

    return x, head


def _temperature(pos, temp):
    return 1.0 + temp["coef"] * torch.log(torch.floor((pos.double() + 1) / temp["every"]) + 1)


def _felovik_exact(c, w, b):
    W, eps, n = c["width"], c["norm"]["eps"], len(b.ids)
    x = w("embed", c["vocab"], W)[b.ids] * c["embedding"]["scale"] + w("pos", c["max_positions"], W)[b.pos]
    for i, layer in enumerate(c["layers"]):
        p, mlp = f"l{i}.", layer["mlp"]
        m, q = layer["mixer"]["left"], p + "mix.left."
        H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        qq = _rms((x @ w(q + "q", H * D, W).T).view(n, H, D), None, eps) \
            * _temperature(b.pos, m["q_temp"])[:, None, None]
        kk = _rms((x @ w(q + "k", G * D, W).T).view(n, G, D), None, eps)
        o = b.attention(qq, kk, (x @ w(q + "v", G * Dv, W).T).view(n, G, Dv), m["scale"])
        o = o.reshape(n, H * Dv) * torch.sigmoid(x @ w(q + "g", H * Dv, W).T)
        left = _rms(o @ w(q + "o", W, H * Dv).T, w(q + "out", W, init="ones"), eps)
        m, q = layer["mixer"]["right"], p + "mix.right."
        H, Dv, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, ch = H * Dv, H * Dv + 2 * G * N
        z, xbc, dt = (x @ w(q + "in", inner + ch + H, W).T).split([inner, ch, H], 1)
        xbc = b.conv(xbc, w(q + "conv", ch, m["conv"]), w(q + "conv.b", ch))
        xx, B, C = xbc.split([inner, G * N, G * N], 1)
        xx = xx.reshape(n, H, Dv)
        B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        dt = torch.nn.functional.softplus(dt + w(q + "dt_bias", H, init="uniform", span=(-4.0, -1.0)))
        fade = torch.exp(-torch.exp(w(q + "A_log", H, init="uniform", span=(-2.0, 1.0))) * dt)

        def step(S, t):
            S = fade[t][..., None, None] * S + (dt[t][..., None] * B[t])[..., None] * xx[t][:, :, None]
            return S, torch.einsum("bhnv,bhn->bhv", S, C[t])

        y = b.walk(step, x.new_zeros(len(b.spans), H, N, Dv), (H, Dv)) \
            + w(q + "D", H, init="ones")[:, None] * xx
        y = (y.reshape(n, inner) * _silu(z)).view(n, m["norm_groups"], -1)
        y = _rms(y, None, eps).reshape(n, inner) * w(q + "norm", inner, init="ones")
        right = _rms(y @ w(q + "o", W, inner).T, w(q + "out", W, init="ones"), eps)
        x = _rms(c["postln_alpha"] * x + 0.5 * (left + right), w(p + "norm1", W, init="ones"), eps)
        y = _gated(x, w, p + "mlp.", W, mlp["ff"], mlp["limit"]) if mlp["kind"] == "dense" else \
            _routed(x, w, p + "mlp.", W, mlp, lambda z: torch.softmax(z, -1))
        x = _rms(c["postln_alpha"] * x + y, w(p + "norm2", W, init="ones"), eps)
    return x, lambda y: _rms(y, w("final.norm", W, init="ones"), eps) @ w("head", c["vocab"], W).T


def _gozolix_exact(c, w, b):
    W, eps, n = c["width"], c["norm"]["eps"], len(b.ids)
    t2 = c["embedding"]["bigram"]
    pair = (b.before(b.ids, 1) * t2["mul_prev"] + b.ids * t2["mul_cur"]) % t2["buckets"]
    pair[b.pos == 0] = t2["buckets"]
    x = w("embed", c["vocab"], W)[b.ids] * c["embedding"]["scale"] \
        + w("bigram", t2["buckets"] + 1, W)[pair]
    kept = {}
    for i, layer in enumerate(c["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        q = p + "mix."
        h = _rms(x, w(p + "norm1", W, init="ones"), eps)
        H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        if layer["type"] == "delta":
            qq, kk, vv = (b.conv(h @ w(q + t, r * d, W).T,
                                 w(q + t + ".conv", r * d, m["conv"], init="uniform", span=(-0.7, 0.7))).view(n, r, d)
                          for t, r, d in (("q", G, D), ("k", G, D), ("v", H, Dv)))
            unit = lambda y: (y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
            qq, kk = unit(qq) * D ** -0.5, unit(kk)
            beta = torch.sigmoid(h @ w(q + "b", H, W).T)
            fade = torch.exp(-torch.exp(w(q + "A_log", H, init="uniform", span=(-2.0, 1.0)))
                             * torch.nn.functional.softplus(
                                 h @ w(q + "a", H, W).T + w(q + "dt_bias", H, init="uniform", span=(-4.0, -1.0))))

            def step(S, t):
                S = fade[t][..., None, None] * S
                u = beta[t][..., None] * (vv[t] - torch.einsum("bhdv,bhd->bhv", S, kk[t]))
                S = S + kk[t][..., None] * u[:, :, None]
                return S, torch.einsum("bhdv,bhd->bhv", S, qq[t])

            o = b.walk(step, x.new_zeros(len(b.spans), H, D, Dv), (H, Dv))
            o = _rms(o, w(q + "norm", Dv, init="ones"), eps).reshape(n, H * Dv) * _silu(h @ w(q + "g", H * Dv, W).T)
        else:
            qq = (h @ w(q + "q", H * D, W).T + w(q + "q.b", H * D)).view(n, H, D) \
                * _temperature(b.pos, m["q_temp"])[:, None, None]
            if "kv_from" not in m:
                kept[i] = ((h @ w(q + "k", G * D, W).T + w(q + "k.b", G * D)).view(n, G, D),
                           (h @ w(q + "v", G * Dv, W).T + w(q + "v.b", G * Dv)).view(n, G, Dv))
            kk, vv = kept[m.get("kv_from", i)]
            o = b.attention(qq, kk, vv, m["scale"], cap=m["softcap"],
                            lose=lambda a, dist: 2.0 ** (-8.0 * (a + 1) / H) * dist).reshape(n, H * Dv)
        y = o @ w(q + "o", W, H * Dv).T
        q = p + "mlp."
        if mlp["kind"] == "dense":
            y = y + (h @ w(q + "up", mlp["ff"], W).T).clamp_min(0) ** 2 @ w(q + "down", W, mlp["ff"]).T
        else:
            y = y + _routed(h, w, q, W, mlp, torch.sigmoid) + _gated(h, w, q + "shared.", W, mlp["shared"]["ff"])
        x = x + y
    return x, lambda y: _rms(y, w("final.norm", W, init="ones"), eps) @ w("head", c["vocab"], W).T


EXACT = {"qwen2": _qwen2_exact, "tebonex": _tebonex_exact, "venanex": _venanex_exact,
         "zodirax": _zodirax_exact, "gesuvik": _gesuvik_exact, "felovik": _felovik_exact,
         "gozolix": _gozolix_exact}


def exact(case, seed):
    config, new = model_of(case), case["new"]
    prompts, after = _tokens(case, seed)
    weights = _Weights(seed, config.get("initializer_range", 0.02))
    forward = EXACT[case["design"].split("_")[0]]
    greedy = case["dtype"] == "float32"
    chosen = []
    while True:
        extra = np.stack(chosen) if greedy and chosen else after[:0 if greedy else new]
        batch = _Batch([np.concatenate([p, extra[:, i]]) for i, p in enumerate(prompts)])
        x, head = forward(config, weights, batch)
        rows = torch.tensor([[a + len(p) - 1 + j for (a, _), p in zip(batch.spans, prompts)]
                             for j in range(len(extra) + 1)], device="cuda")
        logits = torch.cat([head(x[r]) for r in rows])
        if not greedy or len(chosen) == new:
            break
        chosen.append(logits[-len(prompts):].argmax(-1).int().cpu().numpy())
    B = case["batch"]
    out = {"first": logits[:B], "later": logits[B:]}
    if greedy:
        out["tokens"] = None
    return out
