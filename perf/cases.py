"""The work that this library is measured on: prompts and single-token steps of its seven architectures.

A case names an architecture (at layer sizes of the repository's benchmark), a compute dtype, a kind of pass and the
sequences of the batch.  Weights are seeded random numbers, the same for every case of an architecture, as a program that
serves a model loads it once; token ids come from the seed.  Eight layers of the eight-billion-parameter sizes stand for
all 36, which repeat them: with more of them the rounding of bfloat16 alone moves the logits of random weights by more
than the comparison of two implementations allows.

  prompts   one step of whole prompts on an empty cache (``model.step``): logits of the last token of each prompt, or of
            every token (``want`` "all", scoring a text);
  decode    ``steps`` single-token steps of sequences whose prompts are cached, through the decode runner that
            ``generate`` uses.  The tokens of every step are given: logits are then a function of the inputs alone,
            where sampled tokens would turn a last-bit difference into another text.  For the same reason the logits
            are the output and the sampled tokens are not.

``exact`` restates each architecture in plain 64-bit torch over whole sequences.
"""

import hashlib
import json
import math

import torch

import ondeviceinfer_b200 as odi
from ondeviceinfer_b200.api import ResidentModel, decode_runner
from ondeviceinfer_b200.engine.model import DecoderModel
from ondeviceinfer_b200.registry import config_from_dict
from ondeviceinfer_b200.weights import StoredTensor

F64 = torch.float64
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
WEIGHTS_SEED = 20
PAGE = 64
REQUEST_STEPS = 512       # a request of a decode case ends after so many steps and the next one takes its place


# ------------------------------------------------------------------------------ the cases


def _case(name, design, kind, sequences, shortest, longest, *, layers=4, dtype="bfloat16", steps=4, temperature=0.0, want="last"):
    case = {"design": design, "layers": layers, "dtype": dtype, "kind": kind, "sequences": sequences, "shortest": shortest,
            "longest": longest}
    case.update({"want": want} if kind == "prompts" else {"steps": steps, "temperature": temperature})
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user at a keyboard: a single sequence in the middle of a chat, where launches and latency count
        _case("qwen3_decode_b1", "qwen3", "decode", 1, 300, 300, layers=8),
        # the benchmark's headline: eight sequences behind prompts of 2,048 tokens
        _case("qwen3_decode_b8", "qwen3", "decode", 8, 2048, 2048, layers=8),
        # a full server: 48 users at unequal places, with temperature sampling
        _case("qwen3_decode_b48", "qwen3", "decode", 48, 100, 1000, layers=8, temperature=0.7),
        # short questions that arrive together, ragged and off every tile size
        _case("qwen3_prompts_short", "qwen3", "prompts", 5, 23, 211, layers=8),
        # long documents of unequal length: the largest pass
        _case("qwen3_prompts_long", "qwen3", "prompts", 4, 700, 3001, layers=8),
        # scoring every token of a few texts in true float32, as the replay program does
        _case("qwen3_float32_score", "qwen3", "prompts", 3, 37, 90, dtype="float32", want="all"),
        # one prompt of 2,048 tokens through latent attention, the per-channel delta rule and routed experts
        _case("lemesun_prompt", "lemesun", "prompts", 1, 2048, 2048),
        # eight sequences of windowed, squashed attention and table-routed experts in a looped stack
        _case("nulalorn_decode_b8", "nulalorn", "decode", 8, 500, 2048),
        # sixteen sequences of parallel blocks: latent rows shared between layers, attention with a sink
        _case("zigivik_decode_b16", "zigivik", "decode", 16, 128, 1500),
        # one prompt of 2,048 tokens: kept first keys beside the state-space scan, sigmoid-routed experts
        _case("losivik_prompt", "losivik", "prompts", 1, 2048, 2048),
        # three prompts of unequal length: chunked attention with mixed heads beside layers of the per-head delta rule
        _case("noganex_prompts", "noganex", "prompts", 3, 333, 1777),
        # four prompts of a few hundred tokens: parallel streams, biased attention beside retention
        _case("pukinex_prompts", "pukinex", "prompts", 4, 150, 900),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """Any architecture, either direction; lengths and batches over their whole ranges, at most 8,192 prompt tokens
    in a pass (4,096 for the eight-billion-parameter sizes, 400 in float32: less than the largest listed case)."""
    design = rng.choice(["qwen3", "qwen3", "qwen3"] + [d for d in DESIGNS if d != "qwen3"])
    dtype = "float32" if design == "qwen3" and rng.random() < 0.15 else "bfloat16"
    layers = 8 if design == "qwen3" and dtype == "bfloat16" else 4
    if dtype == "float32":
        sequences = rng.randint(1, 4)
        longest = _log_int(rng, 8, 100)
        return _case(None, design, "prompts", sequences, max(1, _log_int(rng, 1, longest)), longest, layers=layers, dtype=dtype,
                     want=rng.choice(["all", "last"]))
    if rng.random() < 0.5:
        sequences = _log_int(rng, 1, 8)
        longest = min(_log_int(rng, 17, 3000), (4096 if design == "qwen3" else 8192) // sequences)
        return _case(None, design, "prompts", sequences, _log_int(rng, 9, longest), longest, layers=layers)
    sequences = _log_int(rng, 1, 56)
    longest = min(_log_int(rng, 40, 2500), 24000 // sequences)
    return _case(None, design, "decode", sequences, _log_int(rng, 20, longest), longest, layers=layers,
                 temperature=rng.choice([0.0, 0.0, 0.7]), steps=rng.randint(2, 6))


def _lengths(case):
    """The prompts' lengths: from the shortest to the longest in equal ratios."""
    n, low, high = case["sequences"], case["shortest"], case["longest"]
    return [high] if n == 1 else [int(round(low * (high / low) ** (i / (n - 1)))) for i in range(n)]


# ------------------------------------------------------------------------------ the architectures at the benchmark's sizes


def _qwen3(layers):
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": layers, "hidden_size": 4096,
            "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": 12288,
            "vocab_size": 151936, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False,
            "max_position_embeddings": 40960, "hidden_act": "silu"}


def _design(name, layers, **more):
    return {"architecture": name, "vocab": 32768, "width": 2048, "norm": {"eps": 1e-6}, "layers": layers, **more}


def _lemesun(layers):
    moe = {"kind": "moe", "expert": {"ff": 1024, "limit": 7.0}, "shared": {"ff": 1024, "limit": 7.0},
           "router": {"experts": 30, "identity": 2, "top": 4, "groups": {"count": 4, "keep": 2}}}
    latent = {"type": "latent_attention", "mlp": moe,
              "mixer": {"heads": 16, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 256, "scale": 96 ** -0.5,
                        "rot": {"base": 10000.0, "dims": 32}}}
    delta = {"type": "channel_delta", "mlp": moe,
             "mixer": {"heads": 16, "kv_heads": 16, "dim": 64, "vdim": 64, "conv": 4, "decay_rank": 64, "gate_rank": 64}}
    return _design("Lemesun", [delta if i % 2 else latent for i in range(layers)])


def _nulalorn(layers):
    mixer = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0, "mask": {"size": 1024},
             "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    moe = {"kind": "moe", "expert": {"ff": 1024}, "shared": {"ff": 1024}, "router": {"experts": 32, "top": 4}}
    entries = [{"type": "attention", "mixer": mixer, "mlp": moe if i else {"kind": "dense", "ff": 5120}} for i in range(layers)]
    return _design("Nulalorn", entries, logit_softcap=40.0, loop={"start": 1, "stop": layers, "times": 2})


def _zigivik(layers):
    attention = {"type": "attention", "mlp": {"kind": "dense", "ff": 5120},
                 "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}}
    mixer = {"heads": 16, "dim": 64, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 768, "scale": 128 ** -0.5,
             "mask": {"size": 1024},
             "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    latent = lambda **more: {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 5120}, "mixer": dict(mixer, **more)}
    return _design("Zigivik", [(latent() if i == 1 else latent(kv_from=1)) if i % 2 else attention for i in range(layers)],
                   residual_mult=0.5, canon={"taps": 4})


def _losivik(layers):
    latent = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 5120, "limit": 7.0},
              "mixer": {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5, "mask": {"size": 1024}}}
    pair = {"type": "parallel",
            "mlp": {"kind": "moe", "expert": {"ff": 1024}, "shared": {"ff": 1024}, "router": {"experts": 32, "top": 4}},
            "mixer": {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                               "mask": {"size": 1024, "keep_first": 64}},
                      "right": {"heads": 32, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1},
                      "left_scale": 0.5, "right_scale": 0.5}}
    return _design("Losivik", [pair if i % 2 else latent for i in range(layers)], embedding={"scale": 1.0}, token_side={"dim": 256})


def _noganex(layers):
    attention = {"type": "attention", "mlp": {"kind": "dense", "ff": 5120},
                 "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                           "rot": {"base": 10000.0, "dims": 128, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    # Experts of equal weight behind a sigmoid router, normed after them: which of two nearly equal scores is fourth would
    # decide the logits of a token, so both kinds of layer have the dense feed-forward here.
    delta = {"type": "delta", "mlp": {"kind": "dense", "ff": 5120},
             "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    return _design("Noganex", [delta if i % 2 else attention for i in range(layers)], logit_scale=0.5)


def _pukinex(layers):
    pair = {"type": "parallel", "mlp": {"kind": "dense", "ff": 7680},
            "mixer": {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias_rows": 32,
                               "bias_max": 512, "q_temp": {"coef": 0.1, "every": 1024}},
                      "right": {"heads": 16, "dim": 128, "vdim": 128, "rot": {"base": 10000.0, "dims": 128},
                                "decay": [1.0 - 2.0 ** (-5.0 - 4.0 * i / 16) for i in range(16)]},
                      "left_scale": 0.5, "right_scale": 0.5}}
    attention = {"type": "attention", "mlp": {"kind": "dense", "ff": 7680},
                 "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0,
                           "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0}}}}
    return _design("Pukinex", [attention if i % 2 else pair for i in range(layers)], embedding={"scale": 1.0}, residual_mult=0.5,
                   streams=2, logit_scale=0.5, logit_softcap=30.0)


DESIGNS = {"qwen3": _qwen3, "lemesun": _lemesun, "nulalorn": _nulalorn, "zigivik": _zigivik, "losivik": _losivik,
           "noganex": _noganex, "pukinex": _pukinex}


def _config(case):
    return DESIGNS[case["design"]](case["layers"])


# ------------------------------------------------------------------------------ weights


class StoredWeights:
    """Seeded tensors in the place of a checkpoint.  Matrices are normal with the customary deviation of 0.02; the
    rates of the recurrent mixers (``A_log``, ``dt_bias``) follow the published start of such models, memories of a
    few to a thousand tokens; taps, norms, stream mixing and the sharpness of the routers have the size of trained ones, and the
    embedding of a design is as large as what its layers add to it."""

    def __init__(self, decls, device):
        self.decls, self.device = {d.name: d for d in decls}, device

    def stored(self):
        return {n: StoredTensor(tuple(d.shape), torch.int32 if d.init.startswith("distinct_below:") else torch.bfloat16)
                for n, d in self.decls.items()}

    def fetch(self, name):
        decl = self.decls[name]
        seed = int.from_bytes(hashlib.sha256(f"{WEIGHTS_SEED}:{name}".encode()).digest()[:7], "little")
        gen = torch.Generator(device=self.device).manual_seed(seed)
        if decl.init.startswith("distinct_below:"):
            order = torch.rand(tuple(decl.shape[:-1]) + (int(decl.init.split(":")[1]),), generator=gen, device=self.device).argsort(-1)
            return order[..., :decl.shape[-1]].to(torch.int32).contiguous()
        if decl.init == "zeros":
            return torch.zeros(decl.shape, dtype=torch.bfloat16, device=self.device)
        if name.endswith("A_log"):
            return torch.log(1.0 + 15.0 * torch.rand(decl.shape, generator=gen, device=self.device)).bfloat16()
        if name.endswith("dt_bias"):
            dt = torch.exp(math.log(1e-3) + math.log(100.0) * torch.rand(decl.shape, generator=gen, device=self.device))
            return (dt + torch.log(-torch.expm1(-dt))).bfloat16()
        t = torch.randn(decl.shape, generator=gen, device=self.device)
        if decl.init == "one_plus_normal":
            t = 1.0 + 0.01 * t
        elif name.endswith((".conv", "canon1")):
            t *= 0.3
        elif name.endswith(".router"):
            t *= 0.1
        elif name == "embed":
            pass
        else:
            t *= 0.02
            if ".hc" in name and name.endswith(".mix"):
                t += torch.eye(decl.shape[0], device=self.device)
        return t.bfloat16()

    def close(self):
        pass


def _decls(case):
    return DecoderModel(config_from_dict(_config(case)).to_plan()).tensor_decls()


_loaded = {}              # the model that the program serves: one at a time


def _model(case):
    key = json.dumps([case["design"], case["layers"], case["dtype"]])
    if key not in _loaded:
        _loaded.clear()
        torch.cuda.empty_cache()
        config = config_from_dict(_config(case))
        decoder = DecoderModel(config.to_plan())
        decoder.load(StoredWeights(decoder.tensor_decls(), torch.device("cuda:0")), dtype=DTYPES[case["dtype"]], device="cuda:0")
        _loaded[key] = ResidentModel(config, decoder)
    return _loaded[key]


# ------------------------------------------------------------------------------ a pass


def _tokens(case, seed):
    """(the prompts, the tokens that each step of a decode case is given)."""
    gen = torch.Generator().manual_seed(seed)
    vocab = 151936 if case["design"] == "qwen3" else 32768
    prompts = [torch.randint(0, vocab, (n,), generator=gen).tolist() for n in _lengths(case)]
    return prompts, torch.randint(0, vocab, (case.get("steps", 0), case["sequences"]), generator=gen).tolist()


def _begin(state):
    """The prompts of a decode case into the cache, and its sequences to the decode runner."""
    cache, prompts = state["cache"], state["prompts"]
    cache.reset()
    state["slots"] = [cache.alloc() for _ in prompts]
    state["model"].step(cache, state["slots"], prompts, "none")
    state["runner"].begin(state["slots"], state["tokens"][0], list(range(len(prompts))), [1] * len(prompts))
    state["left"] = REQUEST_STEPS


def prepare(case, seed):
    model = _model(case)
    prompts, tokens = _tokens(case, seed)
    room = REQUEST_STEPS if case["kind"] == "decode" else 0
    pages = sum(-(-(len(p) + room) // PAGE) for p in prompts)
    cache = model.make_cache(max_tokens=pages * PAGE, max_seqs=len(prompts), max_step_tokens=case["longest"])
    state = {"case": case, "model": model, "cache": cache, "prompts": prompts, "tokens": tokens}
    if case["kind"] == "decode":
        state["runner"] = decode_runner(model, cache, temperature=case["temperature"], seed=seed % 1000)
        _begin(state)
    return state


def run(state):
    case, cache = state["case"], state["cache"]
    if case["kind"] == "prompts":
        slots = [cache.alloc() for _ in state["prompts"]]
        logits = state["model"].step(cache, slots, state["prompts"], case["want"])
        for slot in slots:
            cache.free(slot)
        return logits
    if state["left"] < len(state["tokens"]):
        _begin(state)
    state["left"] -= len(state["tokens"])
    runner, logits = state["runner"], []
    for tokens in state["tokens"]:
        runner.step(tokens)
        logits.append(runner.last_logits().clone())
    return logits


# ------------------------------------------------------------------------------ what a pass cannot do without


def work(case):
    """Bytes: every weight that the pass uses once, cached rows and recurrent state read and written once, the logits
    written once.  Flops: the products of every token, scores and read-outs over the keys that each token sees."""
    cfg, lengths, dtype_bytes = _config(case), _lengths(case), 4 if case["dtype"] == "float32" else 2
    decode = case["kind"] == "decode"
    steps = case["steps"] if decode else 1
    tokens = steps * len(lengths) if decode else sum(lengths)
    rows = tokens if decode or case["want"] == "all" else len(lengths)
    vocab = 151936 if case["design"] == "qwen3" else 32768
    loop = cfg.get("loop")
    runs = lambda layer: loop["times"] if loop and loop["start"] <= layer < loop["stop"] else 1
    number, flops = 0.0, 0.0
    for decl in {d.name: d for d in _decls(case)}.values():
        size = math.prod(decl.shape)
        if "embed" in decl.name or decl.init.startswith("distinct_below:"):
            if case["design"] == "losivik" and decl.name == "embed":      # the head is the table
                number, flops = number + size, flops + 2.0 * size * rows
            continue
        if decl.name.endswith(("head", "lm_head.weight")):
            number, flops = number + size, flops + 2.0 * size * rows
            continue
        layer = decl.name.split(".layers.")[-1].lstrip("l").split(".")[0]
        times = runs(int(layer)) if layer.isdigit() else 1
        share = hit = 1.0
        if ".mlp.e" in decl.name:
            router = cfg["layers"][int(layer)]["mlp"]["router"]
            share = router["top"] / (router["experts"] + router.get("identity", 0))
            hit = 1.0 - (1.0 - share) ** (len(lengths) if decode else tokens)
        number += size * hit
        flops += 2.0 * size * tokens * share * times if len(decl.shape) > 1 else 0.0
    bytes_ = number * dtype_bytes * steps + rows * vocab * 4.0

    def keys_seen(n, window, keep):
        """(keys that the tokens of a sequence of n tokens see in all, rows of its cache that the pass reads)"""
        places = range(n, n + steps) if decode else range(n)
        seen = [p + 1 if window is None else min(p + 1, window + keep) for p in places]
        return float(sum(seen)), float(sum(seen) if decode else n)

    for i in range(case["layers"]):
        if case["design"] == "qwen3":
            mixers = [dict(heads=32, kv_heads=8, dim=128, vdim=128)]
        else:
            mixer = cfg["layers"][i]["mixer"]
            mixers = [mixer["left"], mixer["right"]] if "left" in mixer else [mixer]
        for m in mixers:
            state = "state" in m or "decay" in m or "conv" in m and "kv_rank" not in m
            dim, vdim = m.get("dim", m.get("state", 0)), m.get("vdim", m.get("dim", 0))
            if state:
                flops += 5.0 * tokens * m["heads"] * dim * vdim
                bytes_ += 8.0 * m["heads"] * dim * vdim * len(lengths) * steps
                continue
            mask = m.get("mask") or {}
            row = m["kv_rank"] + m.get("rot_dim", 0) if "kv_rank" in m else m["kv_heads"] * (dim + vdim)
            for n in lengths:
                seen, read = keys_seen(n, mask.get("size"), mask.get("keep_first", 0))
                flops += 2.0 * seen * m["heads"] * (dim + m.get("rot_dim", 0) + vdim) * runs(i)
                bytes_ += read * row * dtype_bytes * runs(i)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Four times what the library's own products against the vendor's (sums in another order) were seen to move the
    logits by: 7e-6 of a norm in float32; in bfloat16 0.004 to 0.008 for the designs, 0.015 for the eight layers, where
    the most that a comparison takes is stated."""
    if case["dtype"] == "float32":
        return {"rel": 2.5e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.3} if case["design"] == "qwen3" else {"rel": 0.025, "max": 0.15}


# ------------------------------------------------------------------------------ plain 64-bit forms


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu_tanh(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _gelu_erf(z):
    return 0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _softplus(z):
    return torch.nn.functional.softplus(z)


def _frequencies(dims, base, scaling):
    """(frequencies, the factor of cosine and sine) of a rotation: plain, divided, slowed by wavelength, or by a ramp."""
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not scaling:
        return f, 1.0
    factor = scaling["factor"]
    if "low" in scaling:
        out = []
        for v in f:
            blend = (scaling["original"] * v / (2.0 * math.pi) - scaling["low"]) / (scaling["high"] - scaling["low"])
            blend = min(max(blend, 0.0), 1.0)
            out.append((1.0 - blend) * v / factor + blend * v)
        return out, 1.0
    if "fast" in scaling:
        index = lambda turns: dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        low, high = max(math.floor(index(scaling["fast"])), 0), min(math.ceil(index(scaling["slow"])), dims - 1)
        ramps = [min(max((i - low) / max(high - low, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        return [v / factor * r + v * (1.0 - r) for v, r in zip(f, ramps)], 0.1 * math.log(factor) + 1.0
    return [v / factor for v in f], 1.0


def _rotate(x, dims, base, scaling=None, *, neighbours):
    """x [T, heads, d]: the first ``dims`` lanes turn, in pairs of neighbours or of halves.  Angles are taken in 32
    bits, as the architectures define them."""
    f, factor = _frequencies(dims, base, scaling)
    position = torch.arange(x.shape[0], dtype=torch.float32, device=x.device)
    angle = (position[:, None] * torch.tensor(f, dtype=F64, device=x.device).float()[None]).to(F64)[:, None]
    cos, sin = torch.cos(angle) * factor, torch.sin(angle) * factor
    turned = x[..., :dims].unflatten(-1, (dims // 2, 2) if neighbours else (2, dims // 2))
    u, v = turned.unbind(-1 if neighbours else -2)
    turned = torch.stack([u * cos - v * sin, v * cos + u * sin], -1 if neighbours else -2).flatten(-2)
    return torch.cat([turned, x[..., dims:]], -1)


def _attend(q, k, v, scale, *, window=None, keep=0, chunk=None, softcap=None, sink=False, bias=None, talk=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv], a block of queries at a time."""
    T, H = q.shape[:2]
    k, v = (t.repeat_interleave(H // t.shape[1], 1).transpose(0, 1) for t in (k, v))
    out, place = [], torch.arange(T, device=q.device)
    for start in range(0, T, 512):
        p = place[start:start + 512, None]
        scores = q[start:start + 512].transpose(0, 1) @ k.transpose(1, 2) * scale
        if talk is not None:
            scores = torch.einsum("hg,gpj->hpj", talk, scores)
        if softcap:
            scores = softcap * torch.tanh(scores / softcap)
        if bias is not None:
            scores = scores + bias[(p - place[None]).clamp(min=0)].permute(2, 0, 1)
        seen = place[None] <= p
        if window is not None:
            seen = seen & ((p - place[None] < window) | (place[None] < keep))
        if chunk is not None:
            seen = seen & (place[None] // chunk == p // chunk)
        scores = scores.masked_fill(~seen[None], float("-inf"))
        if sink:
            scores = torch.cat([torch.zeros_like(scores[..., :1]), scores], -1)
        weights = torch.softmax(scores, -1)
        out.append(((weights[..., 1:] if sink else weights) @ v).transpose(0, 1))
    return torch.cat(out, 0)


def _convolution(x, taps):
    """x [T, C], taps [C, n], the last of them for the current token."""
    n = taps.shape[1]
    padded = torch.cat([torch.zeros_like(x[:1]).expand(n - 1, -1), x], 0)
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))


def _recurrence(q, k, v, decay, beta=None):
    """S <- decay S + k u^T, out = S^T q, with u = v, or beta (v - S^T k) of the decayed state.  q, k [T, H, d],
    v [T, H, dv], decay [T, H, d or 1], beta [T, H]."""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=F64, device=k.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = (q[t][:, None] @ S)[:, 0]
    return out


def _heads(h, w, name, heads):
    x = h @ w[name].T
    if name + ".b" in w:
        x = x + w[name + ".b"]
    return x.view(h.shape[0], heads, -1)


def _mixture(h, chosen, weights, expert, count, identity=0):
    """Sum over the chosen experts of weight times output; the last ``identity`` of them hand the row through."""
    out = torch.zeros_like(h)
    for e in range(count + identity):
        share = (weights * (chosen == e)).sum(-1)
        rows = share.nonzero().flatten()
        if len(rows):
            out[rows] += share[rows, None] * (h[rows] if e >= count else expert(f"e{e}.", h[rows]))
    return out


class _Qwen3:
    def __init__(self, cfg, layer):
        self.cfg, self.prefix = cfg, f"model.layers.{layer}."

    def __call__(self, x, w, ids, keep):
        cfg, eps, T = self.cfg, self.cfg["rms_norm_eps"], x.shape[0]
        h = _rms(x, eps) * w["input_layernorm.weight"]
        q, k, v = (_heads(h, w, f"self_attn.{r}_proj.weight", n) for r, n in (("q", 32), ("k", 8), ("v", 8)))
        q, k = (_rms(t, eps) * w[f"self_attn.{r}_norm.weight"] for t, r in ((q, "q"), (k, "k")))
        q, k = (_rotate(t, 128, cfg["rope_theta"], neighbours=False) for t in (q, k))
        x = x + _attend(q, k, v, 128 ** -0.5).reshape(T, -1) @ w["self_attn.o_proj.weight"].T
        h = _rms(x, eps) * w["post_attention_layernorm.weight"]
        return x + (_silu(h @ w["mlp.gate_proj.weight"].T) * (h @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T


class _Layer:
    """One layer of a design on one sequence: ``self(x, w, ids, keep)`` with w the layer's own tensors and ``keep`` what
    the layers of this sequence share."""

    def __init__(self, cfg, layer):
        self.cfg, self.layer, self.entry, self.prefix = cfg, layer, cfg["layers"][layer], f"l{layer}."
        self.m, self.f, self.eps = self.entry["mixer"], self.entry["mlp"], cfg["norm"]["eps"]


class _Lemesun(_Layer):
    def __call__(self, x, w, ids, keep):
        norm = lambda t, name: _rms(t, self.eps) * (1.0 + w[name])
        mix = self.latent if self.entry["type"] == "latent_attention" else self.delta
        x = x + mix(norm(x, "norm1"), w)
        return x + self.experts(norm(x, "norm2"), w)

    def latent(self, h, w):
        m, T = self.m, h.shape[0]
        R, d = m["kv_rank"], m["dim"]
        rotate = lambda t: _rotate(t, m["rot"]["dims"], m["rot"]["base"], neighbours=True)
        q, down = _heads(h, w, "mix.q", m["heads"]), h @ w["mix.dkv"].T
        c, turned = _rms(down[:, :R], self.eps) * w["mix.dkv.norm"], rotate(down[:, None, R:]).expand(-1, m["heads"], -1)
        k = torch.cat([_heads(c, w, "mix.uk", m["heads"]), turned], -1)
        q = torch.cat([q[..., :d], rotate(q[..., d:])], -1)
        return _attend(q, k, _heads(c, w, "mix.uv", m["heads"]), m["scale"]).reshape(T, -1) @ w["mix.o"].T

    def delta(self, h, w):
        m, T = self.m, h.shape[0]
        q, k, v = (_silu(_convolution(h @ w[f"mix.{r}"].T, w[f"mix.{r}.conv"])).view(T, m["heads"], -1) for r in "qkv")
        rate = _softplus((h @ w["mix.a1"].T) @ w["mix.a2"].T + w["mix.dt_bias"]).view(T, m["heads"], -1)
        decay = torch.exp(-torch.exp(w["mix.A_log"])[:, None] * rate)
        out = _recurrence(_unit(q) * m["dim"] ** -0.5, _unit(k), v, decay, torch.sigmoid(h @ w["mix.b"].T))
        gate = torch.sigmoid((h @ w["mix.g1"].T) @ w["mix.g2"].T).view(T, m["heads"], -1)
        return (_rms(out, self.eps) * w["mix.norm"] * gate).reshape(T, -1) @ w["mix.o"].T

    def experts(self, h, w):
        r, limit = self.f["router"], self.f["expert"]["limit"]

        def expert(e, t):
            g, u = torch.clamp(t @ w[f"mlp.{e}gate"].T, max=limit), torch.clamp(t @ w[f"mlp.{e}up"].T, -limit, limit)
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[f"mlp.{e}down"].T

        scores = torch.softmax(h @ w["mlp.router"].T, -1)
        choice = (scores + w["mlp.correction"]).view(h.shape[0], r["groups"]["count"], -1)
        kept = torch.zeros(choice.shape[:2], dtype=torch.bool, device=h.device)
        kept.scatter_(1, choice.max(-1).values.topk(r["groups"]["keep"], -1).indices, True)
        chosen = choice.masked_fill(~kept[..., None], float("-inf")).flatten(1).topk(r["top"], -1).indices
        return _mixture(h, chosen, scores.gather(1, chosen), expert, r["experts"], r["identity"]) + expert("shared.", h)


class _Nulalorn(_Layer):
    def __call__(self, x, w, ids, keep):
        norm = lambda t, name: _rms(t, self.eps) * w[name]
        m, T, h = self.m, x.shape[0], norm(x, "norm1")
        q, k, v = _heads(h, w, "mix.q", m["heads"]), _heads(h, w, "mix.k", m["kv_heads"]), _heads(h, w, "mix.v", m["kv_heads"])
        q, k = (_rms(_rotate(t, m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"], neighbours=True), self.eps) for t in (q, k))
        out = _attend(q, k, v, m["scale"], window=m["mask"]["size"], softcap=m["softcap"]).reshape(T, -1)
        x = x + norm(out @ w["mix.o"].T, "norm1b")
        h, feed = norm(x, "norm2"), lambda e, t: _gelu_erf(t @ w[f"mlp.{e}up"].T) @ w[f"mlp.{e}down"].T
        if self.f["kind"] == "dense":
            return x + norm(feed("", h), "norm2b")
        r = self.f["router"]
        chosen = w["mlp.table"][ids].long()
        y = _mixture(h, chosen, torch.full(chosen.shape, 1.0 / r["top"], dtype=F64, device=h.device), feed, r["experts"])
        return x + norm(y + torch.sigmoid(h @ w["mlp.shared.sg"].T) * feed("shared.", h), "norm2b")


class _Zigivik(_Layer):
    def __call__(self, x, w, ids, keep):
        h = _rms(x, self.eps) * w["norm1"]
        hc = h + _convolution(h, w["canon1"])
        mix = self.attention if self.entry["type"] == "attention" else self.latent
        z = h @ w["mlp.up"].T + w["mlp.up.b"]
        a = w["mlp.act"]
        z = a[0] * _rms(z, self.eps) + a[1] * _rms(z * z, self.eps) + a[2] * _rms(z ** 3, self.eps) + a[3]
        return x + self.cfg["residual_mult"] * (mix(hc, w, keep) + z @ w["mlp.down"].T + w["mlp.down.b"])

    def attention(self, h, w, keep):
        m, T = self.m, h.shape[0]
        q, k = _heads(h, w, "mix.q", m["heads"]), _heads(h, w, "mix.k", m["kv_heads"])
        turned = [_rotate(t, m["rot"]["dims"], m["rot"]["base"], neighbours=True) for t in (q, k)]
        return _attend(*turned, k, m["scale"], sink=True).reshape(T, -1) @ w["mix.o"].T

    def latent(self, h, w, keep):
        m, T = self.m, h.shape[0]
        R, d, rot = m["kv_rank"], m["dim"], m["rot"]
        rotate = lambda t: _rotate(t, rot["dims"], rot["base"], rot["scaling"], neighbours=False)
        if "kv_from" not in m:
            down = h @ w["mix.dkv"].T
            keep[self.layer] = _rms(down[:, :R], self.eps) * w["mix.dkv.norm"], rotate(down[:, None, R:])
        c, turned = keep[m.get("kv_from", self.layer)]
        q = _heads(_rms(h @ w["mix.dq"].T, self.eps) * w["mix.dq.norm"], w, "mix.uq", m["heads"])
        q = torch.cat([q[..., :d], rotate(q[..., d:])], -1)
        k = torch.cat([_heads(c, w, "mix.uk", m["heads"]), turned.expand(-1, m["heads"], -1)], -1)
        out = _attend(q, k, _heads(c, w, "mix.uv", m["heads"]), m["scale"], window=m["mask"]["size"]).reshape(T, -1)
        return (out * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T


class _Losivik(_Layer):
    def __call__(self, x, w, ids, keep):
        norm = lambda t, name: _rms(t, self.eps) * (1.0 + w[name])
        h, g = norm(x, "norm1"), norm(x, "norm2")
        if self.entry["type"] == "latent_attention":
            mixed, limit = self.latent(h, w), self.f["limit"]
            gate = torch.clamp(g @ w["mlp.gate"].T + w["mlp.gate.b"], max=limit)
            up = torch.clamp(g @ w["mlp.up"].T + w["mlp.up.b"], -limit, limit)
            fed = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ w["mlp.down"].T + w["mlp.down.b"]
        else:
            mixed, fed = self.m["left_scale"] * self.attention(h, w) + self.m["right_scale"] * self.state_space(h, w), self.experts(g, w)
        x = x + mixed * w["ls1"] + fed * w["ls2"]
        d = self.cfg["token_side"]["dim"]
        side = keep["side.embed"][ids][:, self.layer * d:(self.layer + 1) * d]
        return x + _rms((_gelu_tanh(x @ w["side.gate"].T) * side) @ w["side.proj"].T, self.eps) * w["side.norm"]

    def latent(self, h, w):
        m, T = self.m, h.shape[0]
        c = _rms(h @ w["mix.dkv"].T, self.eps) * w["mix.dkv.norm"]
        q, k, v = _heads(h, w, "mix.q", m["heads"]), _heads(c, w, "mix.uk", m["heads"]), _heads(c, w, "mix.uv", m["heads"])
        out = _attend(q, k, v, m["scale"], window=m["mask"]["size"]) * torch.sigmoid(h @ w["mix.g"].T)[:, :, None]
        return out.reshape(T, -1) @ w["mix.o"].T

    def attention(self, h, w):
        m, T = self.m["left"], h.shape[0]
        q, k, v = (_heads(h, w, f"mix.left.{r}", n) for r, n in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
        q, k = (_rms(t, self.eps) * w[f"mix.left.{r}.norm"] for t, r in ((q, "q"), (k, "k")))
        out = _attend(q, k, v, m["scale"], window=m["mask"]["size"], keep=m["mask"]["keep_first"])
        return out.reshape(T, -1) @ w["mix.left.o"].T

    def state_space(self, h, w):
        m, T = self.m["right"], h.shape[0]
        H, P, N = m["heads"], m["vdim"], m["state"]
        z, xbc, dt = (h @ w["mix.right.in"].T).split([H * P, H * P + 2 * N, H], -1)
        x, B, C = _silu(_convolution(xbc, w["mix.right.conv"]) + w["mix.right.conv.b"]).split([H * P, N, N], -1)
        x, dt = x.reshape(T, H, P), _softplus(dt + w["mix.right.dt_bias"])
        decay = torch.exp(-torch.exp(w["mix.right.A_log"]) * dt)[..., None]
        B, C = (t[:, None].expand(-1, H, -1) for t in (B, C))
        y = _recurrence(C, B, x * dt[..., None], decay) + w["mix.right.D"][:, None] * x
        return (_rms(y.reshape(T, -1) * _silu(z), self.eps) * w["mix.right.norm"]) @ w["mix.right.o"].T

    def experts(self, h, w):
        r, feed = self.f["router"], lambda e, t: torch.relu(t @ w[f"mlp.{e}up"].T) ** 2 @ w[f"mlp.{e}down"].T
        scores, chosen = torch.sigmoid(h @ w["mlp.router"].T).topk(r["top"], -1)
        out = feed("shared.", h)
        for e in range(r["experts"]):                     # the score multiplies the expert's input
            share = (scores * (chosen == e)).sum(-1)
            rows = share.nonzero().flatten()
            out[rows] += feed(f"e{e}.", share[rows, None] * h[rows])
        return out


class _Noganex(_Layer):
    def __call__(self, x, w, ids, keep):
        mix = self.attention if self.entry["type"] == "attention" else self.delta
        x = x + self.gated(mix(x, w), x, w, "1")
        fed = (_gelu_tanh(x @ w["mlp.gate"].T + w["mlp.gate.b"]) * (x @ w["mlp.up"].T + w["mlp.up.b"])) @ w["mlp.down"].T + w["mlp.down.b"]
        return x + self.gated(fed, x, w, "2")

    def gated(self, y, x, w, n):
        return _rms(y * torch.sigmoid(x @ w[f"rg{n}"].T + w[f"rg{n}.b"]), self.eps) * w[f"norm{n}"]

    def attention(self, h, w):
        m, T, rot = self.m, h.shape[0], self.m["rot"]
        q, k = (_rms(h @ w[f"mix.{r}"].T, self.eps) * w[f"mix.{r}.norm"] for r in "qk")
        q, k = (_rotate(t.view(T, -1, m["dim"]), rot["dims"], rot["base"], rot["scaling"], neighbours=False) for t in (q, k))
        v = _heads(h, w, "mix.v", m["kv_heads"])
        return _attend(q, k, v, m["scale"], chunk=m["mask"]["size"], talk=w["mix.talk"]).reshape(T, -1) @ w["mix.o"].T

    def delta(self, h, w):
        m, T, H, G = self.m, h.shape[0], self.m["heads"], self.m["kv_heads"]
        q, k, v = (_silu(_convolution(h @ w[f"mix.{r}"].T, w[f"mix.{r}.conv"])).view(T, -1, m["dim"]) for r in "qkv")
        q, k = (_unit(t).repeat_interleave(H // G, 1) for t in (q, k))
        decay = torch.exp(-torch.exp(w["mix.A_log"]) * _softplus(h @ w["mix.a"].T + w["mix.dt_bias"]))[..., None]
        out = _recurrence(q / math.sqrt(m["dim"]), k, v, decay, torch.sigmoid(h @ w["mix.b"].T))
        return ((_rms(out, self.eps) * w["mix.norm"]).reshape(T, -1) * _silu(h @ w["mix.g"].T)) @ w["mix.o"].T


class _Pukinex(_Layer):
    """x holds the parallel streams [T, streams, width]."""

    def __call__(self, x, w, ids, keep):
        mix = self.attention if self.entry["type"] == "attention" else self.pair
        for n, part in (("1", mix), ("2", lambda h, w: torch.relu(h @ w["mlp.up"].T) ** 2 @ w["mlp.down"].T)):
            y = part(_layer_norm(torch.einsum("tsw,s->tw", x, w[f"hc{n}.in"]), w[f"norm{n}"], w[f"norm{n}.b"], self.eps), w)
            x = (torch.einsum("tsw,su->tuw", x, w[f"hc{n}.mix"])
                 + self.cfg["residual_mult"] * w[f"hc{n}.out"][None, :, None] * y[:, None])
        return x

    def attention(self, h, w):
        m, T, rot = self.m, h.shape[0], self.m["rot"]
        q, v = _heads(h, w, "mix.q", m["heads"]), _heads(h, w, "mix.k", m["kv_heads"])     # the values are the unrotated keys
        q, k = (_rotate(t, rot["dims"], rot["base"], rot["scaling"], neighbours=True) for t in (q, v))
        out = _attend(q, k, v, m["scale"], softcap=m["softcap"], sink=True) * torch.sigmoid(h @ w["mix.g"].T)[:, :, None]
        return out.reshape(T, -1) @ w["mix.o"].T

    def pair(self, h, w):
        m, T = self.m["left"], h.shape[0]
        q, k, v = (_heads(h, w, f"mix.left.{r}", n) for r, n in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
        q, k = (_rms(t, self.eps) * w[f"mix.left.{r}.norm"] for t, r in ((q, "q"), (k, "k")))
        warm = [1.0 + m["q_temp"]["coef"] * math.log((p + 1) // m["q_temp"]["every"] + 1) for p in range(T)]
        q = q * torch.tensor(warm, dtype=F64, device=h.device)[:, None, None]
        rows, half = m["bias_rows"], m["bias_rows"] // 2
        row = lambda n: n if n < half else min(rows - 1, half + math.floor(
            math.log(n / half) / math.log(m["bias_max"] / half) * (rows - half)))
        bias = w["mix.left.rel"][torch.tensor([row(n) for n in range(T)], device=h.device)]
        left = _attend(q, k, v, m["scale"], sink=True, bias=bias).reshape(T, -1) * torch.sigmoid(h @ w["mix.left.g"].T)
        m = self.m["right"]
        q, k, v = (_heads(h, w, f"mix.right.{r}", m["heads"]) for r in "qkv")
        q, k = (_rotate(t, m["rot"]["dims"], m["rot"]["base"], neighbours=False) for t in (q, k))
        decay = torch.tensor(m["decay"], dtype=F64, device=h.device).expand(T, -1)[..., None]
        out = _rms(_recurrence(q, k * m["dim"] ** -0.5, v, decay), self.eps).reshape(T, -1) * _silu(h @ w["mix.right.g"].T)
        return self.m["left_scale"] * (left @ w["mix.left.o"].T) + self.m["right_scale"] * (out @ w["mix.right.o"].T)


def _layer_norm(x, weight, bias, eps):
    return _rms(x - x.mean(-1, keepdim=True), eps) * weight + bias


PLAIN = {"qwen3": _Qwen3, "lemesun": _Lemesun, "nulalorn": _Nulalorn, "zigivik": _Zigivik, "losivik": _Losivik, "noganex": _Noganex,
         "pukinex": _Pukinex}


def _sinusoid(T, width, device):
    f = torch.tensor([10000.0 ** (-2.0 * i / width) for i in range(width // 2)], dtype=F64, device=device).float()
    angle = (torch.arange(T, dtype=torch.float32, device=device)[:, None] * f[None]).to(F64)
    return torch.stack([torch.sin(angle), torch.cos(angle)], -1).flatten(1)


def _head(cfg, design, fetch, x):
    """Logits of rows x of the stream."""
    if design == "qwen3":
        return (_rms(x, cfg["rms_norm_eps"]) * fetch("model.norm.weight")) @ fetch("lm_head.weight").T
    eps, weight = cfg["norm"]["eps"], fetch("final.norm")
    if design == "pukinex":
        x = _layer_norm(x.sum(1), weight, fetch("final.norm.b"), eps)
    else:
        x = _rms(x, eps) * (1.0 + weight if design in ("lemesun", "losivik") else weight)
    logits = x @ fetch("embed" if design == "losivik" else "head").T * cfg.get("logit_scale", 1.0)
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def exact(case, seed):
    cfg, design, device = _config(case), case["design"], torch.device("cuda:0")
    store = StoredWeights(_decls(case), device)

    def fetch(name):
        t = store.fetch(name)
        return t.to(F64) if t.is_floating_point() else t

    prompts, tokens = _tokens(case, seed)
    texts = [torch.tensor(p + [step[i] for step in tokens], device=device) for i, p in enumerate(prompts)]
    table = store.fetch("model.embed_tokens.weight" if design == "qwen3" else "embed")
    streams = [table[ids].to(F64) for ids in texts]
    if design == "losivik":
        streams = [x * cfg["embedding"]["scale"] + _sinusoid(x.shape[0], x.shape[1], device) for x in streams]
    elif design == "zigivik":
        streams = [_rms(x, cfg["norm"]["eps"]) * fetch("embed.norm") for x in streams]
    elif design == "pukinex":
        streams = [(x * cfg["embedding"]["scale"])[:, None].repeat(1, cfg["streams"], 1) for x in streams]
    first, kept = streams, [{"side.embed": fetch("side.embed")} if design == "losivik" else {} for _ in texts]
    loop = cfg.get("loop") or {"start": 0, "stop": case["layers"], "times": 1}
    order = list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], case["layers"]))
    turn = 0
    for index in order:
        if cfg.get("loop") and index == loop["start"]:    # the embedding joins the stream again before every pass
            streams = [torch.cat([x, x0], -1) @ fetch("loop.in").T + fetch("loop.step")[turn] for x, x0 in zip(streams, first)]
            turn += 1
        layer = PLAIN[design](cfg, index)
        w = {n[len(layer.prefix):]: fetch(n) for n in store.decls if n.startswith(layer.prefix)}
        streams = [layer(x, w, ids, keep) for x, ids, keep in zip(streams, texts, kept)]
        del w
    if case["kind"] == "decode":
        return [_head(cfg, design, fetch, torch.stack([x[len(p) + j] for x, p in zip(streams, prompts)])) for j in range(case["steps"])]
    return _head(cfg, design, fetch, torch.cat([x if case["want"] == "all" else x[-1:] for x in streams]))
