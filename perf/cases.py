"""The workloads that the engine's speed is judged by: whole passes of serving work through the public entry points
(``ModelRunner.step`` / ``step_decode_graph`` / ``finish``, the cache manager's ``truncate``, ``Sampler.sample``), for every
architecture of the package, over the range of sizes that its configurations, shapes and benchmark sections name.

Six kinds of pass:

* ``decode``: some decode steps of a batch whose contexts are in the cache, from recorded graphs; the requests are then cut back
  to where they stood, so that a pass can be repeated;
* ``prefill``: the prompt step of one request;
* ``mixed``: one step that holds a portion of a long prompt beside the decode rows of other long requests;
* ``serve``: requests from their prompts (in steps of at most 2,048 tokens) through some decode steps to their end;
* ``generate``: the same with the tokens that the engine draws greedily, which pass from step to step on the device;
* ``sample``: the ids drawn for the logits rows of a batch.

Tokens are given, not drawn, except in ``generate`` (32-bit) and ``sample``, so that logits can be compared. Weights are random,
in bfloat16 as a checkpoint's are: matrices of standard deviation 0.02, those that write into the residual stream smaller by the
root of the number of sublayers, an embedding of the size of the stream, norms around one, and for the few vectors that decide
how long a state lives or where a sink lies the ranges that trained models of such designs have. Routers choose by the token, as
trained ones mostly do: every token's embedding carries a part along the directions of its experts.
"""
import math
import random

import torch

from llm_steadyinfer_b200.config import config_from_dict
from llm_steadyinfer_b200.engine.step import ModelRunner, StepEntry
from llm_steadyinfer_b200.models import Model
from llm_steadyinfer_b200.sampling import Sampler, SamplingParams
from llm_steadyinfer_b200.weights.loader import place

DEVICE = "cuda:0"
PAGE = 16
BUDGET = 2048                       # most prompt tokens of a step
F64 = torch.float64


# ---- the models ------------------------------------------------------------------------------------------------

def _llama(hidden, ff, layers, heads, kv, head_dim, factor=8.0, tied=False, vocab=128256, original=8192, theta=500000.0, limit=131072):
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_size": hidden, "intermediate_size": ff,
            "num_hidden_layers": layers, "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": head_dim,
            "vocab_size": vocab, "max_position_embeddings": limit, "rms_norm_eps": 1e-5, "rope_theta": theta,
            "rope_scaling": {"rope_type": "llama3", "factor": factor, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                             "original_max_position_embeddings": original},
            "tie_word_embeddings": tied, "hidden_act": "silu", "torch_dtype": "bfloat16", "bos_token_id": 0, "eos_token_id": 1}


# width, dense feed-forward, attention heads and key/value heads of 128, time-mixing heads of 64, experts, expert and shared sizes
SIZES = {"narrow": (1024, 2816, 8, 2, 16, 8, 704, 1408), "base": (2048, 5632, 16, 4, 32, 16, 1408, 2816)}
VOCAB = 32000


def _mivorax(size):
    d, ff, h, g = SIZES[size][:4]
    dense = {"kind": "dense", "ff": ff}
    lat = {"type": "latent_attention", "mlp": dense,
           "mixer": {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 768, "kv_rank": 512, "scale": 192 ** -0.5,
                     "rot": {"base": 10000.0, "dims": 64}}}
    att = {"type": "attention", "mlp": dense,
           "mixer": {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias_max": 4096.0, "bias_buckets": 64}}
    ssm = {"type": "mamba2", "mlp": None,
           "mixer": {"heads": d // 32, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
    return {"architecture": "Mivorax", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-5},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 17}}, "layers": [lat, att, att, ssm] * 2}


def _nufasun(size):
    d, ff, h, g = SIZES[size][:4]
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": h, "kv_heads": g, "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "softcap": 30.0, "diff": 0.2,
                     "mask": {"size": 4096}, "rot": {"base": 10000.0, "dims": 64}}}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": h, "kv_heads": h // 2, "dim": 128, "vdim": 128, "conv": 4}}
    return {"architecture": "Nufasun", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-6}, "embedding": {"scale": 8.0},
            "logit_softcap": 30.0, "loop": {"start": 0, "stop": 8, "times": 1}, "layers": [att, att, delta, att] * 2}


def _vibunex(size):
    d, _, h, g, th, experts, eff, sff = SIZES[size]
    left = {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
            "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    mlp = {"kind": "moe", "expert": {"ff": eff}, "router": {"experts": experts, "top": 2, "scale": 1.5}, "shared": {"ff": sff}}
    one = {"type": "parallel", "mlp": mlp, "mixer": {"left": left, "right": {"heads": th, "dim": 64, "rank": 64},
                                                     "left_scale": 1.0, "right_scale": 0.6}}
    return {"architecture": "Vibunex", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-5}, "residual_mult": 0.5, "layers": [one] * 8}


def _fevosun(size):
    d, ff, h, g, _, experts, eff, sff = SIZES[size]
    window = {"size": 4096}
    att = {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": window,
           "q_temp": {"coef": 0.5, "every": 1024}}
    lat = {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "mask": window,
           "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    lat2 = dict(lat, q_rank=768, rot={"base": 10000.0, "dims": 64})
    mlp = {"kind": "moe", "expert": {"ff": eff, "limit": 7.0}, "router": {"experts": experts, "identity": 2, "top": 2},
           "shared": {"ff": sff, "limit": 7.0}}
    one = [{"type": "attention", "mixer": att, "mlp": mlp}, {"type": "latent_attention", "mixer": lat, "mlp": mlp},
           {"type": "attention", "mixer": att, "mlp": mlp}, {"type": "latent_attention_2", "mixer": lat2, "mlp": mlp}]
    return {"architecture": "Fevosun", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-6}, "embedding": {"scale": 2.0},
            "layers": [dict(one[0], mlp={"kind": "dense", "ff": ff})] + one[1:] + one}


def _risizen(size):
    d, ff, h, g = SIZES[size][:4]
    own = {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "conv": 4, "scale": 128 ** -0.5, "mask": {"size": 8192}}
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    layers = [{"type": "attention", "mixer": dict(own, kv_from=i - 1) if i % 4 == 3 else own, "mlp": mlp} for i in range(8)]
    return {"architecture": "Risizen", "vocab": VOCAB, "width": d, "streams": 4, "norm": {"eps": 1e-5}, "logit_scale": 0.5,
            "layers": layers}


def _samulorn(size):
    d, ff, h, g, _, experts = SIZES[size][:6]
    delta = {"heads": h, "kv_heads": h // 2, "dim": 128, "vdim": 128, "conv": 4, "rank": 128}
    left = {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "conv": 4, "scale": 128 ** -0.5,
            "rot": {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    pair = {"left": left, "right": {"width": d, "blocks": d // 128, "conv": 4}, "left_scale": 1.0, "right_scale": 0.8}
    dense = {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "expert": {"ff": ff // 4},
           "router": {"experts": experts, "top": 4, "scale": 2.0, "groups": {"count": 4, "keep": 2}}}
    one = [{"type": "channel_delta", "mixer": delta, "mlp": dense}, {"type": "channel_delta", "mixer": delta, "mlp": moe},
           {"type": "parallel", "mixer": pair, "mlp": dense}, {"type": "channel_delta", "mixer": delta, "mlp": moe}]
    return {"architecture": "Samulorn", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-5}, "embedding": {"scale": d ** 0.5},
            "token_side": {"dim": 128}, "loop": {"start": 0, "stop": 8, "times": 1}, "layers": one + one}


DESIGNS = {"mivorax": _mivorax, "nufasun": _nufasun, "vibunex": _vibunex, "fevosun": _fevosun, "risizen": _risizen,
           "samulorn": _samulorn}
LLAMAS = {"llama-8b": _llama(4096, 14336, 32, 32, 8, 128), "llama-1b": _llama(2048, 8192, 16, 32, 8, 64, 32.0, True),
          "llama-3b": _llama(3072, 8192, 28, 24, 8, 128, 32.0, True),
          "llama-tiny": _llama(96, 320, 3, 3, 1, 32, 8.0, False, 1000, 64, limit=512)}


def _config(case):
    model = case["model"]
    return LLAMAS[model] if model in LLAMAS else DESIGNS[model](case["size"])


# ---- the cases -------------------------------------------------------------------------------------------------

def listed():
    return [
        # the shortest calls there are: a small model in 32 bits, where launches and the host's work count
        {"name": "tiny fp32 generate", "kind": "generate", "model": "llama-tiny", "requests": 6, "shortest": 3, "longest": 200, "steps": 16},
        # the headline shape: a few long conversations being answered
        {"name": "8b decode 8", "kind": "decode", "model": "llama-8b", "requests": 8, "shortest": 1024, "longest": 2032, "steps": 8},
        # a full prompt step of the headline shape
        {"name": "8b prefill 2048", "kind": "prefill", "model": "llama-8b", "tokens": 2048},
        # a small model serving a full batch of requests of every length
        {"name": "1b decode 61", "kind": "decode", "model": "llama-1b", "requests": 61, "shortest": 32, "longest": 2016, "steps": 8},
        # long documents: a portion of one prompt beside the decode rows of others
        {"name": "3b mixed 16k", "kind": "mixed", "model": "llama-3b", "requests": 5, "shortest": 12000, "longest": 16128, "tokens": 2043},
        # the end of a step in a service whose requests all draw with temperature and a nucleus
        {"name": "sample 64 top-p", "kind": "sample", "rows": 64, "vocab": 128256, "temperature": 0.7, "top_p": 0.9, "top_k": 0},
        # the other architectures, each a few requests from prompt to end: one long prompt, some, or a full batch of ragged ones
        {"name": "mivorax serve", "kind": "serve", "model": "mivorax", "size": "base", "requests": 1, "shortest": 2048, "longest": 2048, "steps": 16},
        {"name": "nufasun serve", "kind": "serve", "model": "nufasun", "size": "base", "requests": 2, "shortest": 700, "longest": 1500, "steps": 16},
        {"name": "vibunex serve", "kind": "serve", "model": "vibunex", "size": "base", "requests": 3, "shortest": 300, "longest": 1200, "steps": 8},
        {"name": "fevosun serve", "kind": "serve", "model": "fevosun", "size": "base", "requests": 1, "shortest": 3001, "longest": 3001, "steps": 16},
        {"name": "risizen serve", "kind": "serve", "model": "risizen", "size": "base", "requests": 8, "shortest": 60, "longest": 1000, "steps": 16},
        {"name": "samulorn serve", "kind": "serve", "model": "samulorn", "size": "base", "requests": 2, "shortest": 900, "longest": 1100, "steps": 16},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["serve"] * 6 + ["decode"] * 3 + ["prefill"] * 2 + ["mixed", "sample", "generate"])
    if kind == "sample":
        return {"kind": kind, "rows": _log_int(rng, 1, 128), "vocab": rng.choice([1000, 32000, 128256]),
                "temperature": round(rng.uniform(0.5, 1.2), 2), "top_p": rng.choice([1.0, 0.95, 0.9, 0.8]),
                "top_k": rng.choice([0, 0, 50, 200])}
    if kind == "generate":
        low = _log_int(rng, 1, 40)
        return {"kind": kind, "model": "llama-tiny", "requests": rng.randint(1, 8), "shortest": low,
                "longest": _log_int(rng, low, 250), "steps": rng.randint(4, 24)}
    if kind == "decode":
        model = rng.choice(["llama-8b", "llama-1b", "llama-3b"])
        low = _log_int(rng, 32, 1500)
        most = {"llama-8b": 12, "llama-1b": 64, "llama-3b": 24}[model]
        return {"kind": kind, "model": model, "requests": _log_int(rng, 1, most), "shortest": low,
                "longest": _log_int(rng, low, 2032), "steps": rng.randint(2, 8)}
    if kind == "prefill":
        return {"kind": kind, "model": rng.choice(["llama-8b", "llama-1b", "llama-3b"]), "tokens": _log_int(rng, 20, 2048)}
    if kind == "mixed":
        low = _log_int(rng, 1000, 12000)
        return {"kind": kind, "model": rng.choice(["llama-1b", "llama-3b"]), "requests": rng.randint(2, 5), "shortest": low,
                "longest": _log_int(rng, low, 16128), "tokens": _log_int(rng, 64, 2043)}
    n = _log_int(rng, 1, 8)
    high = _log_int(rng, 60, 3600 // n)
    return {"kind": kind, "model": rng.choice(sorted(DESIGNS)), "size": rng.choice(["narrow", "base", "base"]), "requests": n,
            "shortest": max(17, high // rng.choice([1, 2, 8])), "longest": max(17, high), "steps": rng.randint(4, 16)}


def _lengths(case):
    """The requests' lengths: spread over the logarithm of the range, ragged, in an order of their own, the case's alone."""
    n, low, high = case["requests"], case["shortest"], case["longest"]
    rng = random.Random(f"{n} {low} {high}")
    out = [_log_int(rng, low, high) for _ in range(n)]
    out[rng.randrange(n)] = high
    if case["kind"] in ("decode", "mixed"):        # requests are cut back to whole pages after a pass
        out = [max(PAGE, x // PAGE * PAGE) for x in out]
    return out


def _portions(lengths):
    """[(request, from, to)] a step: prompts first come, first served, at most BUDGET tokens a step."""
    steps, room = [[]], BUDGET
    for r, n in enumerate(lengths):
        a = 0
        while a < n:
            if room == 0:
                steps.append([])
                room = BUDGET
            b = min(n, a + room)
            steps[-1].append((r, a, b))
            room -= b - a
            a = b
    return steps


# ---- weights and inputs ------------------------------------------------------------------------------------------

def _generator(seed, salt):
    return torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + salt) % (1 << 62))


def _softplus_inverse(y):
    return torch.log(torch.expm1(y))


def _weights(case, seed):
    """Every tensor of the checkpoint, by name, as it would be stored (bfloat16)."""
    cfg = _config(case)
    shapes_of = Model(config_from_dict(cfg), torch.float32, "cpu")
    gen = _generator(seed, 1)
    depth = cfg["num_hidden_layers"] if "hidden_size" in cfg else len(cfg["layers"])
    tied = cfg.get("tie_word_embeddings") or cfg.get("architecture") == "Samulorn"
    embed_std = 0.05 if tied else 0.7 / ((cfg.get("embedding") or {}).get("scale") or 1.0)
    if cfg.get("architecture") == "Samulorn":
        embed_std = 1.0 / cfg["embedding"]["scale"]
    out = {}
    for name, shape in sorted(shapes_of.weight_shapes().items()):
        last = name.rsplit(".", 1)[-1]
        z = lambda: torch.randn(shape, generator=gen, device=DEVICE)                     # noqa: E731
        u = lambda a, b: a + (b - a) * torch.rand(shape, generator=gen, device=DEVICE)   # noqa: E731
        if last == "dt_bias":                  # steps of 0.001 to 0.1
            t = _softplus_inverse(torch.exp(u(math.log(0.001), math.log(0.1))))
        elif last == "A_log":
            t = torch.log(u(1.0, 16.0))
        elif last == "lam":                    # decays of 0.9 to 0.999 where the gate stands at one half
            t = _softplus_inverse(-torch.log(u(0.9, 0.999)) / 4.0)
        elif last == "w0":                     # decays of 0.7 to 0.999 a step
            t = u(-7.0, -1.0)
        elif last == "sink" or last == "u":
            t = z()
        elif last == "rel":
            t = 0.5 * z()
        elif last == "talk":
            t = torch.eye(shape[0], device=DEVICE) + 0.1 * z()
        elif last == "conv":
            t = 0.4 * z()
        elif ".mu." in name:
            t = u(0.0, 1.0)
        elif last in ("lq1", "lk1", "lq2", "lk2"):
            t = 0.1 * z()
        elif last == "correction":
            t = 0.01 * z()
        elif shapes_of.norm_like(name):
            t = 1.0 + 0.1 * z()
        elif shapes_of.identity_like(name):
            t = torch.eye(shape[0], device=DEVICE) + 0.02 * z()
        else:
            std = 0.02
            if last in ("o", "down") or name.endswith(("o_proj.weight", "down_proj.weight")):
                std /= math.sqrt(2.0 * depth)
            elif last == "router":
                std = 0.005
            elif name in ("embed", "model.embed_tokens.weight"):
                std = embed_std
            t = torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, std, generator=gen)
        out[name] = t.to(torch.bfloat16)
    _route_by_token(cfg, out, gen, embed_std)
    return out


def _route_by_token(cfg, weights, gen, embed_std):
    """Give every token its experts: a direction an expert, added to the token's embedding and, in another order in every layer,
    to the router's rows. With groups of experts a token's experts lie two by two in as many groups as are kept."""
    router = next((x["mlp"]["router"] for x in cfg.get("layers", []) if x.get("mlp") and "router" in x["mlp"]), None)
    if router is None:
        return
    embed, groups = weights["embed"], router.get("groups")
    V, d = embed.shape
    rows = router["experts"] + router.get("identity", 0)
    way = torch.nn.functional.normalize(torch.randn(rows, d, generator=gen, device=DEVICE), dim=-1)
    if groups:
        size = rows // groups["count"]
        pick = torch.rand(V, groups["count"], generator=gen, device=DEVICE).topk(groups["keep"], -1).indices
        each = router["top"] // groups["keep"]
        within = torch.rand(V, groups["keep"], size, generator=gen, device=DEVICE).topk(each, -1).indices
        own = (pick[:, :, None] * size + within).flatten(1)
    else:
        own = torch.rand(V, rows, generator=gen, device=DEVICE).topk(router["top"], -1).indices
    weights["embed"] = (embed + 0.45 * embed_std * math.sqrt(d) * way[own].sum(1)).to(torch.bfloat16)
    for name in weights:
        if name.endswith(".router"):
            order = torch.arange(rows, device=DEVICE)
            if groups:                             # groups change places as a whole
                turn = torch.randint(0, groups["count"], (1,), generator=gen, device=DEVICE)
                order = (order + turn * (rows // groups["count"])) % rows
            else:
                order = torch.randperm(rows, generator=gen, device=DEVICE)
            weights[name] = (weights[name] + 0.2 * way[order]).to(torch.bfloat16)


def _model(case, seed):
    model = Model(config_from_dict(_config(case)), torch.float32 if case["kind"] == "generate" else torch.bfloat16, DEVICE)
    stored = _weights(case, seed)
    tensors = {}
    for name in sorted(stored):
        tensors[name] = place(stored.pop(name), model.keeps_dtype(name), model.dtype, model.device)
    model.load_weights(tensors)
    return model


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _tokens(case, seed):
    """Per request the tokens of its prompt (or context) and the given tokens behind it."""
    vocab = _vocab(_config(case))
    gen = torch.Generator().manual_seed(seed * 7919 + 5)
    rand = lambda n: torch.randint(0, vocab, (n,), generator=gen).tolist()              # noqa: E731
    if case["kind"] == "prefill":
        return [rand(case["tokens"])]
    lengths = _lengths(case)
    if case["kind"] == "mixed":                    # the last request brings a portion, the others a row each
        return [rand(n + 1) for n in lengths[:-1]] + [rand(lengths[-1] + case["tokens"])]
    if case["kind"] == "generate":
        return [rand(n) for n in lengths]
    return [rand(n + case["steps"]) for n in lengths]


class _State:
    """A runner with its model, and the steps of a pass: lists of step entries, made of the given tokens."""


def _plan(case, seed):
    """(prompt steps, decode steps) of a pass: lists of entry lists."""
    seqs = _tokens(case, seed)
    kind = case["kind"]
    if kind == "prefill":
        return [[StepEntry("r0", seqs[0], [len(seqs[0]) - 1])]], []
    lengths = _lengths(case)
    if kind == "mixed":
        rows = [StepEntry(f"r{i}", [s[-1]], [0]) for i, s in enumerate(seqs[:-1])]
        tail = seqs[-1][lengths[-1]:]
        return [[StepEntry(f"r{len(seqs) - 1}", tail, [len(tail) - 1])] + rows], []
    prompt = [[StepEntry(f"r{r}", seqs[r][a:b], [b - a - 1] if b == lengths[r] else []) for r, a, b in step]
              for step in _portions(lengths)]
    given = (lambda r, i: seqs[r][lengths[r] + i]) if kind != "generate" else (lambda r, i: 0)
    decode = [[StepEntry(f"r{r}", [given(r, i)], [0]) for r in range(len(seqs))] for i in range(case["steps"])]
    return ([] if kind == "decode" else prompt), decode


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    if s.kind == "sample":
        gen = _generator(seed, 3)
        # a head's logits: a bell of width two and a few tokens that stand out
        s.logits = 2.0 * torch.randn(case["rows"], case["vocab"], generator=gen, device=DEVICE)
        lead = torch.randint(0, case["vocab"], (case["rows"], 8), generator=gen, device=DEVICE)
        s.logits.scatter_add_(1, lead, 6.0 + 3.0 * torch.randn(case["rows"], 8, generator=gen, device=DEVICE))
        s.sampler = Sampler(DEVICE, case["rows"])
        p = SamplingParams(temperature=case["temperature"], top_p=case["top_p"], top_k=case["top_k"])
        s.rows = [(p, seed * 1000 + r, r % 97) for r in range(case["rows"])]
        return s
    torch.cuda.set_device(0)
    seqs = _tokens(case, seed)
    longest = max(len(t) for t in seqs) + case.get("steps", 0)
    pages = sum(-(-(len(t) + case.get("steps", 0)) // PAGE) + 1 for t in seqs)
    s.runner = ModelRunner(_model(case, seed), page_size=PAGE, num_pages=pages, max_requests=len(seqs),
                           max_step_tokens=BUDGET + len(seqs), max_seq_len=longest)
    s.names = [f"r{i}" for i in range(len(seqs))]
    s.sampler = Sampler(DEVICE, len(seqs)) if s.kind == "generate" else None
    s.keep = None
    if s.kind in ("decode", "mixed"):              # the contexts are in the cache before the pass
        s.keep = _lengths(case)
        for step in _portions(s.keep):
            s.runner.step([StepEntry(f"r{r}", seqs[r][a:b], []) for r, a, b in step])
    rows = [len(e.want) for step in sum(_plan(case, seed), []) for e in step]
    s.logits = torch.empty(sum(rows), _vocab(_config(case)), device=DEVICE)
    s.ids = torch.empty(sum(rows), dtype=torch.int32, device=DEVICE)
    s.prompt, s.decode = _plan(case, seed + 1)     # a server has run before: its graphs are recorded, its scratch is there
    run(s)
    s.prompt, s.decode = _plan(case, seed)
    s.runner.check_status()
    return s


def run(s):
    if s.kind == "sample":
        return s.sampler.sample(s.logits, s.rows)
    runner, at = s.runner, 0
    greedy = [(SamplingParams(), 0, 0)] * len(s.names)
    rows = list(range(len(s.names)))

    def keep(logits):
        nonlocal at
        n = logits.shape[0]
        s.logits[at:at + n].copy_(logits)
        if s.sampler is not None:
            s.ids[at:at + n].copy_(s.sampler.sample(logits, greedy))
        at += n

    for entries in s.prompt:
        logits = runner.step(entries)
        if logits is not None:
            keep(logits)
    for entries in s.decode:
        # drawn tokens pass to the next step on the device
        keep(runner.step_decode_graph(entries, feed=None if s.sampler is None else (s.sampler.last_ids(), rows, rows)))
    for i, name in enumerate(s.names):
        if s.keep is None:
            runner.finish(name)
        else:
            runner.manager.truncate(name, s.keep[i])
    return {"logits": s.logits} if s.sampler is None else {"logits": s.logits, "ids": s.ids}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _attention_layers(cfg):
    """[(query heads x (key + value size), cached numbers a token)] per layer that attends."""
    if "hidden_size" in cfg:
        h, g, hs = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        return [(h * 2 * hs, g * 2 * hs)] * cfg["num_hidden_layers"]
    out = []
    for layer in cfg["layers"]:
        m = layer["mixer"].get("left", layer["mixer"])
        if layer["type"].startswith("latent"):
            out.append((m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["kv_rank"] + m["rot_dim"]))
        elif "attention" in layer["type"] or layer["type"] == "parallel":
            maps = 2 if "diff" in m else 1
            values = 0 if cfg["architecture"] == "Fevosun" else m["vdim"]
            out.append((m["heads"] * maps * (m["dim"] + m["vdim"]), m["kv_heads"] * (maps * m["dim"] + values)))
    return out


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * (case["vocab"] + 1), "flops": 0.0}
    cfg = _config(case)
    shapes = Model(config_from_dict(cfg), torch.float32, "cpu").weight_shapes()
    item = 4 if case["kind"] == "generate" else 2
    count = lambda keep: sum(math.prod(s) for n, s in shapes.items() if len(s) >= 2 and keep(n))     # noqa: E731
    table = lambda n: "embed" in n or n == "bigram"                                   # noqa: E731
    is_expert = lambda n: ".mlp.e" in n                                               # noqa: E731
    is_head = lambda n: n in ("head", "lm_head.weight")                               # noqa: E731
    dense, experts = count(lambda n: not (table(n) or is_expert(n) or is_head(n))), count(is_expert)
    head = _vocab(cfg) * (cfg.get("hidden_size") or cfg["width"])
    router = next((x["mlp"]["router"] for x in cfg.get("layers", []) if x.get("mlp") and "router" in x["mlp"]), None)
    prompt, decode = _plan(case, 0)
    held = dict.fromkeys(f"r{i}" for i in range(64))
    if case["kind"] in ("decode", "mixed"):
        held.update({f"r{i}": n for i, n in enumerate(_lengths(case))})
    nbytes = flops = 0.0
    for entries in prompt + decode:
        T, R = sum(len(e.tokens) for e in entries), sum(len(e.want) for e in entries)
        used = top = 0.0
        if router:
            rows = router["experts"] + router.get("identity", 0)
            top = router["top"] / rows
            used = 1.0 - (1.0 - top) ** T
        nbytes += item * (dense + used * experts + (head if R else 0)) + 4.0 * R * _vocab(cfg)
        flops += 2.0 * (T * (dense + top * experts) + R * head)
        for e in entries:
            n, before = len(e.tokens), held[e.req] or 0
            for sums, cached in _attention_layers(cfg):
                flops += 2.0 * sums * (n * before + n * (n + 1) / 2)
                nbytes += item * cached * (before + 2 * n)
            held[e.req] = before + n
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":                   # a draw on the border of two tokens may fall either way
        return {"rel": 0.0, "max": 0.0, "differ": 0.01}
    if case["kind"] == "generate":                 # 2e-7 from the exact sums
        return {"rel": 2e-6, "max": 2e-5, "differ": 0.0}
    # bfloat16 against the exact sums: 0.010 to 0.017 for these depths of Llama, 0.009 for Nufasun, 0.002 to 0.006 for the others
    if case["model"] in LLAMAS or case["model"] == "nufasun":
        return {"rel": 0.03, "max": 0.3, "differ": 0.0}
    return {"rel": 0.015, "max": 0.3, "differ": 0.0}


# ---- the same in 64 bits, as plain torch -----------------------------------------------------------------------------
# Whole sequences, no cache: ``x`` holds the rows of all sequences one after another, ``segs`` where each lies.

def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _limited(g, u, limit):
    g, u = torch.clamp(g, max=limit), torch.clamp(u, -limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _frequencies(dims, base, sc=None):
    """(angle a position of every pair, factor on sines and cosines), with either of the two rules that lower long waves."""
    i = torch.arange(dims // 2, dtype=F64, device=DEVICE)
    f = base ** (-2.0 * i / dims)
    if not sc:
        return f, 1.0
    if "fast" in sc:
        edge = lambda t: dims * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))   # noqa: E731
        lo, hi = max(math.floor(edge(sc["fast"])), 0), min(math.ceil(edge(sc["slow"])), dims - 1)
        r = torch.clamp((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
        return f / sc["factor"] * r + f * (1.0 - r), 0.1 * math.log(sc["factor"]) + 1.0
    s = torch.clamp((sc["original"] * f / (2.0 * math.pi) - sc["low"]) / (sc["high"] - sc["low"]), 0.0, 1.0)
    return (1.0 - s) * f / sc["factor"] + s * f, 1.0


def _rotate(x, dims, base, sc=None, pairs=False):
    """x [T, heads, size], rows at positions 0 .. T - 1; ``pairs``: neighbours are turned together, else halves."""
    f, mag = _frequencies(dims, base, sc)
    a = torch.arange(x.shape[0], dtype=F64, device=DEVICE)[:, None, None] * f
    c, s = mag * torch.cos(a), mag * torch.sin(a)
    one, two = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., one], x[..., two]
    out = x.clone()
    out[..., one], out[..., two] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, sink=None, cap=None, change=None, window=None, chunk=None):
    """q [T, H, dk], k [T, G, dk], v [T, G, dv] -> [T, H, dv]. ``change(scores, head, i, j)``: what joins the scaled scores."""
    T, H = q.shape[:2]
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=DEVICE)
    j = torch.arange(T, device=DEVICE)[None, :]
    block = max(1, (1 << 27) // max(T, 1))
    for a in range(0, T, block):
        i = torch.arange(a, min(T, a + block), device=DEVICE)[:, None]
        seen = j <= i
        if window:
            seen &= i - j < window
        if chunk:
            seen &= i // chunk == j // chunk
        for h in range(H):
            g = h * k.shape[1] // H
            s = (q[a:a + block, h] @ k[:, g].T) * scale
            s = cap * torch.tanh(s / cap) if cap else s
            s = change(s, h, i, j) if change else s
            s = s.masked_fill_(~seen, -math.inf)
            m = s.amax(-1, keepdim=True)
            if sink is not None:
                m = torch.maximum(m, sink[h])
            e = torch.exp(s - m)
            den = e.sum(-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(sink[h] - m)
            out[a:a + block, h] = (e / den) @ v[:, g]
    return out


def _conv(x, taps):
    """Causal convolution over time of every channel: x [T, C], taps [C, K]."""
    K = taps.shape[1]
    xp = torch.cat([torch.zeros(K - 1, x.shape[1], dtype=F64, device=DEVICE), x])
    return sum(xp[n:n + x.shape[0]] * taps[:, n] for n in range(K))


class _Plain:
    def __init__(self, cfg, weights, seqs):
        self.cfg, self.weights = cfg, weights
        self.tokens = torch.tensor([t for s in seqs for t in s], device=DEVICE)
        self.segs, a = [], 0
        for s in seqs:
            self.segs.append(slice(a, a + len(s)))
            a += len(s)
        self.eps = cfg["rms_norm_eps"] if "hidden_size" in cfg else cfg["norm"]["eps"]

    def w(self, name):
        return self.weights[name].to(F64)

    def mm(self, x, name):
        return x @ self.w(name).T

    def each(self, fn, *rows):
        """``fn`` on every sequence's rows, put together again."""
        return torch.cat([fn(*(r[s] for r in rows)) for s in self.segs])

    # -- llama

    def llama(self, want):
        c = self.cfg
        H, G, hs, sc = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rope_scaling"]
        rot = (hs, c["rope_theta"], {"original": sc["original_max_position_embeddings"], "factor": sc["factor"],
                                     "low": sc["low_freq_factor"], "high": sc["high_freq_factor"]})
        x = self.weights["model.embed_tokens.weight"][self.tokens].to(F64)
        for n in range(c["num_hidden_layers"]):
            p = f"model.layers.{n}."
            h = _rms(x, self.eps, self.w(p + "input_layernorm.weight"))
            q, k, v = (self.mm(h, p + f"self_attn.{o}_proj.weight").view(len(h), -1, hs) for o in "qkv")
            x = x + self.mm(self.each(lambda q, k, v: _attend(_rotate(q, *rot), _rotate(k, *rot), v, hs ** -0.5), q, k, v).flatten(1),
                            p + "self_attn.o_proj.weight")
            h = _rms(x, self.eps, self.w(p + "post_attention_layernorm.weight"))
            x = x + self.mm(_silu(self.mm(h, p + "mlp.gate_proj.weight")) * self.mm(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        return self.mm(_rms(x[want], self.eps, self.w("model.norm.weight")),
                       "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight")

    # -- mixers

    def latent(self, h, p, m, sink=False, pairs=False, window=None):
        H, dk, dr, dv, rk = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        q = self.mm(_rms(self.mm(h, p + "dq"), self.eps, self.w(p + "dq.norm")), p + "uq") if m.get("q_rank") else self.mm(h, p + "q")
        q = q.view(-1, H, dk + dr)
        kv = self.mm(h, p + "dkv")
        c = _rms(kv[:, :rk], self.eps, self.w(p + "dkv.norm"))
        kp, v, kr = self.mm(c, p + "uk").view(-1, H, dk), self.mm(c, p + "uv").view(-1, H, dv), kv[:, rk:].view(-1, 1, dr)
        turn = lambda t: _rotate(t, m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"), pairs)       # noqa: E731

        def one(q, kp, kr, v):
            k = torch.cat([kp, turn(kr).expand(-1, H, -1)], -1)
            return _attend(torch.cat([q[..., :dk], turn(q[..., dk:])], -1), k, v, m["scale"], self.w(p + "sink") if sink else None, window=window)
        return self.mm(self.each(one, q, kp, kr, v).flatten(1), p + "o")

    def biased(self, h, p, m):
        q, k, v = (self.mm(h, p + n).view(len(h), -1, s) for n, s in (("q", m["dim"]), ("k", m["dim"]), ("v", m["vdim"])))
        rel = self.w(p + "rel")
        rows = rel.shape[0]
        half = rows // 2
        far = torch.arange(max(s.stop - s.start for s in self.segs), device=DEVICE).to(F64)
        log = half + torch.floor(torch.log(far.clamp(min=half) / half) / math.log(m["bias_max"] / half) * (rows - half))
        bucket = torch.where(far < half, far, log.clamp(max=rows - 1)).long()
        change = lambda s, hd, i, j: s + rel[:, hd][bucket[(i - j).clamp(min=0)]]                             # noqa: E731
        return self.mm(self.each(lambda q, k, v: _attend(q, k, v, m["scale"], change=change), q, k, v).flatten(1), p + "o")

    def state_space(self, h, p, m):
        heads, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = heads * P
        z, xbc, dt = self.mm(h, p + "in").split([inner, inner + 2 * G * N, heads], -1)
        xbc = _silu(self.each(lambda t: _conv(t, self.w(p + "conv")) + self.w(p + "conv.b"), xbc))
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias"))
        decay = torch.exp(-torch.exp(self.w(p + "A_log")) * dt)

        def scan(xbc, dt, decay):
            x, B, C = xbc.split([inner, G * N, G * N], -1)
            x = x.reshape(-1, heads, P)
            B, C = (t.reshape(-1, G, N).repeat_interleave(heads // G, 1) for t in (B, C))
            S, y = torch.zeros(heads, N, P, dtype=F64, device=DEVICE), []
            for t in range(x.shape[0]):
                S = decay[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
                y.append(torch.einsum("hnp,hn->hp", S, C[t]))
            return torch.stack(y) + self.w(p + "D")[:, None] * x
        y = self.each(scan, xbc, dt, decay).flatten(1) * _silu(z)
        y = _rms(y.view(len(h), m["norm_groups"], -1), self.eps).flatten(1) * self.w(p + "norm")
        return self.mm(y, p + "o")

    def differential(self, h, p, m):
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        turn = lambda t: _rotate(t, m["rot"]["dims"], m["rot"]["base"], pairs=True)                           # noqa: E731
        q = _rms(self.mm(h, p + "q").view(-1, H * 2, dk), self.eps, self.w(p + "q.norm"))
        k = _rms(self.mm(h, p + "k").view(-1, G * 2, dk), self.eps, self.w(p + "k.norm"))
        v = self.mm(h, p + "v").view(-1, G, dv)
        lam = (torch.exp((self.w(p + "lq1") * self.w(p + "lk1")).sum()) - torch.exp((self.w(p + "lq2") * self.w(p + "lk2")).sum()) + m["diff"])

        def one(q, k, v):
            q, k = turn(q), turn(k)
            a = [_attend(q[:, n::2], k[:, n::2], v, m["scale"], cap=m["softcap"], window=m["mask"]["size"]) for n in range(2)]
            return a[0] - lam * a[1]
        o = _rms(self.each(one, q, k, v), self.eps) * (1.0 - m["diff"]) * torch.sigmoid(self.mm(h, p + "g"))[:, :, None]
        return self.mm(o.flatten(1), p + "o")

    def delta(self, h, p, m, channel=False):
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        conv = lambda n: _silu(self.each(lambda t: _conv(t, self.w(p + n + ".conv")), self.mm(h, p + n)))     # noqa: E731
        q, k = (_unit(conv(n).view(-1, G, dk)).repeat_interleave(H // G, 1) for n in "qk")
        v = conv("v").view(-1, H, dv)
        beta = torch.sigmoid(self.mm(h, p + "b"))
        dt = self.mm(self.mm(h, p + "a1"), p + "a2") if channel else self.mm(h, p + "a")
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias")).view(len(h), H, -1)
        decay = torch.exp(-torch.exp(self.w(p + "A_log"))[None, :, None] * dt)

        def scan(q, k, v, beta, decay):
            S, out = torch.zeros(H, dk, dv, dtype=F64, device=DEVICE), []
            for t in range(q.shape[0]):
                S = decay[t][:, :, None] * S
                u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
                S = S + k[t][:, :, None] * u[:, None, :]
                out.append(torch.einsum("hkv,hk->hv", S, q[t]))
            return torch.stack(out)
        o = _rms(self.each(scan, q * dk ** -0.5, k, v, beta, decay), self.eps) * self.w(p + "norm")
        gate = torch.sigmoid(self.mm(self.mm(h, p + "g1"), p + "g2")) if channel else _silu(self.mm(h, p + "g"))
        return self.mm((o * gate.view(-1, H, dv)).flatten(1), p + "o")

    def talking(self, h, p, m):
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q = _rms(self.mm(h, p + "q"), self.eps, self.w(p + "q.norm")).view(-1, H, dk)
        k = _rms(self.mm(h, p + "k"), self.eps, self.w(p + "k.norm")).view(-1, G, dk)
        v = self.mm(h, p + "v").view(-1, G, dv)
        turn = lambda t: _rotate(t, m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))              # noqa: E731
        talk, own = self.w(p + "talk"), torch.arange(H, device=DEVICE) // (H // G)

        def one(q, k, v):                          # every head's weights on every value head, then the mix
            wide = v.flatten(1)[:, None, :].expand(-1, G, -1)
            a = _attend(turn(q), turn(k), wide, m["scale"], self.w(p + "sink")).view(-1, H, G, dv)
            return torch.einsum("hg,tghd->thd", talk, a[:, :, own])
        return self.mm(self.each(one, q, k, v).flatten(1) * torch.sigmoid(self.mm(h, p + "g")), p + "o")

    def time_mix(self, h, p, m):
        H, n = m["heads"], m["dim"]
        prev = self.each(lambda t: torch.cat([torch.zeros_like(t[:1]), t[:-1]]), h)
        mix = lambda s: h + (prev - h) * self.w(p + "mu." + s)                                                # noqa: E731
        r, k, v = (self.mm(mix(s), p + s).view(-1, H, n) for s in "rkv")
        gate = _silu(self.mm(mix("g"), p + "g"))
        decay = torch.exp(-torch.exp(self.mm(torch.tanh(self.mm(mix("w"), p + "w1")), p + "w2") + self.w(p + "w0"))).view(-1, H, n)
        u = self.w(p + "u")

        def scan(r, k, v, decay):
            S, out = torch.zeros(H, n, n, dtype=F64, device=DEVICE), []
            for t in range(r.shape[0]):
                kv = k[t][:, :, None] * v[t][:, None, :]
                out.append(torch.einsum("hkv,hk->hv", S + u[:, :, None] * kv, r[t]))
                S = decay[t][:, :, None] * S + kv
            return torch.stack(out)
        return self.mm(_rms(self.each(scan, r, k, v, decay), self.eps).flatten(1) * self.w(p + "norm") * gate, p + "o")

    def keys_as_values(self, h, p, m):
        H, G, dk = m["heads"], m["kv_heads"], m["dim"]
        q, k = self.mm(h, p + "q").view(-1, H, dk), self.mm(h, p + "k").view(-1, G, dk)
        penalty = lambda s, hd, i, j: s - 2.0 ** (-8.0 * (hd + 1) / H) * (i - j)                              # noqa: E731

        def one(q, k):
            pos = torch.arange(len(q), device=DEVICE).to(F64)
            warm = 1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / m["q_temp"]["every"]) + 1.0)
            return _attend(q * warm[:, None, None], k, k, m["scale"], change=penalty, window=m["mask"]["size"])
        return self.mm(self.each(one, q, k).flatten(1) * torch.sigmoid(self.mm(h, p + "g")), p + "o")

    def recurrence(self, h, p, m):
        y = _gelu(self.mm(h, p + "y") + self.w(p + "y.b"))
        u = self.each(lambda t: _conv(t, self.w(p + "conv")) + self.w(p + "conv.b"), self.mm(h, p + "x") + self.w(p + "x.b"))
        ub = u.view(len(h), m["blocks"], -1)
        gate = lambda n: torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, self.w(p + n)) + self.w(p + n + ".b")).flatten(1)   # noqa: E731
        la = -8.0 * gate("ra") * torch.nn.functional.softplus(self.w(p + "lam"))
        add = torch.sqrt(1.0 - torch.exp(2.0 * la)) * gate("ri") * u

        def scan(a, add):
            S, out = torch.zeros_like(add[0]), []
            for t in range(len(a)):
                S = a[t] * S + add[t]
                out.append(S)
            return torch.stack(out)
        return self.mm(self.each(scan, torch.exp(la), add) * y, p + "o")

    def rotated(self, h, p, m):
        """Attention behind biases, a short convolution and a rotation, heads over their root mean square."""
        q, k, v = (self.each(lambda t: _conv(t, self.w(p + n + ".conv")), self.mm(h, p + n) + self.w(p + n + ".b")) for n in "qkv")
        turn = lambda t: _rotate(t, m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"], True)            # noqa: E731
        heads = lambda t, n: t.view(len(t), n, -1)                                                            # noqa: E731

        def one(q, k, v):
            q, k = (_rms(turn(heads(t, n)), self.eps) for t, n in ((q, m["heads"]), (k, m["kv_heads"])))
            return _attend(q, k, heads(v, m["kv_heads"]), m["scale"])
        return self.mm(self.each(one, q, k, v).flatten(1), p + "o")

    def chunked(self, h, p, m, kept):
        """Attention behind biases and short convolutions, in chunks, one more in the denominator; may read kept keys."""
        take = lambda n: self.each(lambda t: _conv(t, self.w(p + n + ".conv")), self.mm(h, p + n) + self.w(p + n + ".b"))   # noqa: E731
        if kept is None:
            kept = _rms(take("k").view(len(h), m["kv_heads"], -1), self.eps), take("v").view(len(h), m["kv_heads"], -1)
        q = _rms(take("q").view(len(h), m["heads"], -1), self.eps)
        sink = torch.zeros(m["heads"], dtype=F64, device=DEVICE)
        o = self.each(lambda q, k, v: _attend(q, k, v, m["scale"], sink, chunk=m["mask"]["size"]), q, *kept)
        return self.mm(o.flatten(1), p + "o"), kept

    # -- feed-forwards

    def experts(self, h, p, mlp, chosen, weights, fn):
        out = torch.zeros_like(h)
        for e in range(mlp["router"]["experts"]):
            rows, place_ = (chosen == e).nonzero(as_tuple=True)
            if len(rows):
                out.index_add_(0, rows, fn(h[rows], f"{p}e{e}.") * weights[rows, place_][:, None])
        return out

    def squared(self, h, p):
        return self.mm(torch.relu(self.mm(h, p + "up")) ** 2, p + "down")

    def gated(self, h, p):
        return self.mm(_silu(self.mm(h, p + "gate")) * self.mm(h, p + "up"), p + "down")

    def limited(self, h, p, limit, biased=False):
        b = (lambda n: self.w(p + n + ".b")) if biased else (lambda n: 0.0)
        return self.mm(_limited(self.mm(h, p + "gate") + b("gate"), self.mm(h, p + "up") + b("up"), limit), p + "down") + b("down")

    # -- the designs

    def mivorax(self, x):
        bg = self.cfg["embedding"]["bigram"]
        pair = self.each(lambda t: torch.cat([torch.full_like(t[:1], bg["buckets"]),
                                              (t[:-1] * bg["mul_prev"] + t[1:] * bg["mul_cur"]) % bg["buckets"]]), self.tokens)
        x = x + self.weights["bigram"][pair].to(F64)
        for n, layer in enumerate(self.cfg["layers"]):
            p, m = f"l{n}.", layer["mixer"]
            h = _rms(x, self.eps, self.w(p + "norm1"))
            x = x + {"attention": self.biased, "mamba2": self.state_space,
                     "latent_attention": lambda h, p, m: self.latent(h, p, m, sink=True)}[layer["type"]](h, p + "mix.", m)
            if layer["mlp"] is not None:
                x = x + self.squared(_rms(x, self.eps, self.w(p + "norm2")), p + "mlp.")
        return _rms(x, self.eps, self.w("final.norm"))

    def nufasun(self, x):
        x = x * self.cfg["embedding"]["scale"] + self.w("loop.step")[0]
        for n, layer in enumerate(self.cfg["layers"]):
            p = f"l{n}."
            h = _rms(x, self.eps, self.w(p + "norm1"))
            y = (self.differential if layer["type"] == "attention" else self.delta)(h, p + "mix.", layer["mixer"])
            x = x + _rms(y, self.eps, self.w(p + "norm1b"))
            h = _rms(x, self.eps, self.w(p + "norm2"))
            x = x + _rms(self.limited(h, p + "mlp.", layer["mlp"]["limit"], True), self.eps, self.w(p + "norm2b"))
        return _rms(x, self.eps, self.w("final.norm"))

    def vibunex(self, x):
        for n, layer in enumerate(self.cfg["layers"]):
            p, m, mlp = f"l{n}.", layer["mixer"], layer["mlp"]
            h1, h2 = (_rms(x, self.eps) * self.w(p + k) for k in ("norm1", "norm2"))
            mixed = m["left_scale"] * self.talking(h1, p + "mix.left.", m["left"]) + m["right_scale"] * self.time_mix(h1, p + "mix.right.", m["right"])
            s = torch.sigmoid(self.mm(h2, p + "mlp.router"))
            top = torch.topk(s, mlp["router"]["top"], dim=-1)
            ff = self.experts(h2, p + "mlp.", mlp, top.indices, top.values * mlp["router"]["scale"], self.squared)
            ff = ff + self.squared(h2, p + "mlp.shared.") * torch.sigmoid(self.mm(h2, p + "mlp.shared.sg"))
            gate = lambda h, k: torch.sigmoid(self.mm(h, p + k) + self.w(p + k + ".b"))                       # noqa: E731
            x = x + self.cfg["residual_mult"] * (mixed * gate(h1, "rg1") + ff * gate(h2, "rg2"))
        return _rms(x, self.eps) * self.w("final.norm")

    def fevosun(self, x):
        x = x * self.cfg["embedding"]["scale"]
        for n, layer in enumerate(self.cfg["layers"]):
            p, m, mlp = f"l{n}.", layer["mixer"], layer["mlp"]
            h = _rms(x, self.eps, 1.0 + self.w(p + "norm1"))
            if layer["type"] == "attention":
                d = self.keys_as_values(h, p + "mix.", m)
            else:
                d = self.latent(h, p + "mix.", m, pairs=layer["type"].endswith("2"), window=m["mask"]["size"])
            if mlp["kind"] == "dense":
                d = d + self.gated(h, p + "mlp.")
            else:
                s = torch.softmax(self.mm(h, p + "mlp.router"), -1)
                ids = torch.topk(s + self.w(p + "mlp.correction"), mlp["router"]["top"], dim=-1).indices
                kept, limit = torch.gather(s, 1, ids), mlp["expert"]["limit"]
                d = d + self.experts(h, p + "mlp.", mlp, ids, kept, lambda r, q: self.limited(r, q, limit))
                d = d + h * (kept * (ids >= mlp["router"]["experts"])).sum(-1, keepdim=True)
                d = d + self.limited(h, p + "mlp.shared.", mlp["shared"]["limit"])
            x = x + d
        return _rms(x, self.eps, 1.0 + self.w("final.norm"))

    def risizen(self, x):
        x = _rms(x, self.eps, self.w("embed.norm"))[None].repeat(self.cfg["streams"], 1, 1)
        kept = {}
        read = lambda x, p: torch.einsum("s,std->td", self.w(p + "in"), x)                                    # noqa: E731
        write = lambda x, y, p: torch.einsum("sz,std->ztd", self.w(p + "mix"), x) + self.w(p + "out").view(-1, 1, 1) * y   # noqa: E731
        for n, layer in enumerate(self.cfg["layers"]):
            p, m = f"l{n}.", layer["mixer"]
            h = _rms(read(x, p + "hc1."), self.eps, self.w(p + "norm1"))
            y, kept[n] = self.chunked(h, p + "mix.", m, kept.get(m.get("kv_from")))
            x = write(x, y, p + "hc1.")
            h = _rms(read(x, p + "hc2."), self.eps, self.w(p + "norm2"))
            x = write(x, self.limited(h, p + "mlp.", layer["mlp"]["limit"]), p + "hc2.")
        return _rms(x.sum(0), self.eps, self.w("final.norm")) * self.cfg["logit_scale"]

    def samulorn(self, x):
        x = x * self.cfg["embedding"]["scale"]
        dim = self.cfg["token_side"]["dim"]
        side = self.weights["side.embed"][self.tokens].to(F64)
        soft = lambda x, n: torch.tanh(self.w(n + ".alpha") * x) * self.w(n) + self.w(n + ".b")               # noqa: E731
        for n, layer in enumerate(self.cfg["layers"]):
            p, m, mlp = f"l{n}.", layer["mixer"], layer["mlp"]
            h = soft(x, p + "norm1")
            if layer["type"] == "parallel":
                y = m["left_scale"] * self.rotated(h, p + "mix.left.", m["left"]) + m["right_scale"] * self.recurrence(h, p + "mix.right.", m["right"])
            else:
                y = self.delta(h, p + "mix.", m, channel=True)
            x = x + soft(y, p + "norm1b")
            h = soft(x, p + "norm2")
            if mlp["kind"] == "dense":
                f = self.gated(h, p + "mlp.")
            else:
                r = mlp["router"]
                s = torch.sigmoid(self.mm(h, p + "mlp.router"))
                c = s + self.w(p + "mlp.correction")
                best = c.view(len(c), r["groups"]["count"], -1)
                keep = torch.topk(torch.topk(best, min(2, best.shape[-1]), dim=-1).values.sum(-1), r["groups"]["keep"], dim=-1).indices
                off = torch.ones(best.shape[:2], dtype=torch.bool, device=DEVICE).scatter_(1, keep, False)
                ids = torch.topk(best.masked_fill(off[:, :, None], -math.inf).flatten(1), r["top"], dim=-1).indices
                kept = torch.gather(s, 1, ids)
                f = self.experts(h, p + "mlp.", mlp, ids, r["scale"] * kept / (kept.sum(-1, keepdim=True) + 1e-20), self.gated)
            x = x + soft(f, p + "norm2b")
            own = _gelu(self.mm(x, p + "side.gate")) * side[:, n * dim:(n + 1) * dim]
            x = x + _rms(self.mm(own, p + "side.proj"), self.eps, self.w(p + "side.norm"))
        return soft(x, "final.norm")

    def logits(self, model, want):
        if model in LLAMAS:
            return self.llama(want)
        h = getattr(self, model)(self.weights["embed"][self.tokens].to(F64))[want]
        y = self.mm(h, "embed" if model == "samulorn" else "head")
        cap = self.cfg.get("logit_softcap")
        return cap * torch.tanh(y / cap) if cap else y


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "sample":
        return None
    cfg = _config(case)
    seqs = _tokens(case, seed)
    total = sum(len(t) for t in seqs)
    if case["model"] in LLAMAS:
        per_token = 2.0 * sum(math.prod(s) for s in Model(config_from_dict(cfg), torch.float32, "cpu").weight_shapes().values())
        square = sum(len(t) ** 2 for t in seqs) * 2.0 * sum(a for a, _ in _attention_layers(cfg))
        if total * per_token + square > 3e14:      # more than some ten seconds of 64-bit sums
            return None
    weights = _weights(case, seed)
    names = {f"r{i}": i for i in range(len(seqs))}
    out = []
    if case["kind"] == "generate":
        ids = [list(s) for s in seqs]
        for _ in range(case["steps"] + 1):
            plain = _Plain(cfg, weights, ids)
            out.append(plain.logits(case["model"], torch.tensor([s.stop - 1 for s in plain.segs], device=DEVICE)))
            for r, t in zip(ids, out[-1].argmax(-1).tolist()):
                r.append(t)
        return {"logits": torch.cat(out), "ids": None}
    # the tokens that the pass brings to the cache, and the rows whose logits it asks for
    prompt, decode = _plan(case, seed)
    seen = _lengths(case) if case["kind"] in ("decode", "mixed") else [0] * len(seqs)
    plain = _Plain(cfg, weights, seqs)
    rows = []
    for entries in prompt + decode:
        for e in entries:
            r = names[e.req]
            rows += [plain.segs[r].start + seen[r] + w for w in e.want]
            seen[r] += len(e.tokens)
    return {"logits": plain.logits(case["model"], torch.tensor(rows, device=DEVICE))}
