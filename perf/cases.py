"""What this engine is asked to do, as cases that can be timed and checked.

A case is one step of the engine's step function (``Runtime`` and ``Executor.step``, which
``Engine.step``, ``bin/inferx-generate`` and ``bin/trace_run`` all go through): a batch of
requests that each bring one decoded token or a portion of a prompt, run against the cache
that earlier steps left.  The models are the seven designs the engine serves, at the sizes
of ``bench.py``: Qwen2-MoE at the Qwen1.5-MoE-A2.7B layer sizes, a dense Qwen2 for the 32-bit
mode, and the six other designs at widths 1024, 2048 and 4096 with their kinds of layers in
one stack.  Weights and the context that a request already holds are random, scaled so that
activations, gates and decays lie where trained models have them.

Outputs are the logits of the wanted rows, the pages of the cache and the per-request state.
"""
import math
import zlib

import numpy as np
import torch

from inferx_b200.config.registry import config_from_json
from inferx_b200.engine import Runtime, StepEntry, load_model
from inferx_b200.parts.base import BuildContext
from inferx_b200.parts.block import DecoderModel
from inferx_b200.weights.loader import WeightSource

PAGE = 16
VOCAB = 32000
LAYERS = 4


# -- the models ------------------------------------------------------------------------
# heads of 128 over `kv` key/value heads; experts, how many are chosen, their inner width and
# the shared expert's; the dense inner width; latent attention's plain, rotated and value
# entries per head, its latent and its query latent; the window of latent attention
SIZES = {
    1024: dict(heads=8, kv=2, experts=16, top=2, ff=512, shared=2048, dense=2816,
               latent=(96, 32, 128, 256, 384), window=1024),
    2048: dict(heads=16, kv=4, experts=32, top=4, ff=1024, shared=4096, dense=5632,
               latent=(128, 64, 128, 512, 768), window=4096),
    4096: dict(heads=32, kv=8, experts=32, top=4, ff=1408, shared=5632, dense=11008,
               latent=(128, 64, 128, 512, 1536), window=4096),
}


def qwen2_moe(width):
    """Qwen2-MoE at the Qwen1.5-MoE-A2.7B layer sizes (width 2048), 8 of its 24 layers."""
    return {"architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe",
            "num_hidden_layers": 8, "hidden_size": 2048, "num_attention_heads": 16,
            "num_key_value_heads": 16, "head_dim": 128, "num_experts": 60,
            "num_experts_per_tok": 4, "moe_intermediate_size": 1408,
            "shared_expert_intermediate_size": 5632, "intermediate_size": 5632,
            "decoder_sparse_step": 1, "mlp_only_layers": [], "norm_topk_prob": False,
            "vocab_size": 151936, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6,
            "use_sliding_window": False, "tie_word_embeddings": False}


def qwen2_dense(width):
    """Qwen2 with dense layers and a sliding window over half of them."""
    z = SIZES[width]
    return {"architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe",
            "num_hidden_layers": LAYERS, "hidden_size": width, "num_attention_heads": z["heads"],
            "num_key_value_heads": z["kv"], "head_dim": 128, "num_experts": 1,
            "num_experts_per_tok": 1, "moe_intermediate_size": 64,
            "shared_expert_intermediate_size": 0, "intermediate_size": z["dense"],
            "decoder_sparse_step": 1, "mlp_only_layers": list(range(LAYERS)),
            "norm_topk_prob": False, "vocab_size": VOCAB, "rope_theta": 1000000.0,
            "rms_norm_eps": 1e-6, "use_sliding_window": True, "sliding_window": 512,
            "layer_types": ["full_attention", "sliding_attention"] * (LAYERS // 2),
            "tie_word_embeddings": False}


def zuzisun(width):
    z = SIZES[width]
    dim, rot, vdim, rank, _ = z["latent"]
    mixer = {"heads": z["heads"], "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank,
             "scale": 1.0 / math.sqrt(dim + rot), "mask": {"size": z["window"]},
             "rot": {"base": 10000.0, "dims": rot,
                     "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    return {"architecture": "Zuzisun", "vocab": VOCAB, "width": width,
            "embedding": {"scale": math.sqrt(width)}, "norm": {"eps": 1e-6, "groups": 8},
            "layers": [{"type": "latent_attention", "mixer": mixer,
                        "mlp": {"kind": "dense", "ff": z["dense"], "limit": 7.0}}] * LAYERS}


def tinapel(width):
    z = SIZES[width]
    mlp = {"kind": "moe", "expert": {"ff": z["ff"]},
           "router": {"experts": z["experts"], "top": z["top"], "scale": 1.0},
           "shared": {"ff": z["shared"]}}
    wkv = {"type": "wkv", "mixer": {"heads": width // 64, "dim": 64, "rank": 64}, "mlp": mlp}
    gla = {"type": "gla", "mixer": {"heads": width // 128, "dim": 64, "vdim": 128, "tau": 8.0,
                                    "rank": 32}, "mlp": mlp}
    attn = {"type": "attention", "mixer": {
        "heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128,
        "scale": 1.0 / math.sqrt(128.0), "softcap": 30.0,
        "q_temp": {"coef": 0.1, "every": 1024}}, "mlp": mlp}
    return {"architecture": "Tinapel", "vocab": VOCAB, "width": width,
            "embedding": {"scale": math.sqrt(width)}, "norm": {"eps": 1e-6},
            "layers": [wkv, gla, attn, attn]}


def mapovik(width):
    z = SIZES[width]
    mlp = {"kind": "moe", "expert": {"ff": z["ff"]},
           "router": {"experts": z["experts"], "top": z["top"]}}
    both = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128,
                 "scale": 1.0 / math.sqrt(128.0),
                 "rot": {"dims": 64, "base": 10000.0, "scaling": {"factor": 2.0}}},
        "right": {"heads": width // 64, "vdim": 64, "state": 128, "groups": 2, "conv": 4,
                  "norm_groups": 2}}}
    delta = {"type": "channel_delta", "mlp": mlp, "mixer": {
        "heads": width // 128, "kv_heads": width // 128, "dim": 64, "vdim": 128, "conv": 4,
        "rank": 64, "gate_rank": 64}}
    return {"architecture": "Mapovik", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5},
            "residual_mult": 0.5, "logit_scale": 1.0, "layers": [both, delta, delta, both]}


def fudulix(width):
    z = SIZES[width]
    heads = {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128,
             "scale": 1.0 / math.sqrt(128.0), "v_mix": True}
    second = {"type": "attention_2", "mlp": {"kind": "dense", "ff": z["shared"]}, "mixer": dict(
        heads, conv=4, mask={"size": 1024, "keep_first": 4},
        rot={"dims": 128, "base": 1000000.0,
             "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}})}
    first = {"type": "attention", "mixer": dict(
        heads, mask={"size": 1024},
        rot={"dims": 64, "base": 10000.0,
             "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 2048}}),
        "mlp": {"kind": "moe", "expert": {"ff": z["ff"]}, "shared": {"ff": z["shared"]},
                "router": {"experts": z["experts"] - 2, "identity": 2, "top": z["top"],
                           "groups": {"count": 4, "keep": 2}}}}
    return {"architecture": "Fudulix", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
            "layers": [second, first, second, first]}


def dominex(width):
    z = SIZES[width]
    dim, rot, vdim, rank, q_rank = z["latent"]
    mlp = {"kind": "moe", "expert": {"ff": z["ff"]},
           "router": {"experts": z["experts"], "top": z["top"]}}
    both = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128,
                 "scale": 1.0 / math.sqrt(128.0), "mask": {"size": 8192}},
        "right": {"width": width}, "left_scale": 0.7, "right_scale": 0.7}}
    latent = {"heads": z["heads"], "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank,
              "q_rank": q_rank, "scale": 1.0 / math.sqrt(dim + rot),
              "rot": {"base": 10000.0, "dims": rot}}
    return {"architecture": "Dominex", "vocab": VOCAB, "width": width,
            "embedding": {"scale": math.sqrt(width)}, "norm": {"eps": 1e-6},
            "logit_softcap": 30.0,
            "layers": [both, {"type": "latent_attention", "mlp": mlp, "mixer": latent}, both,
                       {"type": "latent_attention", "mlp": mlp,
                        "mixer": dict(latent, kv_from=1)}]}


def biguzen(width):
    z = SIZES[width]
    mlp = {"kind": "moe", "expert": {"ff": z["ff"]}, "shared": {"ff": z["shared"]},
           "router": {"experts": z["experts"], "top": z["top"], "scale": 1.5,
                      "groups": {"count": 4, "keep": 2}}}
    memory = {"type": "mlstm", "mlp": mlp, "mixer": {
        "heads": width // 128, "dim": 64, "vdim": 128, "gate_cap": 15.0}}
    attn = {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128,
            "scale": 1.0 / math.sqrt(128.0), "conv": 4, "mask": {"size": 1024},
            "rot": {"dims": 64, "base": 10000.0, "scaling": {"factor": 2.0}}}
    return {"architecture": "Biguzen", "vocab": VOCAB, "width": width, "streams": 4,
            "norm": {"eps": 1e-6},
            "layers": [memory, {"type": "attention", "mlp": mlp, "mixer": attn}, memory,
                       {"type": "attention", "mlp": mlp, "mixer": dict(attn, kv_from=1)}]}


MODELS = {f.__name__: f for f in (qwen2_moe, qwen2_dense, zuzisun, tinapel, mapovik, fudulix,
                                  dominex, biguzen)}


# -- the cases -------------------------------------------------------------------------
def case_of(model, width=2048, decode=0, context=0, prompt=0, before=0, dtype="bfloat16"):
    """``decode`` requests bring one token each, the longest with ``context`` tokens before it;
    one request brings ``prompt`` tokens behind ``before`` earlier ones."""
    return {"model": model, "width": width, "dtype": dtype, "decode": decode,
            "context": context, "prompt": prompt, "before": before}


def listed():
    return [dict(case, name=name) for name, case in [
        # one user's chat: a token at a time, every launch and every weight counts
        ("qwen2_moe decode 1", case_of("qwen2_moe", decode=1, context=517)),
        # the headline of bench.py: eight sequences at 4,096 tokens of context
        ("qwen2_moe decode 8", case_of("qwen2_moe", decode=8, context=4096)),
        # a prompt in one step (the other headline)
        ("qwen2_moe prompt 2048", case_of("qwen2_moe", prompt=2048)),
        # continuous batching: a portion of a prompt beside sequences that decode
        ("qwen2_moe mixed", case_of("qwen2_moe", decode=20, context=1500, prompt=701, before=512)),
        # the 32-bit mode, in which a result is checked: a short prompt
        ("qwen2_dense fp32 prompt", case_of("qwen2_dense", prompt=600, dtype="float32")),
        # latent attention and token shift: a long prompt
        ("zuzisun prompt 3000", case_of("zuzisun", prompt=3000)),
        # wkv, gated linear attention, squashed attention: a prompt of an odd length
        ("tinapel prompt 1777", case_of("tinapel", prompt=1777)),
        # state space and delta rule: a prompt, and a full batch decoding
        ("mapovik prompt 2048", case_of("mapovik", prompt=2048)),
        ("mapovik decode 48", case_of("mapovik", decode=48, context=2000)),
        # windowed attention with prepared q, k, v: a batch decoding behind a long context
        ("fudulix decode 32", case_of("fudulix", decode=32, context=3000)),
        # attention with a distance penalty, gated recurrence, query latents: a wide model
        ("dominex prompt 1500", case_of("dominex", width=4096, prompt=1500)),
        # several streams, matrix memory, sinks and head gates: a prompt
        ("biguzen prompt 1024", case_of("biguzen", prompt=1024)),
    ]]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        model = rng.choice(["qwen2_moe", "qwen2_moe", "qwen2_moe", "qwen2_dense", "zuzisun",
                            "tinapel", "mapovik", "fudulix", "dominex", "biguzen"])
        width = 2048 if model == "qwen2_moe" else rng.choice([1024, 2048, 2048, 4096])
        if model == "qwen2_dense":
            case = case_of(model, width, prompt=_log_uniform(rng, 40, 800), dtype="float32")
        else:
            kind = rng.choice(["decode", "prompt", "prompt", "mixed"])
            decode = _log_uniform(rng, 1, 64)
            context = _log_uniform(rng, 100, min(8192, 131072 // decode))
            prompt = _log_uniform(rng, 33, 3000)
            if kind == "decode":
                case = case_of(model, width, decode=decode, context=context)
            elif kind == "prompt":
                case = case_of(model, width, prompt=prompt,
                               before=rng.choice([0, 0, _log_uniform(rng, 64, 2048)]))
            else:
                case = case_of(model, width, decode=min(decode, 32), context=min(context, 3000),
                               prompt=min(prompt, 1024), before=rng.choice([0, 512]))
        if _cost(case) <= most:
            return case


def sequences(case):
    """[(tokens already in the cache, new tokens)] of the batch: decoding requests of uneven
    lengths, the portion of a prompt last."""
    c = case["context"]
    out = [(max(1, c - (i * 37) % max(1, c // 3)), 1) for i in range(case["decode"])]
    if case["prompt"]:
        out.append((case["before"], case["prompt"]))
    return out


def config_of(case):
    return MODELS[case["model"]](case["width"])


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


# -- weights and contents ----------------------------------------------------------------
def _generator(seed, name):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) << 32) ^ zlib.crc32(name.encode()))
    return g


class RandomWeights(WeightSource):
    """Weights by (seed, name), drawn on the GPU: matrices scaled by their inner size, gains
    near one, and what shapes decays and gates where trained models have it."""

    def __init__(self, seed, tied):
        self.seed, self.tied = seed, tied

    def names(self):
        return None

    def fetch(self, decl):
        g = _generator(self.seed, decl.name)
        shape = tuple(decl.shape)

        def normal(std=1.0, mean=0.0):
            return torch.randn(shape, generator=g, device="cuda") * std + mean

        def uniform(low, high):
            return torch.rand(shape, generator=g, device="cuda") * (high - low) + low

        name, last = decl.name, decl.name.split(".")[-1]
        if decl.keep == "int32":                         # a token's experts
            start = torch.randint(0, decl.high, (shape[0], 1), generator=g, device="cuda")
            step = torch.arange(shape[1], device="cuda")[None, :]
            return ((start + step) % decl.high).to(torch.int32)
        if name in ("embed", "model.embed_tokens.weight", "bigram"):
            return normal(shape[1] ** -0.5 if self.tied else 1.0)
        if last in ("shift",) or ".mu." in name:
            return uniform(0.0, 1.0)
        if last == "w0":
            return uniform(-6.0, -1.0)
        if name.endswith("a2.b"):
            return normal(1.0, 1.0)
        if last == "dt_bias":
            return uniform(-6.0, -2.0)
        if last == "A_log":
            return uniform(0.0, math.log(16.0))
        if last == "vmix":
            return uniform(0.2, 0.8)
        if name.endswith("right.z.b"):
            return normal(0.5, -2.0)
        if name.endswith("mix.i.b"):
            return normal(0.3, -2.0)
        if name.endswith("mix.f.b"):
            return uniform(3.0, 6.0)
        if last == "correction":
            return normal(0.01)
        if ".hc" in name and last == "in":
            return normal(0.05, 0.25)
        if ".hc" in name and last == "mix":
            return normal(0.03, 0.025) + 0.9 * torch.eye(shape[0], device="cuda")
        if decl.init == "gain":
            return normal(0.1, 1.0)
        if decl.init == "bias":
            return normal(0.1)
        std = shape[-1] ** -0.5                          # a matrix, or a convolution's taps
        if last == "router" or name.endswith("mlp.gate.weight"):
            std *= 4.0                                   # trained routers are decisive
        if last == "down" or name.endswith(("down_proj.weight", ".o", "o_proj.weight")):
            # a sublayer adds less than it reads, one expert of several less still
            std *= 0.1 if "experts." in name or ".e" in name else 0.25
        return normal(std)


def _weights(case, seed):
    tied = case["model"] in ("zuzisun", "tinapel", "dominex")
    return RandomWeights(seed, tied)


def _context(seed, what, shape, dtype):
    """What earlier steps left in the cache: keys, values, latents and states of unit size."""
    g = _generator(seed, "context " + what)
    name = what.split(".")[-1]
    if name == "previous_token":
        return torch.randint(0, VOCAB, shape, generator=g, device="cuda").to(dtype)
    t = torch.randn(shape, generator=g, device="cuda")
    if name in ("memory_maximum", "min_gru_state"):
        t = t.abs()
    elif name in ("recurrent_state", "ssd_state", "delta_state", "memory", "memory_normaliser"):
        t = t * 0.5
    return t.to(dtype)


def _tokens(case, seed):
    rng = np.random.RandomState(seed % (1 << 32))
    cfg = config_of(case)
    vocab = cfg.get("vocab") or cfg["vocab_size"]
    return [rng.randint(0, vocab, n).tolist() for _, n in sequences(case)]


# -- a user's program ----------------------------------------------------------------------
def prepare(case, seed):
    """A loaded model with its cache; the requests that already hold tokens are open."""
    _, model = load_model(dtype=case["dtype"], device="cuda", config_json=config_of(case),
                          source=_weights(case, seed))
    seqs = sequences(case)
    pages = sum(-(-(c + n) // PAGE) for c, n in seqs)
    rt = Runtime(model, page_size=PAGE, num_pages=pages, max_slots=len(seqs), use_graphs=True)
    mgr, storage = rt.manager, rt.storage
    for unit, per in storage.paged.items():
        for name, t in per.items():
            t.copy_(_context(seed, f"{unit}.{name}", t.shape, t.dtype))
    earlier = [i for i, (before, _) in enumerate(seqs) if before]
    held = [mgr.open(i) for i in earlier]
    for i in earlier:
        mgr.reserve(i, sum(seqs[i]))
    for i in earlier:
        mgr.advance(i, seqs[i][0])
    mgr.take_fresh_slots()
    for unit, per in storage.state.items():
        for name, t in per.items():
            t[held] = _context(seed, f"{unit}.{name}", t.shape, t.dtype)[held]
    return {"rt": rt, "seqs": seqs, "tokens": _tokens(case, seed)}


def run(state):
    """One step.  A request that starts with this step is opened before it and closed behind
    it; the others stay where they are, so that the same step can be taken again."""
    rt, mgr = state["rt"], state["rt"].manager
    fresh = [i for i, (before, _) in enumerate(state["seqs"]) if not before]
    for i in fresh:
        mgr.open(i)
        mgr.reserve(i, state["seqs"][i][1])
    logits = rt.executor.step([StepEntry(i, t, [len(t) - 1])
                               for i, t in enumerate(state["tokens"])])
    for i in fresh:
        mgr.advance(i, state["seqs"][i][1])
        mgr.close(i)
    out = {"logits": logits}
    for kind, units in (("pages", rt.storage.paged), ("state", rt.storage.state)):
        for unit, per in units.items():
            for name, t in per.items():
                out[f"{kind}.{unit}.{name}"] = t
    return out


# -- what a step cannot do without -----------------------------------------------------------
_DECLS = {}


def _model_of(case):
    key = (case["model"], case["width"])
    if key not in _DECLS:
        _, spec = config_from_json(config_of(case))
        model = DecoderModel(spec, BuildContext(dtype=torch.bfloat16, device=torch.device("cpu"),
                                                ops=None))
        _DECLS[key] = (list(model.tensors()), model.cache_needs())
    return _DECLS[key]


def _pairs(before, n, window):
    """Query-key pairs of ``n`` new tokens behind ``before`` earlier ones."""
    if not window:
        return n * before + n * (n + 1) // 2
    return sum(min(p + 1, window) for p in range(before, before + n))


def work(case):
    """Every weight that is used once, the visible records of every request once, new records
    and logits once; the products of the tokens with the weights they use, scores and weighted
    values, and the recurrences' multiply-adds."""
    cfg, (decls, needs), seqs = config_of(case), _model_of(case), sequences(case)
    size = 4 if case["dtype"] == "float32" else 2
    tokens, rows = sum(n for _, n in seqs), len(seqs)
    qwen = "layers" not in cfg
    moved = flops = 0.0
    for d in decls:
        numel = math.prod(d.shape)
        each = size if d.keep == "param" else 4
        parts = d.name.split(".")
        if d.name in ("embed", "model.embed_tokens.weight", "bigram"):
            moved += min(numel, tokens * d.shape[1]) * each
            if d.name == "embed" and not any(x.name == "head" for x in decls):
                moved += numel * each
                flops += 2.0 * rows * numel
            continue
        if d.name in ("head", "lm_head.weight"):
            moved += numel * each
            flops += 2.0 * rows * numel
            continue
        if d.name.endswith("table"):
            continue
        share = 1.0
        if "experts" in parts or any(p[:1] == "e" and p[1:].isdigit() for p in parts):
            if qwen:
                experts, top = cfg["num_experts"], cfg["num_experts_per_tok"]
            else:
                r = cfg["layers"][int(parts[0][1:])]["mlp"]["router"]
                experts, top = r["experts"] + r.get("identity", 0), r["top"]
            share = top / experts
        moved += numel * each * (1.0 - (1.0 - share) ** tokens)
        if len(d.shape) == 2:
            flops += 2.0 * tokens * share * numel
    # one entry per layer: (heads, entries of a score, entries of a value, window)
    for i in range(cfg["num_hidden_layers"] if qwen else len(cfg["layers"])):
        if qwen:
            windowed = cfg["use_sliding_window"] and cfg["layer_types"][i] == "sliding_attention"
            mixers = [{"heads": cfg["num_attention_heads"], "kv_heads": cfg["num_key_value_heads"],
                       "dim": cfg["head_dim"], "scale": 1.0,
                       "mask": {"size": cfg["sliding_window"] if windowed else 0}}]
        else:
            m = cfg["layers"][i]["mixer"]
            mixers = [m["left"], m["right"]] if "left" in m else [m]
        for m in mixers:
            window = (m.get("mask") or {}).get("size", 0)
            if "kv_rank" in m or "scale" in m:
                dk = m["dim"] + m.get("rot_dim", 0)
                dv = m.get("vdim", m["dim"])
                record = (m["kv_rank"] + m["rot_dim"] if "kv_rank" in m
                          else m["kv_heads"] * (dk + dv))
                for before, n in seqs:
                    flops += 2.0 * m["heads"] * (dk + dv) * _pairs(before, n, window)
                    moved += record * size * (min(before, window or before) + n)
            elif "dim" in m or "state" in m:
                entries = m["heads"] * m.get("dim", m.get("state")) * m.get("vdim", m["dim"]
                                                                            if "dim" in m else 0)
                flops += 6.0 * tokens * entries
                moved += 8.0 * rows * entries
    moved += rows * (cfg.get("vocab") or cfg["vocab_size"]) * 4
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """32-bit sums in another order; in bfloat16 the rounding of every stored activation, and
    a router's close calls that it decides."""
    return {"rel": 2e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# -- the same in 64 bits -----------------------------------------------------------------------
def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _conv(u, w, earlier):
    """u [n, C] behind the rows ``earlier`` [taps - 1, C]; w [C, taps]."""
    rows = torch.cat([earlier, u], 0)
    return sum(rows[j:j + u.shape[0]] * w[:, j] for j in range(w.shape[1]))


def _turn(x, angle, magnitude=1.0, halves=False):
    """The leading entries of x [n, heads, d], two per angle [n, pairs], turned in pairs."""
    r = 2 * angle.shape[1]
    c, s = (torch.cos(angle) * magnitude)[:, None], (torch.sin(angle) * magnitude)[:, None]
    x = x.clone()
    a, b = ((slice(0, r // 2), slice(r // 2, r)) if halves else
            (slice(0, r, 2), slice(1, r, 2)))
    u, v = x[..., a].clone(), x[..., b].clone()
    x[..., a], x[..., b] = u * c - v * s, v * c + u * s
    return x


def _stretched(dims, base, sc):
    """(frequency of every pair, factor on cosine and sine) under the kinds of scaling."""
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f = base ** (-2.0 * i / dims)
    if not sc:
        return f, 1.0
    if "fast" in sc:
        at = [dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base))
              for t in (sc["fast"], sc["slow"])]
        lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    if "low" in sc:
        turns = sc["original"] * f / (2 * math.pi)
        s = ((turns - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
        return (1 - s) * f / sc["factor"] + s * f, 1.0
    return f / sc["factor"], 1.0


class _Plain:
    """A whole step in double precision, one function per mechanism, from the equations."""

    def __init__(self, case, seed):
        self.cfg, self.case = config_of(case), case
        self.decls = {d.name: d for d in _model_of(case)[0]}
        self.source = _weights(case, seed)
        self.seqs, base, row = [], 0, 0
        for i, (before, n) in enumerate(sequences(case)):
            self.seqs.append((i, before, n, base, slice(row, row + n)))
            base += -(-(before + n) // PAGE) * PAGE
            row += n
        # slots go to the requests that were opened first: the ones that hold tokens
        order = ([s[0] for s in self.seqs if s[1]] + [s[0] for s in self.seqs if not s[1]])
        self.slot = {i: k for k, i in enumerate(order)}
        self.ids = torch.tensor(sum(_tokens(case, seed), []), device="cuda")
        self.pos = torch.cat([torch.arange(b, b + n, device="cuda", dtype=torch.float64)
                              for _, b, n, _, _ in self.seqs])
        self.pages, self.state = {}, {}
        dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
        for unit, layer in enumerate(_model_of(case)[1]):
            for need in layer:
                if hasattr(need, "window"):
                    dims = need.entry_dims or [need.head_dim] * len(need.entries)
                    for name, d in zip(need.entries, dims):
                        t = _context(seed, f"{unit}.{name}", (base // PAGE, need.kv_heads, PAGE, d),
                                     dtype)
                        self.pages[unit, name] = t.float().transpose(1, 2).reshape(base, -1, d)
                else:
                    shape = (len(self.seqs),) + tuple(need.shape)
                    t = _context(seed, f"{unit}.{need.name}", shape, need.dtype)
                    t[[self.slot[s[0]] for s in self.seqs if not s[1]]] = 0
                    self.state[unit, need.name] = t.double()

    def w(self, name):
        d = self.decls[name]
        t = self.source.fetch(d)
        if d.keep == "param" and self.case["dtype"] != "float32":
            t = t.bfloat16()
        return t.double()

    def lin(self, x, name):
        return x @ self.w(name).T

    # -- cache and state
    def recorded(self, unit, name, seq, new):
        """All records of a request, the new ones included; they are stored too."""
        _, before, n, base, _ = seq
        buf = self.pages[unit, name]
        old = buf[base:base + before].double()
        buf[base + before:base + before + n] = new.float()
        return torch.cat([old, new], 0)

    def of(self, unit, name, seq):
        return self.state[unit, name][self.slot[seq[0]]]

    def each(self, f):
        return torch.cat([f(s, s[4]) for s in self.seqs], 0)

    def shifted(self, unit, name, h):
        """The row before every row."""
        def one(s, r):
            prev = self.of(unit, name, s)
            out = torch.cat([prev[None], h[r][:-1]], 0)
            prev.copy_(h[r][-1])
            return out
        return self.each(one)

    def conv(self, unit, name, u, w, first=0):
        """Convolution of columns ``first`` onwards of the kept rows."""
        def one(s, r):
            kept = self.of(unit, name, s)[:, first:first + u.shape[1]]
            out = _conv(u[r], w, kept.clone())
            kept.copy_(torch.cat([kept, u[r]], 0)[-kept.shape[0]:])
            return out
        return self.each(one)

    # -- mechanisms
    def attend(self, q, k, v, scale, seq, window=0, keep=0, sink=None, cap=0.0, penalty=None,
               temp=None):
        """q [n, H, d] over k [m, G, d], v [m, G, dv] -> [n, H, dv]."""
        _, before, n, _, _ = seq
        H, G = q.shape[1], k.shape[1]
        i = torch.arange(before, before + n, device="cuda")[:, None]
        j = torch.arange(before + n, device="cuda")[None]
        seen = j <= i
        if window:
            seen &= (i - j < window) | (j < keep)
        out = torch.empty(n, H, v.shape[2], dtype=torch.float64, device="cuda")
        for h in range(H):
            g = h // (H // G)
            s = q[:, h] @ k[:, g].T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            if penalty is not None:
                r1, r2 = penalty
                s = s * temp[h] - r1[h] * torch.log1p(r2[h] * (i - j).clamp(min=0))
            s = s.masked_fill(~seen, -math.inf)
            top = s.max(-1, keepdim=True).values
            if sink is not None:
                top = torch.maximum(top, sink[h])
            e = torch.exp(s - top)
            den = e.sum(-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(sink[h] - top)
            out[:, h] = e @ v[:, g] / den
        return out

    def paged(self, unit, q, k, v, scale, **more):
        def one(s, r):
            keys = self.recorded(unit, "k", s, k[r]) if k is not None else self.all_of(unit, "k", s)
            vals = self.recorded(unit, "v", s, v[r]) if v is not None else self.all_of(unit, "v", s)
            return self.attend(q[r], keys, vals, scale, s, **more)
        return self.each(one).flatten(1)

    def all_of(self, unit, name, s):
        return self.pages[unit, name][s[3]:s[3] + s[1] + s[2]].double()

    def glu(self, x, p, names=("gate", "up", "down")):
        return self.lin(_silu(self.lin(x, f"{p}.{names[0]}")) * self.lin(x, f"{p}.{names[1]}"),
                        f"{p}.{names[2]}")

    def experts(self, x, chosen, weights, run, inside=False):
        """Sum over the chosen experts; ``inside`` multiplies an expert's input."""
        out = torch.zeros_like(x)
        for e in chosen.unique().tolist():
            rows, place = (chosen == e).nonzero(as_tuple=True)
            c = weights[rows, place][:, None]
            out[rows] += run(c * x[rows], e) if inside else c * run(x[rows], e)
        return out

    def grouped_choice(self, scores, correction, r, pair):
        pick = scores + correction
        groups = r.get("groups") or {"count": 1, "keep": 1}
        parts = pick.view(pick.shape[0], groups["count"], -1)
        value = parts.topk(2, -1).values.sum(-1) if pair else parts.max(-1).values
        keep = value.topk(groups["keep"], -1).indices
        allowed = torch.zeros_like(value, dtype=torch.bool).scatter_(1, keep, True)
        parts = parts.masked_fill(~allowed[..., None], -math.inf)
        chosen = parts.flatten(1).topk(r["top"], -1).indices
        w = scores.gather(1, chosen)
        return chosen, w / (w.sum(-1, keepdim=True) + 1e-20)

    def last_rows(self):
        return torch.tensor([s[4].stop - 1 for s in self.seqs], device="cuda")

    # -- Qwen2
    def run_qwen2_moe(self):
        cfg, eps = self.cfg, self.cfg["rms_norm_eps"]
        H, G, d = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        freq, _ = _stretched(d, cfg["rope_theta"], None)
        angle = self.pos[:, None] * freq
        x = self.w("model.embed_tokens.weight")[self.ids]
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}"
            h = _rms(x, eps) * self.w(f"{p}.input_layernorm.weight")
            q, k, v = (self.lin(h, f"{p}.self_attn.{n}_proj.weight")
                       + self.w(f"{p}.self_attn.{n}_proj.bias") for n in "qkv")
            windowed = (cfg["use_sliding_window"]
                        and cfg["layer_types"][i] == "sliding_attention")
            o = self.paged(i, _turn(q.view(-1, H, d), angle, halves=True),
                           _turn(k.view(-1, G, d), angle, halves=True), v.view(-1, G, d),
                           d ** -0.5, window=cfg["sliding_window"] if windowed else 0)
            x = x + self.lin(o, f"{p}.self_attn.o_proj.weight")
            h = _rms(x, eps) * self.w(f"{p}.post_attention_layernorm.weight")
            names = ("gate_proj.weight", "up_proj.weight", "down_proj.weight")
            if i in cfg["mlp_only_layers"]:
                x = x + self.glu(h, f"{p}.mlp", names)
                continue
            s = torch.softmax(self.lin(h, f"{p}.mlp.gate.weight"), -1)
            w, chosen = s.topk(cfg["num_experts_per_tok"], -1)
            y = self.experts(h, chosen, w,
                             lambda t, e: self.glu(t, f"{p}.mlp.experts.{e}", names))
            gate = torch.sigmoid(self.lin(h, f"{p}.mlp.shared_expert_gate.weight"))
            x = x + y + gate * self.glu(h, f"{p}.mlp.shared_expert", names)
        return self.lin(_rms(x[self.last_rows()], eps) * self.w("model.norm.weight"),
                        "lm_head.weight")

    run_qwen2_dense = run_qwen2_moe

    # -- latent attention
    def latent(self, unit, h, q, m, p, eps, own=True):
        H, dim, rot, vd, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        freq, mag = _stretched(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
        angle = self.pos[:, None] * freq
        q = q.view(-1, H, dim + rot)
        q_rot = _turn(q[..., dim:], angle, mag)
        if own:
            down = self.lin(h, f"{p}.dkv")
            c = _rms(down[:, :rank], eps) * self.w(f"{p}.dkv.norm")
            record = torch.cat([c, _turn(down[:, None, rank:], angle, mag)[:, 0]], -1)[:, None]
        uk, uv = (self.w(f"{p}.{n}").view(H, -1, rank) for n in ("uk", "uv"))

        def one(s, r):
            rec = (self.recorded(unit, "latent", s, record[r]) if own
                   else self.all_of(unit, "latent", s))[:, 0]
            k = torch.einsum("jc,hdc->jhd", rec[:, :rank], uk)
            k = torch.cat([k, rec[:, None, rank:].expand(-1, H, -1)], -1)
            v = torch.einsum("jc,hdc->jhd", rec[:, :rank], uv)
            return self.attend(torch.cat([q[r][..., :dim], q_rot[r]], -1), k, v, m["scale"], s,
                               window=(m.get("mask") or {}).get("size", 0))
        return self.each(one).flatten(1)

    def run_zuzisun(self):
        cfg, eps, groups = self.cfg, self.cfg["norm"]["eps"], self.cfg["norm"]["groups"]

        def norm(x, name):
            return _rms(x.view(x.shape[0], groups, -1), eps).flatten(1) * self.w(name)
        x = self.w("embed")[self.ids] * cfg["embedding"]["scale"]
        for i, layer in enumerate(cfg["layers"]):
            m, f, p = layer["mixer"], layer["mlp"], f"l{i}"
            h = x + (self.shifted(i, "shift_prev", x) - x) * self.w(f"{p}.shift")
            o = self.latent(i, h, self.lin(h, f"{p}.mix.q"), m, f"{p}.mix", eps)
            o = o * torch.sigmoid(self.lin(h, f"{p}.mix.g"))
            x = x + norm(self.lin(o, f"{p}.mix.o"), f"{p}.norm1")
            g = self.lin(x, f"{p}.mlp.gate").clamp(max=f["limit"])
            u = self.lin(x, f"{p}.mlp.up").clamp(-f["limit"], f["limit"])
            y = self.lin(g * torch.sigmoid(1.702 * g) * (u + 1), f"{p}.mlp.down")
            x = x + norm(y, f"{p}.norm2")
        return norm(x[self.last_rows()], "final.norm") @ self.w("embed").T

    # -- recurrences: S [H, K, V] of one request walked token by token
    def walk(self, unit, name, step):
        def one(s, r):
            S = self.of(unit, name, s)
            out = []
            for t in range(r.start, r.stop):
                S, o = step(S, t)
                out.append(o)
            self.state[unit, name][self.slot[s[0]]] = S
            return torch.stack(out)
        return self.each(one)

    def run_tinapel(self):
        cfg, eps = self.cfg, self.cfg["norm"]["eps"]
        width = cfg["width"]

        def norm(x, name):
            return _rms(x, eps) * (1 + self.w(name))
        x = self.w("embed")[self.ids] * cfg["embedding"]["scale"]
        even = torch.arange(0, width, 2, dtype=torch.float64, device="cuda")
        a = self.pos[:, None] * 10000.0 ** (-even / width)
        x = x + torch.stack([torch.sin(a), torch.cos(a)], -1).flatten(1)
        for i, layer in enumerate(cfg["layers"]):
            m, f, p = layer["mixer"], layer["mlp"], f"l{i}.mix"
            h = norm(x, f"l{i}.norm1")
            H, K = m["heads"], m["dim"]
            if layer["type"] == "wkv":
                prev = self.shifted(i, "previous_input", h) - h
                r, k, v, g, z = (h + prev * self.w(f"{p}.mu.{n}") for n in "rkvgw")
                r, k, v = (self.lin(t, f"{p}.{n}").view(-1, H, K) for t, n in
                           ((r, "r"), (k, "k"), (v, "v")))
                g = self.lin(g, f"{p}.g")
                z = self.lin(torch.tanh(self.lin(z, f"{p}.w1")), f"{p}.w2") + self.w(f"{p}.w0")
                keep, u = torch.exp(-torch.exp(z)).view(-1, H, K, 1), self.w(f"{p}.u")[..., None]

                def step(S, t):
                    kv = k[t][..., None] * v[t][:, None]
                    return keep[t] * S + kv, ((S + u * kv) * r[t][..., None]).sum(1)
                o = _rms(self.walk(i, "recurrent_state", step), eps).flatten(1)
                y = self.lin(o * self.w(f"{p}.norm") * _silu(g), f"{p}.o")
            elif layer["type"] == "gla":
                q, k, v = (self.lin(h, f"{p}.{n}").view(h.shape[0], H, -1) for n in "qkv")
                z = self.lin(self.lin(h, f"{p}.a1"), f"{p}.a2") + self.w(f"{p}.a2.b")
                keep = torch.sigmoid(z).pow(1.0 / m["tau"]).view(-1, H, K, 1)

                def step(S, t):
                    S = keep[t] * S + k[t][..., None] * v[t][:, None]
                    return S, (S * q[t][..., None]).sum(1) * K ** -0.5
                o = _rms(self.walk(i, "recurrent_state", step), eps) * self.w(f"{p}.norm")
                y = self.lin(o.flatten(1) * _silu(self.lin(h, f"{p}.g")), f"{p}.o")
            else:
                q = self.lin(h, f"{p}.q").view(-1, H, K)
                k = self.lin(h, f"{p}.k").view(-1, m["kv_heads"], K)
                qt = m["q_temp"]
                warm = 1 + qt["coef"] * torch.log(torch.floor((self.pos + 1) / qt["every"]) + 1)
                q = _rms(q, eps) * self.w(f"{p}.q.norm") * warm[:, None, None]
                o = self.paged(i, q, _rms(k, eps) * self.w(f"{p}.k.norm"), k, m["scale"],
                               cap=m["softcap"])
                y = self.lin(o, f"{p}.o")
            h = norm(x, f"l{i}.norm2")
            w, chosen = torch.softmax(self.lin(h, f"l{i}.mlp.router"), -1).topk(
                f["router"]["top"], -1)
            w = w / (w.sum(-1, keepdim=True) + 1e-20) * f["router"]["scale"]
            x = x + y + self.experts(h, chosen, w, lambda t, e: self.glu(t, f"l{i}.mlp.e{e}"))
            x = x + self.glu(h, f"l{i}.mlp.shared")
        return norm(x[self.last_rows()], "final.norm") @ self.w("embed").T

    def run_mapovik(self):
        cfg, eps, mult = self.cfg, self.cfg["norm"]["eps"], self.cfg["residual_mult"]

        def norm(x, name):
            x = x - x.mean(-1, keepdim=True)
            return _rms(x, eps) * self.w(name)
        softplus = torch.nn.functional.softplus
        x = self.w("embed")[self.ids]
        for i, layer in enumerate(cfg["layers"]):
            m, f, p = layer["mixer"], layer["mlp"], f"l{i}.mix"
            h = norm(x, f"l{i}.norm1")
            T = h.shape[0]
            if layer["type"] == "parallel":
                a, s = m["left"], m["right"]
                q, k, v = (self.lin(h, f"{p}.left.{n}").view(T, -1, a["dim"]) for n in "qkv")
                freq, _ = _stretched(a["rot"]["dims"], a["rot"]["base"], a["rot"]["scaling"])
                angle = self.pos[:, None] * freq
                o = self.paged(i, _turn(q, angle, halves=True), _turn(k, angle, halves=True), v,
                               a["scale"])
                left = self.lin(o, f"{p}.left.o")
                H, V, N, G = s["heads"], s["vdim"], s["state"], s["groups"]
                z, xbc, dt = self.lin(h, f"{p}.right.in").split(
                    [H * V, H * V + 2 * G * N, H], -1)
                xbc = _silu(self.conv(i, "ssd_conv_inputs", xbc, self.w(f"{p}.right.conv"))
                            + self.w(f"{p}.right.conv.b"))
                u, B, C = xbc.split([H * V, G * N, G * N], -1)
                u = u.view(T, H, V)
                B, C = (t.view(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
                dt = softplus(dt + self.w(f"{p}.right.dt_bias"))
                keep = torch.exp(-torch.exp(self.w(f"{p}.right.A_log")) * dt)
                D = self.w(f"{p}.right.D")[:, None]

                def step(S, t):
                    S = keep[t][:, None, None] * S + (dt[t][:, None] * B[t])[..., None] * u[t][:, None]
                    return S, (S * C[t][..., None]).sum(1) + D * u[t]
                y = self.walk(i, "ssd_state", step).flatten(1) * _silu(z)
                y = _rms(y.view(T, s["norm_groups"], -1), eps).flatten(1)
                right = self.lin(y * self.w(f"{p}.right.norm"), f"{p}.right.o")
                y = 0.5 * (_rms(left, eps) * self.w(f"{p}.left.out")
                           + _rms(right, eps) * self.w(f"{p}.right.out"))
            else:
                H, K, V = m["heads"], m["dim"], m["vdim"]
                at, got = 0, []
                for n in "qkv":
                    u = self.lin(h, f"{p}.{n}")
                    got.append(_silu(self.conv(i, "delta_conv_inputs", u, self.w(f"{p}.{n}.conv"),
                                               at)).view(T, H, -1))
                    at += u.shape[1]
                q, k, v = got
                q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
                beta = torch.sigmoid(self.lin(h, f"{p}.b"))
                z = self.lin(self.lin(h, f"{p}.a1"), f"{p}.a2") + self.w(f"{p}.dt_bias")
                rate = torch.exp(self.w(f"{p}.A_log"))[:, None]
                keep = torch.exp(-rate * softplus(z.view(T, H, K)))

                def step(S, t):
                    S = keep[t][..., None] * S
                    u = beta[t][:, None] * (v[t] - (S * k[t][..., None]).sum(1))
                    S = S + k[t][..., None] * u[:, None]
                    return S, (S * q[t][..., None]).sum(1) * K ** -0.5
                o = _rms(self.walk(i, "delta_state", step), eps) * self.w(f"{p}.norm")
                gate = torch.sigmoid(self.lin(self.lin(h, f"{p}.g1"), f"{p}.g2"))
                y = self.lin(o.flatten(1) * gate, f"{p}.o")
            x = x + mult * y
            h = norm(x, f"l{i}.norm2")
            table = self.source.fetch(self.decls[f"l{i}.mlp.table"]).long()
            chosen = table[self.ids]
            even = torch.full(chosen.shape, 1.0 / chosen.shape[1], dtype=torch.float64,
                              device="cuda")
            x = x + mult * self.experts(h, chosen, even,
                                        lambda t, e: self.glu(t, f"l{i}.mlp.e{e}"))
        return norm(x[self.last_rows()], "final.norm") @ self.w("head").T * cfg["logit_scale"]

    def run_fudulix(self):
        cfg, eps = self.cfg, self.cfg["norm"]["eps"]
        b, unit = cfg["embedding"]["bigram"], len(cfg["layers"])

        def pair(s, r):
            kept = self.of(unit, "previous_token", s)
            prev = torch.cat([kept.long(), self.ids[r][:-1]], 0)
            kept[0] = self.ids[r][-1].double()
            row = (prev * b["mul_prev"] + self.ids[r] * b["mul_cur"]) % b["buckets"]
            if not s[1]:
                row[0] = b["buckets"]
            return row
        x = _rms(self.w("embed")[self.ids] + self.w("bigram")[self.each(pair)], eps)
        x = x * self.w("embed.norm")
        first = None
        zero = torch.zeros(64, dtype=torch.float64, device="cuda")
        for i, layer in enumerate(cfg["layers"]):
            m, f, p = layer["mixer"], layer["mlp"], f"l{i}.mix"
            H, G, d, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
            h = _rms(x, eps) * self.w(f"l{i}.norm1")
            q, k, v = (self.lin(h, f"{p}.{n}") for n in "qkv")
            freq, mag = _stretched(rot["dims"], rot["base"], rot["scaling"])
            angle = self.pos[:, None] * freq
            second = layer["type"] == "attention_2"
            if second:
                at, got = 0, []
                for u, n in ((q, "q"), (k, "k"), (v, "v")):
                    got.append(self.conv(i, "attention_conv_inputs", u, self.w(f"{p}.{n}.conv"),
                                         at))
                    at += u.shape[1]
                q, k, v = got
                q, k = (_rms(t, eps) * self.w(f"{p}.{n}.norm") for t, n in ((q, "q"), (k, "k")))
            q, k = (_turn(t.view(-1, n, d), angle, mag, halves=second)
                    for t, n in ((q, H), (k, G)))
            if not second:
                q, k = _rms(q, eps), _rms(k, eps)
            if first is None:
                first = v
            else:
                lam = self.w(f"{p}.vmix")
                v = (1 - lam) * v + lam * first
            o = self.paged(i, q, k, v.view(-1, G, m["vdim"]), m["scale"],
                           window=m["mask"]["size"], keep=m["mask"].get("keep_first", 0),
                           sink=None if second else zero)
            x = x + self.lin(o, f"{p}.o")
            h, p = _rms(x, eps) * self.w(f"l{i}.norm2"), f"l{i}.mlp"
            if f["kind"] == "dense":
                g = torch.nn.functional.gelu(self.lin(h, f"{p}.gate") + self.w(f"{p}.gate.b"),
                                             approximate="tanh")
                u = self.lin(h, f"{p}.up") + self.w(f"{p}.up.b")
                x = x + self.lin(g * u, f"{p}.down") + self.w(f"{p}.down.b")
                continue
            scores = torch.softmax(self.lin(h, f"{p}.router"), -1)
            chosen, w = self.grouped_choice(scores, self.w(f"{p}.correction"), f["router"], False)
            real = f["router"]["experts"]
            x = x + self.experts(h, chosen, w, lambda t, e: (
                self.glu(t, f"{p}.e{e}") if e < real else t)) + self.glu(h, f"{p}.shared")
        return self.lin(_rms(x[self.last_rows()], eps) * self.w("final.norm"), "head")

    def run_dominex(self):
        cfg, eps = self.cfg, self.cfg["norm"]["eps"]

        def norm(x, name):
            return _rms(x, eps) * (1 + self.w(name))
        x = self.w("embed")[self.ids] * cfg["embedding"]["scale"]
        for i, layer in enumerate(cfg["layers"]):
            m, p = layer["mixer"], f"l{i}.mix"
            h = norm(x, f"l{i}.norm1")
            if layer["type"] == "parallel":
                a = m["left"]
                q, k, v = (self.lin(h, f"{p}.left.{n}").view(h.shape[0], -1, a["dim"])
                           for n in "qkv")
                o = self.paged(i, q, k, v, a["scale"], temp=self.w(f"{p}.left.temp"), penalty=(
                    self.w(f"{p}.left.r1"), self.w(f"{p}.left.r2")))
                z = torch.sigmoid(self.lin(h, f"{p}.right.z") + self.w(f"{p}.right.z.b"))
                u = self.lin(h, f"{p}.right.x") + self.w(f"{p}.right.x.b")
                u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))

                def step(S, t):
                    S = (1 - z[t]) * S + z[t] * u[t]
                    return S, S
                r = self.walk(i, "min_gru_state", step) * _silu(self.lin(h, f"{p}.right.g"))
                y = (m["left_scale"] * self.lin(o, f"{p}.left.o")
                     + m["right_scale"] * self.lin(r, f"{p}.right.o"))
            else:
                c = _rms(self.lin(h, f"{p}.dq"), eps) * self.w(f"{p}.dq.norm")
                src = m.get("kv_from")
                o = self.latent(i if src is None else src, h, self.lin(c, f"{p}.uq"), m, p, eps,
                                own=src is None)
                y = self.lin(o, f"{p}.o")
            x = x + y
            h, f = norm(x, f"l{i}.norm2"), layer["mlp"]
            z, chosen = self.lin(h, f"l{i}.mlp.router").topk(f["router"]["top"], -1)
            x = x + self.experts(h, chosen, torch.sigmoid(z),
                                 lambda t, e: self.glu(t, f"l{i}.mlp.e{e}"), inside=True)
        z = norm(x[self.last_rows()], "final.norm") @ self.w("embed").T
        return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])

    def run_biguzen(self):
        cfg, eps = self.cfg, self.cfg["norm"]["eps"]

        def norm(x, name):
            return torch.tanh(self.w(f"{name}.alpha") * x) * self.w(name) + self.w(f"{name}.b")

        def two(h, p):
            return self.lin(torch.nn.functional.gelu(self.lin(h, f"{p}.up")), f"{p}.down")
        streams = self.w("embed")[self.ids].expand(cfg["streams"], -1, -1)
        for i, layer in enumerate(cfg["layers"]):
            m, f, p = layer["mixer"], layer["mlp"], f"l{i}.mix"

            def read(q):
                u = torch.einsum("s,stw->tw", self.w(f"l{i}.hc{q}.in"), streams)
                return norm(u, f"l{i}.norm{q}")

            def write(q, y):
                return (torch.einsum("su,stw->utw", self.w(f"l{i}.hc{q}.mix"), streams)
                        + self.w(f"l{i}.hc{q}.out")[:, None, None] * y)
            h = read(1)
            T, H, d = h.shape[0], m["heads"], m["dim"]
            if layer["type"] == "mlstm":
                q, k, v = (self.lin(h, f"{p}.{n}").view(T, H, -1) for n in "qkv")
                cap = m["gate_cap"]
                gi, gf = (cap * torch.tanh((self.lin(h, f"{p}.{n}") + self.w(f"{p}.{n}.b")) / cap)
                          for n in "if")
                gf = torch.nn.functional.logsigmoid(gf)
                now = {}

                def step(S, t):
                    n, top = now["n"], now["m"]
                    new = torch.maximum(gf[t] + top, gi[t])
                    keep, put = torch.exp(gf[t] + top - new), torch.exp(gi[t] - new)
                    S = keep[:, None, None] * S + (put[:, None] * k[t])[..., None] * v[t][:, None]
                    n = keep[:, None] * n + put[:, None] * k[t]
                    now["n"], now["m"] = n, new
                    qt = q[t] * d ** -0.5
                    den = torch.maximum((n * qt).sum(-1).abs(), torch.exp(-new)) + 1e-6
                    return S, (S * qt[..., None]).sum(1) / den[:, None]

                def one(s, r):
                    slot = self.slot[s[0]]
                    now["n"] = self.state[i, "memory_normaliser"][slot]
                    now["m"] = self.state[i, "memory_maximum"][slot]
                    S, out = self.state[i, "memory"][slot], []
                    for t in range(r.start, r.stop):
                        S, o = step(S, t)
                        out.append(o)
                    self.state[i, "memory"][slot] = S
                    self.state[i, "memory_normaliser"][slot] = now["n"]
                    self.state[i, "memory_maximum"][slot] = now["m"]
                    return torch.stack(out)
                o = _rms(self.each(one), eps).flatten(1) * self.w(f"{p}.norm")
                y = self.lin(o * torch.sigmoid(self.lin(h, f"{p}.g")), f"{p}.o")
            else:
                src, rot, at, got = m.get("kv_from"), m["rot"], 0, []
                freq, _ = _stretched(rot["dims"], rot["base"], rot["scaling"])
                angle = self.pos[:, None] * freq
                for n in "qkv" if src is None else "q":
                    u = self.lin(h, f"{p}.{n}") + self.w(f"{p}.{n}.b")
                    u = self.conv(i, "attention_conv_inputs", u, self.w(f"{p}.{n}.conv"), at)
                    at += u.shape[1]
                    u = u.view(T, -1, d)
                    got.append(u if n == "v" else _turn(u, angle))
                q, k, v = got if src is None else (got[0], None, None)
                o = self.paged(i if src is None else src, q, k, v, m["scale"],
                               window=m["mask"]["size"], sink=self.w(f"{p}.sink"))
                gate = torch.sigmoid(self.lin(h, f"{p}.g"))
                y = self.lin((o.view(T, H, -1) * gate[..., None]).flatten(1), f"{p}.o")
            streams = write(1, y)
            h, p = read(2), f"l{i}.mlp"
            scores = torch.sigmoid(self.lin(h, f"{p}.router"))
            chosen, w = self.grouped_choice(scores, self.w(f"{p}.correction"), f["router"], True)
            y = self.experts(h, chosen, w * f["router"]["scale"],
                             lambda t, e: two(t, f"{p}.e{e}"))
            y = y + torch.sigmoid(self.lin(h, f"{p}.shared.sg")) * two(h, f"{p}.shared")
            streams = write(2, y)
        return norm(streams.sum(0)[self.last_rows()], "final.norm") @ self.w("embed").T


def exact(case, seed):
    plain = _Plain(case, seed)
    out = {"logits": getattr(plain, "run_" + case["model"])()}
    for (unit, name), t in plain.pages.items():
        t = t.view(-1, PAGE, t.shape[1], t.shape[2]).transpose(1, 2)
        out[f"pages.{unit}.{name}"] = t.contiguous()
    for (unit, name), t in plain.state.items():
        out[f"state.{unit}.{name}"] = t.long().to(torch.int32) if name == "previous_token" else t
    return out
