"""The work whose speed is watched: steps of the engine's step function on models of several architectures, and the
choice of tokens from logits.

Each case builds a model from a config.json's content and seeded weights, an engine around it, and requests, as a
serving program holds them; a pass is what such a program does per step (or, for ``replay``, per short run of steps):
``runner.step`` on a list of entries, or ``sampler.sample`` on logits.  ``exact`` computes the same logits for whole
sequences in 64 bits with plain torch.

Kinds of case:

* ``step``: one batch of decoded tokens (``decode`` requests whose caches hold up to ``context`` tokens) and, or, prompt
  portions (``prompts`` of up to ``tokens`` tokens, ``before`` tokens of each already cached).  Pools are filled with
  random keys and values for what is cached.
* ``replay``: ``prompts`` prompts from their first token, then ``steps`` decode steps with given tokens; the logits of
  every step.
* ``sample``: one token per row of logits, with rows of all sampling options in turn.
"""
from __future__ import annotations

import math
import random

import torch

from lyapunov_engine_b200 import EngineConfig, LLMEngine, LoadedModel, SamplingParams, build
from lyapunov_engine_b200.engine.runtime import Runtime
from lyapunov_engine_b200.models.model import Model
from lyapunov_engine_b200.registry import spec_for
from lyapunov_engine_b200.sampling import Sampler

DEVICE = "cuda:0"
VOCAB = 128256
PAGE = 16
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ------------------------------------------------------------------ the cases
def listed():
    step, bf16 = {"kind": "step", "dtype": "bfloat16"}, "bfloat16"
    none = {"decode": 0, "context": 0, "ragged": False, "prompts": 0, "tokens": 0, "before": 0, "want": 1}
    return [
        # one user's chat: a token at a time, a short context; launches and weights are all there is
        {"name": "llama_1b_decode_1", **step, "model": "llama_1b", "layers": 16, **none, "decode": 1, "context": 517},
        # the benchmark's serving step
        {"name": "llama_1b_decode_8", **step, "model": "llama_1b", "layers": 16, **none, "decode": 8, "context": 4096},
        # a busy server: many requests of different ages, a batch that does not fill its captured step
        {"name": "llama_1b_decode_61", **step, "model": "llama_1b", "layers": 16, **none, "decode": 61, "context": 4096,
         "ragged": True},
        # a prompt read in one step
        {"name": "llama_1b_prompt_2048", **step, "model": "llama_1b", "layers": 16, **none, "prompts": 1, "tokens": 2048},
        # a long document into a larger model
        {"name": "llama_3b_prompt_8192", **step, "model": "llama_3b", "layers": 28, **none, "prompts": 1, "tokens": 8192},
        # continuous batching: a portion of a prompt beside the decoding requests
        {"name": "llama_1b_mixed", **step, "model": "llama_1b", "layers": 16, **none, "decode": 23, "context": 2500,
         "ragged": True, "prompts": 1, "tokens": 777, "before": 1024},
        # the 32-bit engine, as used to check a checkpoint's logits
        {"name": "llama_f32_prompt", "kind": "step", "dtype": "float32", "model": "llama_1b", "layers": 4, **none,
         "decode": 3, "context": 500, "ragged": True, "prompts": 1, "tokens": 333},
        # recurrent and attention layers in turn: reading a prompt and scoring it
        {"name": "ribozen_prompt_2048", **step, "model": "ribozen_1b", "layers": 8, **none, "prompts": 1, "tokens": 2048,
         "want": 64},
        # the same model answering eight requests at once
        {"name": "ribozen_replay_8", "kind": "replay", "dtype": bf16, "model": "ribozen_1b", "layers": 8, "prompts": 8,
         "tokens": 61, "steps": 8},
        # a prompt of an odd length through the gated delta rule, attention and latent attention
        {"name": "zepilix_prompt_3001", **step, "model": "zepilix_1b", "layers": 8, **none, "prompts": 1, "tokens": 3001,
         "want": 16},
        # several prompts in one step through lightning attention, attention and experts
        {"name": "zuzenex_prompts_4", **step, "model": "zuzenex_1b", "layers": 8, **none, "prompts": 4, "tokens": 700,
         "want": 64},
        # the choice of the next tokens of a full batch
        {"name": "sample_64", "kind": "sample", "rows": 64, "vocab": VOCAB},
    ]


def draw(rng):
    def size(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    case = {"kind": "step", "dtype": "bfloat16", "model": "llama_1b", "layers": 16, "decode": 0, "context": 0,
            "ragged": rng.random() < 0.7, "prompts": 0, "tokens": 0, "before": 0, "want": 1}
    what = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "float32", "ribozen", "ribozen", "zepilix",
                       "zepilix", "zuzenex", "replay", "replay", "sample"])
    if what == "sample":
        return {"kind": "sample", "rows": size(1, 64), "vocab": rng.choice([VOCAB, 32000, size(1000, VOCAB)])}
    if what == "replay":
        return {"kind": "replay", "dtype": "bfloat16", "model": rng.choice(["ribozen_1b", "zepilix_1b", "zuzenex_1b"]),
                "layers": 8, "prompts": size(1, 16), "tokens": size(4, 200), "steps": rng.randint(4, 8)}
    if what == "decode":
        case.update(decode=size(1, 64), context=size(16, 4096))
    elif what == "prompt":
        case.update(prompts=rng.choice([1, 1, 2, 3]), tokens=size(16, 2700), before=rng.choice([0, 0, size(16, 1024)]))
        if rng.random() < 0.3:
            case.update(model="llama_3b", layers=28)
    elif what == "mixed":
        case.update(decode=size(1, 48), context=size(64, 4096), prompts=1, tokens=size(16, 2048), before=rng.choice([0, 512]))
    elif what == "float32":
        case.update(dtype="float32", layers=4, decode=size(1, 8), context=size(16, 1024), prompts=rng.choice([0, 1]),
                    tokens=size(16, 512))
    else:
        case.update(model=what + "_1b", layers=8, prompts=rng.choice([1, 1, 2, 4]), want=32)
        case.update(tokens=size(33, 4096 // case["prompts"]))
    return case


# ------------------------------------------------------------------ the models' config.json
def config_of(case):
    name, layers = case["model"], case["layers"]
    if name.startswith("llama"):
        big = name == "llama_3b"
        return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": VOCAB,
                "hidden_size": 3072 if big else 2048, "intermediate_size": 8192, "num_hidden_layers": layers,
                "num_attention_heads": 24 if big else 32, "num_key_value_heads": 8, "head_dim": 128 if big else 64,
                "max_position_embeddings": 131072, "rms_norm_eps": 1e-5, "rope_theta": 500000.0,
                "rope_scaling": {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                                 "original_max_position_embeddings": 8192},
                "tie_word_embeddings": True, "hidden_act": "silu", "attention_bias": False, "mlp_bias": False}
    W, nh, nkv, hd, ff = 2048, 32, 8, 64, 8192
    if name == "ribozen_1b":
        # recurrent layers as the designs they come from stack them (the mixer alone); experts behind the attention layers
        moe = {"kind": "moe", "expert": {"ff": ff // 4}, "router": {"experts": 8, "top": 2}, "shared": {"ff": ff // 4}}
        duality = {"type": "mamba2", "mlp": None, "mixer": {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4,
                                                            "norm_groups": 8}}
        memory = {"type": "mlstm", "mlp": None, "mixer": {"heads": W // 256, "dim": 128, "vdim": 256, "gate_cap": 15.0}}
        pair = {"type": "parallel", "mlp": moe,
                "mixer": {"left_scale": 0.7, "right_scale": 1.0,
                          "left": {"heads": nh, "kv_heads": nkv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "softcap": 30.0,
                                   "rot": {"dims": hd, "base": 500000.0,
                                           "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}},
                                   "mask": {"size": 1024, "keep_first": 8}},
                          "right": {"inner": W, "state": 16, "dt_rank": W // 16, "conv": 4}}}
        kinds = (duality, duality, memory, pair)
        return {"architecture": "Ribozen", "vocab": VOCAB, "width": W, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
                "layers": [kinds[i % 4] for i in range(layers)]}
    if name == "zepilix_1b":
        mlp = {"kind": "dense", "ff": ff}
        delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": W // 128, "kv_heads": W // 256, "dim": 128, "vdim": 128, "conv": 4}}
        attention = {"type": "attention", "mlp": mlp, "mixer": {"heads": nh, "kv_heads": nkv, "dim": hd, "vdim": hd, "scale": hd ** -0.5,
                                                                "rot": {"dims": hd, "base": 500000.0}}}
        latent = {"type": "latent_attention", "mlp": mlp,
                  "mixer": {"heads": nh, "dim": hd, "rot_dim": 32, "vdim": hd, "kv_rank": 96, "q_rank": W * 3 // 8,
                            "scale": (hd + 32) ** -0.5, "mask": {"size": 2048}, "rot": {"dims": 32, "base": 1000000.0}}}
        kinds = (delta, attention, delta, latent)
        return {"architecture": "Zepilix", "vocab": VOCAB, "width": W, "norm": {"eps": 1e-6}, "token_side": {"dim": 256},
                "layers": [kinds[i % 4] for i in range(layers)]}
    if name == "zuzenex_1b":
        H, fx = W // 128, ff * 3 // 8
        dense = {"kind": "dense", "ff": fx * 3}
        moe = {"kind": "moe", "expert": {"ff": fx}, "shared": {"ff": fx}, "router": {"experts": 8, "identity": 2, "top": 2}}
        memory = {"type": "lightning", "mlp": dense,
                  "mixer": {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-1.0 - 9.0 * h / (H - 1)) for h in range(H)]}}
        attn = {"type": "attention", "mlp": moe, "mixer": {"heads": nh, "kv_heads": nkv, "dim": hd, "vdim": hd, "scale": hd ** -0.5,
                                                           "q_temp": {"coef": 0.1, "every": 2048}}}
        return {"architecture": "Zuzenex", "vocab": VOCAB, "width": W, "norm": {"eps": 1e-5},
                "layers": [attn if i % 4 == 3 else memory for i in range(layers)]}
    raise ValueError(f"no model {name!r}")


def tensor_shapes(c):
    """name -> shape of every tensor of a checkpoint of this config."""
    out = {}
    if "hidden_size" in c:
        W, F, V = c["hidden_size"], c["intermediate_size"], c["vocab_size"]
        q, kv = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
        out["model.embed_tokens.weight"], out["model.norm.weight"] = (V, W), (W,)
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out.update({p + "self_attn.q_proj.weight": (q, W), p + "self_attn.k_proj.weight": (kv, W),
                        p + "self_attn.v_proj.weight": (kv, W), p + "self_attn.o_proj.weight": (W, q),
                        p + "mlp.gate_proj.weight": (F, W), p + "mlp.up_proj.weight": (F, W), p + "mlp.down_proj.weight": (W, F),
                        p + "input_layernorm.weight": (W,), p + "post_attention_layernorm.weight": (W,)})
        return out
    W, V, arch = c["width"], c["vocab"], c["architecture"]
    out["embed"], out["final.norm"] = (V, W), (W,)
    if arch != "Zepilix":
        out["head"] = (V, W)
    side = c["token_side"]["dim"] if c.get("token_side") else 0
    if side:
        out["side.embed"] = (V, side * len(c["layers"]))
    for i, layer in enumerate(c["layers"]):
        p, m, kind = f"l{i}.mix.", layer["mixer"], layer["type"]
        out[f"l{i}.norm1"] = (W,)
        if kind in ("mlstm", "mamba2", "parallel"):
            out[f"l{i}.ls1"] = (W,)
        if kind == "mlstm":
            d, e, H = m["heads"] * m["dim"], m["heads"] * m["vdim"], m["heads"]
            out.update({p + "q": (d, W), p + "k": (d, W), p + "v": (e, W), p + "g": (e, W), p + "o": (W, e), p + "norm": (e,),
                        p + "i": (H, W), p + "i.b": (H,), p + "f": (H, W), p + "f.b": (H,)})
        elif kind == "mamba2":
            H, inner, gn = m["heads"], m["heads"] * m["vdim"], m["groups"] * m["state"]
            out.update({p + "in": (2 * inner + 2 * gn + H, W), p + "conv": (inner + 2 * gn, m["conv"]), p + "conv.b": (inner + 2 * gn,),
                        p + "dt_bias": (H,), p + "A_log": (H,), p + "D": (H,), p + "norm": (inner,), p + "o": (W, inner)})
        elif kind == "parallel":
            a, s, l, r = m["left"], m["right"], p + "left.", p + "right."
            q, k, v, o = a["heads"] * a["dim"], a["kv_heads"] * a["dim"], a["kv_heads"] * a["vdim"], a["heads"] * a["vdim"]
            out.update({l + "q": (q, W), l + "q.b": (q,), l + "k": (k, W), l + "k.b": (k,), l + "v": (v, W), l + "v.b": (v,),
                        l + "q.norm": (q,), l + "k.norm": (k,), l + "g": (o, W), l + "o": (W, o)})
            C, N, R = s["inner"], s["state"], s["dt_rank"]
            out.update({r + "in": (2 * C, W), r + "conv": (C, s["conv"]), r + "conv.b": (C,), r + "x": (R + 2 * N, C), r + "dt": (C, R),
                        r + "dt.b": (C,), r + "A_log": (C, N), r + "D": (C,), r + "o": (W, C)})
        elif kind == "delta":
            H, qk, e, n = m["heads"], m["kv_heads"] * m["dim"], m["heads"] * m["vdim"], m["conv"]
            out.update({p + "q": (qk, W), p + "k": (qk, W), p + "v": (e, W), p + "q.conv": (qk, n), p + "k.conv": (qk, n),
                        p + "v.conv": (e, n), p + "b": (H, W), p + "a": (H, W), p + "g": (e, W), p + "o": (W, e), p + "A_log": (H,),
                        p + "dt_bias": (H,), p + "norm": (m["vdim"],)})
        elif kind == "latent_attention":
            H, d, t, e, r, qr = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
            out.update({p + "dq": (qr, W), p + "dq.norm": (qr,), p + "uq": (H * (d + t), qr), p + "dkv": (r + t, W), p + "dkv.norm": (r,),
                        p + "uk": (H * d, r), p + "uv": (H * e, r), p + "o": (W, H * e)})
        elif kind == "lightning":
            d, e = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            out.update({p + "q": (d, W), p + "k": (d, W), p + "v": (e, W), p + "g": (e, W), p + "o": (W, e), p + "norm": (e,)})
        else:
            q, k, e = m["heads"] * m["dim"], m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
            out.update({p + "q": (q, W), p + "k": (k, W), p + "o": (W, e)})
            if arch == "Zuzenex":
                out.update({p + "v": (m["kv_heads"] * m["vdim"], W), p + "q.norm": (m["dim"],), p + "k.norm": (m["dim"],),
                            p + "sink": (m["heads"],)})
        f, mlp = f"l{i}.mlp.", layer["mlp"]
        gated = arch != "Zuzenex"

        def feed_forward(prefix, F):
            out.update({prefix + "up": (F, W), prefix + "down": (W, F)})
            if gated:
                out[prefix + "gate"] = (F, W)

        if mlp is not None and mlp["kind"] == "dense":
            feed_forward(f, mlp["ff"])
            if arch == "Zepilix":
                out.update({f + "gate.b": (mlp["ff"],), f + "up.b": (mlp["ff"],), f + "down.b": (W,)})
        elif mlp is not None:
            for x in range(mlp["router"]["experts"]):
                feed_forward(f"{f}e{x}.", mlp["expert"]["ff"])
            feed_forward(f + "shared.", mlp["shared"]["ff"])
            total = mlp["router"]["experts"] + mlp["router"].get("identity", 0)
            out[f + "router"] = (total, W)
            if arch == "Zuzenex":
                out[f + "correction"] = (total,)
        if mlp is not None and arch != "Zuzenex":
            out[f"l{i}.norm2"] = (W,)
            if arch == "Ribozen":
                out[f"l{i}.ls2"] = (W,)
        if side:
            out.update({f"l{i}.side.gate": (side, W), f"l{i}.side.proj": (W, side), f"l{i}.side.norm": (W,)})
    return out


def tensors_of(case, seed):
    """The checkpoint: matrices N(0, 1 / fan-in), decays and step sizes spread so that some channels remember hundreds
    of tokens and others a few, scores sharp enough that single keys count.  A token's embedding leans towards the
    directions of two experts and the routers follow them, so that, as in a trained model, most choices of experts are
    clear (and none hangs on a rounding).  Matrices in the case's type, vectors in 32 bits."""
    g = torch.Generator(device=DEVICE).manual_seed(1000003 * int(seed) + 17)
    out = {}
    c = config_of(case)
    routers = [layer["mlp"]["router"] for layer in c.get("layers", []) if layer["mlp"] and layer["mlp"]["kind"] == "moe"]
    experts = routers[0]["experts"] + routers[0].get("identity", 0) if routers else 0
    lean = torch.randn(max(experts, 1), c.get("width", 1), generator=g, device=DEVICE) / math.sqrt(c.get("width", 1))
    for name, shape in tensor_shapes(c).items():
        tail = name.split(".", 1)[1] if name[0] == "l" and name[1:2].isdigit() else name

        def normal(scale=1.0, around=0.0):
            return around + scale * torch.randn(shape, generator=g, device=DEVICE)

        def between(lo, hi):
            return lo + (hi - lo) * torch.rand(shape, generator=g, device=DEVICE)

        if tail.endswith((".q.norm", ".k.norm")):
            t = normal(0.3, 1.3)
        elif tail.endswith(("norm", "norm1", "norm2", "norm.weight", "layernorm.weight")):
            around_zero = c.get("architecture") == "Zepilix" and (tail in ("norm1", "norm2") or name == "final.norm")
            t = normal(0.2, 0.0 if around_zero else 1.0)
        elif tail in ("ls1", "ls2"):
            t = between(0.4, 1.3)
        elif tail.endswith("conv"):
            t = normal(0.6)
        elif tail == "mix.A_log":
            t = between(-4.0, 0.5)
        elif tail == "mix.right.A_log":
            t = between(-3.0, 1.0)
        elif tail in ("mix.dt_bias", "mix.right.dt.b"):
            t = between(-4.0, 0.0)
        elif tail in ("mix.D", "mix.right.D"):
            t = normal(0.3, 1.0)
        elif tail == "mix.f.b":
            t = between(1.0, 5.0)
        elif tail == "mlp.router":
            t = lean + normal(0.3 / math.sqrt(shape[1]))
        elif tail == "mlp.correction":
            t = normal(0.02)
        elif len(shape) == 1:
            t = normal(0.3)
        elif "embed" in tail:
            t = normal()
            if experts and name == "embed":
                ids = torch.arange(shape[0], device=DEVICE)
                first = ids % experts
                t += 16.0 * (lean[first] + lean[(first + 1 + ids // experts % (experts - 1)) % experts])
        else:
            wide = 0.5 if tail.endswith((".o", "down", "o_proj.weight", "down_proj.weight")) else 1.0
            t = normal(wide / math.sqrt(shape[1]))
        vector = len(shape) == 1 or tail.endswith((".conv", "A_log", "mlp.router"))
        out[name] = t.to(torch.bfloat16).float() if vector else t.to(TYPES[case["dtype"]])
        del t
    return out


# ------------------------------------------------------------------ requests
def requests_of(case, seed):
    """(cached tokens, ids of the tokens that come next, places among them whose logits are wanted) of every request."""
    rng = random.Random(7919 * int(seed) + 3)
    sizes = random.Random(11)                       # the sizes are the case's, not the seed's
    out = []

    def ids(n):
        return [rng.randrange(VOCAB) for _ in range(n)]

    def ragged(n):
        return sizes.randint(max(1, n // 4), n) if case.get("ragged", True) else n

    if case["kind"] == "replay":
        for _ in range(case["prompts"]):
            n = ragged(case["tokens"])
            out.append((0, ids(n + case["steps"]), list(range(n - 1, n + case["steps"]))))
        return out
    for i in range(case["prompts"]):
        n = case["tokens"] if i == 0 else ragged(case["tokens"])
        want = sorted({(j + 1) * n // min(case["want"], n) - 1 for j in range(min(case["want"], n))})
        out.append((case["before"], ids(n), want))
    for i in range(case["decode"]):
        n = case["context"] if i == 0 else ragged(case["context"])
        out.append((n - 1, ids(1), [0]))
    return out


def cached_rows(case, c, seed, layer, total):
    """Keys and values [total cached tokens, kv heads, head size] of one layer."""
    g = torch.Generator(device=DEVICE).manual_seed(900007 * int(seed) + layer)
    shape = (2, total, c["num_key_value_heads"], c["head_dim"])
    return torch.randn(shape, generator=g, device=DEVICE).to(TYPES[case["dtype"]])


def prepare(case, seed):
    if case["kind"] == "sample":
        return prepare_sample(case, seed)
    c = config_of(case)
    dtype = TYPES[case["dtype"]]
    reqs = requests_of(case, seed)
    longest = max(n + len(t) for n, t, _ in reqs)
    limit = (longest + 63) // 64 * 64 + 64
    host = build.load_host()
    tensors = tensors_of(case, seed)
    spec = spec_for(c)
    runtime = Runtime(DEVICE, dtype, max_model_len=limit)
    model = Model(spec)
    model.bind(lambda name: tensors["model.embed_tokens.weight" if name == "lm_head.weight" else name], runtime)
    del tensors
    pages = sum((n + len(t) + PAGE - 1) // PAGE + 1 for n, t, _ in reqs) + limit // PAGE
    engine = LLMEngine(LoadedModel(spec, model, runtime),
                       EngineConfig(num_blocks=pages, block_size=PAGE, max_num_seqs=max(4, len(reqs)), dtype=dtype, device=DEVICE,
                                    max_num_batched_tokens=max(2048, sum(len(t) for _, t, _ in reqs)), max_model_len=limit))
    seqs = []
    for i, (cached, ids, _) in enumerate(reqs):
        seq = host.Sequence(i, [0] * cached + ids, host.SamplingParams())
        if not engine.block_manager.grow(seq, cached + len(ids)):
            raise RuntimeError("the pool is too small for the case")
        seq.set_num_computed_tokens(cached)
        seqs.append(seq)
    total = sum(n for n, _, _ in reqs)
    if total:
        page = torch.cat([torch.tensor(s.get_block_table(), device=DEVICE)[torch.arange(n, device=DEVICE) // PAGE]
                          for s, (n, _, _) in zip(seqs, reqs) if n])
        place = torch.cat([torch.arange(n, device=DEVICE) % PAGE for n, _, _ in reqs if n])
        for layer, pools in enumerate(engine.cache.streams[0]):
            rows = cached_rows(case, c, seed, layer, total)
            pools.k.permute(0, 2, 1, 3)[page, place] = rows[0]
            pools.v.permute(0, 2, 1, 3)[page, place] = rows[1]
    if case["kind"] == "replay" or not case["prompts"]:
        engine.warm_up([longest], [len(reqs)])       # as a server does before its first request
    return {"case": case, "engine": engine, "host": host, "seqs": seqs, "requests": reqs}


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return state["sampler"].sample(state["logits"], state["params"], state["indices"])
    host, step = state["host"], state["engine"].runner.step
    if case["kind"] == "step":
        return step([host.StepEntry(s, n, len(ids), want) for s, (n, ids, want) in zip(state["seqs"], state["requests"])])
    pairs = list(zip(state["seqs"], state["requests"]))
    first = [len(ids) - case["steps"] for _, (_, ids, _) in pairs]
    for s in state["seqs"]:
        s.set_num_computed_tokens(0)
    out = [step([host.StepEntry(s, 0, n, [n - 1]) for (s, _), n in zip(pairs, first)]).clone()]
    for j in range(case["steps"]):
        for (s, _), n in zip(pairs, first):
            s.set_num_computed_tokens(n + j)
        out.append(step([host.StepEntry(s, n + j, 1, [0]) for (s, _), n in zip(pairs, first)]).clone())
    return out


# ------------------------------------------------------------------ choosing tokens
def sample_rows(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(int(seed) + 5)
    logits = 3.0 * torch.randn(case["rows"], case["vocab"], generator=g, device=DEVICE)
    options = [(0.0, 1.0, 0), (1.0, 1.0, 0), (0.8, 0.95, 0), (1.0, 1.0, 50), (0.7, 0.9, 40)]
    return logits, [options[i % len(options)] for i in range(case["rows"])]


def prepare_sample(case, seed):
    logits, options = sample_rows(case, seed)
    params = [SamplingParams(temperature=t, top_p=p, top_k=k, seed=1000 * int(seed) + i) for i, (t, p, k) in enumerate(options)]
    return {"case": case, "logits": logits, "params": params, "indices": list(range(case["rows"])),
            "sampler": Sampler(torch.device(DEVICE), 64)}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 1), "flops": 2 * case["rows"] * case["vocab"]}
    c = config_of(case)
    reqs = requests_of(case, 0)
    if case["kind"] == "step":
        return step_work(case, c, [(n, len(t), len(w)) for n, t, w in reqs])
    first = [len(t) - case["steps"] for _, t, _ in reqs]
    parts = [step_work(case, c, [(0, n, 1) for n in first])]
    parts += [step_work(case, c, [(n + j, 1, 1) for n in first]) for j in range(case["steps"])]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def step_work(case, c, reqs):
    """``reqs``: (cached tokens, tokens of this step, wanted logits) of every request."""
    width = 2 if case["dtype"] == "bfloat16" else 4
    T, wanted = sum(n for _, n, _ in reqs), sum(w for _, _, w in reqs)
    shapes = tensor_shapes(c)
    W, V = c.get("hidden_size", c.get("width")), VOCAB
    nbytes, flops = width * V * W + 4 * wanted * V, 2 * wanted * V * W
    layers = c.get("layers") or [{"type": "llama", "mlp": None}] * c["num_hidden_layers"]

    def pairs(window):
        """keys that all queries see"""
        return sum(min(p + 1, window) if window else p + 1 for n, t, _ in reqs for p in range(n, n + t))

    def keys(window):
        """keys that are read once: all cached ones in sight of the request's first query, and the step's own"""
        return sum((min(n, window) if window else n) + t for n, t, _ in reqs)

    reach = {}

    def attention(window, heads, d, e, kv_entries):
        nonlocal nbytes, flops
        if window not in reach:
            reach[window] = pairs(window), keys(window)
        flops += 2 * heads * (d + e) * reach[window][0]
        nbytes += width * kv_entries * reach[window][1]

    for i, layer in enumerate(layers):
        top = all_experts = None
        if layer["mlp"] and layer["mlp"]["kind"] == "moe":
            r = layer["mlp"]["router"]
            top, all_experts = r["top"], r["experts"]
        prefix = f"model.layers.{i}." if layer["type"] == "llama" else f"l{i}."
        for name, shape in shapes.items():
            if not name.startswith(prefix) or len(shape) < 2 or name.endswith(("conv", "A_log")):
                continue
            n = shape[0] * shape[1]
            share, used = 1.0, 1.0
            if top and name.startswith(prefix + "mlp.e"):
                share, used = top / all_experts, min(1.0, T * top / all_experts)
            nbytes += width * n * used
            flops += 2 * T * n * share
        m = layer.get("mixer")
        states = lambda n: 2 * 4 * n * len(reqs)      # read and written, in 32 bits
        if layer["type"] == "llama":
            h, k, d = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
            attention(0, h, d, d, 2 * k * d)
        elif layer["type"] == "attention":
            own = 1 if c["architecture"] == "Zepilix" else 2
            attention(0, m["heads"], m["dim"], m["vdim"], own * m["kv_heads"] * m["dim"])
        elif layer["type"] == "latent_attention":
            attention(m["mask"]["size"], m["heads"], m["kv_rank"] + m["rot_dim"], m["kv_rank"], m["kv_rank"] + m["rot_dim"])
        elif layer["type"] == "parallel":
            a, s = m["left"], m["right"]
            attention(a["mask"]["size"], a["heads"], a["dim"], a["vdim"], a["kv_heads"] * (a["dim"] + a["vdim"]))
            nbytes += states(s["inner"] * s["state"])
            flops += 6 * T * s["inner"] * s["state"]
        else:
            entries = m["heads"] * m["vdim"] * m.get("dim", m.get("state", 0))
            nbytes += states(entries)
            flops += (6 if layer["type"] in ("mamba2", "delta") else 4) * T * entries
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.05}           # (a sum in another order moves a boundary between two tokens)
    if case["dtype"] == "float32":
        return {"rel": 1e-5}                          # (1.5e-6 against 64 bits)
    return {"rel": 2.4e-2}                            # (0.004 to 0.006)


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    if case["kind"] == "sample":
        return None                                    # (the random numbers are the framework's own)
    c = config_of(case)
    w = tensors_of(case, seed)
    reqs = requests_of(case, seed)
    forward = exact_llama if "hidden_size" in c else exact_layers
    with torch.no_grad():
        rows = forward(case, c, w, reqs, seed)
    if case["kind"] == "step":
        return torch.cat(rows)
    return [torch.stack([r[j] for r in rows]) for j in range(case["steps"] + 1)]


def f64(t):
    return t.double()


def unit_rms(x, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def attend(q, k, v, scale, window=0, keep=0, cap=0.0, sink=None):
    """q [T, H, d] of the last T positions, k [S, G, d], v [S, G, e]; heads in groups share keys."""
    T, H, _ = q.shape
    S, G, _ = k.shape
    out = q.new_empty(T, H, v.shape[-1])
    at = torch.arange(S, device=q.device)
    for lo in range(0, T, 1024):
        hi = min(T, lo + 1024)
        gap = (torch.arange(lo, hi, device=q.device) + S - T)[:, None] - at[None, :]
        seen = gap >= 0
        if window:
            seen &= (gap < window) | (at[None, :] < keep)
        for g in range(G):
            heads = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("thd,sd->hts", q[lo:hi, heads], k[:, g]) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[heads][:, None, None].expand(-1, hi - lo, 1)], dim=-1)
            p = torch.softmax(s, dim=-1)[..., :S]
            out[lo:hi, heads] = torch.einsum("hts,se->the", p, v[:, g])
    return out


def rotate_halves(x, positions, rates, size=1.0):
    half = rates.numel()
    angle = positions.double()[:, None, None] * rates
    c, s = torch.cos(angle) * size, torch.sin(angle) * size
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], dim=-1)


def rotate_pairs(x, positions, rot, base):
    rates = base ** (-2.0 * torch.arange(rot // 2, device=x.device, dtype=torch.float64) / rot)
    angle = positions.double()[:, None, None] * rates
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., 0:rot:2], x[..., 1:rot:2]
    out = x.clone()
    out[..., 0:rot:2], out[..., 1:rot:2] = a * c - b * s, b * c + a * s
    return out


def llama_rates(c):
    hd, r = c["head_dim"], c["rope_scaling"]
    out = []
    for j in range(0, hd, 2):
        f = c["rope_theta"] ** (-j / hd)
        turns = r["original_max_position_embeddings"] * f / (2.0 * math.pi)
        smooth = (turns - r["low_freq_factor"]) / (r["high_freq_factor"] - r["low_freq_factor"])
        smooth = min(1.0, max(0.0, smooth))
        out.append((1.0 - smooth) * f / r["factor"] + smooth * f)
    return torch.tensor(out, device=DEVICE, dtype=torch.float64)


def exact_llama(case, c, w, reqs, seed):
    eps, H, G, d = c["rms_norm_eps"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    rates, total = llama_rates(c), sum(n for n, _, _ in reqs)
    counts = [len(t) for _, t, _ in reqs]
    positions = torch.cat([torch.arange(n, n + t, device=DEVICE) for (n, _, _), t in zip(reqs, counts)])
    embed = w["model.embed_tokens.weight"]
    x = f64(embed[torch.tensor([i for _, t, _ in reqs for i in t], device=DEVICE)])
    for i in range(c["num_hidden_layers"]):
        lin = lambda y, name: y @ f64(w[f"model.layers.{i}.{name}.weight"]).T
        h = unit_rms(x, eps) * f64(w[f"model.layers.{i}.input_layernorm.weight"])
        q = rotate_halves(lin(h, "self_attn.q_proj").view(-1, H, d), positions, rates)
        k = rotate_halves(lin(h, "self_attn.k_proj").view(-1, G, d), positions, rates)
        v = lin(h, "self_attn.v_proj").view(-1, G, d)
        cached = cached_rows(case, c, seed, i, total) if total else None
        o, at, before = [], 0, 0
        for (n, _, _), t in zip(reqs, counts):
            kk, vv = k[at:at + t], v[at:at + t]
            if n:
                kk = torch.cat([f64(cached[0, before:before + n]), kk])
                vv = torch.cat([f64(cached[1, before:before + n]), vv])
            o.append(attend(q[at:at + t], kk, vv, d ** -0.5))
            at, before = at + t, before + n
        x = x + lin(torch.cat(o).reshape(-1, H * d), "self_attn.o_proj")
        h = unit_rms(x, eps) * f64(w[f"model.layers.{i}.post_attention_layernorm.weight"])
        x = x + lin(torch.nn.functional.silu(lin(h, "mlp.gate_proj")) * lin(h, "mlp.up_proj"), "mlp.down_proj")
    x = unit_rms(x, eps) * f64(w["model.norm.weight"])
    return by_request(x, reqs, embed)


def by_request(x, reqs, head):
    out, at = [], 0
    for _, t, want in reqs:
        rows = x[[at + p for p in want]]
        out.append(torch.cat([rows @ f64(part).T for part in head.split(32768)], dim=1))
        at += len(t)
    return out


def exact_layers(case, c, w, reqs, seed):
    """The architectures whose config.json lists its layers; whole sequences (nothing is cached before)."""
    eps, arch = c["norm"]["eps"], c["architecture"]
    out = []
    for _, ids, want in reqs:
        at = torch.tensor(ids, device=DEVICE)
        x = f64(w["embed"][at]) * c.get("embedding", {}).get("scale", 1.0)
        plus = 1.0 if arch == "Zepilix" else 0.0
        for i, layer in enumerate(c["layers"]):
            g = lambda name: f64(w[f"l{i}.{name}"])
            m, mlp = layer["mixer"], layer["mlp"]
            h = unit_rms(x, eps) * (plus + g("norm1"))
            mixer = {"mlstm": matrix_memory, "mamba2": duality, "parallel": side_by_side, "delta": delta_rule,
                     "latent_attention": latent_attention, "lightning": lightning}.get(layer["type"])
            if mixer is None:
                mixer = normed_attention if arch == "Zuzenex" else turned_attention
            y = mixer(h, lambda name: g("mix." + name), m, eps)
            if arch == "Ribozen":
                x = x + y * g("ls1")
                if mlp is not None:
                    h = unit_rms(x, eps) * g("norm2")
                    x = x + experts(h, g, mlp, arch) * g("ls2")
            elif arch == "Zepilix":
                h = unit_rms(x, eps) * (1.0 + g("norm2"))
                a = torch.nn.functional.silu(h @ g("mlp.gate").T + g("mlp.gate.b")) * (h @ g("mlp.up").T + g("mlp.up.b"))
                x = x + y + a @ g("mlp.down").T + g("mlp.down.b")
                s = c["token_side"]["dim"]
                e = f64(w["side.embed"][at][:, i * s:(i + 1) * s])
                z = torch.nn.functional.gelu(x @ g("side.gate").T, approximate="tanh") * e
                x = x + unit_rms(z @ g("side.proj").T, eps) * g("side.norm")
            else:
                x = x + y + (plain(h, g, "mlp.") if mlp["kind"] == "dense" else experts(h, g, mlp, arch))
        x = unit_rms(x, eps) * (plus + f64(w["final.norm"]))
        out += by_request(x, [(0, ids, want)], w["head"] if "head" in w else w["embed"])
    return out


def plain(h, g, p):
    return torch.clamp(h @ g(p + "up").T, min=0.0).pow(2) @ g(p + "down").T


def gated(h, g, p):
    return (torch.nn.functional.silu(h @ g(p + "gate").T) * (h @ g(p + "up").T)) @ g(p + "down").T


def experts(h, g, mlp, arch):
    r = mlp["router"]
    logits = h @ g("mlp.router").T
    one = gated if arch == "Ribozen" else plain
    if arch == "Ribozen":
        chosen = torch.topk(logits, r["top"], dim=-1).indices
        weight = torch.sigmoid(torch.gather(logits, 1, chosen))
    else:
        s = torch.softmax(logits, dim=-1)
        chosen = torch.topk(s + g("mlp.correction"), r["top"], dim=-1).indices
        weight = torch.gather(s, 1, chosen)
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    out = one(h, g, "mlp.shared.")
    for e in range(logits.shape[1]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            s = weight[rows, place][:, None]
            if arch == "Ribozen":                       # the weight meets the expert's input
                y = one(s * h[rows], g, f"mlp.e{e}.")
            else:
                y = s * (h[rows] if e >= r["experts"] else one(h[rows], g, f"mlp.e{e}."))
            out.index_add_(0, rows, y)
    return out


def causal_conv(x, taps, bias=None):
    T, n = x.shape[0], taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    y = sum(padded[j:j + T] * taps[:, j] for j in range(n))
    return y if bias is None else y + bias


def recurrence(decay, k, v, q, S):
    """Per token t: S <- decay[t] * S + k[t] v[t]^T, out = q[t] S.  decay, k, q broadcast against S [H, N, e]; v [T, H, e]."""
    out = []
    for t in range(v.shape[0]):
        S = torch.addcmul(decay[t] * S, k[t], v[t][:, None, :])
        out.append((S * q[t]).sum(1))
    return torch.stack(out)


def duality(h, g, m, eps):
    T, H, e, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * e
    proj = h @ g("in").T
    z, xbc, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * G * N], proj[:, 2 * inner + 2 * G * N:]
    xbc = torch.nn.functional.silu(causal_conv(xbc, g("conv"), g("conv.b")))
    x = xbc[:, :inner].view(T, H, e)
    B, C = (xbc[:, inner + j * G * N:inner + (j + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for j in range(2))
    dt = torch.nn.functional.softplus(dt + g("dt_bias"))
    decay = torch.exp(-torch.exp(g("A_log")) * dt)
    y = recurrence(decay[:, :, None, None], (dt[..., None] * B)[..., None], x, C[..., None], h.new_zeros(H, N, e))
    y = (y + g("D")[:, None] * x).reshape(T, inner) * torch.nn.functional.silu(z)
    parts = m["norm_groups"]
    y = unit_rms(y.view(T, parts, -1), eps).reshape(T, inner) * g("norm")
    return y @ g("o").T


def matrix_memory(h, g, m, eps):
    T, H, d, e, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q = (h @ g("q").T).view(T, H, d) * d ** -0.5
    k, v = (h @ g("k").T).view(T, H, d), (h @ g("v").T).view(T, H, e)
    i = cap * torch.tanh((h @ g("i").T + g("i.b")) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ g("f").T + g("f.b")) / cap))
    run, tops = h.new_zeros(H), []
    for t in range(T):
        run = torch.maximum(f[t] + run, i[t])
        tops.append(run)
    top = torch.stack(tops)
    before = torch.cat([h.new_zeros(1, H), top[:-1]])
    keep, take = torch.exp(f + before - top), torch.exp(i - top)
    ones = torch.cat([v, v.new_ones(T, H, 1)], dim=-1)      # the last column is n
    o = recurrence(keep[:, :, None, None], (take[..., None] * k)[..., None], ones, q[..., None], h.new_zeros(H, d, e + 1))
    below = torch.maximum(o[..., -1].abs(), torch.exp(-top)) + 1e-6
    o = unit_rms(o[..., :-1] / below[..., None], eps).reshape(T, H * e) * g("norm")
    return (o * torch.sigmoid(h @ g("g").T)) @ g("o").T


def side_by_side(h, g, m, eps):
    T, a, s = h.shape[0], m["left"], m["right"]
    H, G, d, e = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
    l = lambda name: g("left." + name)
    q = unit_rms(h @ l("q").T + l("q.b"), eps) * l("q.norm")
    k = unit_rms(h @ l("k").T + l("k.b"), eps) * l("k.norm")
    v = (h @ l("v").T + l("v.b")).view(T, G, e)
    rot, dims = a["rot"], a["rot"]["dims"]
    r = rot["scaling"]
    j = torch.arange(dims // 2, device=DEVICE, dtype=torch.float64)
    f = rot["base"] ** (-2.0 * j / dims)
    dim_of = lambda turns: dims * math.log(r["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))
    lo, hi = max(math.floor(dim_of(r["fast"])), 0), min(math.ceil(dim_of(r["slow"])), dims - 1)
    ramp = torch.clamp((j - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    rates, size = f / r["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(r["factor"]) + 1.0
    at = torch.arange(T, device=DEVICE)
    q, k = rotate_halves(q.view(T, H, d), at, rates, size), rotate_halves(k.view(T, G, d), at, rates, size)
    o = attend(q, k, v, a["scale"], a["mask"]["size"], a["mask"]["keep_first"], a["softcap"]).reshape(T, H * e)
    left = (o * torch.sigmoid(h @ l("g").T)) @ l("o").T
    r = lambda name: g("right." + name)
    inner, N, R = s["inner"], s["state"], s["dt_rank"]
    xz = h @ r("in").T
    x = torch.nn.functional.silu(causal_conv(xz[:, :inner], r("conv"), r("conv.b")))
    low = x @ r("x").T
    dt = torch.nn.functional.softplus(low[:, :R] @ r("dt").T + r("dt.b"))
    B, C = low[:, R:R + N], low[:, R + N:]
    A, S, ys = -torch.exp(r("A_log")), h.new_zeros(inner, N), []
    dx = dt * x
    for t in range(T):
        S = torch.addcmul(torch.exp(dt[t][:, None] * A) * S, dx[t][:, None], B[t][None, :])
        ys.append(S @ C[t])
    y = torch.stack(ys) + r("D") * x
    right = (y * torch.nn.functional.silu(xz[:, inner:])) @ r("o").T
    return m["left_scale"] * left + m["right_scale"] * right


def delta_rule(h, g, m, eps):
    T, H, G, d, e = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    made = lambda name, n, size: torch.nn.functional.silu(causal_conv(h @ g(name).T, g(name + ".conv"))).view(T, n, size)
    q, k, v = made("q", G, d), made("k", G, d), made("v", H, e)
    q = q / torch.sqrt(q.pow(2).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt(k.pow(2).sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, 1)[..., None], k.repeat_interleave(H // G, 1)[..., None]
    beta = torch.sigmoid(h @ g("b").T)
    keep = torch.exp(-torch.exp(g("A_log")) * torch.nn.functional.softplus(h @ g("a").T + g("dt_bias")))
    S, out = h.new_zeros(H, d, e), []
    for t in range(T):
        S = keep[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - (S * k[t]).sum(1))
        S = torch.addcmul(S, k[t], u[:, None, :])
        out.append((S * q[t]).sum(1))
    o = unit_rms(torch.stack(out), eps) * g("norm") * torch.nn.functional.silu(h @ g("g").T).view(T, H, e)
    return o.reshape(T, H * e) @ g("o").T


def turned_attention(h, g, m, eps):
    T, H, G, d, at = h.shape[0], m["heads"], m["kv_heads"], m["dim"], torch.arange(h.shape[0], device=DEVICE)
    q, v = (h @ g("q").T).view(T, H, d), (h @ g("k").T).view(T, G, d)
    q, k = (unit_rms(rotate_pairs(x, at, m["rot"]["dims"], m["rot"]["base"]), eps) for x in (q, v))
    return attend(q, k, v, m["scale"]).reshape(T, H * d) @ g("o").T


def latent_attention(h, g, m, eps):
    T, H, d, t, e, r = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    at, base = torch.arange(T, device=DEVICE), m["rot"]["base"]
    q = ((unit_rms(h @ g("dq").T, eps) * g("dq.norm")) @ g("uq").T).view(T, H, d + t)
    down = h @ g("dkv").T
    c = unit_rms(down[:, :r], eps) * g("dkv.norm")
    q = torch.cat([q[..., :d], rotate_pairs(q[..., d:], at, t, base)], dim=-1)
    turned = rotate_pairs(down[:, None, r:], at, t, base).expand(T, H, t)
    k = torch.cat([(c @ g("uk").T).view(T, H, d), turned], dim=-1)
    o = attend(q, k, (c @ g("uv").T).view(T, H, e), m["scale"], m["mask"]["size"])
    return o.reshape(T, H * e) @ g("o").T


def normed_attention(h, g, m, eps):
    T, H, G, d, e = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q = unit_rms((h @ g("q").T).view(T, H, d), eps) * g("q.norm")
    k = unit_rms((h @ g("k").T).view(T, G, d), eps) * g("k.norm")
    turns = torch.div(torch.arange(T, device=DEVICE) + 1, m["q_temp"]["every"], rounding_mode="floor").double()
    q = q * (1.0 + m["q_temp"]["coef"] * torch.log(turns + 1.0))[:, None, None]
    o = attend(q, k, (h @ g("v").T).view(T, G, e), m["scale"], sink=g("sink"))
    return o.reshape(T, H * e) @ g("o").T


def lightning(h, g, m, eps):
    T, H, d, e = h.shape[0], m["heads"], m["dim"], m["vdim"]
    silu = torch.nn.functional.silu
    q, k = silu(h @ g("q").T).view(T, H, d, 1), silu(h @ g("k").T).view(T, H, d, 1)
    v = silu(h @ g("v").T).view(T, H, e)
    decay = torch.tensor(m["decay"], device=DEVICE, dtype=torch.float64)[None, :, None, None].expand(T, -1, -1, -1)
    o = recurrence(decay, k, v, q, h.new_zeros(H, d, e)).reshape(T, H * e)
    o = unit_rms(o, eps) * g("norm") * torch.sigmoid(h @ g("g").T)
    return o @ g("o").T
