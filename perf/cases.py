"""The work that is timed: the sublayers that the engine's models are made of, and whole steps of a decoder.

A case of a sublayer builds its mixer (or feed-forward) from the registries as a model plan names it, gives it the context of
one step (prompt portions, or single tokens of running requests with their cached keys or states) and runs
``mixer.forward`` and the norm that takes its update: what a block does between two products of the residual stream.  A case
of kind ``steps`` runs whole requests through ``ModelRunner.step`` as the replay program does: admit, the prompts, then
given tokens one by one, and returns the logits of every step.

Sizes are those of the benchmark's configurations: the 2.2B, 500M and 256M decoders, and the widths 1,024 and 2,048 at which
the other designs are compared.
"""

import math

import torch

from edgerag_b200 import Engine
from edgerag_b200.cache.device import DevicePools
from edgerag_b200.cache.manager import CacheManager
from edgerag_b200.config.registry import architecture_of
from edgerag_b200.engine.engine import EngineOptions
from edgerag_b200.engine.step import ModelRunner, StepEntry
from edgerag_b200.models.decoder import DecoderModel
from edgerag_b200.parts.base import LayerCall, LayerSpec, ModelPlan, PartSpec, build_part

F64 = torch.float64
EPS = 1e-5
PAGE = 16

# hidden, layers, query heads, kv heads, intermediate, vocabulary, rope theta
DECODERS = {"2b": (2048, 24, 32, 32, 8192, 49155, 273768.0), "500m": (960, 32, 15, 5, 2560, 49280, 100000.0),
            "256m": (576, 30, 9, 3, 1536, 49280, 100000.0)}
WIDTHS = {
    "w1024": {"hidden": 1024, "ff": 4096, "latent": {"heads": 8, "dim": 64, "rot": 32, "v": 64, "rank": 256},
              "ssd": {"heads": 32, "p": 64, "state": 64, "groups": 4}, "delta": {"heads": 8, "key_heads": 4, "dim": 128},
              "diff": {"heads": 8, "kv": 2, "dim": 64, "v": 128}},
    "w2048": {"hidden": 2048, "ff": 8192, "latent": {"heads": 16, "dim": 128, "rot": 64, "v": 128, "rank": 512},
              "ssd": {"heads": 64, "p": 64, "state": 128, "groups": 8}, "delta": {"heads": 16, "key_heads": 8, "dim": 128},
              "diff": {"heads": 16, "kv": 4, "dim": 64, "v": 128}},
}
EXPERTS, TOP = 32, 4
DIFF = {"diff": 0.6, "cap": 30.0, "base": 1000000.0}
TAPS = 4


def _case(name, kind, size, lens="", past=0, batch=0, context=0, **more):
    """``lens``: the portions of prompts of the step, each after ``past`` cached tokens; ``batch`` single tokens of requests
    that hold ``context`` cached tokens each."""
    return {"name": name, "kind": kind, "size": size, "lens": lens, "past": past, "batch": batch, "context": context,
            "dtype": "bfloat16", "chunk": 0, "cap": 0.0, "new": 0, **more}


def listed():
    return [
        # one user, a short context, the middle model: latency of one attention sublayer
        _case("attention_1x640", "attention", "500m", batch=1, context=640),
        # the benchmark's decode: eight users at the longest context, as many kv heads as heads
        _case("attention_8x8192", "attention", "2b", batch=8, context=8192),
        # continuous batching with grouped heads, 64 users with 7,472 tokens of prompt behind them; an odd length
        _case("attention_64x7531", "attention", "500m", batch=64, context=7531),
        # chunked prefill: three portions of odd sizes beside one another, each behind 2,048 cached tokens
        _case("attention_portions", "attention", "500m", lens="700+511+130", past=2048),
        # the 32-bit path that checks the 16-bit one: a short prompt
        _case("attention_f32_333", "attention", "256m", lens="333", dtype="float32"),
        # attention through a latent: prompts, one of them short, and eight long contexts
        _case("latent_portions", "latent", "w2048", lens="1531+517"),
        _case("latent_8x8192", "latent", "w2048", batch=8, context=8192),
        # the recurrent mixers over a prompt
        _case("ssd_2048", "ssd", "w2048", lens="2048"),
        _case("delta_2048", "delta", "w2048", lens="2048"),
        # differential attention over a prompt
        _case("diff_2048", "diff", "w2048", lens="2048"),
        # routed experts with a shared one, over a prompt
        _case("experts_2048", "experts", "w2048", lens="2048"),
        # whole requests of the largest decoder: eight prompts of 512, then sixteen tokens each
        _case("steps_2b_8", "steps", "2b", lens="512", batch=8, new=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "latent", "latent", "ssd", "delta", "diff", "experts", "steps"])
    if kind == "steps":
        batch = rng.choice([1, 2, 3, 5, 8])
        return _plain(_case("", kind, rng.choice(["256m", "500m", "2b"]), lens=str(_log(rng, 7, 512)), batch=batch, new=rng.randint(1, 16)))
    single = kind != "experts" and rng.random() < 0.5
    size = rng.choice(list(DECODERS) if kind == "attention" else list(WIDTHS))
    if single:
        batch = _log(rng, 1, 64)
        most = 8192 if kind == "attention" and size != "2b" else min(8192, 65536 // batch)
        most = min(most, 7531) if batch > 48 else most
        case = _case("", kind, size, batch=batch, context=_log(rng, 16, most) if kind in ("attention", "latent", "diff") else 0)
    else:
        total = _log(rng, 2 if kind == "experts" else 17, 2048)
        first = total if kind == "experts" or total < 64 or rng.random() < 0.5 else rng.randint(total // 4, total - 2)
        case = _case("", kind, size, lens=str(total) if first == total else "%d+%d" % (first, total - first))
        if kind in ("attention", "latent", "diff") and rng.random() < 0.4:
            case["past"] = _log(rng, 16, 2048)
    if kind == "attention" and size != "2b" and rng.random() < 0.3:
        case["chunk"], case["cap"] = rng.choice([(1024, 0.0), (1024, 30.0), (0, 30.0)])
    if kind == "attention" and case["lens"] and size == "256m" and rng.random() < 0.3 and sum(_lens(case)) <= 512:
        case["dtype"], case["past"] = "float32", 0
    return _plain(case)


def _plain(case):
    return {k: v for k, v in case.items() if k != "name"}


def _lens(case):
    return [int(n) for n in case["lens"].split("+")] if case["lens"] else []


def _rows(case):
    """Per sequence of the step: (tokens, cached tokens before them)."""
    return [(n, case["past"]) for n in _lens(case)] if case["lens"] else [(1, case["context"])] * case["batch"]


def _hidden(case):
    return DECODERS[case["size"]][0] if case["size"] in DECODERS else WIDTHS[case["size"]]["hidden"]


def _gen(case, seed, which):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + which) & 0x7FFFFFFFFFFFFFFF)


# --- weights and inputs, by the tensors' names ------------------------------------------------------------------------

def _shapes(case):
    """Name -> (shape, kind of values) of the sublayer's checkpoint tensors."""
    h = _hidden(case)
    kind = case["kind"]
    if kind == "attention":
        _, _, nq, nkv, _, _, _ = DECODERS[case["size"]]
        return {"q_proj.weight": ((nq * 64, h), "sharp"), "k_proj.weight": ((nkv * 64, h), "m"), "v_proj.weight": ((nkv * 64, h), "m"),
                "o_proj.weight": ((h, nq * 64), "m")}
    m = WIDTHS[case["size"]]
    if kind == "experts":
        ff = m["ff"] // 8
        out = {"router": ((EXPERTS, h), "m")}
        for e in range(EXPERTS):
            out.update({f"e{e}.gate": ((ff, h), "m"), f"e{e}.up": ((ff, h), "m"), f"e{e}.down": ((h, ff), "m")})
        out.update({"shared.gate": ((m["ff"] // 2, h), "m"), "shared.up": ((m["ff"] // 2, h), "m"), "shared.down": ((h, m["ff"] // 2), "m")})
        return out
    m = m[kind]
    H = m["heads"]
    if kind == "latent":
        d, dr, dv, r = m["dim"], m["rot"], m["v"], m["rank"]
        return {"q": ((H * (d + dr), h), "sharp"), "dkv": ((r + dr, h), "m"), "dkv.norm": ((r,), "norm"), "uk": ((H * d, r), "m"),
                "uv": ((H * dv, r), "m"), "g": ((H, h), "m"), "o": ((h, H * dv), "m")}
    if kind == "ssd":
        inner, ch = H * m["p"], H * m["p"] + 2 * m["groups"] * m["state"]
        return {"in": ((inner + ch + H, h), "m"), "conv": ((ch, TAPS), "conv"), "conv.b": ((ch,), "small"), "dt_bias": ((H,), "dt"),
                "A_log": ((H,), "decay"), "D": ((H,), "norm"), "norm": ((inner,), "norm"), "o": ((h, inner), "m")}
    if kind == "delta":
        qk, inner = m["key_heads"] * m["dim"], H * m["dim"]
        return {"q": ((qk, h), "m"), "k": ((qk, h), "m"), "v": ((inner, h), "m"), "g": ((inner, h), "m"), "b": ((H, h), "m"), "a": ((H, h), "m"),
                "q.conv": ((qk, TAPS), "conv"), "k.conv": ((qk, TAPS), "conv"), "v.conv": ((inner, TAPS), "conv"), "dt_bias": ((H,), "dt"),
                "A_log": ((H,), "decay"), "norm": ((m["dim"],), "norm"), "o": ((h, inner), "m")}
    d = m["dim"]
    widths = {"q": H * 2 * d, "k": m["kv"] * 2 * d, "v": m["kv"] * m["v"]}
    out = {n: ((w, h), "sharp" if n == "q" else "m") for n, w in widths.items()}
    out.update({n + ".conv": ((w, TAPS), "conv") for n, w in widths.items()})
    out.update({n: ((d,), "tiny") for n in ("lq1", "lk1", "lq2", "lk2")})
    return {**out, "o": ((h, H * m["v"]), "m")}


def _tensors(case, seed):
    """The sublayer's weights, rounded to 16 bits on both paths (so that both see the same values).  The query projection is
    scaled so that a token's scores spread as a trained model's do: a few of its keys carry most of the weight."""
    g = _gen(case, seed, 1)
    out = {}
    for name, (shape, kind) in _shapes(case).items():
        t = torch.randn(shape, generator=g, device="cuda")
        if kind in ("m", "sharp"):
            t *= (2.0 if kind == "sharp" else 1.0) / math.sqrt(shape[1])
        elif kind == "conv":
            t *= 0.4
        elif kind == "norm":
            t = 1.0 + 0.2 * t
        elif kind == "decay":
            t = torch.log(0.5 + 3.0 * torch.rand(shape, generator=g, device="cuda"))
        elif kind == "dt":
            t -= 1.0
        else:
            t *= 0.2 if kind == "small" else 0.1
        out[name] = t.to(torch.bfloat16)
    return out


def _inputs(case, seed):
    """Normed rows, the residual stream beside them, the next norm's weight; cached rows per sequence; states."""
    g = _gen(case, seed, 2)
    h, kind = _hidden(case), case["kind"]
    dtype = getattr(torch, case["dtype"])
    rows = _rows(case)
    n = sum(a for a, _ in rows)
    rand = lambda *shape: torch.randn(shape, generator=g, device="cuda")     # noqa: E731
    out = {"x": rand(n, h).to(torch.bfloat16).to(dtype), "hidden": 0.5 * rand(n, h), "norm": 1.0 + 0.1 * rand(h), "cached": [], "state": {}}
    if kind in ("attention", "latent", "diff"):
        for _, past in rows:
            if kind == "attention":
                nkv = DECODERS[case["size"]][3]
                kv = (rand(past, nkv, 64), rand(past, nkv, 64))
            elif kind == "latent":
                m = WIDTHS[case["size"]]["latent"]
                kv = (rand(past, 1, m["rank"] + m["rot"]), None)
            else:
                m = WIDTHS[case["size"]]["diff"]
                kv = (rand(past, m["kv"], 2 * m["dim"]), rand(past, m["kv"], m["v"]))
            out["cached"].append(tuple(None if t is None else t.to(torch.bfloat16).to(dtype) for t in kv))
    running = not case["lens"] or case["past"] > 0       # requests that have seen tokens hold a state
    if kind == "ssd":
        m = WIDTHS[case["size"]]["ssd"]
        ch = m["heads"] * m["p"] + 2 * m["groups"] * m["state"]
        out["state"] = {"conv": rand(len(rows), TAPS - 1, ch), "ssm": 0.5 * rand(len(rows), m["heads"], m["state"], m["p"])}
    elif kind == "delta":
        m = WIDTHS[case["size"]]["delta"]
        ch = 2 * m["key_heads"] * m["dim"] + m["heads"] * m["dim"]
        out["state"] = {"conv": rand(len(rows), TAPS - 1, ch), "delta": 0.3 * rand(len(rows), m["heads"], m["dim"], m["dim"])}
    elif kind == "diff":
        m = WIDTHS[case["size"]]["diff"]
        ch = m["heads"] * 2 * m["dim"] + m["kv"] * (2 * m["dim"] + m["v"])
        out["state"] = {"qkv_conv": rand(len(rows), TAPS - 1, ch)}
    for name, t in out["state"].items():
        t.mul_(1.0 if running else 0.0)
        if name.endswith("conv"):                        # (inputs of the convolution were rows of the element type)
            out["state"][name] = t.to(dtype).float()
    return out


# --- what a program keeps ---------------------------------------------------------------------------------------------

def _mixer(case):
    """The part as a model plan names it (for the experts: a mixer that is never run)."""
    h, kind = _hidden(case), case["kind"]
    if kind == "attention":
        _, _, nq, nkv, _, _, theta = DECODERS[case["size"]]
        return PartSpec("attention", {"hidden": h, "n_q_heads": nq, "n_kv_heads": nkv, "head_dim": 64, "chunk": case["chunk"],
                                      "softcap": case["cap"], "position": PartSpec("rope_halves", {"head_dim": 64, "theta": theta})})
    if kind == "experts":
        return PartSpec("attention", {"hidden": h, "n_q_heads": 1, "n_kv_heads": 1, "head_dim": 64, "position": PartSpec("none")})
    m = WIDTHS[case["size"]][kind]
    if kind == "latent":
        return PartSpec("latent_attention", {"hidden": h, "n_heads": m["heads"], "dim": m["dim"], "rot_dim": m["rot"], "v_dim": m["v"],
                                             "kv_rank": m["rank"], "scale": (m["dim"] + m["rot"]) ** -0.5, "rot_base": 10000.0,
                                             "rot_dims": m["rot"], "eps": EPS})
    if kind == "ssd":
        return PartSpec("ssd", {"hidden": h, "n_heads": m["heads"], "head_dim": m["p"], "state": m["state"], "groups": m["groups"],
                                "conv": TAPS, "norm_groups": m["groups"], "eps": EPS})
    if kind == "delta":
        return PartSpec("gated_delta", {"hidden": h, "n_heads": m["heads"], "n_key_heads": m["key_heads"], "key_dim": m["dim"],
                                        "v_dim": m["dim"], "conv": TAPS, "eps": EPS})
    return PartSpec("diff_attention", {"hidden": h, "n_q_heads": m["heads"], "n_kv_heads": m["kv"], "dim": m["dim"], "v_dim": m["v"],
                                       "scale": m["dim"] ** -0.5, "diff": DIFF["diff"], "eps": EPS, "softcap": DIFF["cap"], "conv": TAPS,
                                       "rot_base": DIFF["base"], "rot_dims": m["dim"]})


def _prepare_sublayer(case, seed):
    device, dtype, h = torch.device("cuda:0"), getattr(torch, case["dtype"]), _hidden(case)
    norm = PartSpec("rmsnorm", {"size": h, "eps": EPS})
    plan = ModelPlan(hidden_size=h, vocab_size=16, embedding=PartSpec("table", {"vocab": 16, "hidden": h}, "embed."),
                     layers=[LayerSpec("l.", PartSpec("prenorm"), norm, _mixer(case), None, None)], schedule=[LayerCall(0, 0)],
                     final_norm=norm, head=PartSpec("linear", {"vocab": 16, "hidden": h, "tied_to": "embed.weight"}, "head."))
    model = DecoderModel(plan, dtype, device)
    tensors, inputs, rows = _tensors(case, seed), _inputs(case, seed), _rows(case)
    if case["kind"] == "experts":
        ff = WIDTHS[case["size"]]["ff"]
        part = build_part("ffn", PartSpec("routed_experts", {
            "hidden": h, "intermediate": ff // 8, "n_experts": EXPERTS, "top": TOP,
            "shared": PartSpec("glu_bounded", {"hidden": h, "intermediate": ff // 2}, "shared.")}), dtype, device)
    else:
        part = model.blocks[0].mixer
    part.load_weights(tensors)
    model.final_norm.load_weights({"weight": inputs["norm"]})
    pages = [sum(-(-(a + past) // PAGE) for a, past in rows)] * len(model.cache_layout.groups)
    cache = CacheManager(model.cache_layout, PAGE, pages, max_requests=len(rows))
    pools = DevicePools(model.cache_layout, PAGE, pages, len(rows), dtype, device)
    runner = ModelRunner(model, cache, pools, max_step_tokens=4096, pad_decodes=False)
    for s, (_, past) in enumerate(rows):
        request = cache.admit(s)
        if past:
            cache.grow(s, past)
            cache.advance(s, past)
        if past and inputs["cached"]:
            ids = torch.from_numpy(request.tables[0].array().copy()).long().to(device)
            live = ids >= 0                              # (pages behind the chunk have gone back)
            for pool, t in zip(pools.pages_of(0), inputs["cached"][s]):
                if t is not None:
                    full = torch.zeros((ids.numel() * PAGE,) + tuple(t.shape[1:]), dtype=dtype, device=device)
                    full[:past] = t
                    pool[ids[live]] = full.view(ids.numel(), PAGE, t.shape[1], t.shape[2]).transpose(1, 2)[live]
        for name, t in inputs["state"].items():
            pools.states[f"{name}@0"][request.slot] = t[s]
    ctx, _ = runner.prepare([StepEntry(s, tokens=[0] * a) for s, (a, _) in enumerate(rows)])
    return {"part": part, "norm": model.final_norm, "ctx": ctx, "x": inputs["x"], "hidden": inputs["hidden"],
            "out": torch.empty_like(inputs["x"]), "call": None if case["kind"] == "experts" else LayerCall(0, 0), "runner": runner}


def _decoder_tensors(case, seed, specs):
    """A decoder's weights by name, ``N(0, 0.02)`` as the benchmark's random ones (a generator walks them in order)."""
    g = _gen(case, seed, 3)
    for name, shape in specs:
        yield name, (1.0 + 0.1 * torch.randn(shape, generator=g, device="cuda") if len(shape) == 1
                     else 0.02 * torch.randn(shape, generator=g, device="cuda")).to(torch.bfloat16)


def _decoder_specs(case):
    h, layers, nq, nkv, ff, vocab, _ = DECODERS[case["size"]]
    out = [("embed_tokens.weight", (vocab, h)), ("norm.weight", (h,))]
    for i in range(layers):
        p = f"layers.{i}."
        out += [(p + "input_layernorm.weight", (h,)), (p + "self_attn.q_proj.weight", (nq * 64, h)), (p + "self_attn.k_proj.weight", (nkv * 64, h)),
                (p + "self_attn.v_proj.weight", (nkv * 64, h)), (p + "self_attn.o_proj.weight", (h, nq * 64)),
                (p + "post_attention_layernorm.weight", (h,)), (p + "mlp.gate_proj.weight", (ff, h)), (p + "mlp.up_proj.weight", (ff, h)),
                (p + "mlp.down_proj.weight", (h, ff))]
    return out


def _token_ids(case, seed):
    g = torch.Generator().manual_seed(int(seed) * 7919 + 5)
    vocab, n = DECODERS[case["size"]][5], int(case["lens"])
    return torch.randint(0, vocab, (case["batch"], n + case["new"]), generator=g).tolist()


def _prepare_steps(case, seed):
    h, layers, nq, nkv, ff, vocab, theta = DECODERS[case["size"]]
    raw = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": layers, "hidden_size": h,
           "num_attention_heads": nq, "num_key_value_heads": nkv, "head_dim": 64, "intermediate_size": ff, "vocab_size": vocab,
           "rope_theta": theta, "rms_norm_eps": EPS, "tie_word_embeddings": True, "max_position_embeddings": 8192,
           "hidden_act": "silu", "pad_token_id": 0}
    arch = architecture_of(raw)
    config = arch.read_config(raw, "config")
    model = DecoderModel(arch.make_plan(config), torch.bfloat16, torch.device("cuda:0"))
    tensors = dict(_decoder_tensors(case, seed, _decoder_specs(case)))
    tensors["lm_head.weight"] = tensors["embed_tokens.weight"]
    model.load_weights(tensors)
    n = int(case["lens"]) + case["new"]
    engine = Engine(model, config, EngineOptions(num_blocks=case["batch"] * (n // PAGE + 1) + 1, max_batch_size=case["batch"],
                                                 max_step_tokens=case["batch"] * n))
    return {"engine": engine, "ids": _token_ids(case, seed), "prompt": int(case["lens"])}


def prepare(case, seed):
    return _prepare_steps(case, seed) if case["kind"] == "steps" else _prepare_sublayer(case, seed)


def run(state):
    if "engine" in state:
        runner, prompt = state["engine"].runner, state["prompt"]
        for r in range(len(state["ids"])):
            runner.admit(r)
        logits = [runner.step([StepEntry(r, tokens=ids[:prompt], want=[prompt - 1]) for r, ids in enumerate(state["ids"])]).clone()]
        for t in range(prompt, len(state["ids"][0])):
            logits.append(runner.step([StepEntry(r, tokens=[ids[t]], want=[0]) for r, ids in enumerate(state["ids"])]).clone())
        for r in range(len(state["ids"])):
            runner.release(r)
        return torch.stack(logits)
    ctx = state["ctx"]
    if state["call"] is None:
        update = state["part"].forward(state["x"], ctx)
    else:
        update = state["part"].forward(state["x"], ctx, state["call"])
    state["norm"].forward(state["hidden"], state["out"], update, write_back=False)
    pools = state["runner"].pools
    return {"rows": state["out"], **{name.split("@")[0]: t for name, t in pools.states.items()}}


# --- bytes and operations that a pass cannot do without ---------------------------------------------------------------

def _pairs(case):
    """(query, key) pairs that the mask lets a step see, and cached tokens read."""
    pairs, read = 0, 0
    for n, past in _rows(case):
        if case["chunk"]:
            lo = past // case["chunk"] * case["chunk"]
            pairs += sum((p % case["chunk"]) + 1 for p in range(past, past + n))
            read += past - lo
        else:
            pairs += n * past + n * (n + 1) // 2
            read += past
    return pairs, read


def work(case):
    if case["kind"] == "steps":
        h, layers, nq, nkv, ff, vocab, _ = DECODERS[case["size"]]
        weights = layers * (h * 64 * (2 * nq + 2 * nkv) + 3 * h * ff)
        b, n, new = case["batch"], int(case["lens"]), case["new"]
        kv = layers * 2 * nkv * 64 * 2
        reads = (new + 1) * 2 * (weights + vocab * h) + sum(b * (n + t) * kv for t in range(new + 1)) + 4 * b * (new + 1) * vocab
        pairs = b * (n * (n + 1) // 2 + sum(n + t + 1 for t in range(new)))
        return {"bytes": reads, "flops": 2 * weights * b * (n + new) + 2 * vocab * h * b * (new + 1) + 4 * 64 * nq * layers * pairs}
    item = 4 if case["dtype"] == "float32" else 2
    h, kind = _hidden(case), case["kind"]
    rows = _rows(case)
    n = sum(a for a, _ in rows)
    params = sum(math.prod(s) for s, _ in _shapes(case).values())
    stream = n * h * (2 * item + 4)                                   # rows in, residual stream in, normed rows out
    if kind == "experts":
        ff = WIDTHS[case["size"]]["ff"]
        used = min(EXPERTS, n * TOP)
        touched = used * 3 * h * ff // 8 + 3 * h * ff // 2 + EXPERTS * h
        return {"bytes": touched * item + stream, "flops": 2 * n * (3 * h * (TOP * ff // 8 + ff // 2) + EXPERTS * h)}
    pairs, read = _pairs(case) if kind in ("attention", "latent", "diff") else (0, 0)
    flops, nbytes = 2 * n * params, params * item + stream
    if kind == "attention":
        _, _, nq, nkv, _, _, _ = DECODERS[case["size"]]
        return {"bytes": nbytes + (read + n) * 2 * nkv * 64 * item, "flops": flops + 4 * 64 * nq * pairs}
    m = WIDTHS[case["size"]][kind]
    H = m["heads"]
    if kind == "latent":
        # per token the keys and values of a head are made from the latent, or the query and the result carried over to it
        flops = 2 * n * (params - 2 * H * m["dim"] * m["rank"]) + 4 * n * H * m["dim"] * m["rank"]
        return {"bytes": nbytes + (read + n) * (m["rank"] + m["rot"]) * item, "flops": flops + 2 * H * (2 * m["dim"] + m["rot"]) * pairs}
    if kind == "diff":
        per = m["kv"] * (2 * m["dim"] + m["v"])
        return {"bytes": nbytes + (read + n) * per * item, "flops": flops + 2 * H * (2 * m["dim"] + 2 * m["v"]) * pairs}
    state = H * (m["state"] * m["p"] if kind == "ssd" else m["dim"] ** 2)
    return {"bytes": nbytes + 8 * len(rows) * state, "flops": flops + (6 if kind == "ssd" else 8) * n * state}


def tolerance(case):
    # About four times what the 64-bit results differ by: 0.5e-6 to 1e-6 for 32-bit rows, 2.5e-3 to 4.5e-3 for a sublayer in
    # 16 bits (states among them), 2.0e-2 to 2.9e-2 for the logits behind 24 layers.
    if case["dtype"] == "float32":
        return {"rel": 4e-6}
    return {"rel": 8e-2 if case["kind"] == "steps" else 1.5e-2}


# --- the same results in 64 bits, in plain torch ------------------------------------------------------------------------

def _rms(x, w, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _halves(x, pos, theta):
    """Pairs (i, i + d / 2) of the last axis turned by ``pos * theta ** (-2 i / d)``, the frequencies in 32 bits."""
    d = x.shape[-1]
    f = (1.0 / (theta ** (torch.arange(0, d, 2).float() / d))).to(x.device, F64)
    a = (pos.to(F64)[:, None] * f).reshape((len(pos),) + (1,) * (x.dim() - 2) + (d // 2,))
    lo, hi = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)


def _pairs_turned(x, pos, theta):
    d = x.shape[-1]
    f = theta ** (-2.0 * torch.arange(d // 2, device=x.device, dtype=F64) / d)
    a = (pos.to(F64)[:, None] * f).reshape((len(pos),) + (1,) * (x.dim() - 2) + (d // 2,))
    out = torch.empty_like(x)
    out[..., 0::2] = x[..., 0::2] * a.cos() - x[..., 1::2] * a.sin()
    out[..., 1::2] = x[..., 1::2] * a.cos() + x[..., 0::2] * a.sin()
    return out


def _seen(n, past, chunk=0):
    i = torch.arange(past, past + n, device="cuda")[:, None]
    j = torch.arange(past + n, device="cuda")[None, :]
    return (j <= i) & (i // chunk == j // chunk) if chunk else j <= i


def _weights(s, seen):
    return torch.softmax(s.masked_fill(~seen, float("-inf")), -1)


def _gqa(q, k, v, seen, cap=0.0):
    """``q`` [n, heads, 64], ``k``, ``v`` [keys, kv heads, 64]; a head at a time."""
    rep = q.shape[1] // k.shape[1]
    out = torch.empty_like(q)
    for hd in range(q.shape[1]):
        s = q[:, hd] @ k[:, hd // rep].T * 64 ** -0.5
        if cap:
            s = cap * torch.tanh(s / cap)
        out[:, hd] = _weights(s, seen) @ v[:, hd // rep]
    return out


def _conv(x, before, w, b=None):
    """Causal convolution per channel behind the rows ``before`` it; the last rows that the next token needs."""
    taps, n = w.shape[1], x.shape[0]
    full = torch.cat([before, x], 0)
    y = sum(full[t: t + n] * w[:, t] for t in range(taps))
    return (y if b is None else y + b), full[n:]


def _silu(x):
    return x * torch.sigmoid(x)


def _attention64(case, w, x, past, cached, state):
    _, _, nq, nkv, _, _, theta = DECODERS[case["size"]]
    n = x.shape[0]
    pos = torch.arange(past, past + n, device="cuda")
    q = _halves((x @ w["q_proj.weight"].T).view(n, nq, 64), pos, theta)
    k = torch.cat([cached[0], _halves((x @ w["k_proj.weight"].T).view(n, nkv, 64), pos, theta)], 0)
    v = torch.cat([cached[1], (x @ w["v_proj.weight"].T).view(n, nkv, 64)], 0)
    return _gqa(q, k, v, _seen(n, past, case["chunk"]), case["cap"]).reshape(n, -1) @ w["o_proj.weight"].T, {}


def _latent64(case, w, x, past, cached, state):
    m, n = WIDTHS[case["size"]]["latent"], x.shape[0]
    H, d, dr, dv, r = m["heads"], m["dim"], m["rot"], m["v"], m["rank"]
    pos = torch.arange(past, past + n, device="cuda")
    q = (x @ w["q"].T).view(n, H, d + dr)
    qr = _pairs_turned(q[..., d:], pos, 10000.0)
    down = x @ w["dkv"].T
    c = torch.cat([cached[0][:, 0, :r], _rms(down[:, :r], w["dkv.norm"])], 0)
    kr = torch.cat([cached[0][:, 0, r:], _pairs_turned(down[:, r:], pos, 10000.0)], 0)
    gate, seen = torch.sigmoid(x @ w["g"].T), _seen(n, past)
    out = []
    for hd in range(H):
        s = (q[:, hd, :d] @ (c @ w["uk"][hd * d: (hd + 1) * d].T).T + qr[:, hd] @ kr.T) * (d + dr) ** -0.5
        out.append(gate[:, hd: hd + 1] * (_weights(s, seen) @ (c @ w["uv"][hd * dv: (hd + 1) * dv].T)))
    return torch.cat(out, -1) @ w["o"].T, {}


def _ssd64(case, w, x, past, cached, state):
    m, n = WIDTHS[case["size"]]["ssd"], x.shape[0]
    H, P, N, G = m["heads"], m["p"], m["state"], m["groups"]
    inner = H * P
    proj = x @ w["in"].T
    z, dt = proj[:, :inner], torch.nn.functional.softplus(proj[:, -H:] + w["dt_bias"], threshold=1e9)
    xbc, kept = _conv(proj[:, inner: -H], state["conv"], w["conv"], w["conv.b"])
    xbc = _silu(xbc)
    u = xbc[:, :inner].view(n, H, P)
    B = xbc[:, inner: inner + G * N].view(n, G, N).repeat_interleave(H // G, 1)
    C = xbc[:, inner + G * N:].view(n, G, N).repeat_interleave(H // G, 1)
    decay, S = torch.exp(-torch.exp(w["A_log"]) * dt), state["ssm"]
    y = torch.empty_like(u)
    for t in range(n):
        S = S * decay[t, :, None, None] + (dt[t, :, None] * B[t])[:, :, None] * u[t, :, None, :]
        y[t] = torch.bmm(C[t][:, None], S)[:, 0]
    y = (y + w["D"][:, None] * u).view(n, inner) * _silu(z)
    y = _rms(y.view(n, G, inner // G), 1.0).view(n, inner) * w["norm"]
    return y @ w["o"].T, {"conv": kept, "ssm": S}


def _delta64(case, w, x, past, cached, state):
    m, n = WIDTHS[case["size"]]["delta"], x.shape[0]
    H, G, d = m["heads"], m["key_heads"], m["dim"]
    qkv, kept = _conv(torch.cat([x @ w[i].T for i in "qkv"], -1), state["conv"], torch.cat([w[i + ".conv"] for i in "qkv"], 0))
    qkv = _silu(qkv)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)      # noqa: E731
    q = (unit(qkv[:, : G * d].reshape(n, G, d)) * d ** -0.5).repeat_interleave(H // G, 1)
    k = unit(qkv[:, G * d: 2 * G * d].reshape(n, G, d)).repeat_interleave(H // G, 1)
    v = qkv[:, 2 * G * d:].reshape(n, H, d)
    beta = torch.sigmoid(x @ w["b"].T)
    g = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"], threshold=1e9))
    S, o = state["delta"], torch.empty_like(v)                                  # S: [heads, value, key]
    for t in range(n):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(S, k[t, :, :, None])[..., 0])
        S = S + u[:, :, None] * k[t, :, None, :]
        o[t] = torch.bmm(S, q[t, :, :, None])[..., 0]
    o = _rms(o, w["norm"]) * _silu(x @ w["g"].T).view(n, H, d)
    return o.reshape(n, H * d) @ w["o"].T, {"conv": kept, "delta": S}


def _diff64(case, w, x, past, cached, state):
    m, n = WIDTHS[case["size"]]["diff"], x.shape[0]
    H, G, d, dv = m["heads"], m["kv"], m["dim"], m["v"]
    qkv, kept = _conv(torch.cat([x @ w[i].T for i in "qkv"], -1), state["qkv_conv"], torch.cat([w[i + ".conv"] for i in "qkv"], 0))
    pos, wq, wk = torch.arange(past, past + n, device="cuda"), H * 2 * d, G * 2 * d
    f = DIFF["base"] ** (-2.0 * torch.arange(d // 2, device="cuda", dtype=F64) / d)
    a = (pos.to(F64)[:, None] * f)[:, None, None, :]

    def turned(t, heads):
        t = t.reshape(n, heads, 2, d)
        lo, hi = t[..., : d // 2], t[..., d // 2:]
        return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)

    q = turned(qkv[:, :wq], H)
    k = torch.cat([cached[0].view(past, G, 2, d), turned(qkv[:, wq: wq + wk], G)], 0)
    v = torch.cat([cached[1], qkv[:, wq + wk:].reshape(n, G, dv)], 0)
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + DIFF["diff"]
    seen, out = _seen(n, past), []
    for hd in range(H):
        kv = hd // (H // G)
        o = [_weights(DIFF["cap"] * torch.tanh(q[:, hd, s] @ k[:, kv, s].T * d ** -0.5 / DIFF["cap"]), seen) @ v[:, kv] for s in (0, 1)]
        out.append(_rms(o[0] - lam * o[1], 1.0 - DIFF["diff"]))
    return torch.cat(out, -1) @ w["o"].T, {"qkv_conv": kept}


def _experts64(w, x):
    glu = lambda t, p: (_silu(t @ w[p + "gate"].T) * (t @ w[p + "up"].T)) @ w[p + "down"].T      # noqa: E731
    score, chosen = torch.topk(torch.sigmoid(x @ w["router"].T), TOP, dim=-1)
    out = glu(x, "shared.")
    for e in range(EXPERTS):
        row, place = torch.nonzero(chosen == e, as_tuple=True)
        if row.numel():
            out[row] += glu(x[row] * score[row, place][:, None], f"e{e}.")
    return out


def _steps64(case, seed):
    """A layer at a time over all requests, so that one layer's weights are held in 64 bits."""
    h, layers, nq, nkv, ff, vocab, theta = DECODERS[case["size"]]
    ids = torch.tensor(_token_ids(case, seed), device="cuda")
    prompt, total = int(case["lens"]), ids.shape[1]
    w = dict(_decoder_tensors(case, seed, _decoder_specs(case)))
    x = w["embed_tokens.weight"][ids].to(F64)                                     # [batch, total, hidden]
    pos, seen = torch.arange(total, device="cuda"), _seen(total, 0)
    for i in range(layers):
        t = {k[len(f"layers.{i}."):]: v.to(F64) for k, v in w.items() if k.startswith(f"layers.{i}.")}
        y = _rms(x, t["input_layernorm.weight"])
        for b in range(x.shape[0]):
            q = _halves((y[b] @ t["self_attn.q_proj.weight"].T).view(total, nq, 64), pos, theta)
            k = _halves((y[b] @ t["self_attn.k_proj.weight"].T).view(total, nkv, 64), pos, theta)
            v = (y[b] @ t["self_attn.v_proj.weight"].T).view(total, nkv, 64)
            x[b] += _gqa(q, k, v, seen).reshape(total, -1) @ t["self_attn.o_proj.weight"].T
        y = _rms(x, t["post_attention_layernorm.weight"])
        x = x + (_silu(y @ t["mlp.gate_proj.weight"].T) * (y @ t["mlp.up_proj.weight"].T)) @ t["mlp.down_proj.weight"].T
    y = _rms(x[:, prompt - 1:], w["norm.weight"].to(F64))
    return (y @ w["embed_tokens.weight"].to(F64).T).transpose(0, 1).contiguous()


def exact(case, seed):
    if case["kind"] == "steps":
        return _steps64(case, seed)
    w = {k: v.to(F64) for k, v in _tensors(case, seed).items()}
    given = _inputs(case, seed)
    x, rows = given["x"].to(F64), _rows(case)
    if case["kind"] == "experts":
        update, states = _experts64(w, x), {}
    else:
        fn = {"attention": _attention64, "latent": _latent64, "ssd": _ssd64, "delta": _delta64, "diff": _diff64}[case["kind"]]
        parts, at = [], 0
        for s, (n, past) in enumerate(rows):
            cached = [None if t is None else t.to(F64) for t in given["cached"][s]] if given["cached"] else None
            parts.append(fn(case, w, x[at: at + n], past, cached, {k: t[s].to(F64) for k, t in given["state"].items()}))
            at += n
        update = torch.cat([p[0] for p in parts], 0)
        states = {k: torch.stack([p[1][k] for p in parts]) for k in given["state"]}
    return {"rows": _rms(given["hidden"].to(F64) + update, given["norm"].to(F64)), **states}
