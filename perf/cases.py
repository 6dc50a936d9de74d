"""What a program does with this framework, in pieces that can be timed and compared.

Twelve listed cases and any number of drawn ones.  Three are whole steps through the step function, which return
logits: decoding a batch, a batch that decodes beside a prompt portion, and the 32-bit path.  They run as generation
runs them, from the graph that the step function captures of a shape it has seen before.  The others are single layers of
the architectures (a mixer or a feed-forward) called with a step's context, on prompt portions kernel by kernel, and on
single tokens from a captured graph, since decode steps always run captured.  Layer sizes are those of the benchmark's
configurations; weights and inputs are random with the spread that trained layers have where it matters (decays near
one, normalised inputs).

A case is a flat dictionary:

    kind      dense | attention | latent | delta | gated_delta | gla | experts
    dtype     bfloat16 | float32 (dense only)
    decode    requests that bring one token each
    portions  requests that bring a portion of a prompt each
    tokens    tokens of a portion, on the mean: with several portions they are of uneven length
    context   tokens of a request before this step, on the mean, likewise uneven

and the sizes of its kind.
"""

from __future__ import annotations

import math
import zlib

import torch

F64 = torch.float64
PAGE = 16
EPS = 1e-6

# The dense decoder at the widths of Qwen2.5 3B and 7B (fewer layers; the vocabulary is the real one), the designs with
# other mixers at the benchmark's two widths.
DENSE = {
    "3b": dict(width=2048, heads=16, kv_heads=2, dim=128, ff=11008, vocab=151936, tied=True),
    "7b": dict(width=3584, heads=28, kv_heads=4, dim=128, ff=18944, vocab=152064, tied=False),
}
ATTENTION = {2048: dict(heads=16, kv_heads=2, dim=128), 4096: dict(heads=32, kv_heads=8, dim=128)}
LATENT = {2048: dict(heads=16, q_rank=768), 4096: dict(heads=32, q_rank=1536)}
LATENT_HEAD = dict(dim=128, rot_dim=64, vdim=128, kv_rank=512)
DELTA = {2048: dict(heads=32, dim=64), 4096: dict(heads=64, dim=64)}
GATED_DELTA = {2048: dict(heads=16, kv_heads=8, dim=128), 4096: dict(heads=32, kv_heads=16, dim=128)}
GLA = {2048: dict(heads=16, dim=128), 4096: dict(heads=32, dim=128)}
EXPERTS = {2048: dict(experts=16, top=4, ff=1376), 4096: dict(experts=32, top=4, ff=2048)}
TAPS = 4
RANK = 64
TAU = 8.0
WINDOW = 1024


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    def step(name, size, layers, dtype="bfloat16", **batch):
        return dict(name=name, kind="dense", size=size, layers=layers, dtype=dtype, **_batch(**batch))

    def layer(name, kind, width, style="", **batch):
        return dict(name=name, kind=kind, width=width, style=style, dtype="bfloat16", **_batch(**batch))

    return [
        # a small server's steady state: eight requests, one token each, on their graph
        step("dense-decode-8", "3b", 8, decode=8, context=2048),
        # a loaded server: decoding requests beside a portion of a newcomer's prompt
        step("dense-mixed-7b", "7b", 4, decode=32, portions=1, tokens=512, context=1024),
        # the 32-bit path, which generation is checked against: a short prompt whole
        step("dense-float32", "3b", 2, dtype="float32", portions=1, tokens=300),
        # a long prompt's attention layer: q/k norm, rotation of half a head, a sink
        layer("attention-prompt", "attention", 2048, "sink", portions=1, tokens=2048),
        # prompts of three requests in portions, over what they have in the cache, under a window with a penalty
        layer("attention-window-portions", "attention", 2048, "penalty", portions=3, tokens=500, context=1500),
        # the same kind of layer while eight requests decode
        layer("attention-decode", "attention", 2048, "sink", decode=8, context=2048),
        # attention on cached latents: a prompt
        layer("latent-prompt", "latent", 2048, portions=1, tokens=2048),
        # the generalized delta rule over a prompt
        layer("delta-prompt", "delta", 2048, portions=1, tokens=2048),
        # the gated delta rule over uneven portions of four prompts, with states from before
        layer("gated-delta-portions", "gated_delta", 2048, portions=4, tokens=333, context=100),
        # gated linear attention over a prompt
        layer("gla-prompt", "gla", 2048, portions=1, tokens=2048),
        # routed experts: a prompt, and a decode step
        layer("experts-prompt", "experts", 2048, portions=1, tokens=2048),
        layer("experts-decode", "experts", 2048, decode=8),
    ]


def _batch(decode=0, portions=0, tokens=0, context=0):
    return dict(decode=decode, portions=portions, tokens=tokens, context=context)


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "attention", "attention", "latent", "delta", "gated_delta", "gla", "experts"])
    context = rng.choice([0, _log_int(rng, 16, 6000)])
    if kind == "dense":
        if rng.random() < 0.2:
            batch = _batch(0, 1, _log_int(rng, 17, 400), 0)
            return dict(kind=kind, size="3b", layers=2, dtype="float32", **batch)
        size, layers = rng.choice(["3b", "7b"]), rng.choice([2, 3])
        if rng.random() < 0.5:
            batch = _batch(_log_int(rng, 1, 64), 0, 0, max(context, 16))
        else:
            batch = _batch(rng.choice([0, _log_int(rng, 1, 32)]), 1, _log_int(rng, 16, 600), min(context, 3000))
        return dict(kind=kind, size=size, layers=layers, dtype="bfloat16", **batch)
    style = rng.choice(["sink", "penalty"]) if kind == "attention" else ""
    if rng.random() < 0.35:
        batch = _batch(_log_int(rng, 1, 48), 0, 0, max(context, 16))
    else:
        portions = rng.choice([1, 1, 2, 3, 5, 8])
        batch = _batch(0, portions, max(8, _log_int(rng, 48, 2300) // portions), min(context, 4000))
    if kind == "experts":
        batch["context"] = 0
    return dict(kind=kind, width=rng.choice([2048, 4096]), style=style, dtype="bfloat16", **batch)


def requests(case):
    """(tokens of this step, tokens before it) per request: decoding requests first, lengths spread about the mean."""
    out = []
    for count, tokens in ((case["decode"], 0), (case["portions"], case["tokens"])):
        for i in range(count):
            share = 0.6 + 0.8 * ((i * 7 + 3) % count) / (count - 1) if count > 1 else 1.0
            other = 0.6 + 0.8 * ((i * 5 + 1) % count) / (count - 1) if count > 1 else 1.0
            out.append((max(2, int(tokens * share)) if tokens else 1, int(case["context"] * other)))
    return out


# ------------------------------------------------------------------------------------------------ random values
def _normal(seed, name, *shape, std=1.0, mean=0.0, dtype=torch.float32):
    generator = torch.Generator(device="cuda")
    generator.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    values = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=generator)
    return values.to(dtype)


def _uniform(seed, name, *shape, low=0.0, high=1.0):
    generator = torch.Generator(device="cuda")
    generator.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(low, high, generator=generator)


def _matrix(case, seed, name, rows, columns):
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    # rounded to bfloat16 either way, as stored models are
    return _normal(seed, name, rows, columns, std=0.02, dtype=torch.bfloat16).to(dtype)


def _gain(seed, name, size):
    return _normal(seed, name, size, std=0.1, mean=1.0)


def _token_ids(case, seed, vocab):
    total = sum(new for new, _ in requests(case))
    return (_uniform(seed, "ids", total) * vocab).long().clamp_(0, vocab - 1).cpu().tolist()


def _inputs(case, seed, width):
    total = sum(new for new, _ in requests(case))
    return _normal(seed, "x", total, width, dtype=torch.bfloat16)


def _cached(case, seed, request, layer, before, heads, dim, which):
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    return _normal(seed, f"{which}.{layer}.{request}", before, heads, dim, dtype=torch.bfloat16).to(dtype)


def _weights(case, seed):
    """The tensors of a layer by the names that its part gives them."""
    kind = case["kind"]
    width = DENSE[case["size"]]["width"] if kind == "dense" else case["width"]

    def m(name, rows, columns=None):
        return _matrix(case, seed, name, rows, columns or width)

    w = {}
    if kind == "dense":
        s = DENSE[case["size"]]
        q, kv = s["heads"] * s["dim"], s["kv_heads"] * s["dim"]
        w["model.embed_tokens.weight"] = m("embed", s["vocab"])
        if not s["tied"]:
            w["lm_head.weight"] = m("head", s["vocab"])
        w["model.norm.weight"] = _gain(seed, "norm", width)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            for name, rows in (("q", q), ("k", kv), ("v", kv)):
                w[f"{p}self_attn.{name}_proj.weight"] = m(f"{i}.{name}", rows)
                w[f"{p}self_attn.{name}_proj.bias"] = _normal(seed, f"{i}.{name}.b", rows, std=0.1)
            w[p + "self_attn.o_proj.weight"] = m(f"{i}.o", width, q)
            w[p + "mlp.gate_proj.weight"] = m(f"{i}.gate", s["ff"])
            w[p + "mlp.up_proj.weight"] = m(f"{i}.up", s["ff"])
            w[p + "mlp.down_proj.weight"] = m(f"{i}.down", width, s["ff"])
            w[p + "input_layernorm.weight"] = _gain(seed, f"{i}.norm1", width)
            w[p + "post_attention_layernorm.weight"] = _gain(seed, f"{i}.norm2", width)
    elif kind == "attention":
        s = ATTENTION[width]
        q, kv = s["heads"] * s["dim"], s["kv_heads"] * s["dim"]
        w.update({"q": m("q", q), "k": m("k", kv), "v": m("v", kv), "o": m("o", width, q),
                  "q.norm": _gain(seed, "q.norm", q), "k.norm": _gain(seed, "k.norm", kv)})
        if case["style"] == "sink":
            w["sink"] = _normal(seed, "sink", s["heads"])
        else:
            w.update({name + ".b": _normal(seed, name + ".b", rows, std=0.1) for name, rows in (("q", q), ("k", kv), ("v", kv))})
            w["r1"], w["r2"] = _uniform(seed, "r1", s["heads"], high=1.0), _uniform(seed, "r2", s["heads"], high=1.0)
    elif kind == "latent":
        s, h = LATENT[width], LATENT_HEAD
        w.update({"dq": m("dq", s["q_rank"]), "dq.norm": _gain(seed, "dq.norm", s["q_rank"]),
                  "uq": m("uq", s["heads"] * (h["dim"] + h["rot_dim"]), s["q_rank"]),
                  "dkv": m("dkv", h["kv_rank"] + h["rot_dim"]), "dkv.norm": _gain(seed, "dkv.norm", h["kv_rank"]),
                  "uk": m("uk", s["heads"] * h["dim"], h["kv_rank"]), "uv": m("uv", s["heads"] * h["vdim"], h["kv_rank"]),
                  "sink": _normal(seed, "sink", s["heads"]), "o": m("o", width, s["heads"] * h["vdim"])})
    elif kind == "delta":
        inner = DELTA[width]["heads"] * DELTA[width]["dim"]
        w.update({name: m(name, inner) for name in ("r", "k", "v", "g", "a")})
        w.update({"a.b": _normal(seed, "a.b", inner), "w1": m("w1", RANK), "w2": m("w2", inner, RANK),
                  "w0": _uniform(seed, "w0", inner, low=-6.0, high=0.0), "norm": _gain(seed, "norm", inner),
                  "o": m("o", width, inner)})
    elif kind == "gated_delta":
        s = GATED_DELTA[width]
        qk, v = s["kv_heads"] * s["dim"], s["heads"] * s["dim"]
        step = torch.exp(_uniform(seed, "dt", s["heads"], low=math.log(0.001), high=math.log(0.1)))
        w.update({"q": m("q", qk), "k": m("k", qk), "v": m("v", v), "g": m("g", v), "b": m("b", s["heads"]),
                  "a": m("a", s["heads"]), "A_log": torch.log(_uniform(seed, "A", s["heads"], low=1.0, high=16.0)),
                  "dt_bias": torch.log(torch.expm1(step)), "norm": _gain(seed, "norm", s["dim"]), "o": m("o", width, v)})
        w.update({name + ".conv": _normal(seed, name + ".conv", rows, TAPS, std=0.5)
                  for name, rows in (("q", qk), ("k", qk), ("v", v))})
    elif kind == "gla":
        inner = GLA[width]["heads"] * GLA[width]["dim"]
        w.update({name: m(name, inner) for name in ("q", "k", "v", "g")})
        w.update({"o": m("o", width, inner), "norm": _gain(seed, "norm", GLA[width]["dim"]), "a1": m("a1", RANK),
                  "a2": m("a2", inner, RANK), "a2.b": _uniform(seed, "a2.b", inner, low=-1.0, high=5.0)})
    else:
        s = EXPERTS[width]
        w["router"] = _normal(seed, "router", s["experts"], width, std=0.02)
        w["router.b"] = _normal(seed, "router.b", s["experts"], std=0.1)
        for e in range(s["experts"]):
            w[f"e{e}.gate"], w[f"e{e}.up"] = m(f"{e}.gate", s["ff"]), m(f"{e}.up", s["ff"])
            w[f"e{e}.down"] = m(f"{e}.down", width, s["ff"])
    return w


def _state_floats(case):
    """(matrix floats, floats of the convolution's history) of one request's state."""
    kind, width = case["kind"], case["width"]
    if kind == "delta":
        return DELTA[width]["heads"] * DELTA[width]["dim"] ** 2, 0
    if kind == "gla":
        return GLA[width]["heads"] * GLA[width]["dim"] ** 2, 0
    s = GATED_DELTA[width]
    return s["heads"] * s["dim"] ** 2, (TAPS - 1) * (2 * s["kv_heads"] + s["heads"]) * s["dim"]


def _state_of(case, seed, request, before):
    """What a request's earlier tokens left: nothing before its first one."""
    matrix, history = _state_floats(case)
    if not before:
        return torch.zeros(matrix + history, dtype=torch.float32, device="cuda")
    return torch.cat([_normal(seed, f"state.{request}", matrix, std=0.3), _normal(seed, f"history.{request}", history)])


# ------------------------------------------------------------------------------------------------ the framework's side
def _configuration(case):
    """The config.json of a model that has the layer."""
    kind = case["kind"]
    if kind == "dense":
        s = DENSE[case["size"]]
        return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=s["width"],
                    num_hidden_layers=case["layers"], num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"],
                    intermediate_size=s["ff"], vocab_size=s["vocab"], rope_theta=1000000.0, rms_norm_eps=EPS,
                    attention_bias=True, tie_word_embeddings=s["tied"], eos_token_id=151643,
                    max_position_embeddings=32768, hidden_act="silu", use_sliding_window=False)
    width = case["width"]
    common = dict(vocab=64, width=width, norm=dict(eps=EPS))
    if kind in ("delta", "latent"):
        if kind == "delta":
            entry = dict(type="general_delta", mixer=dict(DELTA[width], decay_rank=RANK))
        else:
            h = LATENT_HEAD
            entry = dict(type="latent_attention",
                         mixer=dict(LATENT[width], **h, scale=(h["dim"] + h["rot_dim"]) ** -0.5,
                                    rot=dict(base=10000.0, dims=h["rot_dim"])))
        return dict(common, architecture="Lodalix", layers=[dict(entry, mlp=dict(kind="dense", ff=64, limit=7.0))])
    if kind == "gated_delta":
        s = GATED_DELTA[width]
        entry = dict(type="delta", mixer=dict(s, vdim=s["dim"], conv=TAPS), mlp=dict(kind="dense", ff=64))
        return dict(common, architecture="Lazilorn", embedding=dict(scale=1.0), logit_scale=1.0, layers=[entry])
    if kind == "attention" and case["style"] == "penalty":
        s = ATTENTION[width]
        entry = dict(type="attention", mixer=dict(s, vdim=s["dim"], scale=s["dim"] ** -0.5, mask=dict(size=WINDOW)))
        return dict(common, architecture="Zisesun", max_positions=16384, layers=[entry])
    dense = dict(kind="dense", ff=64)
    if kind == "attention":
        s = ATTENTION[width]
        entry = dict(type="attention", mixer=dict(s, vdim=s["dim"], scale=s["dim"] ** -0.5, rot=_rotation(s["dim"])), mlp=dense)
    else:
        s = GLA[width]
        mlp = dense
        if kind == "experts":
            e = EXPERTS[width]
            mlp = dict(kind="moe", expert=dict(ff=e["ff"]), router=dict(experts=e["experts"], top=e["top"]))
        entry = dict(type="gla", mixer=dict(s, vdim=s["dim"], tau=TAU, decay_rank=RANK), mlp=mlp)
    return dict(common, architecture="Bilipel", residual_mult=1.0, layers=[entry])


def _rotation(dim):
    return dict(base=500000.0, dims=dim // 2, scaling=dict(factor=4.0, original=2048, fast=16.0, slow=2.0))


def prepare(case, seed):
    from cloud_inference_from_scratch_b200 import models, parts  # noqa: F401  (fills the registries)
    from cloud_inference_from_scratch_b200.engine.core import build_core
    from cloud_inference_from_scratch_b200.engine.step import StepEntry

    batch = requests(case)
    longest = max(before + new for new, before in batch) + PAGE
    longest += -longest % 256
    pages = sum(-(-(before + new) // PAGE) for new, before in batch) + 2
    tokens = sum(new for new, _ in batch)
    core = build_core(None, dtype=case["dtype"], page_size=PAGE, num_pages=pages, max_requests=len(batch),
                      max_model_len=longest, max_tokens_per_step=0, random_config=_configuration(case), seed=1,
                      random_device="cuda")
    step, runtime = core.step, core.runtime
    weights = _weights(case, seed)
    dense = case["kind"] == "dense"
    if dense:
        core.model.bind(lambda name: weights[name], runtime)
        vocab = core.spec.vocab_size
        ids = _token_ids(case, seed, vocab)
    else:
        layer = core.model.layers[0]
        part = layer.feed_forward if case["kind"] == "experts" else layer.mixer
        part.bind(weights, runtime)
        ids = [0] * tokens
    del weights

    # the requests as the steps before this one have left them
    for i, (_, before) in enumerate(batch):
        step.admit(i)
    core.cache.ensure_capacity_batch({i: (0, before) for i, (_, before) in enumerate(batch)})
    core.cache.commit_lengths({i: before for i, (_, before) in enumerate(batch)})
    entries, first = [], 0
    for i, (new, _) in enumerate(batch):
        entries.append(StepEntry(i, ids[first:first + new], want=(new - 1,) if dense else ()))
        first += new
    if dense:
        step.enable_graphs(longest)
    host, _, _ = step.prepare(entries)
    for index, binding in enumerate(core.pools.bindings):
        if binding.kv is not None:
            for i, (_, before) in enumerate(batch):
                row = torch.from_numpy(host.tables[binding.kv.group][i].copy()).cuda().long()
                place = torch.arange(before, device="cuda")
                kept = row[place // PAGE] >= 0            # pages behind a window are gone
                page, offset = row[place // PAGE][kept], (place % PAGE)[kept]
                for which, pool in (("k", binding.kv.k), ("v", binding.kv.v)):
                    values = _cached(case, seed, i, index, before, pool.shape[1], pool.shape[3], which)
                    pool[page, :, offset] = values[kept]
        if binding.state is not None and case["kind"] != "experts":      # its mixer is not called
            for i, (_, before) in enumerate(batch):
                slot = core.cache.slot(i)
                binding.state[slot] = _state_of(case, seed, i, before).view(binding.state[slot].shape)
    if dense:
        for _ in range(3):      # the third time a shape comes by, the step function captures it
            step.forward_host(host)
        return dict(core=core, call=lambda: step.forward_host(host)[1])

    ctx = step.upload(host)
    binding = ctx.bindings[0]
    x = _inputs(case, seed, case["width"])
    if case["kind"] == "experts":
        def call():
            return part.forward(x, ctx)
    else:
        def call():
            update = part.forward(x, ctx, binding)
            return (update,) if binding.state is None else (update, binding.state)
    if case["portions"]:
        return dict(core=core, call=call)
    # single tokens: the launches captured once and replayed, as every decode step runs
    kept = None if case["kind"] == "experts" or binding.state is None else binding.state.clone()
    for _ in range(2):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outputs = call()
    if kept is not None:
        binding.state.copy_(kept)

    def replay():
        graph.replay()
        return outputs

    return dict(core=core, call=replay)


def run(state):
    return state["call"]()


# ------------------------------------------------------------------------------------------------ what a pass needs
def _pairs(case, window=0):
    """(query, key) pairs that causal attention weighs, and cached rows that it reads."""
    total = keys = 0
    for new, before in requests(case):
        for_each = [min(before + i + 1, window) if window else before + i + 1 for i in (0, new - 1)]
        if window and before + new > window:
            whole = sum(min(before + i + 1, window) for i in range(new))
        else:
            whole = new * (for_each[0] + for_each[1]) // 2
        total += whole
        keys += min(before, window - 1) if window else before
    return total, keys


def work(case):
    kind = case["kind"]
    batch = requests(case)
    tokens = sum(new for new, _ in batch)
    size = 4 if case["dtype"] == "float32" else 2
    if kind == "dense":
        s = DENSE[case["size"]]
        q, kv = s["heads"] * s["dim"], s["kv_heads"] * s["dim"]
        layer = s["width"] * (2 * q + 2 * kv + 3 * s["ff"])
        pairs, keys = _pairs(case)
        rows = len(batch)
        flops = 2 * tokens * layer * case["layers"] + 4 * pairs * q * case["layers"] + 2 * rows * s["width"] * s["vocab"]
        read = size * (layer * case["layers"] + s["width"] * s["vocab"] + 2 * (keys + tokens) * kv * case["layers"])
        return {"bytes": read + 4 * rows * s["vocab"], "flops": flops}
    width = case["width"]
    rows = tokens * width * (2 + 4)      # bfloat16 in, float32 out
    if kind == "experts":
        s = EXPERTS[width]
        used = s["experts"] * (1.0 - (1.0 - s["top"] / s["experts"]) ** tokens)      # experts that tokens choose at random
        matrix = 3 * width * s["ff"]
        return {"bytes": int(rows + 2 * used * matrix + 4 * width * s["experts"]),
                "flops": 2 * tokens * (s["top"] * matrix + width * s["experts"])}
    if kind == "attention":
        s = ATTENTION[width]
        q, kv = s["heads"] * s["dim"], s["kv_heads"] * s["dim"]
        pairs, keys = _pairs(case, WINDOW if case["style"] == "penalty" else 0)
        matrix = width * (2 * q + 2 * kv)
        return {"bytes": rows + 2 * matrix + 4 * (keys + tokens) * kv, "flops": 2 * tokens * matrix + 4 * pairs * q}
    if kind == "latent":
        s, h = LATENT[width], LATENT_HEAD
        heads = s["heads"]
        expand = heads * (h["dim"] + h["vdim"]) * h["kv_rank"]
        matrix = (width * (s["q_rank"] + h["kv_rank"] + h["rot_dim"] + heads * h["vdim"])
                  + s["q_rank"] * heads * (h["dim"] + h["rot_dim"]))
        pairs, keys = _pairs(case)
        # a portion expands the keys and values of all it sees; a single token takes its query to the latents instead
        if case["portions"]:
            flops = 2 * (keys + tokens) * expand + 2 * pairs * heads * (h["dim"] + h["rot_dim"] + h["vdim"])
        else:
            flops = 2 * tokens * expand + 2 * pairs * heads * (2 * h["kv_rank"] + h["rot_dim"])
        return {"bytes": rows + 2 * (matrix + expand) + 2 * (keys + tokens) * (h["kv_rank"] + h["rot_dim"]),
                "flops": 2 * tokens * matrix + flops}
    matrices, history = _state_floats(case)
    state = 8 * len(batch) * (matrices + history)      # read once, written once
    if kind == "delta":
        inner = DELTA[width]["heads"] * DELTA[width]["dim"]
        matrix = width * (6 * inner + RANK) + inner * RANK
        per_state = 9
    elif kind == "gla":
        inner = GLA[width]["heads"] * GLA[width]["dim"]
        matrix = width * (5 * inner + RANK) + inner * RANK
        per_state = 5
    else:
        s = GATED_DELTA[width]
        matrix = width * (2 * s["kv_heads"] + 3 * s["heads"]) * s["dim"] + 2 * width * s["heads"]
        per_state = 7
    return {"bytes": rows + 2 * matrix + state, "flops": 2 * tokens * matrix + per_state * tokens * matrices}


# Relative errors of a correct implementation: bfloat16 rounds the inputs of every product to 8 bits, and one layer holds
# two to four of them in a row (measured against exact(): 0.0017 to 0.0034; a stack of 4 to 8 layers 0.013; 32-bit 4e-6);
# "max" is the largest single element's, over the root mean square.
def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4}
    if case["kind"] == "dense":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.01, "max": 0.1}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _frequencies(dims, base, scaling=None):
    half = dims // 2
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(half)], dtype=F64, device="cuda")
    if scaling is None:
        return f, 1.0
    factor, original = scaling["factor"], scaling["original"]

    def pair(turns):
        return dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
    ramp = torch.tensor([min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(half)], dtype=F64, device="cuda")
    return f / factor * ramp + f * (1 - ramp), 0.1 * math.log(factor) + 1.0


def _rotate(x, positions, dims, base, scaling=None, interleaved=False):
    """x [T, heads, dim] with its first ``dims`` elements rotated."""
    f, magnitude = _frequencies(dims, base, scaling)
    angle = positions.to(F64).view(-1, 1, 1) * f
    cos, sin = torch.cos(angle) * magnitude, torch.sin(angle) * magnitude
    out = x.clone()
    first, second = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., first], x[..., second]
    out[..., first], out[..., second] = u * cos - v * sin, v * cos + u * sin
    return out


def _attend(q, k, v, before, scale, window=0, sinks=None, distance=None):
    """q [T, H, d] against k, v [before + T, kv, d]: heads in turn, rows in blocks."""
    tokens, heads = q.shape[0], q.shape[1]
    out = torch.empty(tokens, heads, v.shape[2], dtype=F64, device="cuda")
    columns = torch.arange(before + tokens, device="cuda")
    for first in range(0, tokens, 1024):
        rows = torch.arange(first, min(first + 1024, tokens), device="cuda")
        gap = (rows + before).view(-1, 1) - columns.view(1, -1)
        hidden = gap < 0
        if window:
            hidden |= gap >= window
        for h in range(heads):
            kv = h // (heads // k.shape[1])
            s = q[rows, h] @ k[:, kv].T * scale
            if distance is not None:
                s = s - distance[0][h] * torch.log1p(distance[1][h] * gap.clamp(min=0))
            s = s.masked_fill(hidden, -math.inf)
            if sinks is not None:
                s = torch.cat([s, sinks[h].expand(s.shape[0], 1)], dim=1)
            p = torch.softmax(s, dim=1)[:, :before + tokens]
            out[rows, h] = p @ v[:, kv]
    return out


def exact(case, seed):
    batch = requests(case)
    w = {name: tensor.to(F64) for name, tensor in _weights(case, seed).items()}
    kind = case["kind"]
    if kind == "dense":
        return _exact_dense(case, seed, w, batch)
    x = _inputs(case, seed, case["width"]).to(F64)
    if kind == "experts":
        return _exact_experts(case, w, x)
    spans, first = [], 0
    for i, (new, before) in enumerate(batch):
        spans.append((i, first, first + new, before))
        first += new
    if kind in ("attention", "latent"):
        layer = _exact_attention if kind == "attention" else _exact_latent
        return [torch.cat([layer(case, seed, w, x[a:b], i, before) for i, a, b, before in spans])]
    layer = {"delta": _exact_delta, "gated_delta": _exact_gated_delta, "gla": _exact_gla}[kind]
    parts = [layer(case, w, x[a:b], _state_of(case, seed, i, before).to(F64)) for i, a, b, before in spans]
    # request i has slot i: the slots of an empty table are handed out in order
    states = torch.stack([state for _, state in parts])
    if kind != "gated_delta":
        heads, dim = (DELTA if kind == "delta" else GLA)[case["width"]].values()
        states = states.view(-1, heads, dim, dim)
    return [torch.cat([update for update, _ in parts]), states]


def _exact_dense(case, seed, w, batch):
    s = DENSE[case["size"]]
    ids = torch.tensor(_token_ids(case, seed, s["vocab"]), device="cuda")
    h = w["model.embed_tokens.weight"][ids]
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}."
        x = _rms(h) * w[p + "input_layernorm.weight"]
        q, k, v = ((x @ w[f"{p}self_attn.{n}_proj.weight"].T + w[f"{p}self_attn.{n}_proj.bias"]).view(len(ids), -1, s["dim"])
                   for n in "qkv")
        outs, first = [], 0
        for i, (new, before) in enumerate(batch):
            rows = slice(first, first + new)
            first += new
            positions = torch.arange(before, before + new, device="cuda")
            qi, ki = (_rotate(t[rows], positions, s["dim"], 1000000.0) for t in (q, k))
            keys = torch.cat([_cached(case, seed, i, layer, before, s["kv_heads"], s["dim"], "k").to(F64), ki])
            values = torch.cat([_cached(case, seed, i, layer, before, s["kv_heads"], s["dim"], "v").to(F64), v[rows]])
            outs.append(_attend(qi, keys, values, before, s["dim"] ** -0.5))
        h = h + torch.cat(outs).flatten(1) @ w[p + "self_attn.o_proj.weight"].T
        x = _rms(h) * w[p + "post_attention_layernorm.weight"]
        gate = x @ w[p + "mlp.gate_proj.weight"].T
        h = h + (gate * torch.sigmoid(gate) * (x @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    last = torch.tensor([new for new, _ in batch], device="cuda").cumsum(0) - 1
    x = _rms(h[last]) * w["model.norm.weight"]
    return x @ w["model.embed_tokens.weight" if s["tied"] else "lm_head.weight"].T


def _exact_attention(case, seed, w, x, request, before):
    s = ATTENTION[case["width"]]
    tokens, sink = x.shape[0], case["style"] == "sink"
    q, k, v = (x @ w[n].T + (0 if sink else w[n + ".b"]) for n in "qkv")
    q, k = ((_rms(t) * w[n]).view(tokens, -1, s["dim"]) for t, n in ((q, "q.norm"), (k, "k.norm")))
    v = v.view(tokens, -1, s["dim"])
    if sink:
        positions = torch.arange(before, before + tokens, device="cuda")
        rot = _rotation(s["dim"])
        q, k = (_rotate(t, positions, rot["dims"], rot["base"], rot["scaling"]) for t in (q, k))
    else:
        v = _rms(v)
    k = torch.cat([_cached(case, seed, request, 0, before, s["kv_heads"], s["dim"], "k").to(F64), k])
    v = torch.cat([_cached(case, seed, request, 0, before, s["kv_heads"], s["dim"], "v").to(F64), v])
    out = _attend(q, k, v, before, s["dim"] ** -0.5, 0 if sink else WINDOW, w["sink"] if sink else None,
                  None if sink else (w["r1"], w["r2"]))
    return out.flatten(1) @ w["o"].T


def _exact_latent(case, seed, w, x, request, before):
    heads, h = LATENT[case["width"]]["heads"], LATENT_HEAD
    tokens = x.shape[0]
    positions = torch.arange(before, before + tokens, device="cuda")
    q = ((_rms(x @ w["dq"].T) * w["dq.norm"]) @ w["uq"].T).view(tokens, heads, -1)
    q = torch.cat([q[..., :h["dim"]], _rotate(q[..., h["dim"]:], positions, h["rot_dim"], 10000.0, interleaved=True)], -1)
    down = x @ w["dkv"].T
    latent = _rms(down[:, :h["kv_rank"]]) * w["dkv.norm"]
    shared = _rotate(down[:, None, h["kv_rank"]:], positions, h["rot_dim"], 10000.0, interleaved=True)[:, 0]
    latent = torch.cat([_cached(case, seed, request, 0, before, 1, h["kv_rank"], "k")[:, 0].to(F64), latent])
    shared = torch.cat([_cached(case, seed, request, 0, before, 1, h["rot_dim"], "v")[:, 0].to(F64), shared])
    keys = (latent @ w["uk"].T).view(-1, heads, h["dim"])
    keys = torch.cat([keys, shared[:, None].expand(-1, heads, -1)], -1)
    values = (latent @ w["uv"].T).view(-1, heads, h["vdim"])
    out = _attend(q, keys, values, before, (h["dim"] + h["rot_dim"]) ** -0.5, sinks=w["sink"])
    return out.flatten(1) @ w["o"].T


def _exact_delta(case, w, x, state):
    s = DELTA[case["width"]]
    heads, dim, tokens = s["heads"], s["dim"], x.shape[0]
    r, k, v, g, a = (x @ w[n].T for n in ("r", "k", "v", "g", "a"))
    rate = torch.sigmoid(a + w["a.b"]).view(tokens, heads, dim)
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ w["w1"].T) @ w["w2"].T + w["w0"])).view(tokens, heads, dim)
    r, k, v = (t.view(tokens, heads, dim) for t in (r, k, v))
    unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S = state.view(heads, dim, dim).clone()
    out = torch.empty(tokens, heads, dim, dtype=F64, device="cuda")
    for t in range(tokens):
        seen = torch.einsum("hk,hkv->hv", unit[t], S)
        S = decay[t][:, :, None] * S - (rate[t] * unit[t])[:, :, None] * seen[:, None] + k[t][:, :, None] * v[t][:, None]
        out[t] = torch.einsum("hk,hkv->hv", r[t], S)
    gated = _rms(out).flatten(1) * w["norm"] * torch.sigmoid(g)
    return gated @ w["o"].T, S.flatten()


def _exact_gated_delta(case, w, x, state):
    s = GATED_DELTA[case["width"]]
    heads, dim, tokens = s["heads"], s["dim"], x.shape[0]
    qk, group = s["kv_heads"] * dim, heads // s["kv_heads"]
    matrix = heads * dim * dim
    raw = torch.cat([x @ w[n].T for n in "qkv"], dim=1)
    filtered = torch.cat([state[matrix:].view(TAPS - 1, -1), raw])
    taps = torch.cat([w[n + ".conv"] for n in "qkv"])
    conv = sum(filtered[i:i + tokens] * taps[:, i] for i in range(TAPS))
    conv = conv * torch.sigmoid(conv)
    q, k, v = conv[:, :qk], conv[:, qk:2 * qk], conv[:, 2 * qk:]
    q, k = (t.view(tokens, -1, dim) for t in (q, k))
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = ((q * dim ** -0.5).repeat_interleave(group, 1), k.repeat_interleave(group, 1))
    v = v.view(tokens, heads, dim)
    write = torch.sigmoid(x @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))
    S = state[:matrix].view(heads, dim, dim).clone()
    out = torch.empty(tokens, heads, dim, dtype=F64, device="cuda")
    for t in range(tokens):
        S = decay[t][:, None, None] * S
        u = write[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    g = x @ w["g"].T
    gated = (_rms(out) * w["norm"]).flatten(1) * g * torch.sigmoid(g)
    return gated @ w["o"].T, torch.cat([S.flatten(), filtered[tokens:].flatten()])


def _exact_gla(case, w, x, state):
    s = GLA[case["width"]]
    heads, dim, tokens = s["heads"], s["dim"], x.shape[0]
    q, k, v = ((x @ w[n].T).view(tokens, heads, dim) for n in "qkv")
    g = x @ w["g"].T
    z = (x @ w["a1"].T) @ w["a2"].T + w["a2.b"]
    decay = torch.exp(torch.nn.functional.logsigmoid(z) / TAU).view(tokens, heads, dim)
    S = state.view(heads, dim, dim).clone()
    out = torch.empty(tokens, heads, dim, dtype=F64, device="cuda")
    for t in range(tokens):
        S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t] * dim ** -0.5)
    gated = (_rms(out) * w["norm"]).flatten(1) * g * torch.sigmoid(g)
    return gated @ w["o"].T, S.flatten()


def _exact_experts(case, w, x):
    s = EXPERTS[case["width"]]
    logits = x @ w["router"].T + w["router.b"]
    best, chosen = torch.topk(logits, s["top"], dim=1)
    share = torch.softmax(best, dim=1)
    out = torch.zeros_like(x)
    for e in range(s["experts"]):
        token, place = torch.nonzero(chosen == e, as_tuple=True)
        if len(token):
            gate = x[token] @ w[f"e{e}.gate"].T
            inner = gate * torch.sigmoid(gate) * (x[token] @ w[f"e{e}.up"].T)
            out[token] += share[token, place][:, None] * (inner @ w[f"e{e}.down"].T)
    return out
