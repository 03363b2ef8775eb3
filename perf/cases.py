"""The work that users of this package have it do, case by case: inputs, one pass through the public entry points, the bytes and
operations a pass cannot do without, and what the same pass gives in 64 bits.

Kinds of case, and what each stands for in real use:

``decode_step``   one token for every running request of a served model, replayed from the engine's CUDA graphs
``prompt_step``   the first step of new requests: whole prompts in, the logits behind their last tokens out
``attention``     one grouped-query attention layer over the paged cache: prompts and portions of prompts, or one token per request
``mlp``           one SwiGLU feed-forward for a batch of decoding requests, or for a portion of a prompt
``experts``       one routed feed-forward (14 experts and 2 identity experts, 4 per token from 2 of 4 groups)
``delta``         one gated delta rule layer over prompts
``parallel``      softmax attention beside linear attention with a decay per channel, over prompts
``state_space``   one selective state-space layer, over prompts (ragged, behind earlier tokens too) or one token per request
``float32``       both sublayers of a dense layer in the package's 32-bit mode (what numerics are checked with)

Layer sizes are those of the Qwen3 presets and of the benchmark's other designs at the same widths."""

import math
import zlib

import torch

from miniserve_b200.cache import CacheManager
from miniserve_b200.config import preset, resolve
from miniserve_b200.config.spec import LayerSpec, ModelSpec, PartSpec, RunEntry
from miniserve_b200.engine.engine import Engine
from miniserve_b200.engine.step import StepFunction, StepRow
from miniserve_b200.parts.decoder import DecoderModel

DEV = "cuda:0"
PAGE = 16
EPS = 1e-6
SIZES = {"0.6b": (1024, 3072), "1.7b": (2048, 6144), "8b": (4096, 12288)}  # width, feed-forward
HEADS, KV_HEADS, HEAD_DIM, THETA = 16, 8, 128, 1e6  # of the two smaller presets
EXPERTS, IDENTITY, TOP, GROUPS, KEEP, ROUTE_SCALE = 14, 2, 4, 4, 2, 2.0
TAU, TAPS, RANK, STATE, STATE_GROUPS = 16.0, 4, 64, 128, 8


def listed():
    return [
        # eight users reading their answers: the step whose time they wait for, again and again
        {"name": "decode_step_b8", "kind": "decode_step", "size": "0.6b", "contexts": "2048,1800,2300,2111,1933,2048,2205,1999"},
        # a prompt arrives at an idle server: time to first token
        {"name": "prompt_step_1999", "kind": "prompt_step", "size": "0.6b", "rows": "0:1999"},
        # a mixed step's prompts: two new ones and a portion behind a cached prefix
        {"name": "attention_prompts", "kind": "attention", "size": "1.7b", "rows": "0:1531,1024:517,4096:900"},
        # a full house: 64 requests, contexts of all lengths
        {"name": "attention_decode_b64", "kind": "attention", "size": "1.7b", "rows": ",".join("%d:1" % (1024 + 47 * i) for i in range(64))},
        # the feed-forward of a large dense model at a moderate batch
        {"name": "mlp_8b_rows24", "kind": "mlp", "size": "8b", "tokens": 24},
        # routed experts over a prompt of odd length
        {"name": "experts_prompt_1900", "kind": "experts", "size": "1.7b", "tokens": 1900},
        # routed experts when eight requests decode: most experts are touched by a row or two
        {"name": "experts_decode_b8", "kind": "experts", "size": "1.7b", "tokens": 8},
        # recurrent layers over a prompt
        {"name": "delta_prompt_2048", "kind": "delta", "size": "0.6b", "rows": "0:2048"},
        {"name": "parallel_prompt_2048", "kind": "parallel", "size": "0.6b", "rows": "0:2048"},
        # several prompts in one step, one of them in portions
        {"name": "state_space_prompts", "kind": "state_space", "size": "1.7b", "rows": "0:1037,2048:640,0:371"},
        # 32 requests decode through a state-space layer
        {"name": "state_space_decode_b32", "kind": "state_space", "size": "1.7b", "rows": ",".join("%d:1" % (100 + 31 * i) for i in range(32))},
        # the 32-bit mode, a prompt of 700 tokens
        {"name": "float32_layer_700", "kind": "float32", "size": "0.6b", "rows": "0:700"},
    ]


def draw(rng):
    """One more case of the same ranges; sizes spread over their logarithm."""

    def about(lo, hi):
        return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    def prompts(most, longest_prefix):
        rows, left = [], about(64, most)
        while left > 0 and len(rows) < 4:
            n = left if len(rows) == 3 or rng.random() < 0.4 else min(left, max(17, int(left * rng.uniform(0.2, 0.8))))
            rows.append("%d:%d" % (rng.choice([0, 0, about(1, longest_prefix)]) if longest_prefix else 0, n))
            left -= n
        return ",".join(rows)

    kind = rng.choice(["decode_step", "prompt_step", "attention", "attention", "mlp", "experts", "experts", "delta", "parallel", "state_space",
                       "state_space", "float32"])
    size = rng.choice(["0.6b", "1.7b"])
    if kind == "decode_step":
        n = about(1, 32)
        top = about(64, min(3000, 16400 // n))
        return {"kind": kind, "size": "0.6b", "contexts": ",".join(str(rng.randint(max(1, top // 2), top)) for _ in range(n))}
    if kind == "prompt_step":
        return {"kind": kind, "size": "0.6b", "rows": prompts(1999, 0)}
    if kind == "attention":
        if rng.random() < 0.5:
            return {"kind": kind, "size": size, "rows": prompts(2900, 4096)}
        n = about(1, 64)
        top = about(64, min(4000, 160000 // n))
        return {"kind": kind, "size": size, "rows": ",".join("%d:1" % rng.randint(max(1, top // 3), top) for _ in range(n))}
    if kind == "mlp":
        return {"kind": kind, "size": rng.choice(["0.6b", "1.7b", "8b"]), "tokens": about(1, 1500)}
    if kind == "experts":
        return {"kind": kind, "size": size, "tokens": about(1, 2048)}
    if kind == "state_space" and rng.random() < 0.4:
        return {"kind": kind, "size": size, "rows": ",".join("%d:1" % rng.randint(1, 4000) for _ in range(about(1, 32)))}
    if kind == "float32":
        return {"kind": kind, "size": "0.6b", "rows": prompts(700, 0)}
    return {"kind": kind, "size": size, "rows": prompts(2048, 2048 if kind == "state_space" else 0)}


# ------------------------------------------------------------------------------------------------ what a case is made of

def rows_of(case):
    """(tokens already cached, new tokens) of every request of the case's step."""
    if "contexts" in case:
        return [(int(c), 1) for c in case["contexts"].split(",")]
    if "rows" in case:
        return [tuple(int(n) for n in r.split(":")) for r in case["rows"].split(",")]
    return [(0, case["tokens"])]


def made(seed, name, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    """Normal numbers that follow from the seed and the name alone."""
    gen = torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 60))
    t = torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32)
    return (t * std + mean).to(dtype)


def spread(seed, name, *shape, lo, hi):
    """Numbers whose logarithms are uniform, float32."""
    gen = torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 60))
    return torch.exp(torch.rand(shape, generator=gen, device=DEV) * (math.log(hi) - math.log(lo)) + math.log(lo))


def inverse_softplus(y):
    return y + torch.log(-torch.expm1(-y))


def attention_weights(seed, pre, width, heads, kv_heads, dtype=torch.bfloat16):
    d, std = HEAD_DIM, width ** -0.5
    return {pre + "q_proj.weight": made(seed, pre + "q", heads * d, width, std=std, dtype=dtype),
            pre + "k_proj.weight": made(seed, pre + "k", kv_heads * d, width, std=std, dtype=dtype),
            pre + "v_proj.weight": made(seed, pre + "v", kv_heads * d, width, std=std, dtype=dtype),
            pre + "o_proj.weight": made(seed, pre + "o", width, heads * d, std=(heads * d) ** -0.5, dtype=dtype),
            # (queries and keys of a trained model attend: scores a few units apart)
            pre + "q_norm.weight": made(seed, pre + "qn", d, std=0.1, mean=1.5, dtype=dtype),
            pre + "k_norm.weight": made(seed, pre + "kn", d, std=0.1, mean=1.5, dtype=dtype)}


def mlp_weights(seed, pre, width, ff, dtype=torch.bfloat16):
    return {pre + "gate_proj.weight": made(seed, pre + "gate", ff, width, std=width ** -0.5, dtype=dtype),
            pre + "up_proj.weight": made(seed, pre + "up", ff, width, std=width ** -0.5, dtype=dtype),
            pre + "down_proj.weight": made(seed, pre + "down", width, ff, std=ff ** -0.5, dtype=dtype)}


def expert_weights(seed, pre, width, ff):
    w = {pre + "router.weight": made(seed, pre + "router", EXPERTS + IDENTITY, width, std=2 * width ** -0.5, dtype=torch.float32),
         pre + "router.correction": made(seed, pre + "correction", EXPERTS + IDENTITY, std=0.02, dtype=torch.float32)}
    for e in range(EXPERTS):
        w.update(mlp_weights(seed, "%sexperts.%d." % (pre, e), width, ff // 4))
    return w


def delta_sizes(width):
    return width // 64, width // 128, 64, 64  # heads, query/key heads, key and value channels of a head


def delta_weights(seed, pre, width):
    h, g, dk, dv = delta_sizes(width)
    s, f32 = width ** -0.5, torch.float32
    m = lambda name, *shape, **k: made(seed, pre + name, *shape, **k)  # noqa: E731
    return {pre + "q_proj.weight": m("q", g * dk, width, std=s), pre + "k_proj.weight": m("k", g * dk, width, std=s),
            pre + "v_proj.weight": m("v", h * dv, width, std=s), pre + "b_proj.weight": m("b", h, width, std=s),
            pre + "q_conv.weight": m("qc", g * dk, TAPS, std=0.5, dtype=f32), pre + "k_conv.weight": m("kc", g * dk, TAPS, std=0.5, dtype=f32),
            pre + "v_conv.weight": m("vc", h * dv, TAPS, std=0.5, dtype=f32),
            pre + "A_log": torch.log(spread(seed, pre + "A", h, lo=1.0, hi=16.0)),
            pre + "dt_bias": inverse_softplus(spread(seed, pre + "dt", h * dk, lo=1e-3, hi=1e-1)),
            pre + "o_norm.weight": m("norm", dv, std=0.1, mean=1.0, dtype=f32),
            pre + "a_proj.0.weight": m("a1", RANK, width, std=s), pre + "a_proj.1.weight": m("a2", h * dk, RANK, std=RANK ** -0.5),
            pre + "g_proj.0.weight": m("g1", RANK, width, std=s), pre + "g_proj.1.weight": m("g2", h * dv, RANK, std=RANK ** -0.5),
            pre + "o_proj.weight": m("o", width, h * dv, std=(h * dv) ** -0.5)}


def linear_sizes(width):
    return width // 128, 64, 128  # heads, key and value channels of a head


def parallel_weights(seed, pre, width):
    h, dk, dv = linear_sizes(width)
    s, f32 = width ** -0.5, torch.float32
    left = attention_weights(seed, pre + "left.", width, HEADS, KV_HEADS)
    for n in ("q_norm.weight", "k_norm.weight"):  # (the general attention path keeps these in 32 bits)
        left[pre + "left." + n] = left[pre + "left." + n].float()
    m = lambda name, *shape, **k: made(seed, pre + "right." + name, *shape, **k)  # noqa: E731
    right = {"q_proj.weight": m("q", h * dk, width, std=s), "k_proj.weight": m("k", h * dk, width, std=s), "v_proj.weight": m("v", h * dv, width, std=s),
             "g_proj.weight": m("g", h * dv, width, std=s), "o_proj.weight": m("o", width, h * dv, std=(h * dv) ** -0.5),
             "o_norm.weight": m("norm", dv, std=0.1, mean=1.0, dtype=f32), "a_proj.0.weight": m("a1", RANK, width, std=s),
             "a_proj.1.weight": m("a2", h * dk, RANK, std=RANK ** -0.5), "a_proj.1.bias": m("ab", h * dk, std=1.0, mean=1.0, dtype=f32)}
    return {**left, pre + "left.g_proj.weight": made(seed, pre + "left.g", HEADS, width, std=s), **{pre + "right." + n: t for n, t in right.items()}}


def state_space_sizes(width):
    return 2 * width // 64, 64  # heads, channels of a head


def state_space_weights(seed, pre, width):
    h, dv = state_space_sizes(width)
    inner, f32 = h * dv, torch.float32
    channels = inner + 2 * STATE_GROUPS * STATE
    m = lambda name, *shape, **k: made(seed, pre + name, *shape, **k)  # noqa: E731
    return {pre + "in_proj.weight": m("in", inner + channels + h, width, std=width ** -0.5),
            pre + "conv1d.weight": m("conv", channels, TAPS, std=0.5, dtype=f32), pre + "conv1d.bias": m("convb", channels, std=0.1, dtype=f32),
            pre + "dt_bias": inverse_softplus(spread(seed, pre + "dt", h, lo=1e-3, hi=1e-1)),
            pre + "A_log": torch.log(spread(seed, pre + "A", h, lo=1.0, hi=16.0)),
            pre + "D": m("D", h, std=0.1, mean=1.0, dtype=f32), pre + "norm.weight": m("norm", inner, std=0.1, mean=1.0, dtype=f32),
            pre + "out_proj.weight": m("o", width, inner, std=inner ** -0.5)}


def attention_spec(width, **more):
    return PartSpec("gqa_attention", dict(hidden=width, heads=HEADS, kv_heads=KV_HEADS, head_dim=HEAD_DIM, qk_norm=True, qk_norm_eps=EPS,
                                          position=PartSpec("rope_neox", dict(head_dim=HEAD_DIM, theta=THETA)), **more))


def layer_of(case):
    """(mixer, feed-forward) of the one layer that a case runs."""
    width, ff = SIZES[case["size"]]
    kind = case["kind"]
    swiglu = PartSpec("swiglu", dict(hidden=width, intermediate=ff))
    if kind in ("attention", "mlp", "float32"):
        return attention_spec(width), swiglu
    if kind == "experts":
        return attention_spec(width), PartSpec("routed_experts", dict(
            hidden=width, intermediate=ff // 4, experts=EXPERTS, identity=IDENTITY, top=TOP, group_count=GROUPS, group_keep=KEEP,
            weight_scale=ROUTE_SCALE))
    if kind == "delta":
        h, g, dk, dv = delta_sizes(width)
        return PartSpec("gated_delta_rule", dict(hidden=width, heads=h, kv_heads=g, key_dim=dk, value_dim=dv, conv=TAPS, decay_rank=RANK,
                                                 gate_rank=RANK, eps=EPS)), None
    if kind == "parallel":
        h, dk, dv = linear_sizes(width)
        left = attention_spec(width, value_dim=HEAD_DIM, sink=True, out_gate="head_sigmoid")
        left = PartSpec("gqa_attention", {**left.params, "position": PartSpec("rope_pairs", dict(head_dim=HEAD_DIM, theta=THETA, rotary_dim=64))})
        right = PartSpec("decay_linear_attention", dict(hidden=width, heads=h, key_dim=dk, value_dim=dv, tau=TAU, decay_rank=RANK, eps=EPS))
        return PartSpec("parallel", dict(branches=(("left.", left, 1.0), ("right.", right, 0.5)))), None
    h, dv = state_space_sizes(width)
    return PartSpec("mamba2", dict(hidden=width, heads=h, head_dim=dv, state=STATE, groups=STATE_GROUPS, conv=TAPS, norm_groups=8, eps=EPS)), None


def layer_weights(case, seed):
    """Tensors of the layer's sublayers, by the names that a checkpoint of such a layer has."""
    width, ff = SIZES[case["size"]]
    kind = case["kind"]
    if kind == "attention":
        return attention_weights(seed, "mix.", width, HEADS, KV_HEADS)
    if kind == "mlp":
        return mlp_weights(seed, "mlp.", width, ff)
    if kind == "experts":
        return expert_weights(seed, "mlp.", width, ff)
    if kind == "delta":
        return delta_weights(seed, "mix.", width)
    if kind == "parallel":
        return parallel_weights(seed, "mix.", width)
    if kind == "state_space":
        return state_space_weights(seed, "mix.", width)
    return {**attention_weights(seed, "mix.", width, HEADS, KV_HEADS, torch.float32), **mlp_weights(seed, "mlp.", width, ff, torch.float32)}


def model_weights(seed, raw):
    """Tensors of a whole Qwen3 model by name (made layer by layer by ``model_layer_weights``)."""
    w = {"model.embed_tokens.weight": made(seed, "embed", raw["vocab_size"], raw["hidden_size"]),
         "model.norm.weight": made(seed, "norm", raw["hidden_size"], std=0.1, mean=1.0)}
    for i in range(raw["num_hidden_layers"]):
        w.update(model_layer_weights(seed, raw, i))
    return w


def model_layer_weights(seed, raw, i):
    pre, width = "model.layers.%d." % i, raw["hidden_size"]
    w = {pre + n + ".weight": made(seed, pre + n, width, std=0.1, mean=1.0) for n in ("input_layernorm", "post_attention_layernorm")}
    w.update(attention_weights(seed, pre + "self_attn.", width, HEADS, KV_HEADS))
    w.update(mlp_weights(seed, pre + "mlp.", width, raw["intermediate_size"]))
    for n in ("self_attn.o_proj.weight", "mlp.down_proj.weight"):  # a sublayer adds a fraction of the stream, as in a trained model
        w[pre + n] *= 0.25
    return w


def cached(seed, layer, row, tokens, dtype=torch.bfloat16):
    """Keys and values [tokens, kv heads, head size] that a request's earlier tokens left."""
    name = "cached.%d.%d." % (layer, row)
    return (made(seed, name + "k", tokens, KV_HEADS, HEAD_DIM, std=1.5, dtype=dtype), made(seed, name + "v", tokens, KV_HEADS, HEAD_DIM, dtype=dtype))


def put_cached(seed, layer, requests, rows, view):
    """Earlier tokens' keys and values into the pages that the requests hold."""
    for r, (rc, (start, _)) in enumerate(zip(requests, rows)):
        if start == 0:
            continue
        blocks = torch.tensor(rc.tables[view.group].blocks, device=DEV)[:-(-start // PAGE)]
        for pool, dense in zip((view.k, view.v), cached(seed, layer, r, start, view.k.dtype)):
            padded = torch.zeros((len(blocks) * PAGE, KV_HEADS, HEAD_DIM), dtype=dense.dtype, device=DEV)
            padded[:start] = dense
            pool[blocks] = padded.view(-1, PAGE, KV_HEADS, HEAD_DIM).transpose(1, 2)


# ------------------------------------------------------------------------------------------------ a pass

def prepare(case, seed):
    return _prepare_model(case, seed) if case["kind"] in ("decode_step", "prompt_step") else _prepare_layer(case, seed)


def _tokens(seed, rows, vocab):
    gen = torch.Generator().manual_seed(int(seed))
    return [torch.randint(0, vocab, (n,), generator=gen).tolist() for _, n in rows]


def _prepare_model(case, seed):
    rows, raw = rows_of(case), preset(case["size"])
    _, _, spec = resolve(raw)
    model = DecoderModel(spec, torch.bfloat16, DEV)
    model.bind(model_weights(seed, raw))
    pages = sum(-(-(s + n + PAGE) // PAGE) for s, n in rows) + 160
    engine = Engine(model, kv_pool_tokens=pages * PAGE, page_size=PAGE, max_running=max(len(rows), 8))
    requests = [engine.cache.new_request() for _ in rows]
    before = [(rc, s) for rc, (s, _) in zip(requests, rows) if s]
    if before:
        engine.cache.reserve(before)
        for layer, view in enumerate(engine.cache.entry_views):
            put_cached(seed, layer, requests, rows, view)
    step = [StepRow(rc, ids, (len(ids) - 1,)) for rc, ids in zip(requests, _tokens(seed, rows, raw["vocab_size"]))]
    return {"kind": case["kind"], "engine": engine, "rows": step}


def _prepare_layer(case, seed):
    rows, (width, _) = rows_of(case), SIZES[case["size"]]
    dtype = torch.float32 if case["kind"] == "float32" else torch.bfloat16
    mixer, ffn = layer_of(case)
    norm = PartSpec("rmsnorm", dict(size=width, eps=EPS))
    names = dict(mixer="mix.", norm1="norm1.", **(dict(feed_forward="mlp.", norm2="norm2.") if ffn else {}))
    norms = dict(norm1=norm, **(dict(norm2=norm) if ffn else {}))
    spec = ModelSpec(architecture="layer", hidden_size=width, vocab_size=64, embedding=PartSpec("token_embedding", dict(vocab=64, hidden=width, name="embed")),
                     layers=(LayerSpec("", PartSpec("prenorm", dict(names=names)), mixer, ffn, norms),), run_order=(RunEntry(0),), final_norm=norm,
                     final_norm_prefix="norm.", head=PartSpec("linear_head", dict(vocab=64, hidden=width, tied=True, name="head", tied_to="embed")))
    model = DecoderModel(spec, dtype, DEV)
    block = model.layers[0]
    w = layer_weights(case, seed)
    parts = {"mix.": block.mixer} if any(n.startswith("mix.") for n in w) else {}
    if any(n.startswith("mlp.") for n in w):
        parts["mlp."] = block.feed_forward
    for pre, part in parts.items():
        part.bind_all(w, pre)
    pages = sum(-(-(s + n) // PAGE) for s, n in rows) + 2
    cache = CacheManager(model.entry_caches, pages, PAGE, len(rows), dtype=dtype, device=DEV)
    requests = [cache.new_request() for _ in rows]
    before = [(rc, s) for rc, (s, _) in zip(requests, rows) if s]
    if before:
        cache.reserve(before)
    step = StepFunction(model, cache)
    ctx = step.prepare([StepRow(rc, [1] * n) for rc, (_, n) in zip(requests, rows)])
    view = cache.entry_views[0]
    state = {"kind": case["kind"], "step": step, "ctx": ctx, "view": view, "parts": parts, "x": made(seed, "x", sum(n for _, n in rows), width, dtype=dtype)}
    if case["kind"] in ("attention", "parallel", "float32"):
        paged = view[0] if case["kind"] == "parallel" else view
        paged.k.zero_()
        paged.v.zero_()
        put_cached(seed, 0, requests, rows, paged)
    if case["kind"] == "state_space":
        for t, (shape, std) in zip(view, _state_before(case)):
            t.state.zero_()
            for r, (rc, (start, _)) in enumerate(zip(requests, rows)):
                if start:
                    t.state[rc.state_slot] = made(seed, "state.%d.%d" % (r, len(shape)), *shape, std=std, dtype=t.state.dtype)
        # the requests' state before the step: a pass starts from it
        state["before"] = [(t.state, t.state.clone()) for t in view] if before else []
    return state


def _state_before(case):
    width, _ = SIZES[case["size"]]
    h, dv = state_space_sizes(width)
    return ((h, dv, STATE), 0.1), ((TAPS - 1, h * dv + 2 * STATE_GROUPS * STATE), 1.0)


def run(state):
    kind = state["kind"]
    if kind in ("decode_step", "prompt_step"):
        engine, rows = state["engine"], state["rows"]
        if kind == "decode_step":
            engine.graphs.run(rows, None)  # (the sampled tokens are an argmax of these logits, which ties decide)
            out = {"logits": next(iter(engine.graphs._graphs.values())).logits[:len(rows)]}
        else:
            out = {"logits": engine.step_fn.run(rows)}
        for row in rows:  # the requests stay where they were, for another pass
            for table in row.cache.tables:
                table.rewind(len(row.tokens))
        return out
    ctx, parts, x, view = state["ctx"], state["parts"], state["x"], state["view"]
    for held, before in state.get("before", ()):
        held.copy_(before)
    ctx.step_cache.clear()  # as the model does when a pass begins
    ctx.buffers.clear()
    out = {}
    if "mix." in parts:
        out["out"] = parts["mix."].forward(x, ctx, view)
        if kind in ("attention", "float32"):
            out["k"], out["v"] = view.k, view.v
        elif kind == "parallel":
            out["k"], out["v"], out["state"] = view[0].k, view[0].v, view[1].state
        else:
            out["state"], out["inputs"] = view[0].state, view[1].state
    if "mlp." in parts:
        out["mlp"] = parts["mlp."].forward(x, ctx)
    return out


# ------------------------------------------------------------------------------------------------ what a pass cannot do without

def work(case):
    rows, (width, ff) = rows_of(case), SIZES[case["size"]]
    t, kind = sum(n for _, n in rows), case["kind"]
    item = 4 if kind == "float32" else 2
    pairs = sum(n * s + n * (n + 1) / 2 for s, n in rows)
    held = sum(s for s, _ in rows)
    q, kv = HEADS * HEAD_DIM, KV_HEADS * HEAD_DIM
    att_w, mlp_w = width * (2 * q + 2 * kv), 3 * width * ff
    att_bytes, att_flops = (att_w + 2 * (held + t) * kv) * item, 2.0 * t * att_w + 4.0 * pairs * q
    mlp_bytes, mlp_flops = mlp_w * item, 2.0 * t * mlp_w
    io = 2 * t * width * item
    if kind == "attention":
        return {"bytes": att_bytes + io, "flops": att_flops}
    if kind == "mlp":
        return {"bytes": mlp_bytes + io, "flops": mlp_flops}
    if kind == "float32":
        return {"bytes": att_bytes + mlp_bytes + 3 * t * width * item, "flops": att_flops + mlp_flops}
    if kind in ("decode_step", "prompt_step"):
        layers, vocab = preset(case["size"])["num_hidden_layers"], preset(case["size"])["vocab_size"]
        return {"bytes": layers * (att_bytes + mlp_bytes) + vocab * width * 2 + len(rows) * vocab * 4,
                "flops": layers * (att_flops + mlp_flops) + 2.0 * len(rows) * vocab * width}
    if kind == "experts":
        used = min(EXPERTS, t * TOP)
        real = TOP * EXPERTS / (EXPERTS + IDENTITY)
        return {"bytes": used * 3 * width * (ff // 4) * 2 + io + (EXPERTS + IDENTITY) * width * 4, "flops": 2.0 * t * real * 3 * width * (ff // 4)}
    if kind == "delta":
        h, g, dk, dv = delta_sizes(width)
        weights = width * (2 * g * dk + h * dv + h + 2 * RANK) + RANK * (h * dk + h * dv) + width * h * dv
        return {"bytes": weights * 2 + io + len(rows) * h * dk * dv * 4, "flops": 2.0 * t * weights + 7.0 * t * h * dk * dv}
    if kind == "parallel":
        h, dk, dv = linear_sizes(width)
        weights = att_w + width * HEADS + width * (2 * h * dk + 3 * h * dv + RANK) + RANK * h * dk
        return {"bytes": (weights + 2 * (held + t) * kv) * 2 + io + len(rows) * h * dk * dv * 4,
                "flops": 2.0 * t * weights + 4.0 * pairs * q + 5.0 * t * h * dk * dv}
    h, dv = state_space_sizes(width)
    inner = h * dv
    weights = width * (3 * inner + 2 * STATE_GROUPS * STATE + h)
    behind = sum(1 for s, _ in rows if s)
    return {"bytes": weights * 2 + io + (len(rows) + behind) * (inner * STATE * 4 + (TAPS - 1) * (inner + 2 * STATE_GROUPS * STATE) * 2),
            "flops": 2.0 * t * weights + 5.0 * t * inner * STATE}


def tolerance(case):
    """Largest relative errors of another correct implementation at the same precision: about four times what the package's results
    were measured to differ from 64 bits by (bfloat16 between products: 0.0022 to 0.0037 for the feed-forwards and the recurrent layers,
    0.0046 to 0.0061 behind softmax attention, 0.0039 to 0.0049 behind 28 layers; 32 bits: 1.3e-6 to 4.2e-6)."""
    return {"rel": {"float32": 1.7e-5, "attention": 2.4e-2, "parallel": 1.8e-2, "decode_step": 2e-2, "prompt_step": 2e-2, "mlp": 1.5e-2,
                    "experts": 1e-2, "delta": 1.4e-2, "state_space": 1.4e-2}[case["kind"]]}


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def _rms(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _angles(positions, dims):
    i = torch.arange(0, dims, 2, dtype=torch.float64, device=DEV)
    a = positions.double()[:, None] * (THETA ** (-i / dims)).float().double()[None, :]
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _attend(q, k, v, start, sink=False):
    """q [n, heads, d] at positions start.. over k, v [start + n, kv heads, d]; a sink is one more term of score 0."""
    n, heads, d = q.shape
    g = heads // k.shape[1]
    out = torch.empty_like(q)
    for h in range(heads):
        for a in range(0, n, 1024):
            b = min(n, a + 1024)
            s = (q[a:b, h] @ k[:, h // g].T) * d ** -0.5
            at = torch.arange(start + a, start + b, device=DEV)[:, None]
            s = s.masked_fill(torch.arange(k.shape[0], device=DEV)[None, :] > at, -math.inf)
            if sink:
                s = torch.cat((s, torch.zeros((b - a, 1), dtype=s.dtype, device=DEV)), dim=1)
            out[a:b, h] = torch.softmax(s, dim=1)[:, :k.shape[0]] @ v[:, h // g]
    return out


def _heads(x, w, n):
    return (x @ w.double().T).view(x.shape[0], n, -1)


def _attention(x, w, pre, rows, earlier, adjacent=0, sink=False):
    """Before the output product: [T, heads, d]. ``adjacent``: so many channels turn in adjacent pairs, else the whole head by halves."""
    outs, base = [], 0
    for r, (start, n) in enumerate(rows):
        xr = x[base:base + n]
        base += n
        q = _rms(_heads(xr, w[pre + "q_proj.weight"], HEADS)) * w[pre + "q_norm.weight"].double()
        k = _rms(_heads(xr, w[pre + "k_proj.weight"], KV_HEADS)) * w[pre + "k_norm.weight"].double()
        v = _heads(xr, w[pre + "v_proj.weight"], KV_HEADS)
        c, s = _angles(torch.arange(start, start + n, device=DEV), adjacent or HEAD_DIM)
        turned = []
        for y in (q, k):
            y = y.clone()
            one, two = (slice(0, adjacent, 2), slice(1, adjacent, 2)) if adjacent else (slice(0, HEAD_DIM // 2), slice(HEAD_DIM // 2, HEAD_DIM))
            a, b = y[..., one].clone(), y[..., two].clone()
            y[..., one], y[..., two] = a * c - b * s, b * c + a * s
            turned.append(y)
        q, k = turned
        if start:
            ek, ev = earlier(r, start)
            k, v = torch.cat((ek.double(), k)), torch.cat((ev.double(), v))
        outs.append(_attend(q, k, v, start, sink))
    return torch.cat(outs)


def _swiglu(x, w, pre):
    return (_silu(x @ w[pre + "gate_proj.weight"].double().T) * (x @ w[pre + "up_proj.weight"].double().T)) @ w[pre + "down_proj.weight"].double().T


def _experts(x, w, pre):
    s = torch.softmax(x @ w[pre + "router.weight"].double().T, dim=-1)
    choice = s + w[pre + "router.correction"].double()
    per = (EXPERTS + IDENTITY) // GROUPS
    best = choice.view(-1, GROUPS, per).max(-1).values
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, torch.topk(best, KEEP, dim=-1).indices, True)
    choice = choice.masked_fill(~kept.repeat_interleave(per, dim=1), -math.inf)
    chosen = torch.topk(choice, TOP, dim=-1).indices
    weight = torch.zeros_like(s).scatter_(1, chosen, torch.gather(s, 1, chosen) * ROUTE_SCALE)
    out = x * weight[:, EXPERTS:].sum(1, keepdim=True)
    for e in range(EXPERTS):
        rows = torch.nonzero(weight[:, e]).flatten()
        if rows.numel():
            out[rows] += weight[rows, e, None] * _swiglu(x[rows], w, "%sexperts.%d." % (pre, e))
    return out


def _conv(x, w, before=None):
    """A causal convolution over time per channel; ``before``: the inputs ahead of the first one (zeros if None)."""
    taps = w.shape[1]
    ahead = torch.zeros((taps - 1, x.shape[1]), dtype=x.dtype, device=DEV) if before is None else before.double()
    full = torch.cat((ahead, x))
    return sum(full[j:j + x.shape[0]] * w.double()[:, j] for j in range(taps)), full[-(taps - 1):]


def _scan(q, k, v, decay, beta=None, state=None):
    """Token by token over [T, heads, channels]; with ``beta`` the delta rule. Returns (outputs, the state [heads, dk, dv])."""
    S = torch.zeros((q.shape[1], q.shape[2], v.shape[2]), dtype=q.dtype, device=DEV) if state is None else state.clone()
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=q.dtype, device=DEV)
    for t in range(q.shape[0]):
        S *= decay[t][:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.matmul(k[t][:, None, :], S)[:, 0])
        S += k[t][:, :, None] * u[:, None, :]
        out[t] = torch.matmul(q[t][:, None, :], S)[:, 0]
    return out, S


def _delta(x, w, pre, width):
    h, g, dk, dv = delta_sizes(width)
    t = x.shape[0]
    raw = torch.cat([x @ w[pre + n + "_proj.weight"].double().T for n in "qkv"], dim=1)
    y, last = _conv(raw, torch.cat([w[pre + n + "_conv.weight"] for n in "qkv"]))
    y = _silu(y)
    q, k, v = y[:, :g * dk].view(t, g, dk), y[:, g * dk:2 * g * dk].view(t, g, dk), y[:, 2 * g * dk:].view(t, h, dv)
    q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
    q, k = (z.repeat_interleave(h // g, dim=1) for z in (q * dk ** -0.5, k))
    z = (x @ w[pre + "a_proj.0.weight"].double().T) @ w[pre + "a_proj.1.weight"].double().T + w[pre + "dt_bias"].double()
    decay = torch.exp(-torch.exp(w[pre + "A_log"].double())[None, :, None] * torch.nn.functional.softplus(z, threshold=1e9).view(t, h, dk))
    o, S = _scan(q, k, v, decay, torch.sigmoid(x @ w[pre + "b_proj.weight"].double().T))
    gate = torch.sigmoid((x @ w[pre + "g_proj.0.weight"].double().T) @ w[pre + "g_proj.1.weight"].double().T).view(t, h, dv)
    o = _rms(o) * w[pre + "o_norm.weight"].double() * gate
    return o.reshape(t, h * dv) @ w[pre + "o_proj.weight"].double().T, S.transpose(1, 2), last


def _linear(x, w, pre, width):
    h, dk, dv = linear_sizes(width)
    t = x.shape[0]
    q, k, v = (_heads(x, w[pre + n + "_proj.weight"], h) for n in "qkv")
    z = (x @ w[pre + "a_proj.0.weight"].double().T) @ w[pre + "a_proj.1.weight"].double().T + w[pre + "a_proj.1.bias"].double()
    o, S = _scan(q * dk ** -0.5, k, v, (torch.sigmoid(z) ** (1 / TAU)).view(t, h, dk))
    o = (_rms(o) * w[pre + "o_norm.weight"].double()).reshape(t, h * dv) * _silu(x @ w[pre + "g_proj.weight"].double().T)
    return o @ w[pre + "o_proj.weight"].double().T, S.transpose(1, 2)


def _state_space(x, w, pre, width, state, before):
    h, dv = state_space_sizes(width)
    t, inner, gn = x.shape[0], h * dv, STATE_GROUPS * STATE
    proj = x @ w[pre + "in_proj.weight"].double().T
    y, last = _conv(proj[:, inner:2 * inner + 2 * gn], w[pre + "conv1d.weight"], before)
    y = _silu(y + w[pre + "conv1d.bias"].double())
    xs = y[:, :inner].view(t, h, dv)
    b, c = (z.reshape(t, STATE_GROUPS, STATE).repeat_interleave(h // STATE_GROUPS, dim=1) for z in (y[:, inner:inner + gn], y[:, inner + gn:]))
    dt = torch.nn.functional.softplus(proj[:, 2 * inner + 2 * gn:] + w[pre + "dt_bias"].double(), threshold=1e9)
    decay = torch.exp(-torch.exp(w[pre + "A_log"].double()) * dt)[:, :, None].expand(t, h, STATE)
    o, S = _scan(c, b, xs * dt[:, :, None], decay, state=state)
    o = (o + w[pre + "D"].double()[None, :, None] * xs).reshape(t, inner) * _silu(proj[:, :inner])
    o = _rms(o.view(t, 8, -1)).reshape(t, inner) * w[pre + "norm.weight"].double()
    return o @ w[pre + "out_proj.weight"].double().T, S.transpose(1, 2), last


def exact(case, seed):
    kind, rows = case["kind"], rows_of(case)
    width, _ = SIZES[case["size"]]
    if kind in ("decode_step", "prompt_step"):
        return _exact_model(case, seed, rows)
    w = layer_weights(case, seed)
    x = made(seed, "x", sum(n for _, n in rows), width, dtype=torch.float32 if kind == "float32" else torch.bfloat16).double()
    starts = [sum(n for _, n in rows[:i]) for i in range(len(rows))]
    pieces = [x[a:a + n] for a, (_, n) in zip(starts, rows)]
    out = {}
    if kind in ("attention", "float32"):
        o = _attention(x, w, "mix.", rows, lambda r, n: cached(seed, 0, r, n, torch.bfloat16))
        out.update(out=o.reshape(x.shape[0], -1) @ w["mix.o_proj.weight"].double().T, k=None, v=None)
    if kind in ("mlp", "float32"):
        out["mlp"] = _swiglu(x, w, "mlp.")
    if kind == "experts":
        out["mlp"] = _experts(x, w, "mlp.")
    if kind == "delta":
        got = [_delta(p, w, "mix.", width) for p in pieces]
        out.update(out=torch.cat([o for o, _, _ in got]), state=_slots([s for _, s, _ in got]), inputs=_slots([c for _, _, c in got]))
    if kind == "parallel":
        o = _attention(x, w, "mix.left.", rows, None, adjacent=64, sink=True)
        o = o * torch.sigmoid(x @ w["mix.left.g_proj.weight"].double().T)[:, :, None]
        left = o.reshape(x.shape[0], -1) @ w["mix.left.o_proj.weight"].double().T
        got = [_linear(p, w, "mix.right.", width) for p in pieces]
        out.update(out=left + 0.5 * torch.cat([o for o, _ in got]), k=None, v=None, state=_slots([s for _, s in got]))
    if kind == "state_space":
        (shape, std), (taps, _) = _state_before(case)
        got = []
        for r, (p, (start, _)) in enumerate(zip(pieces, rows)):
            state = made(seed, "state.%d.%d" % (r, len(shape)), *shape, std=std, dtype=torch.float32).double().transpose(1, 2) if start else None
            before = made(seed, "state.%d.%d" % (r, len(taps)), *taps) if start else None
            got.append(_state_space(p, w, "mix.", width, state, before))
        out.update(out=torch.cat([o for o, _, _ in got]), state=_slots([s for _, s, _ in got]), inputs=_slots([c for _, _, c in got]))
    return out


def _slots(states):
    """Per-request states as the cache keeps them: request r has slot r, one more slot stays zero."""
    return torch.stack([*states, torch.zeros_like(states[0])])


def _exact_model(case, seed, rows):
    raw = preset(case["size"])
    ids = torch.tensor([i for row in _tokens(seed, rows, raw["vocab_size"]) for i in row], device=DEV)
    embed = made(seed, "embed", raw["vocab_size"], raw["hidden_size"]).double()
    h = embed[ids]
    for i in range(raw["num_hidden_layers"]):
        pre, w = "model.layers.%d." % i, model_layer_weights(seed, raw, i)
        x = _rms(h) * w[pre + "input_layernorm.weight"].double()
        o = _attention(x, w, pre + "self_attn.", rows, lambda r, n, i=i: cached(seed, i, r, n))
        h = h + o.reshape(x.shape[0], -1) @ w[pre + "self_attn.o_proj.weight"].double().T
        h = h + _swiglu(_rms(h) * w[pre + "post_attention_layernorm.weight"].double(), w, pre + "mlp.")
    last = torch.tensor([sum(n for _, n in rows[:i + 1]) - 1 for i in range(len(rows))], device=DEV)
    logits = (_rms(h[last]) * made(seed, "norm", raw["hidden_size"], std=0.1, mean=1.0).double()) @ embed.T
    return {"logits": logits}
