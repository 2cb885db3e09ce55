"""The calls that a diffusion pipeline makes of this framework, as cases that can be timed.

Each case is one pass through the public entry points as a user's program makes it: an attention
call on q, k and v that are in hand, a linear layer, or a whole attention layer of the diffusion
transformer (qkv projection, per-head norm and RoPE with the attention's per-block work, attention).
Sizes are the repository's own (its benchmark, its configurations and its tests' shapes) or generic.
Everything random is drawn on the GPU from the seed.
"""

import math

import torch

from mmh3_b200 import attention, gemm, synthetic
from mmh3_b200.vsa import PackedLayout, VsaPlan

HEAD_DIM = 128
EPSILON = 1e-6
SOL_TAU = 1.3


def listed():
    return [
        # The text encoder reads one prompt: causal, four query heads to a key/value head. The
        # smallest call of the pipeline.
        dict(name="prompt_causal_300", kind="text", tokens=300, heads=32, group=4, batch=1),
        # The VAE decoder attends inside a batch of windows, FP16 heads of 64, with the query's
        # norm and RoPE inside the call.
        dict(name="vae_windows_8x1025", kind="vae", tokens=1025, heads=16, batch=8, pairs=32),
        # The CPU-sized workload of the configurations: a small image's attention by itself.
        dict(name="dense_bf16_4096_h8", kind="dense", tokens=4096, heads=8, precision="bf16"),
        # The headline workload: a 256 x 256 token image and 512 text tokens.
        dict(name="dense_bf16_66048_h32", kind="dense", tokens=66048, heads=32,
             precision="bf16"),
        # A 45 x 45 token image and 60 text tokens in INT8/FP8, quantized by the call itself.
        dict(name="dense_int8_2085_h56", kind="dense", tokens=2085, heads=56,
             precision="int8-fp8"),
        # A whole attention layer of a preview image (32 x 32 tokens and 77 of text) in BF16.
        dict(name="layer_bf16_1101_h56", kind="layer", tokens=1101, heads=56, hidden=5376,
             precision="bf16"),
        # The same of a large image (128 x 128 tokens and 512 of text) in INT8/FP8, the projection
        # leaving the maxima of |v| for the quantizer.
        dict(name="layer_int8_16896_h56", kind="layer", tokens=16896, heads=56, hidden=5376,
             precision="int8-fp8"),
        # The attention layer of a 1344 x 768 clip with the gates that VSA-trained checkpoints
        # have: 37 x 24 x 42 video tokens after 36 of text, nine tenths of the tiles left out.
        dict(name="video_layer_bf16_37332_h56_gated", kind="video_layer", text=36, frames=37,
             rows=24, columns=42, heads=56, hidden=5376, sparsity=0.9, precision="bf16",
             gated=True),
        # The long video of the configurations (31 x 48 x 84 tokens after 512 of text): BF16 from
        # raw q, k and v, and INT8/FP8 from the fused input pass on.
        dict(name="video_bf16_125504_h32", kind="video", text=512, frames=31, rows=48, columns=84,
             heads=32, sparsity=0.875, precision="bf16", gated=False),
        dict(name="video_int8_125504_h32", kind="video", text=512, frames=31, rows=48, columns=84,
             heads=32, sparsity=0.875, precision="int8-fp8", gated=False),
        # Sol-Attn, for checkpoints that were not trained for VSA, on the headline workload.
        dict(name="sol_bf16_66048_h32", kind="sol", tokens=66048, heads=32, sinks=8,
             precision="bf16"),
        # The gated half of a feed-forward network with a low-rank adapter.
        dict(name="ffn_swiglu_adapter_4213", kind="linear", tokens=4213, features=28672,
             hidden=5376, swiglu=True, rank=384),
    ]


def _spread(rng, low, high):
    """A whole number spread over the logarithm of the range."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["text", "vae", "dense", "dense", "layer", "video_layer", "video", "sol",
                       "linear"])
    if kind == "text":
        return dict(kind=kind, tokens=_spread(rng, 16, 2048), heads=rng.choice([16, 32]),
                    group=rng.choice([1, 2, 4, 8]), batch=rng.choice([1, 1, 2]))
    if kind == "vae":
        return dict(kind=kind, tokens=_spread(rng, 64, 4096), heads=rng.choice([8, 12, 16]),
                    batch=rng.randint(1, 12), pairs=rng.choice([20, 32]))
    if kind == "dense":
        heads = rng.choice([8, 16, 24, 32, 56])
        # No more work than the headline workload.
        most = int(66048 * min(1.0, math.sqrt(32 / heads)))
        return dict(kind=kind, tokens=_spread(rng, 200, most), heads=heads,
                    precision=rng.choice(["bf16", "int8-fp8"]))
    if kind == "layer":
        heads = rng.choice([24, 32, 56])
        return dict(kind=kind, tokens=_spread(rng, 256, 32768), heads=heads,
                    hidden=96 * heads if heads == 56 else 128 * heads,
                    precision=rng.choice(["bf16", "int8-fp8"]))
    if kind in ("video_layer", "video"):
        whole = kind == "video_layer"
        heads = rng.choice([32, 56]) if whole else rng.choice([8, 16, 32])
        rows, columns = rng.choice([(15, 26), (24, 42), (34, 60), (48, 84)])
        most = min(37, (37332 if whole else 124992) // (rows * columns))
        case = dict(kind=kind, text=rng.randint(20, 512), frames=rng.randint(5, most), rows=rows,
                    columns=columns, heads=heads)
        if whole:
            case["hidden"] = 96 * heads if heads == 56 else 128 * heads
        case.update(sparsity=rng.choice([0.8, 0.875, 0.9]),
                    precision=rng.choice(["bf16", "int8-fp8"]), gated=rng.random() < 0.5)
        return case
    if kind == "sol":
        return dict(kind=kind, tokens=_spread(rng, 2048, 66048), heads=rng.choice([8, 16, 32]),
                    sinks=rng.randint(1, 9), precision=rng.choice(["bf16", "int8-fp8"]))
    swiglu = rng.random() < 0.5
    return dict(kind="linear", tokens=_spread(rng, 64, 32768),
                features=rng.choice([28672, 14336]) if swiglu else rng.choice([5376, 12288, 21504]),
                hidden=rng.choice([4096, 5376, 7168]), swiglu=swiglu, rank=rng.choice([0, 64, 384]))


# -------------------------------------------------------------------------------------------------
# Inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(generator, shape, dtype=torch.float32):
    return torch.randn(shape, generator=generator, device="cuda", dtype=dtype)


def _random_qkv(generator, tokens, heads):
    """q, v ~ N(0, 1); k ~ N(0, 1) plus an offset of each channel with variance 2."""
    qkv = _randn(generator, (tokens, 3, heads, HEAD_DIM), torch.bfloat16)
    qkv[:, 1] += (_randn(generator, (heads, HEAD_DIM)) * math.sqrt(2.0)).bfloat16()
    return qkv


def _output(tokens, heads):
    return torch.zeros((tokens, heads, HEAD_DIM), dtype=torch.bfloat16, device="cuda")


def _norm(generator, tokens, positions=None):
    """Norm weights near one, and the angles of 64 rotary pairs over the tokens' positions."""
    weights = [(1.0 + 0.1 * _randn(generator, (HEAD_DIM,))).bfloat16() for _ in range(2)]
    if positions is None:
        positions = torch.arange(tokens, device="cuda", dtype=torch.float32)[:, None]
    axes = positions.shape[1]
    pairs = HEAD_DIM // 2
    axis = torch.arange(pairs, device="cuda") * axes // pairs
    step = torch.arange(pairs, device="cuda") % (pairs // axes) / (pairs // axes)
    angles = positions[:, axis] * torch.exp(-math.log(10000.0) * step)[None, :]
    return attention.HeadNorm(weights[0], weights[1], angles.float().contiguous(), pairs, EPSILON)


def _video(case):
    layout = PackedLayout.text_to_video(case["text"], case["frames"], 2 * case["rows"],
                                        2 * case["columns"], 0)
    return layout, VsaPlan.for_layout(layout)


def _video_positions(case, layout, plan):
    """(frame, row, column) of every token in the plan's order; text counts along the frames."""
    order = torch.tensor(plan.video_order, device="cuda", dtype=torch.int64)
    grid = torch.stack((order // (case["rows"] * case["columns"]),
                        order // case["columns"] % case["rows"], order % case["columns"]), 1)
    text = torch.arange(plan.video_start, device="cuda")[:, None].expand(-1, 3)
    return torch.cat((text, grid)).float(), order


def _projection(generator, tokens, heads, hidden, smooth=None):
    """An INT8 block input with a scale a row, an INT8 qkv weight with a scale a column, and the
    buffers the projection fills. Outputs are of the order of one. `smooth` (rows, values) is added
    to the block input before it is quantized."""
    inner = heads * HEAD_DIM
    rows = _randn(generator, (tokens, hidden))
    if smooth is not None:
        start, values = smooth
        rows[start:start + values.shape[0]] += values
    row_scales = rows.abs().amax(dim=1) / 127.0
    activations = torch.round(rows / row_scales[:, None]).to(torch.int8)
    del rows
    weights = torch.randint(-127, 128, (3 * inner, hidden), dtype=torch.int8, device="cuda",
                            generator=generator)
    column_scales = (torch.rand(3 * inner, generator=generator, device="cuda") + 0.5) / \
        (73.0 * math.sqrt(hidden))
    return dict(activations=activations, weights=weights, row_scales=row_scales,
                column_scales=column_scales, hidden=hidden,
                qkv=torch.zeros((tokens, 3, heads, HEAD_DIM), dtype=torch.bfloat16, device="cuda"),
                maxima=torch.zeros(heads, dtype=torch.float32, device="cuda"))


def prepare(case, seed):
    generator = _generator(seed)
    kind = case["kind"]
    state = dict(case=case)
    if kind in ("text", "vae"):
        dim = 64 if kind == "vae" else HEAD_DIM
        dtype = torch.float16 if kind == "vae" else torch.bfloat16
        tokens, heads, batch = case["tokens"], case["heads"], case["batch"]
        group = case.get("group", 1)
        shape = (batch, tokens, heads, dim)
        key_shape = (batch, tokens, heads // group, dim)
        state.update(query=_randn(generator, shape, dtype), key=_randn(generator, key_shape, dtype),
                     value=_randn(generator, key_shape, dtype),
                     output=torch.zeros(shape, dtype=dtype, device="cuda"))
        inner, key_inner = heads * dim, heads // group * dim
        state["layout"] = attention.make_layout(
            (inner, key_inner, key_inner, inner), head_stride=(dim,) * 4,
            batch_stride=(tokens * inner, tokens * key_inner, tokens * key_inner, tokens * inner),
            heads_per_key_value=group, causal=int(kind == "text"))
        state["scale"] = 1.0 / math.sqrt(dim)
        if kind == "vae":
            state["angles"] = (torch.rand((tokens, case["pairs"]), generator=generator,
                                          device="cuda") * 6.0 - 3.0)
        return state
    if kind == "linear":
        tokens, features, hidden = case["tokens"], case["features"], case["hidden"]
        columns = features // 2 if case["swiglu"] else features
        random_int8 = dict(dtype=torch.int8, device="cuda", generator=generator)
        state.update(
            activations=torch.randint(-127, 128, (tokens, hidden), **random_int8),
            weights=torch.randint(-127, 128, (features, hidden), **random_int8),
            row_scales=torch.rand(tokens, generator=generator, device="cuda") + 0.5,
            column_scales=(torch.rand(features, generator=generator, device="cuda") + 0.5) /
            (73.0 * 73.0 * math.sqrt(hidden)),
            output=torch.zeros((tokens, columns), dtype=torch.bfloat16, device="cuda"))
        if case["rank"]:
            rank = case["rank"]
            state["adapter"] = gemm.Adapter(_randn(generator, (tokens, rank), torch.bfloat16),
                                            _randn(generator, (features, rank), torch.bfloat16),
                                            rank, rank, 0.3 / math.sqrt(rank))
        return state

    heads = case["heads"]
    state["scale"] = synthetic.softmax_scale()
    if kind in ("video", "video_layer"):
        layout, plan = _video(case)
        tokens = len(layout)
        state.update(tokens=tokens, kept=plan.kept_video_tiles(case["sparsity"]),
                     layout=attention.qkv_layout(heads), gate=None)
        positions, order = _video_positions(case, layout, plan)
        if kind == "video":
            state["qkv"] = synthetic.video_qkv_device(layout, plan, heads, seed)
        else:
            grid = (case["frames"], case["rows"], case["columns"])
            coarse = _randn(generator, (1, case["hidden"], 4, 6, 11))
            smooth = torch.nn.functional.interpolate(coarse, size=grid, mode="trilinear",
                                                     align_corners=True)
            smooth = smooth.reshape(case["hidden"], -1).t()[order]
            state.update(_projection(generator, tokens, heads, case["hidden"],
                                     (plan.video_start, smooth)))
            del smooth, coarse
        state["norm"] = _norm(generator, tokens, positions)
        if case["gated"]:
            state["gate"] = _randn(generator, (tokens, heads * HEAD_DIM), torch.bfloat16)
        state["workspace"] = attention.VsaWorkspace(plan, tokens, heads,
                                                    quantized=case["precision"] == "int8-fp8")
    else:
        tokens = case["tokens"]
        state["tokens"] = tokens
        quantized = case["precision"] == "int8-fp8"
        if kind == "layer":
            state.update(_projection(generator, tokens, heads, case["hidden"]))
            state["norm"] = _norm(generator, tokens)
        else:
            state["qkv"] = _random_qkv(generator, tokens, heads)
        if kind == "sol":
            state.update(layout=attention.qkv_layout(heads),
                         sinks=attention.SparseSinks((0, case["sinks"]), (0, 0)),
                         workspace=attention.SparseWorkspace(tokens, heads, quantized=quantized))
        elif quantized:
            state["workspace"] = attention.QuantizedWorkspace(tokens, heads)
    state["output"] = _output(tokens, heads)
    return state


# -------------------------------------------------------------------------------------------------
# One pass


def _project(state, maxima):
    """The qkv projection, with the maxima of |v| when the next step quantizes."""
    heads = state["case"]["heads"]
    inner = heads * HEAD_DIM
    column_maxima = None
    if maxima:
        state["maxima"].zero_()
        column_maxima = gemm.ColumnMaxima(state["maxima"], 2 * inner)
    gemm.int8(None, state["activations"], state["weights"], state["row_scales"],
              state["column_scales"], gemm.Output(state["qkv"], column_maxima=column_maxima),
              state["tokens"], 3 * inner, state["hidden"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "text":
        attention.attention(0, HEAD_DIM, state["query"], state["key"], state["value"],
                            state["output"], case["tokens"], case["heads"], case["batch"],
                            state["layout"], state["scale"])
        return state["output"]
    if kind == "vae":
        attention.attention_roped(1, 64, state["query"], state["key"], state["value"],
                                  state["output"], case["tokens"], case["heads"], case["batch"],
                                  state["layout"], state["scale"], state["angles"], case["pairs"],
                                  EPSILON)
        return state["output"]
    if kind == "linear":
        gemm.int8(None, state["activations"], state["weights"], state["row_scales"],
                  state["column_scales"], gemm.Output(state["output"], swiglu=case["swiglu"]),
                  case["tokens"], case["features"], case["hidden"], state.get("adapter"))
        return state["output"]

    qkv, output, scale = state["qkv"], state["output"], state["scale"]
    tokens, heads = state["tokens"], case["heads"]
    quantized = case["precision"] == "int8-fp8"
    if kind == "dense":
        if quantized:
            attention.dense_quantized(qkv, output, scale, state["workspace"])
        else:
            attention.dense_bf16(qkv, output, tokens, heads, scale)
        return output
    if kind == "sol":
        attention.sparse(qkv, output, state["layout"], scale, SOL_TAU, state["sinks"],
                         state["workspace"])
        return output
    if kind == "layer":
        _project(state, quantized)
        if quantized:
            attention.prepare_inputs(qkv, state["norm"], tokens, heads, state["workspace"],
                                     value_head_maxima=state["maxima"])
            attention.dense_quantized(qkv, output, scale, state["workspace"],
                                      attention.AttentionInputs.PREPARED_WITH_VALUES)
        else:
            attention.qk_norm_rope(qkv, state["norm"], tokens, heads)
            attention.dense_bf16(qkv, output, tokens, heads, scale)
        return {"qkv": qkv, "output": output}
    if kind == "video_layer":
        _project(state, quantized)
        attention.prepare_inputs(qkv, state["norm"], tokens, heads, vsa=state["workspace"],
                                 value_head_maxima=state["maxima"] if quantized else None)
        attention.vsa(qkv, state["gate"], output, state["layout"], scale, state["kept"],
                      state["workspace"],
                      attention.AttentionInputs.PREPARED_WITH_VALUES if quantized
                      else attention.AttentionInputs.PREPARED)
        return {"qkv": qkv, "output": output}
    inputs = attention.AttentionInputs.RAW
    if quantized:
        # Leaves q, k and v in qkv as they are: what it norms goes to the INT8 workspace.
        attention.prepare_inputs(qkv, state["norm"], tokens, heads, vsa=state["workspace"])
        inputs = attention.AttentionInputs.PREPARED
    attention.vsa(qkv, state["gate"], output, state["layout"], scale, state["kept"],
                  state["workspace"], inputs)
    return output


# -------------------------------------------------------------------------------------------------
# What a pass cannot do without


def work(case):
    kind = case["kind"]
    if kind == "linear":
        tokens, features, hidden, rank = (case[name] for name in
                                          ("tokens", "features", "hidden", "rank"))
        columns = features // 2 if case["swiglu"] else features
        return {"bytes": (tokens + features) * (hidden + 4 + 2 * rank) + 2 * tokens * columns,
                "flops": 2 * tokens * features * (hidden + rank)}
    heads = case["heads"]
    if kind in ("text", "vae"):
        dim = 64 if kind == "vae" else HEAD_DIM
        tokens, batch = case["tokens"], case["batch"]
        pairs = tokens * (tokens + 1) // 2 if kind == "text" else tokens * tokens
        operands = 2 * heads + 2 * (heads // case.get("group", 1))
        return {"bytes": 2 * batch * tokens * operands * dim + 4 * tokens * case.get("pairs", 0),
                "flops": 4 * batch * heads * pairs * dim}
    inner = heads * HEAD_DIM
    if kind in ("video", "video_layer"):
        layout, plan = _video(case)
        tokens = len(layout)
        fraction = plan.expected_selected_fraction(plan.kept_video_tiles(case["sparsity"]))
    else:
        tokens, fraction = case["tokens"], 1.0
        if kind == "sol":
            # About a tenth of the pairs of blocks pass the threshold on these values.
            blocks = -(-tokens // 64)
            fraction = min(1.0, 0.1 + case["sinks"] / blocks)
    flops = int(4 * tokens * tokens * inner * fraction)
    moved = 2 * tokens * 4 * inner
    if kind in ("layer", "video_layer"):
        # The block input and the weight in; qkv and the output out.
        hidden = case["hidden"]
        flops += 2 * tokens * 3 * inner * hidden
        moved += tokens * hidden + 3 * inner * hidden
    if kind == "layer" or (kind in ("video", "video_layer") and
                           (kind == "video_layer" or case["precision"] == "int8-fp8")):
        moved += 4 * tokens * (HEAD_DIM // 2)
    if case.get("gated"):
        moved += 2 * tokens * inner
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """About four times the error of these entry points against 64-bit restatements of the same
    calls (2-norms, 300 to 16,896 tokens), and less for the low-precision ones."""
    if case["kind"] == "linear":
        # Without an adapter the sums are whole numbers and the operations after them are fixed.
        # With one, 3.0e-3 (the output's own rounding is 1.7e-3 of it).
        return {"rel": 6e-3} if case["rank"] else "exact"
    if case.get("precision") == "int8-fp8":
        # Probabilities of three mantissa bits are 2.6e-2 from unrounded ones over the same INT8 q,
        # k and FP8 v; rounded about two different maxima of a row, 3.6e-2 from each other.
        return {"rel": 6e-2}
    # 2.3e-3 in BF16 (over routes 2.0e-3), 3.6e-4 in FP16.
    return {"rel": 1.5e-3} if case["kind"] == "vae" else {"rel": 1e-2}
