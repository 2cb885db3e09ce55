"""Parity of the dense BF16 attention kernel, through the C ABI, on a B200.

Mirrors crates/mmh3-cuda/tests/attention.rs: the same generator, seeds, shapes and tolerance against
an f64 softmax attention, plus ragged sizes around the kernel's 128/256-row tiles, the benchmark's
value distribution, and the reference's own CUDA kernel on the same device buffers.
"""

import ctypes

import numpy as np
import pytest
import torch

import oracle_lib
from mmh3_b200 import _lib, attention, synthetic

pytestmark = pytest.mark.gpu

SCALE = synthetic.softmax_scale()


def lcg_qkv(oracle, tokens, heads, seed):
    values, _ = oracle_lib.lcg(oracle, seed, tokens * 3 * heads * 128, -2.0, 2.0)
    return synthetic.to_bf16_bits(values).reshape(tokens, 3, heads, 128)


def run_dense(bits, tokens, heads):
    qkv = synthetic.bf16_tensor(bits, "cuda")
    output = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    attention.dense_bf16(qkv, output, tokens, heads, SCALE)
    assert attention.take_status() == 0
    return output.float().cpu().numpy()


def cosine(a, b):
    a, b = a.astype(np.float64).ravel(), b.astype(np.float64).ravel()
    return float(a @ b / (np.linalg.norm(a) * np.linalg.norm(b) + 1e-300))


def load_selftest():
    library = ctypes.CDLL(str(_lib.SELFTEST_LIBRARY))
    library.mmh3_b200_umma_selftest.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 6
    library.mmh3_b200_umma_selftest.restype = ctypes.c_int
    return library


def test_a_wait_that_runs_out_is_reported_and_the_context_survives():
    """Failure detection without a fault: every wait in the kernels is bounded; one that runs out
    (here: on a barrier nothing completes) leaves its code in the status word, the kernel returns,
    take_status reads and clears the word, and the next launch on the same context works."""
    library = load_selftest()
    library.mmh3_b200_expired_wait_selftest.argtypes = [ctypes.c_uint]
    library.mmh3_b200_expired_wait_selftest.restype = ctypes.c_int
    library.mmh3_b200_take_status.restype = ctypes.c_int
    code = 0x00770001
    assert library.mmh3_b200_take_status() == 0
    assert library.mmh3_b200_expired_wait_selftest(code) == 64  # every thread gave up
    assert library.mmh3_b200_take_status() == code
    assert library.mmh3_b200_take_status() == 0
    test_umma_bf16_building_blocks()
    tokens, heads = 300, 2
    bits = synthetic.dense_qkv(tokens, heads, seed=3).view(torch.int16).numpy().view(np.uint16)
    run_dense(bits, tokens, heads)
    assert attention.take_status() == 0


def test_umma_bf16_building_blocks():
    """scores = A.B^T from shared memory and output = P.V with P in tensor memory, BF16."""
    library = load_selftest()
    generator = torch.Generator().manual_seed(11)
    a = torch.randn((128, 128), generator=generator).bfloat16().cuda()
    b = torch.randn((128, 128), generator=generator).bfloat16().cuda()
    v = torch.randn((128, 128), generator=generator).bfloat16().cuda()
    p = torch.rand((128, 128), generator=generator).bfloat16().cuda()
    scores = torch.zeros((128, 128), dtype=torch.float32, device="cuda")
    output = torch.zeros((128, 128), dtype=torch.float32, device="cuda")
    code = library.mmh3_b200_umma_selftest(0, a.data_ptr(), b.data_ptr(), v.data_ptr(),
                                           p.data_ptr(), scores.data_ptr(), output.data_ptr())
    assert code == 0
    assert attention.take_status() == 0
    expected_scores = a.float().cpu() @ b.float().cpu().t()
    expected_output = p.float().cpu() @ v.float().cpu()
    assert torch.allclose(scores.cpu(), expected_scores, atol=1e-3, rtol=1e-4)
    assert torch.allclose(output.cpu(), expected_output, atol=1e-3, rtol=1e-4)


def test_umma_int8_fp8_building_blocks(oracle):
    """INT8 A.B^T with INT32 accumulators (exact) and E4M3 P.V^T with P in tensor memory."""
    library = load_selftest()
    rng = np.random.default_rng(12)
    a = rng.integers(-127, 128, size=(128, 128), dtype=np.int8)
    b = rng.integers(-127, 128, size=(128, 128), dtype=np.int8)
    p = rng.integers(0, 0x7F, size=(128, 128), dtype=np.uint8)  # positive finite E4M3
    v = rng.integers(0, 0x7F, size=(128, 128), dtype=np.uint8)
    v |= (rng.integers(0, 2, size=(128, 128), dtype=np.uint8) << 7)
    table = np.array([oracle.oracle_e4m3_to_f32(code) for code in range(256)], dtype=np.float64)
    device = [torch.from_numpy(x.view(np.uint8).copy()).cuda() for x in (a, b, v, p)]
    scores = torch.zeros((128, 128), dtype=torch.int32, device="cuda")
    output = torch.zeros((128, 128), dtype=torch.float32, device="cuda")
    code = library.mmh3_b200_umma_selftest(1, *(x.data_ptr() for x in device), scores.data_ptr(),
                                           output.data_ptr())
    assert code == 0
    assert attention.take_status() == 0
    expected_scores = a.astype(np.int32) @ b.astype(np.int32).T
    assert np.array_equal(scores.cpu().numpy(), expected_scores)
    # v is V^T [dims][keys]: output[m][d] = sum_k p[m][k] v[d][k]
    expected_output = table[p] @ table[v].T
    assert np.allclose(output.cpu().numpy(), expected_output, rtol=2e-3, atol=1e-2)


@pytest.mark.parametrize("tokens,heads", [(1, 1), (64, 2), (200, 3)])
def test_matches_cpu_reference(oracle, tokens, heads):
    """attention.rs:27-90: LCG data uniform in [-2, 2), seed tokens * 31 + heads."""
    bits = lcg_qkv(oracle, tokens, heads, tokens * 31 + heads)
    actual = run_dense(bits, tokens, heads)
    expected = oracle_lib.attention_bf16(oracle, bits, tokens, heads, SCALE)
    assert np.all(np.abs(actual - expected) <= 0.02 + 0.01 * np.abs(expected))


@pytest.mark.parametrize("tokens", [127, 128, 129, 255, 256, 257, 384, 1000])
def test_ragged_sizes(oracle, tokens):
    heads = 2
    bits = synthetic.dense_qkv(tokens, heads, seed=tokens).view(torch.int16).numpy().view(np.uint16)
    actual = run_dense(bits, tokens, heads)
    expected = oracle_lib.attention_bf16(oracle, bits, tokens, heads, SCALE)
    assert np.max(np.abs(actual - expected)) <= 2e-2
    assert cosine(actual, expected) >= 0.9995


def test_cpu_workload_sampled(oracle):
    """B=1, H=8, L=4096 with the benchmark's distribution, every 29th query row on the CPU."""
    tokens, heads = synthetic.CONFIGS["C0"]
    bits = synthetic.dense_qkv(tokens, heads, seed=0).view(torch.int16).numpy().view(np.uint16)
    actual = run_dense(bits, tokens, heads)
    rows = list(range(0, tokens, 29))
    for row in rows:
        expected = oracle_lib.attention_bf16(oracle, bits, tokens, heads, SCALE, row, row + 1)
        assert np.max(np.abs(actual[row] - expected[0])) <= 2e-2
    expected = np.concatenate([
        oracle_lib.attention_bf16(oracle, bits, tokens, heads, SCALE, row, row + 1) for row in rows[:32]
    ])
    assert cosine(actual[rows[:32]], expected) >= 0.9995


def test_agrees_with_the_reference_kernel(reference_kernels):
    """The reference's mma.sync kernel and this one on the same device buffers."""
    tokens, heads = 1000, 3
    inner = heads * 128
    qkv = synthetic.dense_qkv(tokens, heads, seed=5).cuda()
    ours = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    theirs = torch.zeros_like(ours)
    attention.dense_bf16(qkv, ours, tokens, heads, SCALE)
    base = qkv.data_ptr()
    code = reference_kernels.mmh3_attention_bf16(base, base + 2 * inner, base + 4 * inner,
                                                 theirs.data_ptr(), tokens, heads, 3 * inner,
                                                 3 * inner, 3 * inner, inner, SCALE, None)
    assert code == 0
    torch.cuda.synchronize()
    assert attention.take_status() == 0
    a, b = ours.float().cpu().numpy(), theirs.float().cpu().numpy()
    assert np.max(np.abs(a - b)) <= 2e-2
    assert cosine(a, b) >= 0.9995


def test_grouped_heads_and_batches(oracle):
    """mmh3_attention with two query heads per key/value head and a batch of two."""
    tokens, heads, group, batch = 130, 4, 2, 2
    generator = torch.Generator().manual_seed(3)
    q = torch.randn((batch, tokens, heads, 128), generator=generator).bfloat16()
    k = torch.randn((batch, tokens, heads // group, 128), generator=generator).bfloat16()
    v = torch.randn((batch, tokens, heads // group, 128), generator=generator).bfloat16()
    output = torch.zeros((batch, tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    kv_inner = heads // group * 128
    layout = attention.make_layout(
        (heads * 128, kv_inner, kv_inner, heads * 128),
        batch_stride=(tokens * heads * 128, tokens * kv_inner, tokens * kv_inner,
                      tokens * heads * 128),
        heads_per_key_value=group)
    attention.attention(0, 128, q.cuda(), k.cuda(), v.cuda(), output, tokens, heads, batch, layout,
                        SCALE)
    assert attention.take_status() == 0
    scores = torch.einsum("bqhd,bkhd->bhqk", q.double(),
                          k.double().repeat_interleave(group, dim=2)) * SCALE
    expected = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1),
                            v.double().repeat_interleave(group, dim=2))
    assert torch.max(torch.abs(output.cpu().double() - expected)) <= 2e-2


@pytest.mark.parametrize("element_type,head_dim,tokens,batch,causal,order", [
    (0, 128, 130, 3, 1, "items"),       # [batch, tokens, heads, dim]
    (1, 64, 257, 9, 0, "items"),
    (1, 64, 300, 2, 0, "tokens"),       # [tokens, batch, heads, dim]
    (0, 128, 1, 4, 0, "heads"),         # [heads, batch, tokens, dim]
    (0, 64, 140, 3, 0, "shared"),       # one key and value for all items: a stride of zero
    (0, 128, 140, 3, 0, "off grid"),    # items that do not start on 16 bytes
    (1, 128, 40, 3, 0, "overlapping"),  # outputs that the next item partly writes over
])
@pytest.mark.parametrize("rope", [False, True])
def test_a_batch_equals_its_items(element_type, head_dim, tokens, batch, causal, order, rope):
    """A batch that TMA can describe goes in one launch, the others item by item: the same bits as
    one call per item, in order, either way."""
    heads, group = 4, 2
    dtype = torch.float16 if element_type == 1 else torch.bfloat16
    generator = torch.Generator().manual_seed(tokens + batch)
    pairs = 20
    angles = (torch.rand((tokens, pairs), generator=generator) * 6.0 - 3.0).cuda()

    def strides(count):
        if order == "tokens":
            return batch * count * head_dim, head_dim, count * head_dim
        if order == "heads":
            return head_dim, batch * tokens * head_dim, tokens * head_dim
        return count * head_dim, head_dim, tokens * count * head_dim

    counts = (heads, heads // group, heads // group, heads)
    layout = [list(strides(count)) for count in counts]
    if order == "shared":
        layout[1][2] = layout[2][2] = 0
    if order == "off grid":
        for operand in layout:
            operand[2] += 4
    if order == "overlapping":
        layout[3][2] //= 2
    sizes = [1 + (tokens - 1) * t + (count - 1) * h + (batch - 1) * b + head_dim
             for (t, h, b), count in zip(layout, counts)]
    query, key, value = (torch.randn(size, generator=generator).to(dtype).cuda()
                         for size in sizes[:3])

    def run(whole):
        output = torch.zeros(sizes[3], dtype=dtype, device="cuda")
        operands = (query, key, value, output)
        described = attention.make_layout(*zip(*layout), heads_per_key_value=group, causal=causal)
        for item in range(1 if whole else batch):
            views = [tensor[item * operand[2]:] for tensor, operand in zip(operands, layout)]
            arguments = (element_type, head_dim, *views, tokens, heads, batch if whole else 1,
                         described, SCALE)
            if rope:
                attention.attention_roped(*arguments, angles, pairs, 1e-6)
            else:
                attention.attention(*arguments)
        assert attention.take_status() == 0
        return output

    assert torch.equal(run(True).view(torch.int16), run(False).view(torch.int16))


@pytest.mark.parametrize("operand,shift", [(0, -1), (0, 0), (0, 1), (1, -1), (1, 1), (2, -1), (2, 1)])
def test_a_batch_whose_output_lies_over_its_operands(operand, shift):
    """Item i's output over the query, keys or values of item i - 1 or i + 1, or in its own query's
    place: the bits of one call per item, in order."""
    tokens, heads, batch, head_dim = 700, 4, 3, 64
    size = tokens * heads * head_dim
    layout = attention.make_layout((heads * head_dim,) * 4, head_stride=(head_dim,) * 4,
                                   batch_stride=(size,) * 4)
    generator = torch.Generator().manual_seed(operand)
    source = torch.randn((3, batch + 2, size), generator=generator).bfloat16().cuda()

    def run(whole):
        buffers = source.clone()
        for item in range(1 if whole else batch):
            views = [buffers[index, 1 + item:] for index in range(3)]
            attention.attention(0, head_dim, *views, buffers[operand, 1 + item + shift:], tokens,
                                heads, batch if whole else 1, layout, 0.125)
        assert attention.take_status() == 0
        return buffers

    assert torch.equal(run(True).view(torch.int16), run(False).view(torch.int16))


def reference_attention(q, k, v, group, causal):
    """softmax(q k^T * scale) v in float64 with torch, [batch, tokens, heads, 128] operands."""
    keys = k.double().repeat_interleave(group, dim=2)
    values = v.double().repeat_interleave(group, dim=2)
    scores = torch.einsum("bqhd,bkhd->bhqk", q.double(), keys) * SCALE
    if causal:
        tokens = q.shape[1]
        future = torch.triu(torch.ones((tokens, tokens), dtype=torch.bool), diagonal=1)
        scores = scores.masked_fill(future, float("-inf"))
    return torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), values)


@pytest.mark.parametrize("element_type", [0, 1])
@pytest.mark.parametrize("tokens,causal", [(77, 1), (256, 1), (700, 1), (1000, 0), (513, 1)])
def test_causal_and_fp16_variants(reference_kernels, element_type, tokens, causal):
    """The other users of mmh3_attention at heads of 128 (crates/mmh3-cuda/kernels/attention.cu:
    502-536): the text encoder's causal attention with grouped key/value heads
    (src/text_encoder.rs:653-666), in BF16 and in FP16, against float64 and against the reference's
    kernel on the same buffers."""
    heads, group, batch = 4, 2, 2
    dtype = torch.float16 if element_type == 1 else torch.bfloat16
    generator = torch.Generator().manual_seed(tokens + element_type)
    q = torch.randn((batch, tokens, heads, 128), generator=generator).to(dtype)
    k = torch.randn((batch, tokens, heads // group, 128), generator=generator).to(dtype)
    v = torch.randn((batch, tokens, heads // group, 128), generator=generator).to(dtype)
    kv_inner = heads // group * 128
    layout = attention.make_layout(
        (heads * 128, kv_inner, kv_inner, heads * 128),
        batch_stride=(tokens * heads * 128, tokens * kv_inner, tokens * kv_inner,
                      tokens * heads * 128),
        heads_per_key_value=group, causal=causal)
    device = [tensor.cuda() for tensor in (q, k, v)]
    ours = torch.zeros((batch, tokens, heads, 128), dtype=dtype, device="cuda")
    theirs = torch.zeros_like(ours)
    attention.attention(element_type, 128, *device, ours, tokens, heads, batch, layout, SCALE)
    assert reference_kernels.mmh3_attention(
        element_type, 128, *(tensor.data_ptr() for tensor in device), theirs.data_ptr(), tokens,
        heads, batch, ctypes.byref(layout), SCALE, None) == 0
    torch.cuda.synchronize()
    assert attention.take_status() == 0
    expected = reference_attention(q, k, v, group, causal)
    assert torch.max(torch.abs(ours.cpu().double() - expected)) <= 2e-2
    a, b = ours.float().cpu().numpy(), theirs.float().cpu().numpy()
    assert np.max(np.abs(a - b)) <= 2e-2
    assert cosine(a, b) >= 0.9995


def normalized_rotated(q, angles, pairs, epsilon, dtype):
    """The query after the fused RMS norm and RoPE, rounded to the element type as the kernel
    rounds it (crates/mmh3-cuda/kernels/attention.cu:62-111)."""
    values = q.double()
    values = values * torch.rsqrt(values.pow(2).mean(dim=-1, keepdim=True) + epsilon)
    first, second = values[..., :pairs], values[..., pairs:2 * pairs]
    cosine = torch.cos(angles.double())[None, :, None, :]
    sine = torch.sin(angles.double())[None, :, None, :]
    rotated = values.clone()
    rotated[..., :pairs] = first * cosine - second * sine
    rotated[..., pairs:2 * pairs] = first * sine + second * cosine
    return rotated.to(dtype)


@pytest.mark.parametrize("element_type", [0, 1])
@pytest.mark.parametrize("head_dim,tokens,causal,pairs", [
    (64, 300, 0, None), (64, 513, 1, None), (64, 700, 0, 32), (64, 129, 0, 20),
    (128, 300, 0, 64), (128, 257, 1, 40),
])
def test_heads_of_64_and_the_fused_query_rope(reference_kernels, element_type, head_dim, tokens,
                                              causal, pairs):
    """The VAE decoder's use of mmh3_attention_roped (src/vae.rs:1008): FP16 heads of 64 in a
    batched layout with the query's RMS norm and RoPE inside the attention; and the same options in
    every other combination the reference's kernel takes, against float64 and against that kernel
    on the same buffers."""
    heads, batch, epsilon = 3, 2, 1e-6
    scale = 1.0 / head_dim ** 0.5
    dtype = torch.float16 if element_type == 1 else torch.bfloat16
    generator = torch.Generator().manual_seed(tokens + head_dim + element_type)
    q, k, v = (torch.randn((batch, tokens, heads, head_dim), generator=generator).to(dtype)
               for _ in range(3))
    inner = heads * head_dim
    layout = attention.make_layout((inner,) * 4, head_stride=(head_dim,) * 4,
                                   batch_stride=(tokens * inner,) * 4, causal=causal)
    device = [tensor.cuda() for tensor in (q, k, v)]
    ours = torch.zeros((batch, tokens, heads, head_dim), dtype=dtype, device="cuda")
    theirs = torch.zeros_like(ours)
    angles = None
    if pairs is not None:
        angles = (torch.rand((tokens, pairs), generator=generator) * 6.0 - 3.0).cuda()
        attention.attention_roped(element_type, head_dim, *device, ours, tokens, heads, batch,
                                  layout, scale, angles, pairs, epsilon)
    else:
        attention.attention(element_type, head_dim, *device, ours, tokens, heads, batch, layout,
                            scale)
    assert reference_kernels.mmh3_attention_roped(
        element_type, head_dim, *(tensor.data_ptr() for tensor in device), theirs.data_ptr(),
        tokens, heads, batch, ctypes.byref(layout), scale,
        angles.data_ptr() if angles is not None else None, pairs or 0, epsilon, None) == 0
    torch.cuda.synchronize()
    assert attention.take_status() == 0
    query = normalized_rotated(q, angles.cpu(), pairs, epsilon, dtype) if pairs else q
    scores = torch.einsum("bqhd,bkhd->bhqk", query.double(), k.double()) * scale
    if causal:
        future = torch.triu(torch.ones((tokens, tokens), dtype=torch.bool), diagonal=1)
        scores = scores.masked_fill(future, float("-inf"))
    expected = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), v.double())
    assert torch.max(torch.abs(ours.cpu().double() - expected)) <= 2e-2
    a, b = ours.float().cpu().numpy(), theirs.float().cpu().numpy()
    assert np.max(np.abs(a - b)) <= 2e-2
    assert cosine(a, b) >= 0.9995


@pytest.mark.parametrize("head_dim,tokens,pairs", [
    (64, 1, 32), (64, 127, 20), (64, 129, 1), (64, 257, 31), (64, 518, 32),
    (128, 5, 64), (128, 131, 33), (128, 300, 40), (128, 255, 3),
])
@pytest.mark.parametrize("element_type,span", [(0, 40.0), (1, 40.0), (1, 2e5)])
def test_fused_query_rope_against_float64(element_type, span, head_dim, tokens, pairs):
    """Every split of a head into pairs and the rest, rows that fill a warp's turn and rows that do
    not, angles past what is reduced without a branch; the bound of the tests above."""
    heads, batch, epsilon = 3, 2, 1e-6
    scale = 1.0 / head_dim ** 0.5
    dtype = torch.float16 if element_type == 1 else torch.bfloat16
    generator = torch.Generator().manual_seed(tokens + head_dim + pairs)
    q, k, v = (torch.randn((batch, tokens, heads, head_dim), generator=generator).to(dtype)
               for _ in range(3))
    q = q * 3
    inner = heads * head_dim
    layout = attention.make_layout((inner,) * 4, head_stride=(head_dim,) * 4,
                                   batch_stride=(tokens * inner,) * 4)
    angles = torch.rand((tokens, pairs), generator=generator) * (2 * span) - span
    ours = torch.zeros((batch, tokens, heads, head_dim), dtype=dtype, device="cuda")
    attention.attention_roped(element_type, head_dim, q.cuda(), k.cuda(), v.cuda(), ours, tokens,
                              heads, batch, layout, scale, angles.cuda(), pairs, epsilon)
    assert attention.take_status() == 0
    query = normalized_rotated(q, angles, pairs, epsilon, dtype)
    scores = torch.einsum("bqhd,bkhd->bhqk", query.double(), k.double()) * scale
    expected = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), v.double())
    assert torch.max(torch.abs(ours.cpu().double() - expected)) <= 2e-2


@pytest.mark.parametrize("span", [0.8, 40.0, 1000.0, 47999.0])
def test_sines_and_cosines_without_a_branch(span):
    """Against float64, to two units in the last place of the result (what sincosf is allowed): over the
    span, and next to the multiples of pi/4 in it, where the quadrant changes and where all three parts
    of pi/2 are needed."""
    library = load_selftest()
    generator = torch.Generator().manual_seed(int(span))
    angles = torch.rand(1 << 21, generator=generator, dtype=torch.float64) * (2 * span) - span
    turns = torch.randint(-int(span / 0.7854), int(span / 0.7854) + 1, (1 << 20,),
                          generator=generator).double() * (np.pi / 4)
    near = turns * (1 + (torch.randint(-3, 4, turns.shape, generator=generator) * 2.0 ** -24))
    angles = torch.cat([angles, near.clamp(-span, span)]).float().cuda()
    result = torch.empty((angles.numel(), 2), dtype=torch.float32, device="cuda")
    assert library.mmh3_b200_sine_and_cosine_selftest(
        ctypes.c_void_p(angles.data_ptr()), ctypes.c_void_p(result.data_ptr()),
        angles.numel()) == 0
    torch.cuda.synchronize()
    exact = torch.stack([torch.sin(angles.double()), torch.cos(angles.double())], dim=1)
    unit = torch.exp2(torch.floor(torch.log2(exact.abs().clamp_min(2.0 ** -126))) - 23)
    # pi/2 in three floats is right to 2^-24 of the third, 1.7e-15 * 6e-8 a quarter turn, at most
    # 48,000 * 0.64 of them: far below a unit of the smallest sine of a float up to the limit.
    assert float(((result.double() - exact).abs() / unit).max()) <= 2.0


@pytest.mark.parametrize("span", [1000.0, 47900.0])
@pytest.mark.parametrize("head_dim,pairs", [(64, 32), (64, 20), (128, 64), (128, 33)])
def test_fused_query_rope_of_large_angles_seen_through_one_key(span, head_dim, pairs):
    """A key of one dimension at a time reads a rotated query's dimension out of the attention: two
    keys whose scores differ by the dimension alone, and values of one and zero, give its logistic
    function."""
    tokens, heads = 256, 2
    dims = 24  # heads of the batch: a dimension each
    generator = torch.Generator().manual_seed(pairs)
    q = torch.randn((1, tokens, heads, head_dim), generator=generator).half()
    angles = torch.rand((tokens, pairs), generator=generator) * (2 * span) - span
    read = torch.linspace(0, head_dim - 1, dims).long()
    query = q.expand(dims, -1, -1, -1).contiguous()
    key = torch.zeros((dims, tokens, heads, head_dim)).half()
    value = torch.zeros_like(key)
    for item, dimension in enumerate(read.tolist()):
        key[item, ::2, :, dimension] = 4.0
        value[item, ::2] = 1.0
    inner = heads * head_dim
    layout = attention.make_layout((inner,) * 4, head_stride=(head_dim,) * 4,
                                   batch_stride=(tokens * inner,) * 4)
    output = torch.zeros((dims, tokens, heads, head_dim), dtype=torch.float16, device="cuda")
    attention.attention_roped(1, head_dim, query.cuda(), key.cuda(), value.cuda(), output, tokens,
                              heads, dims, layout, 0.25, angles.cuda(), pairs, 1e-6)
    assert attention.take_status() == 0
    rotated = normalized_rotated(q, angles, pairs, 1e-6, torch.float16)[0].double()
    expected = torch.sigmoid(rotated[:, :, read]).permute(2, 0, 1)[..., None]
    # The rotated query may round to the next FP16 value (2^-10 below two, where the logistic passes on
    # a quarter of it, 2^-9 below four, where it passes on a tenth); P and the output are rounded once
    # each (2^-11): 1.3e-3 in all.
    assert float((output.cpu().double() - expected).abs().max()) <= 1.3e-3


@pytest.mark.parametrize("element_type", [0, 1])
def test_heads_of_64_whose_exponentials_come_two_ways(element_type):
    """Two of eight pairs of keys take a polynomial: every key alone in turn holds a row's weight or a
    NaN, and scores far below the maximum weigh nothing."""
    tokens, heads, head_dim = 128, 2, 64
    dtype = torch.float16 if element_type == 1 else torch.bfloat16
    layout = attention.make_layout((heads * head_dim,) * 4, head_stride=(head_dim,) * 4)
    q = torch.zeros((tokens, heads, head_dim))
    k = torch.zeros_like(q)
    # Row i points at key i: 60 * 8 / 8 above the others, 2^-86 of the weight left to them.
    for row in range(tokens):
        q[row, :, row // 2] = 60.0
        k[row, :, row // 2] = 8.0 if row % 2 else -8.0
    q[0::2] = -q[0::2]
    v = torch.randn(q.shape, generator=torch.Generator().manual_seed(1))

    def run(key):
        output = torch.zeros(q.shape, dtype=dtype, device="cuda")
        attention.attention(element_type, head_dim, q.to(dtype).cuda(), key.to(dtype).cuda(),
                            v.to(dtype).cuda(), output, tokens, heads, 1, layout, 0.125)
        assert attention.take_status() == 0
        return output.cpu().float()

    # One probability of one, whose value is then the output to the bit.
    assert torch.equal(run(k), v.to(dtype).float())
    for column in (0, 1, 6, 7, 12, 13, 127):
        poisoned = k.clone()
        poisoned[column, 0, 0] = float("nan")
        result = run(poisoned)
        assert torch.isnan(result[:, 0]).all() and torch.isfinite(result[:, 1]).all()


def test_the_polynomial_exponential_is_as_close_as_the_unit_it_relieves():
    """exp2_polynomial against float64. Its fit is off by 2.0e-9, the rounding of its coefficients by
    1e-8; the last FMA rounds by half a unit of a result of 0.707 to 1.415 (6.0e-8 of it at most), the
    one before by half a unit of a number under one, times a fraction of a half over the result (2.1e-8),
    and the others by less: 1.1e-7 in all. ex2.approx is within 1.45e-7."""
    library = load_selftest()
    count = 1 << 22
    generator = torch.Generator().manual_seed(5)
    x = torch.rand(count, generator=generator, dtype=torch.float64) * 133.0 - 125.0
    # Near the whole numbers and half-way between them, where n changes.
    x[:4096] = torch.arange(4096).double() / 32.0 - 120.0
    x[4096:8192] = x[:4096] * (1.0 + 2.0 ** -23)
    x = x.float().cuda()

    def evaluate(values):
        result = torch.empty_like(values)
        assert library.mmh3_b200_exp2_selftest(
            ctypes.c_void_p(values.data_ptr()), ctypes.c_void_p(result.data_ptr()),
            values.numel() // 2) == 0
        torch.cuda.synchronize()
        return result

    exact = torch.exp2(x.double())
    assert float(((evaluate(x).double() - exact) / exact).abs().max()) <= 1.1e-7
    # Nothing is left of what the MUFU gives zero for, but for denormals above -127.
    low = torch.tensor([-127.0, -127.5, -1e4, -3e38, float("-inf"), float("nan")], device="cuda")
    assert torch.equal(evaluate(low).view(torch.int32), torch.zeros(6, dtype=torch.int32).cuda())
    between = torch.linspace(-126.999, -125.0, 1000, device="cuda")
    values = evaluate(between).double()
    assert (values >= 0).all() and (values <= torch.exp2(between.double()) * (1 + 1.1e-7)).all()


@pytest.mark.parametrize("tokens", [1, 63, 64, 130, 300])
def test_later_values_do_not_reach_causal_rows_of_heads_of_64(tokens):
    """A masked key weighs exactly nothing in BF16, whose smallest numbers times the largest values
    are not small: rows are the same bits whatever finite values the tokens after them have."""
    heads, head_dim, later = 2, 64, 300
    layout = attention.make_layout((heads * head_dim,) * 4, head_stride=(head_dim,) * 4, causal=1)
    generator = torch.Generator().manual_seed(tokens)
    q, k, v = (torch.randn((tokens + later, heads, head_dim), generator=generator).bfloat16().cuda()
               for _ in range(3))

    def run(values):
        output = torch.zeros_like(q)
        attention.attention(0, head_dim, q, k, values, output, tokens + later, heads, 1, layout,
                            0.125)
        assert attention.take_status() == 0
        return output[:tokens].view(torch.int16)

    huge = v.clone()
    huge[tokens:] = 3e38
    assert torch.equal(run(huge), run(v))


def test_unsupported_combinations_report_an_error():
    tokens, heads = 64, 1
    qkv = torch.zeros((tokens, 3, heads, 128), dtype=torch.bfloat16, device="cuda")
    output = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    layout = attention.qkv_layout(heads)
    library = _lib.library()
    arguments = (qkv.data_ptr(), qkv.data_ptr() + 256, qkv.data_ptr() + 512, output.data_ptr(),
                 tokens, heads, 1, ctypes.byref(layout), SCALE)
    assert library.mmh3_attention(2, 128, *arguments, None) == _lib.CUDA_ERROR_INVALID_VALUE
    assert library.mmh3_attention(0, 96, *arguments, None) == _lib.CUDA_ERROR_INVALID_VALUE
    angles = torch.zeros((tokens, 64), dtype=torch.float32, device="cuda")
    # more rotary pairs than half a head
    assert library.mmh3_attention_roped(0, 64, *arguments, angles.data_ptr(), 33, 1e-6,
                                        None) == _lib.CUDA_ERROR_INVALID_VALUE


@pytest.mark.parametrize("element_type,head_dim,group,causal",
                         [(0, 128, 1, 0), (1, 64, 1, 0), (0, 128, 2, 1)])
def test_layouts_off_the_tma_grid_equal_aligned_ones(element_type, head_dim, group, causal):
    """Operands whose base or strides are not multiples of 16 bytes: the reference copies them with
    cp.async instead of TMA and asks for the same bits either way
    (crates/mmh3-cuda/tests/attention.rs:91-114). Here they are gathered into dense arrays first,
    and the output must be the bits of the same values in an aligned layout."""
    tokens, heads = 200, 4
    kv_heads = heads // group
    dtype = torch.float16 if element_type else torch.bfloat16
    generator = torch.Generator(device="cpu").manual_seed(31)
    query = (torch.rand((tokens, heads, head_dim), generator=generator) * 4 - 2).to(dtype).cuda()
    key = (torch.rand((tokens, kv_heads, head_dim), generator=generator) * 4 - 2).to(dtype).cuda()
    value = (torch.rand((tokens, kv_heads, head_dim), generator=generator) * 4 - 2).to(dtype).cuda()
    library = _lib.library()
    scale = 1.0 / head_dim ** 0.5

    def run(operands, token_strides, head_strides):
        output = torch.zeros((tokens, heads, head_dim), dtype=dtype, device="cuda")
        layout = attention.make_layout(tuple(token_strides) + (heads * head_dim,),
                                       tuple(head_strides) + (head_dim,),
                                       heads_per_key_value=group if group > 1 else 0,
                                       causal=causal)
        assert library.mmh3_attention(element_type, head_dim, *operands, output.data_ptr(), tokens,
                                      heads, 1, ctypes.byref(layout), scale, None) == 0
        torch.cuda.synchronize()
        assert attention.take_status() == 0
        return output

    aligned = run([tensor.data_ptr() for tensor in (query, key, value)],
                  [heads * head_dim, kv_heads * head_dim, kv_heads * head_dim], [head_dim] * 3)

    # The same values two bytes off a 16-byte boundary, with a token stride of an odd number of
    # elements and heads head_dim + 2 elements apart.
    def shifted(tensor):
        count = tensor.shape[1]
        head_stride = head_dim + 2
        token_stride = count * head_stride + 1
        storage = torch.zeros(tokens * token_stride + 16, dtype=dtype, device="cuda")
        view = torch.as_strided(storage, (tokens, count, head_dim), (token_stride, head_stride, 1), 1)
        view.copy_(tensor)
        return storage, storage.data_ptr() + 2, token_stride, head_stride

    storages = [shifted(tensor) for tensor in (query, key, value)]
    moved = run([entry[1] for entry in storages], [entry[2] for entry in storages],
                [entry[3] for entry in storages])
    assert torch.equal(moved.view(torch.int16), aligned.view(torch.int16))
    # One operand off the grid is enough to take the copy, and the others are left where they are.
    mixed = run([storages[0][1], key.data_ptr(), value.data_ptr()],
                [storages[0][2], kv_heads * head_dim, kv_heads * head_dim],
                [storages[0][3], head_dim, head_dim])
    assert torch.equal(mixed.view(torch.int16), aligned.view(torch.int16))


@pytest.mark.parametrize("groups", [1, 4, 0])
def test_host_pipeline_equals_one_call(groups):
    """Pinned host buffers in and out, a group of heads at a time on four streams (the first and
    the last group one head each): the same bits as one call over device buffers, twice in a row
    over the same buffers."""
    tokens, heads = 700, 6
    host_qkv = synthetic.dense_qkv(tokens, heads, seed=21, pinned=True)
    expected = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    attention.dense_bf16(host_qkv.cuda(), expected, tokens, heads, SCALE)
    qkv = torch.zeros((tokens, 3, heads, 128), dtype=torch.bfloat16, device="cuda")
    output = torch.zeros_like(expected)
    host_output = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16).pin_memory()
    pipeline = attention.HostPipeline(tokens, heads, groups=groups)
    # One group; four, the first and the last of one head; or runs that double and drain.
    assert [span for _, span in pipeline.groups] == ([6] if groups == 1 else [1, 2, 2, 1])
    for _ in range(2):
        host_output.zero_()
        pipeline.run(host_qkv, qkv, output, host_output, SCALE)
        torch.cuda.synchronize()
        assert attention.take_status() == 0
        assert torch.equal(host_output, expected.cpu())


def test_sharded_host_pipeline_on_one_rank():
    """World size 1: the sharded pipeline is one copy in, the dense layer, one copy out. (With
    more ranks `bench.py --gpus N` compares it with the resident run on every rank.)"""
    from mmh3_b200.shard import HostUlyssesPipeline, Shard

    tokens, heads = 500, 3
    host_qkv = synthetic.dense_qkv(tokens, heads, seed=22, pinned=True)
    expected = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16, device="cuda")
    attention.dense_bf16(host_qkv.cuda(), expected, tokens, heads, SCALE)

    def dense(qkv, output, count, span):
        attention.dense_bf16(qkv, output, count, span, SCALE)

    pipeline = HostUlyssesPipeline(Shard.even(0, 1, tokens, heads), tokens, heads, dense, 2)
    qkv = torch.zeros((tokens, 3, heads, 128), dtype=torch.bfloat16, device="cuda")
    output = torch.zeros_like(expected)
    host_output = torch.zeros((tokens, heads, 128), dtype=torch.bfloat16).pin_memory()
    pipeline.run(host_qkv, qkv, output, host_output)
    torch.cuda.synchronize()
    assert attention.take_status() == 0
    assert torch.equal(host_output, expected.cpu())
