"""The rule by which a batch of dense attention goes in one launch (items_are_independent), against the
sets of elements that the items read and write. It looks at addresses and strides alone, so that it
runs without a GPU.
"""

import ctypes
import itertools
import random

import pytest

from mmh3_b200 import _lib, attention

BASE = 1 << 20


def rule(bases, tokens, heads, group, head_dim, batch, strides):
    """`bases` in elements; `strides` (token, head, batch) of q, k, v and the output."""
    function = ctypes.CDLL(str(_lib.SELFTEST_LIBRARY)).mmh3_b200_batch_items_selftest
    function.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_int] * 5 + [ctypes.c_void_p]
    function.restype = ctypes.c_int
    layout = attention.make_layout(*zip(*strides), heads_per_key_value=group)
    return bool(function(*(BASE + 2 * base for base in bases), tokens, heads, group, head_dim, batch,
                         ctypes.byref(layout)))


def elements(base, tokens, heads, head_dim, strides, item):
    token_stride, head_stride, batch_stride = strides
    return {base + item * batch_stride + token * token_stride + head * head_stride + index
            for token, head, index in itertools.product(range(tokens), range(heads),
                                                        range(head_dim))}


def independent(bases, tokens, heads, group, head_dim, batch, strides):
    written = [elements(bases[3], tokens, heads, head_dim, strides[3], item) for item in range(batch)]
    for item in range(batch):
        touched = set(written[item])
        for operand in range(3):
            touched |= elements(bases[operand], tokens, heads if operand == 0 else heads // group,
                                head_dim, strides[operand], item)
        if any(touched & written[other] for other in range(batch) if other != item):
            return False
    return True


def packed(order, sizes, head_dim, gap):
    """Strides (token, head, batch) of an array whose dimensions are `order`, outermost first."""
    strides, step = {}, head_dim
    for dimension in reversed(order):
        strides[dimension] = step
        step = step * sizes[dimension] + gap
    return strides["tokens"], strides["heads"], strides["batch"]


@pytest.mark.parametrize("seed", range(8))
def test_no_batch_whose_items_meet_goes_in_one_launch(seed):
    rng = random.Random(seed)
    answers = {True: 0, False: 0}
    for _ in range(400):
        tokens, batch = rng.randint(1, 4), rng.randint(2, 4)
        group = rng.choice([1, 1, 2])
        heads = group * rng.randint(1, 2)
        head_dim = 4
        sizes = {"tokens": tokens, "heads": heads, "batch": batch}
        order = rng.sample(sorted(sizes), 3)
        gap = rng.choice([0, 0, 3])
        strides = [packed(order if rng.random() < 0.7 else rng.sample(sorted(sizes), 3), sizes,
                          head_dim, gap) for _ in range(4)]
        if rng.random() < 0.5:  # q, k, v and the output as parts of one row, or of one head
            width = rng.choice([1, 2, 3, 4])
            strides = [tuple(width * stride for stride in strides[3])] * 4
        if rng.random() < 0.1:
            strides[3] = (strides[3][0], strides[3][1], max(strides[3][2] // 2, 1))
        reach = rng.choice([8, 200, 2000])
        bases = [rng.choice([0, head_dim, 2 * head_dim, heads * head_dim, strides[3][2],
                             rng.randint(0, reach)]) for _ in range(4)]
        arguments = (bases, tokens, heads, group, head_dim, batch, strides)
        answer = rule(*arguments)
        answers[answer] += 1
        assert not answer or independent(*arguments), arguments
    assert answers[True] >= 40 and answers[False] >= 40


def test_the_usual_layouts_go_in_one_launch():
    tokens, heads, head_dim, batch = 5, 4, 64, 3
    inner = heads * head_dim
    apart = 10 ** 6
    row = (inner, head_dim, tokens * inner)
    kv = (inner // 2, head_dim, tokens * inner // 2)
    fused = (3 * inner, head_dim, 3 * tokens * inner)
    interleaved = (3 * batch * inner, head_dim, 3 * inner)
    by_head = (head_dim, batch * tokens * head_dim, tokens * head_dim)
    for group, bases, strides in [
        (2, (0, apart, 2 * apart, 3 * apart), (row, kv, kv, row)),
        (1, (0, inner, 2 * inner, apart), (fused,) * 3 + (row,)),
        (1, (0, inner, 2 * inner, 0), (fused,) * 4),              # the output in q's place
        (1, (0, inner, 2 * inner, 0), (interleaved,) * 4),
        (1, (0, apart, 2 * apart, 3 * apart), (by_head,) * 4),
        (2, (0, apart, 2 * apart, 0), (row, kv, kv, row)),        # over a query of its own
    ]:
        arguments = (bases, tokens, heads, group, head_dim, batch, strides)
        assert independent(*arguments) and rule(*arguments), (group, bases, strides)


def test_an_output_over_another_items_operands_goes_item_by_item():
    tokens, heads, head_dim, batch = 5, 2, 64, 3
    row = (heads * head_dim, head_dim, tokens * heads * head_dim)
    apart = 10 ** 6
    for operand, shift in itertools.product(range(3), (-2, -1, 1, 2)):
        bases = [apart, 2 * apart, 3 * apart, 0]
        bases[3] = bases[operand] + shift * row[2]
        arguments = (bases, tokens, heads, 1, head_dim, batch, (row,) * 4)
        assert not independent(*arguments) and not rule(*arguments), (operand, shift)
