// Which items of a batch may be worked on at the same time: host rules over the layout alone.
#pragma once

#include <algorithm>
#include <cstdint>
#include <utility>

#include "common.cuh"

namespace mmh3 {

// Whether the elements of an array whose innermost dimension is `span` contiguous ones are all
// different, whatever the order of its other dimensions: taken from the smallest stride up, each
// steps over all that the ones before it span. (Some arrays whose elements are different fail it.)
template <int DIMENSIONS>
bool elements_differ(int64_t span, int64_t (&&strides)[DIMENSIONS], int64_t (&&sizes)[DIMENSIONS]) {
    for (int taken = 0; taken < DIMENSIONS; taken++) {
        int next = taken;
        for (int index = taken + 1; index < DIMENSIONS; index++) {
            next = strides[index] < strides[next] ? index : next;
        }
        std::swap(strides[taken], strides[next]);
        std::swap(sizes[taken], sizes[next]);
        if (sizes[taken] > 1 && strides[taken] < span) {
            return false;
        }
        span += strides[taken] * (sizes[taken] - 1);
    }
    return true;
}

// Whether no item's output shares an element with another item's output, query, key or value, so that
// the items give the same results at the same time as one after the other. What an item's output does
// to its own operands is the same either way (over its own query it does no harm). `bases` are q, k,
// v and the output; the batch strides of q, k and v are positive.
inline bool items_are_independent(const void *const (&bases)[4], int tokens, int heads, int group,
                                  int head_dim, int batch, const Mmh3AttentionLayout &layout) {
    if (!elements_differ<3>(head_dim,
                            {layout.token_stride[OUTPUT], layout.head_stride[OUTPUT],
                             layout.batch_stride[OUTPUT]},
                            {tokens, heads, batch})) {
        return false;
    }
    // In bytes: where an operand begins, what one of its items spans, and the step to the next.
    auto begin = [&](int operand) { return reinterpret_cast<intptr_t>(bases[operand]); };
    auto span = [&](int operand) {
        const int its_heads = operand == KEY || operand == VALUE ? heads / group : heads;
        return 2 * ((tokens - 1) * layout.token_stride[operand] +
                    (its_heads - 1) * layout.head_stride[operand] + head_dim);
    };
    auto step = [&](int operand) { return 2 * layout.batch_stride[operand]; };
    auto end = [&](int operand) {
        return begin(operand) + (batch - 1) * step(operand) + span(operand);
    };
    for (int operand = 0; operand < 3; operand++) {
        // Apart altogether: the usual case.
        if (end(OUTPUT) <= begin(operand) || end(operand) <= begin(OUTPUT)) {
            continue;
        }
        // Item by item in one window that steps over itself, such as [batch][tokens][q | k | v] with
        // the output in the place of q.
        if (step(OUTPUT) == step(operand) &&
            std::max(begin(OUTPUT) + span(OUTPUT), begin(operand) + span(operand)) -
                    std::min(begin(OUTPUT), begin(operand)) <=
                step(operand)) {
            continue;
        }
        // With the same strides, in the same place or as the two halves of one array with different
        // elements, such as [tokens][batch][q | k | v].
        const int64_t distance = begin(OUTPUT) > begin(operand) ? begin(OUTPUT) - begin(operand)
                                                                : begin(operand) - begin(OUTPUT);
        if (layout.token_stride[OUTPUT] == layout.token_stride[operand] &&
            layout.head_stride[OUTPUT] == layout.head_stride[operand] &&
            step(OUTPUT) == step(operand) && distance % 2 == 0 &&
            (distance == 0 ||
             elements_differ<4>(head_dim,
                                {layout.token_stride[OUTPUT], layout.head_stride[OUTPUT],
                                 layout.batch_stride[OUTPUT], distance / 2},
                                {tokens, heads, batch, 2}))) {
            continue;
        }
        return false;
    }
    return true;
}

} // namespace mmh3
