"""The order in which the kernels that are launched behind one another (launch_behind) do what they
owe one another, read from their sources: broken, it shows as a hang or a stale read on some other
device or at some other size, if at all.
"""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "mmh3_b200" / "csrc"


def kernels():
    """(name, body without comments) of every __global__ function."""
    for path in sorted(CSRC.glob("*.cu")):
        source = re.sub(r"//[^\n]*", "", path.read_text())
        for start in re.finditer(r"__global__ void", source):
            # Attributes with arguments come before the name: the parameter list is the last pair of
            # parentheses before the body.
            brace = source.index("{", start.end())
            name = re.findall(r"(\w*kernel\w*)\s*\(", source[start.end():brace])[-1]
            depth, end = 0, brace
            while True:
                depth += {"{": 1, "}": -1}.get(source[end], 0)
                end += 1
                if depth == 0:
                    break
            yield name, source[brace:end]


def behind():
    found = [(name, body) for name, body in kernels() if "wait_for_kernels_before" in body]
    assert {name for name, _ in found} == {"dense_bf16_kernel", "quantized_dense_kernel",
                                           "int8_gemm_kernel", "inputs_kernel",
                                           "value_scales_kernel"}
    return found


@pytest.mark.parametrize("name,body", behind(), ids=lambda value: value if "{" not in value else "")
def test_tensor_memory_changes_hands_without_a_circle(name, body):
    """A CTA takes tensor memory when the kernels before have ended, and the next kernel may begin when
    every CTA has its own: a CTA of the next one beside it cannot have taken the columns first and wait
    for it."""
    assert body.count("let_next_kernel_begin()") == 1
    assert body.count("wait_for_kernels_before()") == 1
    if "tmem_alloc" not in body:
        return
    begin = body.index("let_next_kernel_begin()")
    wait = body.index("wait_for_kernels_before()")
    first = body.index("tmem_alloc")
    last = body.rindex("tmem_alloc")
    barrier = body.index("__syncthreads", last)
    assert wait < first <= last < barrier < begin


# What each kernel reads through the read-only path of what a kernel before it may have written.
READ_ONLY = {
    "dense_bf16_kernel": {"rope.angles": "behind"},
    "quantized_dense_kernel": {"query_scales[": "behind", "= key_scales +": "behind",
                               "value_scales[": "behind"},
    # Rows and columns follow from the tile, which follows from the wait.
    "int8_gemm_kernel": {"tile = first_tile +": "behind"},
    "inputs_kernel": {"block = blockIdx.x +": "wait_for_kernels_before()"},
    "value_scales_kernel": {"block = threadIdx.x +": "wait_for_kernels_before()"},
}


@pytest.mark.parametrize("name,body", behind(), ids=lambda value: value if "{" not in value else "")
def test_read_only_loads_follow_from_the_wait(name, body):
    """A read-only load may be moved before an asm statement that clobbers memory, but not before the
    value its address is made of: the zero that the wait returns is in each of them."""
    assert not re.search(r"[;{}]\s*wait_for_kernels_before\(\);", body)
    for begin, token in READ_ONLY[name].items():
        places = [match.start() for match in re.finditer(re.escape(begin), body)]
        assert places, begin
        for place in places:
            statement = body[place:body.index(";", place)]
            assert token in statement, statement
