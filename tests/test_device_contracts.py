"""Rules of the device sources that no run shows: what holds today by the compiler's or the hardware's
grace would break silently."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lambent_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("name", ["wavefront.cu", "scene.cu"])
def test_kernels_that_read_one_another_are_launched_in_a_chain(name):
    """A wave's kernels take queue lengths and triangle slots from the kernels before them, whose
    launches may fail: all go through Launches, which stops at the first failure."""
    text = source(name)
    assert "launch_next(" not in text
    assert "<<<" not in text
    assert ".next(" in text


def functions(text):
    """(signature, body) of every kernel definition."""
    for m in re.finditer(r"__global__ void[^{;]*\{", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(0), text[m.end():k]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_dependent_kernels_read_other_kernels_output_by_plain_loads(name):
    """A kernel that waits for the previous one exists while that one writes, so what it reads is not
    read-only for its lifetime: no const __restrict__ parameter, and __ldg for the scene alone."""
    for head, body in functions(source(name)):
        if "wait_previous()" not in body:
            continue
        assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", head), head
        for arg in re.findall(r"__ldg\(([^;]*)", body):
            assert re.match(r"(tp\b|S[.\[]|reinterpret_cast<const uint32_t\*>\(S\[q\]->materials)", arg), (head, arg)


def test_block_barriers_are_not_in_functions_that_halves_of_a_block_call_apart():
    """head_grad<0> and head_grad<1> run at once in the two halves of a block: __syncthreads in one
    and __syncthreads in the other are different barriers to the language."""
    text = source("guide_net.cuh")
    body = text[text.index("float head_grad("):]
    body = body[:body.index("\n}")]
    assert "__syncthreads" not in body and "halves_meet();" in body
