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
