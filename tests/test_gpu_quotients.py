"""The corrected quotients of device_math.cuh and traverse.cuh as the device computes them: the bits of the
division for every argument, zeros, infinities and NaN among them."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "lambent_b200", "csrc")


def test_corrected_quotients_have_the_bits_of_the_division(cuda, tmp_path):
    so = str(tmp_path / "quotients.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o", so, os.path.join(HERE, "data", "quotients.cu")],
                   check=True)
    edge = [0x00000000, 0x80000000, 0x7F800000, 0xFF800000, 0x7FC00000, 0x00000001, 0x80000001, 0x007FFFFF, 0x00800000,
            0x7F7FFFFF, 0xFF7FFFFF, 0x3F800000, 0xBF800000]
    counts = (C.c_ulonglong * 4)()
    assert C.CDLL(so).run(counts, (C.c_uint32 * len(edge))(*edge), len(edge)) == 0
    assert list(counts) == [0, 0, 0, 0]
