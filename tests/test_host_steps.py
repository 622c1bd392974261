"""The host-side sequences of csrc/host_steps.h, compiled alone, with steps and allocations that fail."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lambent_b200", "csrc")


@pytest.fixture
def run(tmp_path):
    def compile_and_run(body):
        src, exe = tmp_path / "t.cpp", tmp_path / "t"
        src.write_text('#include <cstdio>\n#include <vector>\n#include "host_steps.h"\nusing namespace lam;\n'
                       "int main() {\n" + body + "\n}\n")
        subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, "-o", str(exe), str(src)], check=True)
        return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    return compile_and_run


@pytest.mark.parametrize("fails,taken,status", [(-1, "0123", 0), (0, "0", 7), (1, "01", 7), (3, "0123", 7)])
def test_no_step_after_one_that_failed(run, fails, taken, status):
    """A ray query's second kernel indexes triangles with what the first one wrote."""
    out = run(f"""
        enum Status {{ OK = 0, BAD = 7 }};
        Steps<Status> go;
        for (int k = 0; k < 4; ++k) go([&] {{ std::printf("%d", k); return k == {fails} ? BAD : OK; }});
        std::printf(" %d", (int)go.status);""")
    assert out == [taken, str(status)]


@pytest.mark.parametrize("room,want", [(0, "3 1 1"), (15, "3 1 1"), (16, "0 0 0")])
def test_a_pair_is_allocated_whole_or_not_at_all(run, room, want):
    """The class order's two lists: with one of them alone, the next batch wrote through the other."""
    out = run(f"""
        std::vector<int> store(16);
        int *a = nullptr, *b = nullptr;
        int rc = alloc_pair(&a, &b, 8, [&](int** p, size_t n) {{
            if (n > {room}) return 3;
            *p = store.data();
            return 0;
        }});
        std::printf("%d %d %d", rc, a == nullptr, b == nullptr);
        return a && b != a + 8;""")
    assert " ".join(out) == want


@pytest.mark.parametrize("fits,tried,status", [(148, "148", 0), (147, "148,74", 0), (40, "148,74,37", 0),
                                               (0, "148,74,37,19,10,5,3,2,1", 9), (-1, "148", 4)])
def test_a_grid_that_must_be_resident_shrinks_to_fit(run, fits, tried, status):
    """Training on a partition of the device with fewer multiprocessors; other errors (-1) stay."""
    out = run(f"""
        enum Status {{ OK = 0, OTHER = 4, TOO_LARGE = 9 }};
        const Status s = launch_resident(148u, TOO_LARGE, [](unsigned grid) {{
            std::printf(grid == 148 ? "%u" : ",%u", grid);
            return {fits} < 0 ? OTHER : (int)grid <= {fits} ? OK : TOO_LARGE;
        }});
        std::printf(" %d", (int)s);""")
    assert out == [tried, str(status)]
