"""Device arrays laid out in one block (csrc/arena.h), compiled alone, with an allocator that runs out."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lambent_b200", "csrc")

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "arena.h"
using namespace lam;
int main(int, char** argv) {
    const size_t limit = strtoull(argv[1], nullptr, 0), room = strtoull(argv[2], nullptr, 0), n = strtoull(argv[3], nullptr, 0);
    size_t given = 0, calls = 0;
    uintptr_t next = 1u << 20;
    // an address of its own for each allocation of at most `limit` bytes, `room` in all
    ArenaAlloc alloc = [&](void** p, size_t bytes) {
        ++calls;
        if (bytes > limit || given + bytes > room) return 3;
        given += bytes;
        *p = reinterpret_cast<void*>(next);
        next += (bytes + 0xFFFFFu) / 0x100000u * 0x100000u + (uintptr_t(1) << 32);
        return 0;
    };
    double *a, *d;
    uint32_t* b;
    char* c;
    auto layout = [&](Arena& m) {
        m.take(&a, n);
        m.take(&b, n + 1);
        m.take(&c, 0);
        m.take(&d, 2 * n);
    };
    const int rc = place(alloc, layout);
    struct { uintptr_t at; size_t bytes; } s[] = {{(uintptr_t)a, 8 * n}, {(uintptr_t)b, 4 * (n + 1)}, {(uintptr_t)d, 16 * n}};
    bool apart = true, aligned = true;
    for (int i = 0; i < 3; ++i) {
        aligned = aligned && s[i].at % 256 == 0;
        for (int j = 0; j < i; ++j) apart = apart && (s[i].at + s[i].bytes <= s[j].at || s[j].at + s[j].bytes <= s[i].at);
    }
    std::printf("%d %zu %d %d %d %d", rc, calls, apart, aligned, c == nullptr, given == arena_bytes(layout));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("arena")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, "-o", str(d / "t"), str(d / "t.cpp")], check=True)
    return str(d / "t")


NO_LIMIT = 1 << 60


@pytest.mark.parametrize("limit,room,n,want", [
    (NO_LIMIT, NO_LIMIT, 1 << 20, "0 1 1 1 1 1"),      # one block, of the measured size
    (NO_LIMIT, NO_LIMIT, 1000, "0 3 1 1 1 0"),         # small arrays one by one
    (20 << 20, NO_LIMIT, 1 << 20, "0 4 1 1 1 0"),      # no block of 28 MB: one by one
    (20 << 20, 13 << 20, 1 << 20, "3 4"),              # nor room for all of them
    (NO_LIMIT, 100, 1000, "3 1"),
])
def test_place(program, limit, room, n, want):
    out = subprocess.run([program, str(limit), str(room), str(n)], check=True, capture_output=True, text=True).stdout
    assert out.split()[:len(want.split())] == want.split()
