"""The handle's growing result buffers (mnhack8_b200/csrc/hs_grow.h), on the CPU
with a fake allocator: a growth that finds no memory is refused and leaves the
buffer as it was (kernels of later calls write through it), and no memory is
given back twice or lost."""
import os
import subprocess

from tests.conftest import ROOT

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "hs_grow.h"
static size_t limit = 1 << 12;
static int live = 0;
struct Mem {
    static constexpr int ok = 0;
    static int get(void** p, size_t bytes) {
        if (bytes > limit) return 2;
        *p = std::malloc(bytes);
        ++live;
        return 0;
    }
    static void put(void* p) { std::free(p); --live; }
};
#define CHECK(c) if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; }
int main() {
    {
        hs::GrowBuf<double, Mem> b;
        CHECK(b.need(64) == 0 && b.n == 64 && b.p && live == 1);
        b.p[63] = 7.0;
        double* const p = b.p;
        CHECK(b.need(10) == 0 && b.p == p && b.n == 64 && live == 1);
        CHECK(b.need(1 << 20) == 2);                       // no memory for more
        CHECK(b.p == p && b.n == 64 && b.p[63] == 7.0 && live == 1);
        CHECK(b.need(64) == 0 && b.p == p);
        CHECK(b.need(65) == 0 && b.n == 65 && live == 1);
        b.p[64] = 1.0;
        hs::GrowBuf<int, Mem> never;
        CHECK(never.need(1 << 20) == 2 && !never.p && never.n == 0);
    }
    CHECK(live == 0);
    return 0;
}
"""


def test_growth_that_fails_leaves_the_buffer(tmp_path):
    src, exe = tmp_path / "grow.cpp", tmp_path / "grow"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "mnhack8_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
