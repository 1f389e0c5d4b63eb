"""The cache of encoded tensor maps, compiled by itself with the host compiler: as many buffers as it has entries are encoded once
each, whatever a call needs of a buffer, and what a call was given stays valid for the call."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "map_cache.h"
using namespace eider::gemm;

struct Maps { int rows128, rows64, rows32; };  // (stand-ins for what the grouped GEMM encodes of one buffer)
static int made = 0;
static int make(int buffer, Maps* m) {
    if (buffer < 0) return 1;
    *m = {3 * buffer, 3 * buffer + 1, 3 * buffer + 2};
    ++made;
    return 0;
}
static FifoCache<Maps> cache;  // (zero-initialized as in a plan)
static char memory[64];
static const Maps* get(int buffer, int status = 0) {
    const Maps* out = nullptr;
    const MapKey key{buffer < 0 ? nullptr : memory + buffer, 128, 64, 64, 128};
    const MapKey bad{memory + 63, 1, 64, 64, 128};
    if (cache.get(&out, buffer < 0 ? bad : key, [&](Maps* m) { return make(buffer, m); }) != status) return nullptr;
    return out;
}
#define CHECK(x) if (!(x)) { std::printf("line %d\n", __LINE__); return 1; }
int main() {
    for (int round = 0; round < 10; ++round)
        for (int b = 0; b < kMapEntries; ++b) {
            const Maps* m = get(b);
            CHECK(m && m->rows128 == 3 * b && m->rows64 == 3 * b + 1 && m->rows32 == 3 * b + 2)
        }
    CHECK(made == kMapEntries)
    CHECK(get(-1, 1) == nullptr && made == kMapEntries)   // (a failure is reported and nothing is kept under its key)
    CHECK(get(-1, 1) == nullptr)
    const Maps* held = get(kMapEntries);                  // replaces the oldest
    for (int b = kMapEntries + 1; b < 2 * kMapEntries; ++b) {
        CHECK(get(b) && held->rows128 == 3 * kMapEntries)  // ... and stays while seven others are made
    }
    CHECK(get(0) && held->rows128 == 0)
    std::printf("ok\n");
    return 0;
}
"""


def test_every_buffer_is_encoded_once_and_stays_put(tmp_path):
    source, program = tmp_path / "cache.cpp", tmp_path / "cache"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "eider_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True)
    assert done.returncode == 0 and done.stdout == "ok\n", done.stdout
