"""The raster's triangle order (csrc/bfx_raster_order.h, host-only, compiled with g++): a permutation
whose first eighth is every eighth triangle along the curve, whatever the coordinates are, and false
instead of an exception where host memory is missing.  CPU only."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numi-gpu-physics_b200", "csrc")
DRIVER = r'''
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "bfx_raster_order.h"
using namespace bfx;
static int fail_at = -1, news = 0;
void* operator new[](size_t n, const std::nothrow_t&) noexcept { return news++ == fail_at ? nullptr : std::malloc(n); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete[](void* p, size_t) noexcept { std::free(p); }
#define CHECK(c) do { if (!(c)) { std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c); return 1; } } while (0)
static int check(uint32_t nv, uint32_t nt, float special) {
    std::vector<float> pts(3 * nv);
    std::vector<uint32_t> tris(3 * nt);
    std::vector<uint8_t> segment(nv);
    uint32_t x = 12345;
    auto next = [&] { return x = x * 1664525u + 1013904223u, x >> 8; };
    for (float& p : pts) p = (float)(next() % 2000) * 0.01f - 10.0f;
    if (special == special) pts[4] = special; else pts[5] = special;
    for (uint32_t& t : tris) t = next() % nv;
    for (uint32_t i = 0; i < nv; ++i) segment[i] = (uint8_t)(next() % 3);
    bfx_mesh m;
    std::memset(&m, 0, sizeof(m));
    m.local_vertices = pts.data();
    m.vertex_segment = segment.data();
    m.vertex_count = nv;
    m.triangles = tris.data();
    m.triangle_count = nt;
    RasterOrder o;
    fail_at = -1;
    CHECK(o.build(&m));
    std::vector<char> seen(nt, 0);
    for (uint32_t i = 0; i < nt; ++i) {
        const RasterOrder::Triangle& t = o.triangles()[i];
        CHECK(t.id < nt && !seen[t.id]);
        seen[t.id] = 1;
        CHECK(std::memcmp(t.vertex, tris.data() + 3 * t.id, 12) == 0);
    }
    // within the two passes the segments ascend
    const uint32_t first = (nt + 7) / 8;
    for (uint32_t i = 1; i < nt; ++i)
        if (i != first) CHECK(segment[o.triangles()[i - 1].vertex[0]] <= segment[o.triangles()[i].vertex[0]]);
    for (int k = 0; k < 2; ++k) {
        fail_at = k;
        news = 0;
        RasterOrder none;
        CHECK(!none.build(&m));
    }
    return 0;
}
int main() {
    const float inf = INFINITY;
    const uint32_t sizes[] = {0, 1, 7, 8, 9, 64, 1000};
    for (uint32_t n : sizes)
        if (check(50, n, 3.0f) || check(50, n, inf) || check(50, n, -inf) || check(50, n, NAN)) return 1;
    std::printf("OK\n");
    return 0;
}
'''


def test_raster_order_is_a_permutation_and_throws_nothing(tmp_path):
    src, exe = tmp_path / "o.cpp", tmp_path / "o"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fno-exceptions", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
