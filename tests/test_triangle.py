"""The triangle distance of the raster and the link search (csrc/bfx_triangle.h, compiled with g++ as
the library's host side is): closest_distance equals |p - closest_point| bit for bit, and both hold a
finite distance for triangles without area.  CPU only."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numi-gpu-physics_b200", "csrc")
SOURCE = r'''
#include "bfx_triangle.h"
using namespace bfx;
static V3 at(const float* p) { return v3(p[0], p[1], p[2]); }
extern "C" void distances(const float* p, const float* tri, long n, float* branchless, float* literal, float* bary) {
    for (long i = 0; i < n; ++i) {
        const V3 q = at(p + 3 * i), a = at(tri + 9 * i), b = at(tri + 9 * i + 3), c = at(tri + 9 * i + 6);
        V3 w;
        literal[i] = length(q - closest_point(q, a, b, c, w));
        branchless[i] = closest_distance(q, a, b, c);
        bary[3 * i] = w.x;
        bary[3 * i + 1] = w.y;
        bary[3 * i + 2] = w.z;
    }
}
'''
N = 300_000


@pytest.fixture(scope="module")
def distances(tmp_path_factory):
    d = tmp_path_factory.mktemp("triangle")
    src, so = d / "t.cpp", d / "t.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def call(p, tri):
        p, tri = np.ascontiguousarray(p, np.float32), np.ascontiguousarray(tri, np.float32)
        out = np.empty(len(p), np.float32), np.empty(len(p), np.float32), np.empty((len(p), 3), np.float32)
        lib.distances(*(ctypes.c_void_p(v.ctypes.data) for v in (p, tri)), ctypes.c_long(len(p)),
                      *(ctypes.c_void_p(v.ctypes.data) for v in out))
        return out
    return call


def unit(rng, n):
    u = rng.standard_normal((n, 3))
    return u / np.linalg.norm(u, axis=1)[:, None]


def triangles(rng, size, aspect, offset):
    """Triangles of longest edge about `size`, a height or a shortest edge of size * aspect, vertices in
    random order, and cell centres around them."""
    a = offset + rng.uniform(0, 32, (N, 3))
    u, w = unit(rng, N), unit(rng, N)
    kind = rng.integers(0, 3, N)[:, None]
    b = a + size * u
    c = np.where(kind == 0, a + u * size * rng.uniform(0, 1, (N, 1)) + w * size * aspect,
                 np.where(kind == 1, a + w * size * aspect, b + w * size * aspect))
    order = (np.arange(3)[None] + rng.integers(0, 3, (N, 1))) % 3
    tri = np.stack([a, b, c], 1).astype(np.float32)[np.arange(N)[:, None], order]
    p = np.floor(tri.mean(1) + rng.uniform(-1, 1, (N, 3)) * (size + 4.0)) + 0.5
    return p.astype(np.float32), tri


def exact(p, tri):
    """Distance in FP64: the plane's foot where it lies inside, else the nearest of the three segments."""
    p, (a, b, c) = p.astype(np.float64), np.moveaxis(tri.astype(np.float64), 1, 0)

    def segment(s, e):
        d, l2 = e - s, ((e - s) ** 2).sum(1)
        t = np.clip(np.divide(((p - s) * d).sum(1), l2, out=np.zeros(len(p)), where=l2 > 0), 0, 1)
        return np.linalg.norm(p - s - t[:, None] * d, axis=1)
    best = np.minimum(segment(a, b), np.minimum(segment(b, c), segment(c, a)))
    n = np.cross(b - a, c - a)
    n2 = (n * n).sum(1)
    inside = n2 > 0
    for s, e in ((a, b), (b, c), (c, a)):
        inside &= (np.cross(e - s, p - s) * n).sum(1) >= 0
    height = np.abs(((p - a) * n).sum(1)) / np.sqrt(np.where(n2 > 0, n2, 1.0))
    return np.where(inside, height, best)


@pytest.mark.parametrize("offset", [0.0, 300.0])
@pytest.mark.parametrize("size", [0.05, 0.5, 4.0, 40.0])
@pytest.mark.parametrize("aspect", [0.7, 1e-2, 1e-4, 1e-6, 0.0])
def test_branchless_distance_is_the_literal_one(distances, size, aspect, offset):
    rng = np.random.default_rng(int(size * 1000) + int(-np.log10(aspect + 1e-9)))
    p, tri = triangles(rng, size, aspect, offset)
    got, literal, bary = distances(p, tri)
    assert np.isfinite(got).all() and np.isfinite(bary).all()
    assert np.array_equal(got, literal)


def test_coincident_vertices_leave_the_edge(distances):
    rng = np.random.default_rng(5)
    p, tri = triangles(rng, 2.0, 0.5, 0.0)
    for keep in ((0, 0, 1), (0, 1, 0), (1, 0, 0), (0, 0, 0)):
        flat = tri[:, list(keep)]
        got, literal, bary = distances(p, flat)
        assert np.array_equal(got, literal) and (bary >= 0).all()
        want = exact(p, flat)
        reach = np.linalg.norm(p[:, None].astype(np.float64) - flat, axis=2).max(1)
        assert (np.abs(got - want) <= 64 * 2.0 ** -24 * (reach + 2.0)).all()
