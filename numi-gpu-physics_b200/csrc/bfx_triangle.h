// float3 arithmetic in the reference's operation order, and the closest point of a
// triangle (BF.metal:1529-1583), for the geometry kernels and for the host.
// Compiled without contraction of a*b+c on both sides (nvcc --fmad=false, gcc
// -ffp-contract=off), so host and device agree bit for bit.
#pragma once

#include <math.h>

#include "bfx_portable_math.h"

namespace bfx {

struct V3 {
    float x, y, z;
};
BFX_HD V3 v3(float x, float y, float z) { return V3{x, y, z}; }
BFX_HD V3 operator+(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
BFX_HD V3 operator-(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
BFX_HD V3 operator*(V3 a, float s) { return v3(a.x * s, a.y * s, a.z * s); }
BFX_HD float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
BFX_HD V3 cross(V3 a, V3 b) {
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
BFX_HD float length(V3 a) { return sqrtf(dot(a, a)); }

// Closest point of triangle (a, b, c) to p and its barycentric coordinates.  An
// edge region needs an edge: where its two end distances are equal (an edge of
// zero length, or one that rounds to it) its quotient would be 0 / 0, and the
// following regions hold the point: with a = b the edge region a-c.  Hence d3 < 0
// and d6 < 0 where the reference has <=: with d3 = 0 the region's other
// conditions leave d1 = 0 alone, as d1 d4 <= 0 and, past b's region, d4 > 0
// (likewise d6 = 0 and d2).
BFX_HD V3 closest_point(V3 p, V3 a, V3 b, V3 c, V3& bary) {
    V3 ab = b - a, ac = c - a, ap = p - a;
    float d1 = dot(ab, ap), d2 = dot(ac, ap);
    if (d1 <= 0.0f && d2 <= 0.0f) {
        bary = v3(1, 0, 0);
        return a;
    }
    V3 bp = p - b;
    float d3 = dot(ab, bp), d4 = dot(ac, bp);
    if (d3 >= 0.0f && d4 <= d3) {
        bary = v3(0, 1, 0);
        return b;
    }
    float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0f && d1 >= 0.0f && d3 < 0.0f) {
        float v = d1 / (d1 - d3);
        bary = v3(1.0f - v, v, 0);
        return v3(a.x + v * ab.x, a.y + v * ab.y, a.z + v * ab.z);
    }
    V3 cp = p - c;
    float d5 = dot(ab, cp), d6 = dot(ac, cp);
    if (d6 >= 0.0f && d5 <= d6) {
        bary = v3(0, 0, 1);
        return c;
    }
    float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0f && d2 >= 0.0f && d6 < 0.0f) {
        float w = d2 / (d2 - d6);
        bary = v3(1.0f - w, 0, w);
        return v3(a.x + w * ac.x, a.y + w * ac.y, a.z + w * ac.z);
    }
    float va = d3 * d6 - d5 * d4;
    if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f && (d4 - d3) + (d5 - d6) > 0.0f) {
        float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        bary = v3(0, 1.0f - w, w);
        return v3(b.x + w * (c.x - b.x), b.y + w * (c.y - b.y), b.z + w * (c.z - b.z));
    }
    float inv = 1.0f / fmaxf(va + vb + vc, 1.0e-20f);
    float v = vb * inv, w = vc * inv;
    bary = v3(1.0f - v - w, v, w);
    return v3(a.x + ab.x * v + ac.x * w, a.y + ab.y * v + ac.y * w, a.z + ab.z * v + ac.z * w);
}

// |p - closest_point(p)| without branches: the region is decided by the same
// comparisons in the same order, and its one division, edge and base point are
// selected, so the value equals closest_point's bit for bit (an unused term
// adds a zero).  A warp whose lanes fall in different regions runs one path
// instead of up to seven, each with its own division.
BFX_HD float closest_distance(V3 p, V3 a, V3 b, V3 c) {
    const V3 ab = b - a, ac = c - a, ap = p - a, bp = p - b, cp = p - c;
    const float d1 = dot(ab, ap), d2 = dot(ac, ap), d3 = dot(ab, bp), d4 = dot(ac, bp), d5 = dot(ab, cp),
                d6 = dot(ac, cp);
    const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
    const bool in_a = d1 <= 0.0f && d2 <= 0.0f;
    const bool in_b = d3 >= 0.0f && d4 <= d3;
    const bool on_ab = vc <= 0.0f && d1 >= 0.0f && d3 < 0.0f;
    const bool in_c = d6 >= 0.0f && d5 <= d6;
    const bool on_ac = vb <= 0.0f && d2 >= 0.0f && d6 < 0.0f;
    const bool on_bc =
        va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f && (d4 - d3) + (d5 - d6) > 0.0f;
    // 0 a, 1 b, 2 ab, 3 c, 4 ac, 5 bc, 6 face
    const int r = in_a ? 0 : (in_b ? 1 : (on_ab ? 2 : (in_c ? 3 : (on_ac ? 4 : (on_bc ? 5 : 6)))));
    const float num = r == 2 ? d1 : (r == 4 ? d2 : (r == 5 ? d4 - d3 : 1.0f));
    const float den = r == 2 ? d1 - d3
                             : (r == 4 ? d2 - d6
                                       : (r == 5 ? (d4 - d3) + (d5 - d6)
                                                 : (r == 6 ? fmaxf(va + vb + vc, 1.0e-20f) : 1.0f)));
    const float quot = num / den;
    const float s = r == 6 ? vb * quot : (r == 2 || r == 4 || r == 5 ? quot : 0.0f);
    const float t = r == 6 ? vc * quot : 0.0f;
    const V3 base = r == 1 || r == 5 ? b : (r == 3 ? c : a);
    const V3 e = r == 4 ? ac : (r == 5 ? c - b : ab);
    const V3 d = v3(p.x - (base.x + e.x * s + ac.x * t), p.y - (base.y + e.y * s + ac.y * t),
                    p.z - (base.z + e.z * s + ac.z * t));
    return length(d);
}

}  // namespace bfx
