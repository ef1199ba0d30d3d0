// Host-only: the order in which the mesh raster takes the triangles (no CUDA, so
// that it can be tested without a GPU; throws nothing, as it runs below a C entry).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <memory>
#include <new>

#include "../../include/bfx.h"

namespace bfx {

// The triangles (vertices, id) along a Morton curve of the centroid within each
// segment (10 bits an axis of the segment-frame coordinates, the first keyframe's
// for a replay), every eighth triangle of the curve first.  Those leave a key near
// the final one in almost every voxel, which lets the others drop most of theirs;
// the order changes no result.
class RasterOrder {
  public:
    struct Triangle {
        uint32_t vertex[3], id;
    };
    // false: no host memory
    bool build(const bfx_mesh* m) {
        const uint32_t n = m->triangle_count;
        struct Keyed {
            uint64_t code;
            uint32_t triangle;
        };
        std::unique_ptr<Keyed[]> keyed(new (std::nothrow) Keyed[(size_t)n + 1]);
        order_.reset(new (std::nothrow) Triangle[(size_t)n + 1]);
        if (!keyed || !order_) return false;
        const float* pts = m->keyframe_count >= 2 ? m->keyframe_points : m->local_vertices;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (uint32_t i = 0; i < m->vertex_count; ++i)
            for (int k = 0; k < 3; ++k) {
                lo[k] = std::min(lo[k], pts[3 * (size_t)i + k]);
                hi[k] = std::max(hi[k], pts[3 * (size_t)i + k]);
            }
        // one scale for the three axes, so that the curve's cells are cubes
        const float extent = std::max(hi[0] - lo[0], std::max(hi[1] - lo[1], hi[2] - lo[2]));
        const float scale = extent > 0.0f ? 1023.0f / (3.0f * extent) : 0.0f;
        const auto spread = [](uint32_t v) {
            uint64_t r = 0;
            for (int b = 0; b < 10; ++b) r |= (uint64_t)((v >> b) & 1u) << (3 * b);
            return r;
        };
        for (uint32_t t = 0; t < n; ++t) {
            const uint32_t* v = m->triangles + 3 * (size_t)t;
            const float *a = pts + 3 * (size_t)v[0], *b = pts + 3 * (size_t)v[1], *c = pts + 3 * (size_t)v[2];
            uint64_t code = (uint64_t)m->vertex_segment[v[0]] << 32;
            for (int k = 0; k < 3; ++k) {
                const float f = ((a[k] - lo[k]) + (b[k] - lo[k]) + (c[k] - lo[k])) * scale;
                const uint32_t i = f >= 0.0f ? (uint32_t)std::min(f, 1023.0f) : 0u;  // a NaN counts as 0
                code |= spread(i) << k;
            }
            keyed[t] = {code, t};
        }
        std::sort(keyed.get(), keyed.get() + n, [](const Keyed& x, const Keyed& y) {
            return x.code != y.code ? x.code < y.code : x.triangle < y.triangle;
        });
        size_t at = 0;
        for (int rest = 0; rest < 2; ++rest)
            for (size_t i = 0; i < n; ++i)
                if ((i % 8 != 0) == (rest != 0)) {
                    const uint32_t t = keyed[i].triangle;
                    const uint32_t* v = m->triangles + 3 * (size_t)t;
                    order_[at++] = {{v[0], v[1], v[2]}, t};
                }
        return true;
    }
    const Triangle* triangles() const { return order_.get(); }

  private:
    std::unique_ptr<Triangle[]> order_;
};

}  // namespace bfx
