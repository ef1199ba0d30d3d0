// Host-only: the rule that lets a step with static geometry fill its halo beside
// the link kernel (no CUDA, so that it can be tested without a GPU).
#pragma once

#include <cstddef>
#include <cstdint>

namespace bfx {

// Cells that a face needs free of solid ones for the fill beside the link
// kernel.  A link writes the slot of a fluid cell next to a solid one (or of the
// solid cell itself, in the representation before an even step), so with the
// solid cells at index 3 or more from a face it stays at 2 or more; the fill
// writes slots of index 0 or the halo, an outflow copy reads slots of index 0
// and 1, and no link's source is a periodic image.
constexpr int kFaceClearance = 3;

// No cell of the mask (bits `part`: a solid part's id) within kFaceClearance
// cells of a lattice face.
inline bool solid_clear_of_faces(const uint8_t* mask, int nx, int ny, int nz, uint8_t part) {
    const int c = kFaceClearance;
    const auto outer = [c](int i, int n) { return i < c || i >= n - c; };
    for (int z = 0; z < nz; ++z)
        for (int y = 0; y < ny; ++y) {
            const uint8_t* row = mask + (size_t)nx * ((size_t)y + (size_t)ny * (size_t)z);
            const bool whole = outer(z, nz) || outer(y, ny);
            for (int x = 0; x < nx; ++x) {
                if (!whole && x == c && nx > 2 * c) x = nx - c;
                if (row[x] & part) return false;
            }
        }
    return true;
}

}  // namespace bfx
