// jacobi_tiles.h — the tiles of the resident Jacobi sweeps (jacobi_resident.cu).  Host arithmetic.
#pragma once

#include <algorithm>
#include <cstddef>

namespace shg {

constexpr size_t kResSmem = 208 * 1024;  // of a tile: 26 planes of 1024 FP64 voxels, 52 of FP32

struct ResidentTiles {
    int ytiles, tz, ztiles;  // tiles along y, planes per tile (the last may have fewer), tiles along z
};

// Tiles of an n x n x nz grid of `real`-byte voxels: rows of 1024 / n (side a power of two, 32 to
// 256, so that 256 threads of 2 x 2 voxels cover a tile's plane) by enough planes for one CTA on each
// of `sms` multiprocessors.  False where a tile outgrows the shared memory, or where the tiles are
// more than the `resident` CTAs that a cooperative launch may have.
inline bool resident_tiles(size_t real, int n, int nz, int sms, int resident, ResidentTiles* t) {
    if ((n != 32 && n != 64 && n != 128 && n != 256) || nz < 1 || sms < 1) return false;
    t->ytiles = n / (1024 / n);
    const int zt = std::max(1, std::min(nz, sms / t->ytiles));
    t->tz = (nz + zt - 1) / zt;
    t->ztiles = (nz + t->tz - 1) / t->tz;
    return real * 1024 * (size_t)t->tz <= kResSmem && t->ytiles * t->ztiles <= resident;
}

}  // namespace shg
