// sp_column.cuh -- the interior sweep of the pointwise kernels (conversions,
// corrections, error sums, widening).
#pragma once

#include <cuda_runtime.h>

#include "sp_internal.h"

namespace sp {

// A block of 32 x 8 threads takes a 32 x 8 patch of (x, y) columns, thread
// (tx, ty) the cells of one column at z = blockIdx.y, blockIdx.y + gridDim.y, ...
// These kernels are bound by memory (L2 for fields below ~100 MB), so a thread
// has to reach its cell in a few instructions: with one flat index per cell,
// split by three 64-bit divisions, converting a 128^3 field took 17-19 us, with
// the columns 10 us.  The grid is `waves` waves of full SMs (8 blocks of 256
// threads per SM): one where every block ends in atomics on the same few words.
constexpr int kColX = 32, kColY = 8;

inline dim3 column_grid(const Geo& g, int items = 1, unsigned waves = 1) {
    const unsigned tiles = (unsigned)((g.ni + kColX - 1) / kColX) * (unsigned)((g.nj + kColY - 1) / kColY);
    const unsigned per = tiles * (unsigned)items, want = 148u * 8u * waves;
    const unsigned nz = per >= want ? 1u : want / per;
    return dim3(tiles, nz < (unsigned)g.nk ? nz : (unsigned)g.nk, (unsigned)items);
}

template <typename F>
__device__ __forceinline__ void for_column(const Geo& g, F&& cell) {
    const int tiles_x = (g.ni + kColX - 1) / kColX;
    const int ty = blockIdx.x / tiles_x;
    const int x = (blockIdx.x - ty * tiles_x) * kColX + threadIdx.x;
    const int y = ty * kColY + threadIdx.y;
    if (x >= g.ni || y >= g.nj) return;
    for (int z = blockIdx.y; z < g.nk; z += gridDim.y) cell(x, y, z);
}

__device__ __forceinline__ long long cell_at(const Geo& g, int x, int y, int z) {
    return g.origin + z * g.plane + y * g.px + x;
}

}  // namespace sp
