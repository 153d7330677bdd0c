// cell_block.cuh -- thread-to-cell mapping of the per-cell kernels: a block of
// 32 * ROWS threads takes 32 cells along j (one warp, one 256-byte line per
// plane row) by ROWS rows along i.  Neighbouring rows' loads then meet in L1,
// and a cell's indices cost one 32-bit division per block; a flat index over
// nx * ny costs a 64-bit division per thread and splits its warps over rows.
#pragma once

#include <cuda_runtime.h>

#include "rmhd2d_internal.h"

namespace rmhd2d {

template <int ROWS> struct CellBlock {
    static constexpr int THREADS = 32 * ROWS;
    static __host__ __device__ __forceinline__ unsigned blocks(const Grid &g)
    {
        return (unsigned)((g.ny + 31) / 32) * (unsigned)((g.nx + ROWS - 1) / ROWS);
    }
    // The calling thread's cell; false beyond the array.
    static __device__ __forceinline__ bool cell(const Grid &g, int &i, int &j)
    {
        const unsigned across = (unsigned)(g.ny + 31) / 32u, bi = blockIdx.x / across;
        j = (int)((blockIdx.x - bi * across) * 32u + (threadIdx.x & 31u));
        i = (int)(bi * ROWS + (threadIdx.x >> 5));
        return i < g.nx && j < g.ny;
    }
};

}  // namespace rmhd2d
