// mixed_solve.cuh -- FP32 parts of the mixed Fermat solve, shared by the back-projection
// (k_mixed.cu) and the crossing points (k_crossings.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "kernels.hpp"
#include "node_lists.cuh"

namespace bsar {

struct Facet32 {
    float x0, y0, dx, dy, z00, b, c, e;
    float idx, idy;     // 1 / dx, 1 / dy
};

struct MixedCtx : ListGrid {
    const float* __restrict__ z32;  // pitch-padded FP32 heights, z32[j * pitch + i]
    int pitch;
    double ox, oy, oz;              // origin of the FP32 frame (first DEM node, DemView::z0)
    double idx64, idy64;            // 1 / spacing, FP64
    int lists;                      // node scans may run on candidate lists
};

__device__ __forceinline__ float zf(const MixedCtx& m, int i, int j) { return __ldg(m.z32 + (int64_t)j * m.pitch + i); }

// FP32 bilinear height (clamped to the DEM) for the flat-interface start.
__device__ __forceinline__ float height32(const MixedCtx& m, float x, float y)
{
    float fx = x * m.istepx, fy = y * m.istepy;
    int i = min(max((int)floorf(fx), 0), m.nx - 2);
    int j = min(max((int)floorf(fy), 0), m.ny - 2);
    float u = fminf(fmaxf(fx - (float)i, 0.f), 1.f), v = fminf(fmaxf(fy - (float)j, 0.f), 1.f);
    float z00 = zf(m, i, j), z01 = zf(m, i + 1, j), z10 = zf(m, i, j + 1), z11 = zf(m, i + 1, j + 1);
    return z00 + (z01 - z00) * u + (z10 - z00) * v + (z11 - z01 - z10 + z00) * u * v;
}

// Branch-free update of a node ranking: best value / position and runner-up value.  G is the
// voxel-side endpoint of the path (index ng), E the other one (index ne); the scans rank
// L' = re |N-E| + |N-G| = L / ng with re = ne / ng.
__device__ __forceinline__ void rank(float L, int i, int j, float& v1, float& v2, int& bi, int& bj)
{
    v2 = fminf(v2, fmaxf(v1, L));
    bool p = L < v1;
    v1 = p ? L : v1;
    bi = p ? i : bi;
    bj = p ? j : bj;
}

struct Rank {
    float v1, v2;
    int bi, bj;
};

}  // namespace bsar
