// diffsoup_b200/csrc/rows.cuh -- short per-pixel rows moved by whole warps.
#pragma once

#include "common.cuh"

namespace dsb {

// Warp-wide copy between 32 rows of K floats, lane's row at tile + lane * K, and
// `live` consecutive rows at g (16-byte aligned when all 32 are live).
template <bool STORE>
__device__ __forceinline__ void warp_rows(float* tile, float* g, int K, int live) {
    const int lane = threadIdx.x & 31;
    if (!STORE) __syncwarp();
    if (live == 32 && ((uintptr_t)g & 15) == 0) {
        for (int i = lane; i < 8 * K; i += 32) {
            float4* t = reinterpret_cast<float4*>(tile) + i;
            float4* o = reinterpret_cast<float4*>(g) + i;
            if (STORE) *o = *t; else *t = __ldg(o);
        }
    } else {
        for (int i = lane; i < live * K; i += 32) {
            if (STORE) g[i] = tile[i]; else tile[i] = __ldg(g + i);
        }
    }
    __syncwarp();
}

}  // namespace dsb
