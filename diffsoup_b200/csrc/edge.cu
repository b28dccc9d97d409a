// diffsoup_b200/csrc/edge.cu -- silhouette/implicit edge gradients and the
// per-fragment opacity auxiliary gradient (kenji-tojo/diffsoup
// src/cuda/rasterize.cu:489-992) behind the C ABI.
#include "edge_math.cuh"

namespace dsb {

// rasterize.cu:653-903: one thread per pixel, 4 neighbours.
__global__ void __launch_bounds__(kThreads) edge_grad_kernel(int B, int H, int W, int C,
                                                             const float* __restrict__ color,
                                                             const float* __restrict__ grad_color,
                                                             const float* __restrict__ rast, int V,
                                                             const float* __restrict__ pos,
                                                             float* __restrict__ grad_pos,
                                                             const int* __restrict__ tri) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t hw = (int64_t)H * W;
    if (idx >= (int64_t)B * hw) return;
    const int b = (int)(idx / hw);
    const int y0 = (int)((idx % hw) / W), x0 = (int)((idx % hw) % W);
    EdgeAccum acc;
    const int it0 = edge_grad_pixel(b, y0, x0, H, W, C, color, grad_color, rast, pos + (size_t)b * V * 4, tri,
                                    b * hw, acc);
    if (it0 < 0 || !acc.any) return;
    float* gp = grad_pos + (size_t)b * V * 4;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int v = __ldg(tri + it0 * 3 + k);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (acc.g[k * 4 + j] != 0.f) atomicAdd(gp + (size_t)v * 4 + j, acc.g[k * 4 + j]);
    }
}

// The same for three channels: one CTA per 16x16 tile of a view, its pixels and
// their border staged in shared memory, the covered pixels compacted onto the
// first threads triangle by triangle, pairs evaluated kind by kind (edge_grad_pixel_tile) and runs of
// one triangle in a warp summed before the atomics.  Two views of 803x601, 15,000
// triangles: 189 -> 101 us (one thread per pixel ran 13.5 of 32 lanes on 98
// registers and 12 atomics a pixel).
constexpr int kEdgeTileThreads = DS_TILE * DS_TILE;

__global__ void __launch_bounds__(kEdgeTileThreads, 3) edge_grad_tile_kernel(
    int H, int W, int tiles_x, int tiles_y, const float* __restrict__ color, const float* __restrict__ grad_color,
    const float* __restrict__ rast, int V, const float* __restrict__ pos, float* __restrict__ grad_pos,
    const int* __restrict__ tri) {
    __shared__ EdgeHalo h;
    __shared__ float s_adj[4 * kEdgeLanes];  // per thread and neighbour: the marked pairs' adjoints
    __shared__ short s_pix[kEdgeTileThreads];
    __shared__ int s_warp_n[kEdgeTileThreads / 32];
    static_assert(kEdgeLanes == kEdgeTileThreads, "one thread per pixel of the tile");
    const int per = tiles_x * tiles_y, b = (int)(blockIdx.x / (unsigned)per), tl = (int)(blockIdx.x - (unsigned)b * per);
    const int tx0 = (tl % tiles_x) * DS_TILE, ty0 = (tl / tiles_x) * DS_TILE;
    const int64_t base = (int64_t)b * H * W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the triangles of the tile's own pixels: nothing to do where all are background
    const int cy = threadIdx.x / DS_TILE, cx = threadIdx.x % DS_TILE;
    const bool own = ty0 + cy < H && tx0 + cx < W;
    const float id = own ? __ldg(rast + (base + (int64_t)(ty0 + cy) * W + tx0 + cx) * 4 + 3) : 0.f;
    const bool cov = (int)id - 1 >= 0;
    if (!__syncthreads_or(cov)) return;
    for (int i = threadIdx.x; i < kHaloN; i += kEdgeTileThreads) {
        const int hy = i / kHaloW, hx = i - (i / kHaloW) * kHaloW;
        const int y = ty0 + hy - 1, x = tx0 + hx - 1;
        int it = kOutside;
        float dep = 0.f, cc[3] = {0.f, 0.f, 0.f}, gg[3] = {0.f, 0.f, 0.f};
        if (y >= 0 && y < H && x >= 0 && x < W) {
            const int64_t p = base + (int64_t)y * W + x;
            const float4 r = reinterpret_cast<const float4*>(rast)[p];
            it = (int)r.w - 1;
            if (it < -1) it = -1;  // any negative ID is background (kOutside marks the view's border)
            dep = r.z;
#pragma unroll
            for (int k = 0; k < 3; ++k) { cc[k] = color[p * 3 + k]; gg[k] = grad_color[p * 3 + k]; }
        }
        h.it[i] = it;
        h.dep[i] = dep;
#pragma unroll
        for (int k = 0; k < 3; ++k) { h.c[k][i] = cc[k]; h.g[k][i] = gg[k]; }
    }
    __syncthreads();
    const int n = edge_tile_order(h, s_pix, s_warp_n);
    if (warp * 32 >= n) return;  // warp-uniform: no covered pixel left for this warp
    const bool active = (int)threadIdx.x < n;
    const int src = active ? s_pix[threadIdx.x] : 0;
    const int ly = src / DS_TILE, lx = src % DS_TILE;
    EdgeAccum acc;
    const int it0 = edge_grad_pixel_tile(h, (ly + 1) * kHaloW + lx + 1, ty0 + ly, tx0 + lx, H, W,
                                         pos + (size_t)b * V * 4, tri, acc, s_adj + threadIdx.x, active);
    const int key = (it0 >= 0 && acc.any) ? it0 : -1 - lane;
    if (__ballot_sync(0xffffffffu, key >= 0) == 0) return;
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != key);
    const int seg = __popc(heads & ((2u << lane) - 1u));
    int oseg[5];
#pragma unroll
    for (int s = 0; s < 5; ++s) oseg[s] = __shfl_down_sync(0xffffffffu, seg, 1 << s);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        float v = acc.g[k];
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            const float ov = __shfl_down_sync(0xffffffffu, v, 1 << s);
            if (lane + (1 << s) < 32 && oseg[s] == seg) v += ov;
        }
        acc.g[k] = v;
    }
    if (!((heads >> lane) & 1u) || key < 0) return;
    float* gp = grad_pos + (size_t)b * V * 4;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int v = __ldg(tri + it0 * 3 + k);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (acc.g[k * 4 + j] != 0.f) atomicAdd(gp + (size_t)v * 4 + j, acc.g[k * 4 + j]);
    }
}

// rasterize.cu:923-971: one thread per fragment.
__global__ void __launch_bounds__(kThreads) aux_fragment_kernel(int H, int W, int C, const float* __restrict__ color,
                                                                const float* __restrict__ target,
                                                                const float* __restrict__ rast, int n,
                                                                const int* __restrict__ frag_pix,
                                                                const float* __restrict__ frag_attrs,
                                                                const float* __restrict__ frag_alpha,
                                                                float* __restrict__ grad_frag_alpha) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = frag_pix[(size_t)i * 3];
    if (b < 0) return;
    const int64_t p = (int64_t)b * H * W + (int64_t)frag_pix[(size_t)i * 3 + 1] * W + frag_pix[(size_t)i * 3 + 2];
    const float4 fa = reinterpret_cast<const float4*>(frag_attrs)[i];
    const float4 rp = reinterpret_cast<const float4*>(rast)[p];
    const int tf = (int)fa.w - 1, tp = (int)rp.w - 1;
    if (tp >= 0 && fa.z > rp.z) return;
    float loss = 0.f;
    for (int c = 0; c < C; ++c) loss += fabsf(color[p * C + c] - target[p * C + c]);
    grad_frag_alpha[i] += aux_alpha_grad(loss, frag_alpha[i], tp >= 0 && tf == tp);
}

}  // namespace dsb

using namespace dsb;

extern "C" {

int ds_backward_edge_grad(int B, int H, int W, int C, const float* color, const float* grad_color, const float* rast,
                          int V, const float* pos, float* grad_pos, const int* tri, ds_stream_t stream) {
    DS_CHECK_ARG(B >= 0 && H >= 0 && W >= 0 && C > 0 && V >= 0, "backward_edge_grad: bad sizes");
    const int64_t n = (int64_t)B * H * W;
    if (n == 0) return DS_OK;
    DS_CHECK_ARG(((uintptr_t)rast & 15) == 0 && ((uintptr_t)pos & 15) == 0,
                 "backward_edge_grad: rast/pos not 16-byte aligned");
    // three channels (a colour) take the staged kernel; other widths one thread per pixel
    const int64_t tiles_x = (W + DS_TILE - 1) / DS_TILE, tiles_y = (H + DS_TILE - 1) / DS_TILE;
    if (C == 3 && tiles_x * tiles_y * B <= 0x7fffffff) {
        edge_grad_tile_kernel<<<(unsigned)(tiles_x * tiles_y * B), kEdgeTileThreads, 0, (cudaStream_t)stream>>>(
            H, W, (int)tiles_x, (int)tiles_y, color, grad_color, rast, V, pos, grad_pos, tri);
        return check_launch("backward_edge_grad");
    }
    edge_grad_kernel<<<blocks_for(n), kThreads, 0, (cudaStream_t)stream>>>(B, H, W, C, color, grad_color, rast, V, pos,
                                                                          grad_pos, tri);
    return check_launch("backward_edge_grad");
}

int ds_backward_opacity_aux_loss(int B, int H, int W, int C, const float* color, const float* target,
                                 const float* rast, int num_frags, const int* frag_pix, const float* frag_attrs,
                                 const float* frag_alpha, float* grad_frag_alpha, ds_stream_t stream) {
    DS_CHECK_ARG(B >= 0 && H >= 0 && W >= 0 && C > 0 && num_frags >= 0, "backward_opacity_aux_loss: bad sizes");
    if (num_frags == 0) return DS_OK;
    DS_CHECK_ARG(((uintptr_t)rast & 15) == 0 && ((uintptr_t)frag_attrs & 15) == 0,
                 "backward_opacity_aux_loss: rast/frag_attrs not 16-byte aligned");
    aux_fragment_kernel<<<blocks_for(num_frags), kThreads, 0, (cudaStream_t)stream>>>(
        H, W, C, color, target, rast, num_frags, frag_pix, frag_attrs, frag_alpha, grad_frag_alpha);
    return check_launch("backward_opacity_aux_loss");
}

}  // extern "C"
