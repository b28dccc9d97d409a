// diffsoup_b200/csrc/step.cu -- the batched training step of DiffSoup
// (examples/02_synthetic.py:354-388 with an MSE photometric loss) as one
// graph-capturable sequence of sm_100a kernels:
//
//   accumulate_to_level(...).sigmoid() for opacity and features   (prep)
//   project_vertices (examples/utils.py:412-426)                   (prep)
//   screen-tile binning + tiled stochastic-opacity rasterizer      (tiled.cu)
//   fused shading forward + backward, BF16 MLP on tensor cores     (shade.cuh)
//   opacity auxiliary gradient, recomputed tile by tile            (tiled.cu)
//   edge gradients to clip-space vertices                          (edge)
//   adjoints of the sigmoid, the level accumulation and projection (finish)
//
// Views may differ in resolution; their pixels are packed back to back.
#include <cmath>
#include <cstdio>

#include "edge_math.cuh"
#include "lattice_map.cuh"
#include "shade.cuh"
#include "shade_reg.cuh"
#include "shade_tc.cuh"
#include "tiled.cuh"

namespace dsb {

// ---------------------------------------------------------------------------
// Level accumulation + sigmoid, one warp per triangle (multires.cu:329-369).
// The triangle's source samples are staged in shared memory; outputs are
// sigmoid(sum over levels of the lattice interpolation at each target vertex).
// ---------------------------------------------------------------------------
constexpr int kPrepWarps = 4;
constexpr int kMaxSrc = 2048;  // floats of one triangle's samples per warp (S*C)

// Outputs have a channel stride of CP >= C (padding channels written as zero).
template <bool BF16OUT>
__global__ void __launch_bounds__(kPrepWarps * 32) accum_sigmoid_kernel(int T, int lo, int hi, int target, int S,
                                                                       int ST, int C, int CP,
                                                                       const float* __restrict__ src,
                                                                       float* __restrict__ out_f32,
                                                                       __nv_bfloat16* __restrict__ out_bf16) {
    __shared__ float s_src[kPrepWarps][kMaxSrc];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * kPrepWarps + warp;
    if (t >= T) return;
    const int n = S * C;
    const float* ts = src + (size_t)t * n;
    for (int i = lane; i < n; i += 32) s_src[warp][i] = ts[i];
    __syncwarp();
    const float R = (float)(1u << target);
    for (int e = lane; e < ST * CP; e += 32) {
        const int k = e / CP, c = e % CP;
        if (c >= C) {
            out_f32[(size_t)t * ST * CP + e] = 0.f;
            if (BF16OUT) out_bf16[(size_t)t * ST * CP + e] = __float2bfloat16_rn(0.f);
            continue;
        }
        uint32_t x, y;
        index_to_xy((uint32_t)k, x, y);
        const float b0 = __fdiv_rn((float)x, R), b1 = __fdiv_rn((float)y, R);
        float acc = 0.f;
        uint32_t off = 0;
        for (int l = lo; l <= hi; ++l) {
            uint32_t idx[3]; float w[3];
            lattice_cell(b0, b1, (uint32_t)l, idx, w);
#pragma unroll
            for (int j = 0; j < 3; ++j) acc = madd(acc, w[j], s_src[warp][(off + idx[j]) * C + c]);
            off += feats_at_level((uint32_t)l);
        }
        const float s = 1.f / (1.f + expf(-acc));
        out_f32[(size_t)t * ST * CP + e] = s;
        if (BF16OUT) out_bf16[(size_t)t * ST * CP + e] = __float2bfloat16_rn(s);
    }
}

// Adjoint of accum_sigmoid: grad_src[t] = sum_k lattice^T (grad_out * s (1-s)).
// Accumulated per warp in shared memory, written once (no global atomics).
// sig and grad_out have the channel stride CP, grad_src the stride C.
__global__ void __launch_bounds__(kPrepWarps * 32) accum_sigmoid_backward_kernel(
    int T, int lo, int hi, int target, int S, int ST, int C, int CP, const float* __restrict__ sig,
    const float* __restrict__ grad_out, float* __restrict__ grad_src) {
    __shared__ float s_acc[kPrepWarps][kMaxSrc];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * kPrepWarps + warp;
    if (t >= T) return;
    const int n = S * C;
    for (int i = lane; i < n; i += 32) s_acc[warp][i] = 0.f;
    __syncwarp();
    const float R = (float)(1u << target);
    for (int e = lane; e < ST * C; e += 32) {
        const int k = e / C, c = e % C;
        const size_t o = ((size_t)t * ST + k) * CP + c;
        const float s = sig[o];
        const float gz = grad_out[o] * s * (1.f - s);
        if (gz == 0.f) continue;
        uint32_t x, y;
        index_to_xy((uint32_t)k, x, y);
        const float b0 = __fdiv_rn((float)x, R), b1 = __fdiv_rn((float)y, R);
        uint32_t off = 0;
        for (int l = lo; l <= hi; ++l) {
            uint32_t idx[3]; float w[3];
            lattice_cell(b0, b1, (uint32_t)l, idx, w);
#pragma unroll
            for (int j = 0; j < 3; ++j) atomicAdd(&s_acc[warp][(off + idx[j]) * C + c], gz * w[j]);
            off += feats_at_level((uint32_t)l);
        }
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) grad_src[(size_t)t * n + i] = s_acc[warp][i];
}

// ---------------------------------------------------------------------------
// Level accumulation of the step through the map's rows (lattice_map.cuh),
// opacity and features in one launch each way.  A group of one or two warps takes G
// triangles at a time; a lane takes four channels of one output sample, so a row's entry and
// one 16-byte shared load feed four products.  Features sit in the group's tile
// as [triangle][sample][CP], opacities as [sample][triangle] (with G = 4 they
// are one more group of four).  The sources are copied with cp.async; the adjoint
// forms g s (1 - s) on the way in.  Only pairs of nonzero weight are used.
// Issue slots (0.7 a cycle) and the tile's shared loads share the bound: a second
// tile per warp for copies ahead halved the resident warps (637 us forward), one
// triangle a warp put half of the loads on the banks of another row (493 us).
//
// 200,000 triangles, levels 0..3, 16 channels (1.8 GB read and written forward,
// 2.1 GB in the adjoint): forward 1014 -> 447 us, adjoint 756 -> 496 us; 60,000
// triangles of 7 channels, levels 0..2: 50 -> 38 and 40 -> 41 us, against one
// lane per channel with a 4-byte load and a table read per product.  Four
// triangles interleaved in the tile instead of four channels (the layout of the
// operators, which take any channel count) left too few warps on an SM: 1038
// and 1673 us.
// ---------------------------------------------------------------------------
constexpr int kTabMax = 1024;  // (target sample, level, corner) pairs

__device__ __forceinline__ float sigmoid_ref(float x) { return 1.f / (1.f + expf(-x)); }

// Triangles a group takes at a time and warps of a group, by channel stride: 4
// triangles on one warp where they have 8 channels, 2 on two warps where they
// have 16 (their tile is too large for one tile a warp).
template <int CP>
constexpr int kTabGroup = CP == 8 ? 4 : 2;
template <int CP>
constexpr int kTabGroupWarps = CP == 8 ? 1 : 2;

// Floats between the triangles of a tile: the eight lanes of a quarter warp read
// the same sample of G triangles, so their rows must fall in different banks.
__host__ __device__ constexpr int tab_triangle_floats(int samples, int CP) {
    return ((samples * CP - CP + 31) / 32) * 32 + CP;
}

// Tile floats of a group: the triangles' features, then their opacities.
__host__ __device__ constexpr int tab_tile_floats(int samples, int CP, int G) {
    return G * tab_triangle_floats(samples, CP) + ((samples * G + 31) & ~31);
}

// Barrier of a group's lanes.
template <int GW>
__device__ __forceinline__ void tab_group_sync(int group) {
    if (GW == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GW * 32) : "memory");
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
                 "n"(BYTES)
                 : "memory");
}

// Output rows of the features of G triangles and of their opacities, over the
// group's lanes: feature(triangle, row, quad, value4), opacity(row, triangle,
// value).
template <int CP, int G, int GW, class Feature, class Opacity>
__device__ __forceinline__ void tab_rows(const MapRows& m, const float* tile, int samples, int rows, Feature feature,
                                         Opacity opacity) {
    constexpr int Q = CP / 4;
    const int lane = threadIdx.x % (32 * GW);
    const int ts = tab_triangle_floats(samples, CP);
    const float* ta = tile + G * ts;
    const int nf = G * Q * rows;
    // with G = 4 the opacity rows go on where the feature rows end, with the same loads
    for (int s = lane; s < nf + (G == 4 ? rows : 0); s += 32 * GW) {
        const bool f = G != 4 || s < nf;
        const int q = s % Q, g = s / Q % G;
        const int row = f ? s / (Q * G) : s - nf;
        const float* x0 = f ? tile + g * ts + q * 4 : ta;
        const int stride = f ? CP : 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        const int end = m.row[row + 1];
#pragma unroll 2
        for (int n = m.row[row]; n < end; ++n) {
            const int2 e = m.ent[n];
            const float w = __int_as_float(e.y);
            const float4 x = *reinterpret_cast<const float4*>(x0 + e.x * stride);
            v.x = madd(v.x, w, x.x); v.y = madd(v.y, w, x.y); v.z = madd(v.z, w, x.z); v.w = madd(v.w, w, x.w);
        }
        if (f) {
            feature(g, row, q, v);
        } else {
            opacity(row, 0, v.x); opacity(row, 1, v.y); opacity(row, 2, v.z); opacity(row, 3, v.w);
        }
    }
    if (G == 2)
        for (int row = lane; row < rows; row += 32 * GW) {
            float2 v = make_float2(0.f, 0.f);
            const int end = m.row[row + 1];
            for (int n = m.row[row]; n < end; ++n) {
                const int2 e = m.ent[n];
                const float w = __int_as_float(e.y);
                const float2 x = *reinterpret_cast<const float2*>(ta + e.x * 2);
                v.x = madd(v.x, w, x.x); v.y = madd(v.y, w, x.y);
            }
            opacity(row, 0, v.x); opacity(row, 1, v.y);
        }
}

// alpha_out[t] = sigmoid(accumulate(alpha_src[t])), feat_out[t] likewise
// per channel (+ a bf16 copy; both with the channel stride CP >= C, padding
// channels zero).  The grid's last CTA builds the adjoint's rows meanwhile and
// leaves them in adj_ent [N], adj_row [S + 1].
template <int C, int CP>
__global__ void __launch_bounds__(kMapWarps * 32) accum_tab_kernel(int T, int lo, int hi, int S, int ST,
                                                                   const float* __restrict__ alpha_src,
                                                                   const float* __restrict__ feat_src,
                                                                   float* __restrict__ alpha_out,
                                                                   float* __restrict__ feat_out,
                                                                   __nv_bfloat16* __restrict__ feat_bf16,
                                                                   int2* __restrict__ adj_ent, int* __restrict__ adj_row) {
    constexpr int G = kTabGroup<CP>, GW = kTabGroupWarps<CP>, L = 32 * GW;
    extern __shared__ __align__(16) unsigned char map_smem[];
    const int N = ST * (hi - lo + 1) * 3;
    if (blockIdx.x == gridDim.x - 1) {
        const MapTables a = map_tables_at(map_smem, N, S);
        build_adjoint_rows(a, lo, hi, hi, ST, S);
        for (int i = threadIdx.x; i < N; i += blockDim.x) adj_ent[i] = a.nonzero.ent[i];
        for (int i = threadIdx.x; i <= S; i += blockDim.x) adj_row[i] = a.nonzero.row[i];
        return;
    }
    const MapTables m = map_tables_at(map_smem, N, ST);
    const int group = (threadIdx.x >> 5) / GW, lane = threadIdx.x % L;
    const int ts = tab_triangle_floats(S, CP), tf = tab_tile_floats(S, CP, G);
    float* tile = reinterpret_cast<float*>(map_smem + map_table_bytes(N, ST > S ? ST : S)) + (size_t)group * tf;
    if (C < CP)
        for (int i = lane; i < tf; i += L) tile[i] = 0.f;  // the padding channels stay zero
    tab_group_sync<GW>(group);
    const bool wide = C % 4 == 0 && ((uintptr_t)feat_src & 15) == 0;
    auto stage = [&](int64_t t) {
        for (int g = 0; g < G && t + g < T; ++g) {
            const float* fs = feat_src + (size_t)(t + g) * S * C;
            float* dst = tile + g * ts;
            if (wide) {
                for (int e = lane; e < S * (C / 4); e += L) cp_async<16>(dst + e * 4, fs + e * 4);
            } else {
                for (int e = lane; e < S * C; e += L) cp_async<4>(dst + (C == CP ? e : e / C * CP + e % C), fs + e);
            }
            for (int d = lane; d < S; d += L) cp_async<4>(tile + G * ts + d * G + g, alpha_src + (size_t)(t + g) * S + d);
        }
    };
    const int64_t step = (int64_t)(gridDim.x - 1) * (kMapWarps / GW) * G;
    int64_t t = ((int64_t)blockIdx.x * (kMapWarps / GW) + group) * G;
    stage(t);
    build_forward_rows(m, lo, hi, hi, ST);
    for (; t < T; t += step) {
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        tab_group_sync<GW>(group);
        tab_rows<CP, G, GW>(
            m.nonzero, tile, S, ST,
            [&](int g, int row, int q, float4 v) {
                if (t + g >= T) return;
                float4 y = make_float4(sigmoid_ref(v.x), sigmoid_ref(v.y), sigmoid_ref(v.z), sigmoid_ref(v.w));
                if (C == 7 && q == 1) y.w = 0.f;
                const size_t o = ((size_t)(t + g) * ST + row) * CP + q * 4;
                *reinterpret_cast<float4*>(feat_out + o) = y;
                const __nv_bfloat162 a = __floats2bfloat162_rn(y.x, y.y), c = __floats2bfloat162_rn(y.z, y.w);
                *reinterpret_cast<uint2*>(feat_bf16 + o) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&c));
            },
            [&](int row, int g, float v) {
                if (t + g < T) alpha_out[(size_t)(t + g) * ST + row] = sigmoid_ref(v);
            });
        tab_group_sync<GW>(group);
        stage(t + step);
    }
}

// Adjoint of accum_tab_kernel: grad_src[t][d] = sum over the targets k that
// read d of w * grad_out[t][k] * s (1 - s); a gather, written once.  feat_sig and
// feat_grad have the channel stride CP (padding channels zero), feat_src_grad
// the stride C.
template <int C, int CP>
__global__ void __launch_bounds__(kMapWarps * 32) accum_tab_backward_kernel(
    int T, int lo, int hi, int S, int ST, const float* __restrict__ alpha_sig, const float* __restrict__ alpha_grad,
    const float* __restrict__ feat_sig, const float* __restrict__ feat_grad, float* __restrict__ alpha_src_grad,
    float* __restrict__ feat_src_grad, const int2* __restrict__ adj_ent, const int* __restrict__ adj_row) {
    constexpr int G = kTabGroup<CP>, GW = kTabGroupWarps<CP>, L = 32 * GW, Q = CP / 4;
    extern __shared__ __align__(16) unsigned char map_smem[];
    chain_wait();
    const int N = ST * (hi - lo + 1) * 3;
    MapRows m;
    m.ent = reinterpret_cast<int2*>(map_smem);
    m.row = reinterpret_cast<int*>(m.ent + N);
    const int group = (threadIdx.x >> 5) / GW, lane = threadIdx.x % L;
    const int ts = tab_triangle_floats(ST, CP);
    float* tile = reinterpret_cast<float*>(map_smem + (((size_t)N * 8 + (size_t)(S + 1) * 4 + 127) & ~(size_t)127)) +
                  (size_t)group * tab_tile_floats(ST, CP, G);
    for (int i = threadIdx.x; i <= S; i += blockDim.x) m.row[i] = adj_row[i];
    for (int i = threadIdx.x; i < adj_row[S]; i += blockDim.x) m.ent[i] = adj_ent[i];
    __syncthreads();
    const bool wide = C % 4 == 0 && ((uintptr_t)feat_src_grad & 15) == 0;
    const int64_t step = (int64_t)gridDim.x * (kMapWarps / GW) * G;
    for (int64_t t = ((int64_t)blockIdx.x * (kMapWarps / GW) + group) * G; t < T; t += step) {
        for (int g = 0; g < G && t + g < T; ++g) {
            const float4* sp = reinterpret_cast<const float4*>(feat_sig + (size_t)(t + g) * ST * CP);
            const float4* gp = reinterpret_cast<const float4*>(feat_grad + (size_t)(t + g) * ST * CP);
            for (int e0 = lane; e0 < ST * Q; e0 += 3 * L) {  // three (sigmoid, gradient) pairs in flight
                float4 y[3], v[3];
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (e0 + L * u < ST * Q) { y[u] = __ldg(sp + e0 + L * u); v[u] = __ldg(gp + e0 + L * u); }
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (e0 + L * u < ST * Q) {
                        v[u].x = v[u].x * y[u].x * (1.f - y[u].x); v[u].y = v[u].y * y[u].y * (1.f - y[u].y);
                        v[u].z = v[u].z * y[u].z * (1.f - y[u].z); v[u].w = v[u].w * y[u].w * (1.f - y[u].w);
                        *reinterpret_cast<float4*>(tile + g * ts + (e0 + L * u) * 4) = v[u];
                    }
            }
            for (int k = lane; k < ST; k += L) {
                const size_t o = (size_t)(t + g) * ST + k;
                const float y = __ldg(alpha_sig + o);
                tile[G * ts + k * G + g] = __ldg(alpha_grad + o) * y * (1.f - y);
            }
        }
        tab_group_sync<GW>(group);
        tab_rows<CP, G, GW>(
            m, tile, ST, S,
            [&](int g, int row, int q, float4 v) {
                if (t + g >= T) return;
                float* o = feat_src_grad + ((size_t)(t + g) * S + row) * C + q * 4;
                if (wide) {
                    *reinterpret_cast<float4*>(o) = v;
                    return;
                }
                o[0] = v.x; o[1] = v.y; o[2] = v.z;
                if (C % 4 == 0 || q < Q - 1) o[3] = v.w;
            },
            [&](int row, int g, float v) {
                if (t + g < T) alpha_src_grad[(size_t)(t + g) * S + row] = v;
            });
        tab_group_sync<GW>(group);
    }
}

// Dynamic shared memory of the table kernels: rows and each group's tile.
template <int CP>
static size_t lattice_tab_smem(int lo, int hi, int S, int ST, bool backward) {
    const int N = ST * (hi - lo + 1) * 3;
    const size_t tables = backward ? (((size_t)N * 8 + (size_t)(S + 1) * 4 + 127) & ~(size_t)127)
                                   : map_table_bytes(N, ST > S ? ST : S);
    return tables + (size_t)(kMapWarps / kTabGroupWarps<CP>) * tab_tile_floats(backward ? ST : S, CP, kTabGroup<CP>) *
                        sizeof(float);
}

// Whether the table kernels cover this configuration (two CTAs per SM).
static bool lattice_tab_fits(int lo, int hi, int S, int ST, int CP) {
    if (ST * (hi - lo + 1) * 3 > kTabMax) return false;
    return (CP == 8 && lattice_tab_smem<8>(lo, hi, S, ST, false) <= 110 * 1024) ||
           (CP == 16 && lattice_tab_smem<16>(lo, hi, S, ST, false) <= 110 * 1024);
}

// clip[b][v] = mvp[b] . (verts[v], 1)  (examples/utils.py:412-426)
__global__ void __launch_bounds__(kThreads) project_kernel(int B, int V, const float* __restrict__ verts,
                                                           const float* __restrict__ mvp, float* __restrict__ pos) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)B * V) return;
    const int b = (int)(i / V), v = (int)(i % V);
    const float* M = mvp + (size_t)b * 16;
    const float x = verts[(size_t)v * 3], y = verts[(size_t)v * 3 + 1], z = verts[(size_t)v * 3 + 2];
    // fixed evaluation order: ((M[r][3] + M[r][0] x) + M[r][1] y) + M[r][2] z, fused
    float4 o;
    o.x = __fmaf_rn(M[2], z, __fmaf_rn(M[1], y, __fmaf_rn(M[0], x, M[3])));
    o.y = __fmaf_rn(M[6], z, __fmaf_rn(M[5], y, __fmaf_rn(M[4], x, M[7])));
    o.z = __fmaf_rn(M[10], z, __fmaf_rn(M[9], y, __fmaf_rn(M[8], x, M[11])));
    o.w = __fmaf_rn(M[14], z, __fmaf_rn(M[13], y, __fmaf_rn(M[12], x, M[15])));
    reinterpret_cast<float4*>(pos)[i] = o;
}

// grad_verts[v] = sum_b mvp[b][:, :3]^T grad_pos[b][v]; the first thread also
// closes the step: the loss, the next iteration of the opacity-threshold RNG
// and the status of re-enumerated blocks.
__global__ void __launch_bounds__(kThreads) project_backward_kernel(int B, int V, const float* __restrict__ mvp,
                                                                    const double* __restrict__ grad_pos,
                                                                    float* __restrict__ grad_verts,
                                                                    const double* __restrict__ loss_sum, float inv_n,
                                                                    float* __restrict__ loss, uint64_t* __restrict__ rng,
                                                                    const int* __restrict__ rec_counters,
                                                                    int* __restrict__ status) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        *loss = (float)(*loss_sum * (double)inv_n);
        if (rng) rng[1] += 1;
        if (status && rec_counters[1] > 0) atomicOr(status, DS_STATUS_RECORD_FALLBACK);
    }
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    double gx = 0.0, gy = 0.0, gz = 0.0;
    for (int b = 0; b < B; ++b) {
        const float* M = mvp + (size_t)b * 16;
        const double2* gp = reinterpret_cast<const double2*>(grad_pos + ((size_t)b * V + v) * 4);
        const double2 g01 = gp[0], g23 = gp[1];
        const double g[4] = {g01.x, g01.y, g23.x, g23.y};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            gx += (double)M[r * 4 + 0] * g[r];
            gy += (double)M[r * 4 + 1] * g[r];
            gz += (double)M[r * 4 + 2] * g[r];
        }
    }
    grad_verts[(size_t)v * 3] = (float)gx;
    grad_verts[(size_t)v * 3 + 1] = (float)gy;
    grad_verts[(size_t)v * 3 + 2] = (float)gz;
}

// Edge gradients over packed views (rasterize.cu:653-903): one CTA per
// 16x16 screen tile, one thread per pixel.  The tile and its one-pixel
// border are staged in shared memory first (triangle, depth, colour,
// dL/dcolour and the triangle's far depth bound), so the four neighbours of
// every pixel are shared-memory reads.  Pixels of a warp (two rows of 16)
// mostly share a triangle along a row: a segmented warp reduction sums runs
// of equal triangles before one FP64 atomic per vertex component.  Only
// covered pixels have a contribution, so after staging the tile's covered
// pixels are compacted onto the CTA's first threads, triangle by triangle
// (edge_tile_order): warps run full of covered pixels and the warps left
// without one exit.  In row order, where stochastic opacity alternates
// surfaces from pixel to pixel, half of a dense scene's time went to the atomics of its
// short runs: 200,000 triangles in 3 full-HD views 707 -> 387 us, 6 uneven views
// 292 -> 224 us, 8 views of 800x800 268 -> 265 us.
constexpr int kEdgeThreads = DS_TILE * DS_TILE;
#ifndef DSB_EDGE_MIN_CTAS
#define DSB_EDGE_MIN_CTAS 4  // resident 8-warp CTAs per SM the register budget is sized for (64 registers)
#endif

__device__ __forceinline__ int tile_view(const ds_view_desc* __restrict__ views, int B, int tile) {
    int lo = 0, hi = B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&views[mid].tile_base) <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(kEdgeThreads, DSB_EDGE_MIN_CTAS) edge_step_kernel(
    int B, const ds_view_desc* __restrict__ views, int V, int T, TileTables tab, const int* __restrict__ tri,
    const float* __restrict__ color, const float* __restrict__ grad_color, const float* __restrict__ rast,
    double* __restrict__ grad_pos) {
    __shared__ EdgeHalo h;
    chain_wait();
    const int tile = blockIdx.x;
    // no triangle may cover a pixel centre of the tile (its list is empty): every pixel is background,
    // and background pixels contribute nothing as the centre of a pair
    if (tab.offsets[tile] == tab.offsets[tile + 1]) return;
    const int b = tile_view(views, B, tile);
    const ds_view_desc vd = views[b];
    const int tl = tile - vd.tile_base;
    const int tx0 = (tl % vd.tiles_x) * DS_TILE, ty0 = (tl / vd.tiles_x) * DS_TILE;
    const TriBox* __restrict__ boxes = tab.boxes + (size_t)b * T;
    for (int i = threadIdx.x; i < kHaloN; i += kEdgeThreads) {
        const int hy = i / kHaloW, hx = i - (i / kHaloW) * kHaloW;
        const int y = ty0 + hy - 1, x = tx0 + hx - 1;
        int it = kOutside;
        float dep = 0.f, zh = 0.f, cc[3] = {0.f, 0.f, 0.f}, gg[3] = {0.f, 0.f, 0.f};
        if (y >= 0 && y < vd.H && x >= 0 && x < vd.W) {
            const int64_t p = vd.pix_offset + (int64_t)y * vd.W + x;
            const float4 r = reinterpret_cast<const float4*>(rast)[p];
            it = (int)r.w - 1;
            dep = r.z;
#pragma unroll
            for (int k = 0; k < 3; ++k) { cc[k] = color[p * 3 + k]; gg[k] = grad_color[p * 3 + k]; }
            if (it >= 0) zh = boxes[it].zhi;
        }
        h.it[i] = it;
        h.dep[i] = dep;
        h.zhi[i] = zh;
#pragma unroll
        for (int k = 0; k < 3; ++k) { h.c[k][i] = cc[k]; h.g[k][i] = gg[k]; }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ short s_pix[kEdgeThreads];
    __shared__ int s_warp_n[kEdgeThreads / 32];
    const int n = edge_tile_order(h, s_pix, s_warp_n);
    if (warp * 32 >= n) return;  // warp-uniform: no covered pixel left for this warp
    const bool active = (int)threadIdx.x < n;
    const int src = active ? s_pix[threadIdx.x] : 0;
    const int ly = src / DS_TILE, lx = src % DS_TILE;
    const int y = ty0 + ly, x = tx0 + lx;
    EdgeAccum acc;
    __shared__ float s_adj[4 * kEdgeLanes];  // per thread and neighbour: the marked pairs' adjoints
    static_assert(kEdgeLanes == kEdgeThreads, "one thread per pixel of the tile");
    // every lane of the warp takes part (warp-wide reductions inside); lanes past the covered
    // pixels contribute nothing
    const int it0 = edge_grad_pixel_staged(h, (ly + 1) * kHaloW + lx + 1, y, x, vd.H, vd.W,
                                           tab.verts + (size_t)b * T, acc, s_adj + threadIdx.x, active);
    const int key = (it0 >= 0 && acc.any) ? it0 : -1 - lane;
    if (__ballot_sync(0xffffffffu, key >= 0) == 0) return;  // no lane of the warp has a contribution
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
    const bool head = (heads >> lane) & 1u;
    if (head && key >= 0) {
        double* gp = grad_pos + (size_t)b * V * 4;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int v = __ldg(tri + it0 * 3 + k);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (acc.g[k * 4 + j] != 0.f) atomicAdd(gp + (size_t)v * 4 + j, (double)acc.g[k * 4 + j]);
        }
    }
}

template <class K>
static int launch_shade(const ShadeArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(ShadeSmem<K>);
    static int per_sm = 0;  // set on the first (eager) call, before any graph capture
    if (per_sm == 0) {
        DS_CUDA(cudaFuncSetAttribute(shade_step_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        DS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shade_step_kernel<K>, K::WARPS * 32, smem));
        if (per_sm <= 0) return set_error(DS_ERR_CUDA, "shade_step: kernel does not fit on an SM");
    }
    const int64_t chunks = (a.num_pixels + 31) / 32;
    const int64_t want = (chunks + K::WARPS - 1) / K::WARPS;
    const int64_t cap = (int64_t)sm_count() * (per_sm > 0 ? per_sm : 1);
    const unsigned grid = (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
    launch_chained(shade_step_kernel<K>, dim3(grid), K::WARPS * 32, smem, st, a);
    return check_launch("shade_step");
}

// The register-resident kernels of the width-16 MLPs.
template <class K>
static int launch_shade_reg(const ShadeArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(RegSmem<K>);
    static int per_sm = 0;  // set on the first (eager) call, before any graph capture
    if (per_sm == 0) {
        DS_CUDA(cudaFuncSetAttribute(shade_reg_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        DS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shade_reg_kernel<K>, kShadeRegWarps * 32, smem));
        if (per_sm <= 0) return set_error(DS_ERR_CUDA, "shade_reg: kernel does not fit on an SM");
    }
    const int64_t chunks = (a.num_pixels + 31) / 32;
    const int64_t want = (chunks + kShadeRegWarps - 1) / kShadeRegWarps;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    const unsigned grid = (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
    launch_chained(shade_reg_kernel<K>, dim3(grid), kShadeRegWarps * 32, smem, st, a);
    return check_launch("shade_reg");
}

// The tcgen05 kernel of the wide BF16 MLP: persistent over 128-pixel tiles.
static int launch_shade_tc(const ShadeArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(TcSmem);
    static int per_sm = 0;  // set on the first (eager) call, before any graph capture
    if (per_sm == 0) {
        DS_CUDA(cudaFuncSetAttribute(shade_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        DS_CUDA(cudaFuncSetAttribute(shade_tc_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared));
        DS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shade_tc_kernel, kTcThreads, smem));
        // The query answers 1 for this kernel's 105 KB, while two CTAs fit the SM's shared memory and
        // registers (and run together: measured 1.6x the throughput of one).  Take the count those two
        // limits allow.
        int dev = 0, smem_sm = 0, reserved = 0;
        cudaFuncAttributes fa;
        DS_CUDA(cudaGetDevice(&dev));
        DS_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
        DS_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
        DS_CUDA(cudaFuncGetAttributes(&fa, shade_tc_kernel));
        const int by_smem = smem_sm / (int)(smem + (size_t)reserved);
        const int regs = (fa.numRegs + 7) / 8 * 8;  // allocation granularity per thread
        const int by_regs = regs > 0 ? 65536 / (regs * kTcThreads) : 1;
        const int fit = by_smem < by_regs ? by_smem : by_regs;
        if (fit > per_sm) per_sm = fit;
        if (per_sm <= 0) return set_error(DS_ERR_CUDA, "shade_tc: kernel does not fit on an SM");
        if (per_sm > 2) per_sm = 2;  // 256 TMEM columns per CTA: two CTAs fill an SM's 512
    }
    const int64_t tiles = (a.num_pixels + kTcThreads - 1) / kTcThreads;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    const unsigned grid = (unsigned)(tiles < 1 ? 1 : (tiles < cap ? tiles : cap));
    launch_chained(shade_tc_kernel, dim3(grid), kTcThreads, smem, st, a);
    return check_launch("shade_tc");
}

static inline size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

// Optional phase events (profiling): recorded on the step's stream at the
// boundaries prep | bin | raster | shade | aux | edge | finish.
constexpr int kStepEvents = 8;
static cudaEvent_t g_step_events[kStepEvents];
static int g_step_nevents = 0;

static int mark(int i, cudaStream_t st) {
    if (i < g_step_nevents) DS_CUDA(cudaEventRecord(g_step_events[i], st));
    return DS_OK;
}

// A second stream per device for the parts of the step that do not depend on
// each other (level accumulation beside projection and binning; the opacity
// auxiliary gradient beside the edge gradients).  The caller's stream forks
// to it through an event and joins it back before the dependent kernels, so
// the step stays one ordered unit on the caller's stream and captures into a
// CUDA graph as parallel branches.  Created on a device's first step.
constexpr int kMaxDevices = 64;
struct SideStream {
    cudaStream_t s = nullptr;
    cudaEvent_t fork[2] = {nullptr, nullptr}, join[2] = {nullptr, nullptr};
};
static SideStream g_side[kMaxDevices];

static SideStream* side_stream() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    SideStream& x = g_side[dev];
    if (x.s == nullptr) {
        SideStream n;
        if (cudaStreamCreateWithFlags(&n.s, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
        for (int i = 0; i < 2; ++i)
            if (cudaEventCreateWithFlags(&n.fork[i], cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&n.join[i], cudaEventDisableTiming) != cudaSuccess)
                return nullptr;
        x = n;
    }
    return &x;
}

// The side stream starts after everything issued so far on st.
static int fork_to(SideStream* x, int i, cudaStream_t st) {
    DS_CUDA(cudaEventRecord(x->fork[i], st));
    DS_CUDA(cudaStreamWaitEvent(x->s, x->fork[i], 0));
    return DS_OK;
}

// Work issued on st from now on starts after the side stream's work.
static int join_from(SideStream* x, int i, cudaStream_t st) {
    DS_CUDA(cudaEventRecord(x->join[i], x->s));
    DS_CUDA(cudaStreamWaitEvent(st, x->join[i], 0));
    return DS_OK;
}

struct StepWs {
    float* pos;
    float* alpha_acc;
    float* feat_acc;
    __nv_bfloat16* feat_bf16;
    float* rast;
    float* color;
    float* grad_color;
    float* l1;
    int2* adj_ent;      // rows of the level accumulation's adjoint, left by its forward kernel
    int* adj_row;
    double* grad_pos;
    float* grad_alpha_acc;
    float* grad_feat_acc;
    double* loss_sum;
    int* rec_counters;  // [2], zeroed with the accumulators
    void* tiles;
    size_t tiles_bytes;
    RecordStore rec;    // rec.capacity == 0: no records
};

// Fragment records reserved for P pixels: frag_records per pixel plus one
// chunk for every warp of the rasterizer's grid (each warp's last chunk is
// partly filled), a multiple of the chunk size.
static int64_t record_capacity(const ds_step_config& c, int num_tiles, int64_t P) {
    if (!(c.frag_records > 0.f)) return 0;
    const double n = std::ceil((double)P * (double)c.frag_records / kRecChunk);
    const int64_t items = (int64_t)num_tiles * 8;
    const int64_t warps = max_resident_warps();
    return ((int64_t)n + (items < warps ? items : warps)) * kRecChunk;
}

// Channel stride of the step's accumulated feature tables (and their
// gradients): C rounded up to a multiple of 8, so that a lattice sample is
// one or more 16-byte (bf16) / 32-byte (fp32) vectors.
static int feat_stride(const ds_step_config& c) { return (c.C + 7) & ~7; }

static StepWs carve_step(void* ws, const ds_step_config& c, int num_tiles, int64_t P, int64_t cap, size_t* total) {
    char* base = reinterpret_cast<char*>(ws);
    const int ST = (int)feats_at_level((uint32_t)c.max_level);
    size_t o = 0;
    StepWs w;
    w.pos = reinterpret_cast<float*>(base + o); o += al((size_t)c.B * c.V * 16);
    w.alpha_acc = reinterpret_cast<float*>(base + o); o += al((size_t)c.T * ST * 4);
    const int CP = feat_stride(c);
    w.feat_acc = reinterpret_cast<float*>(base + o); o += al((size_t)c.T * ST * CP * 4);
    w.feat_bf16 = reinterpret_cast<__nv_bfloat16*>(base + o); o += al((size_t)c.T * ST * CP * 2);
    w.rast = reinterpret_cast<float*>(base + o); o += al((size_t)P * 16);
    w.color = reinterpret_cast<float*>(base + o); o += al((size_t)P * 12);
    w.grad_color = reinterpret_cast<float*>(base + o); o += al((size_t)P * 12);
    w.l1 = reinterpret_cast<float*>(base + o); o += al((size_t)P * 4);
    w.adj_ent = reinterpret_cast<int2*>(base + o);
    o += al((size_t)ST * (c.max_level - c.min_level + 1) * 3 * sizeof(int2));
    w.adj_row = reinterpret_cast<int*>(base + o);
    o += al((size_t)(total_feats((uint32_t)c.min_level, (uint32_t)c.max_level) + 1) * sizeof(int));
    // zeroed together each step: grad_pos .. loss_sum
    w.grad_pos = reinterpret_cast<double*>(base + o); o += al((size_t)c.B * c.V * 32);
    w.grad_alpha_acc = reinterpret_cast<float*>(base + o); o += al((size_t)c.T * ST * 4);
    w.grad_feat_acc = reinterpret_cast<float*>(base + o); o += al((size_t)c.T * ST * CP * 4);
    w.loss_sum = reinterpret_cast<double*>(base + o);
    w.rec_counters = reinterpret_cast<int*>(base + o + 64);
    o += 256;
    w.tiles = base + o;
    w.tiles_bytes = ds_tiles_workspace_size(c.B, c.T, num_tiles, cap);
    o += al(w.tiles_bytes);
    const int64_t rcap = record_capacity(c, num_tiles, P);
    w.rec.capacity = rcap;
    w.rec.counters = w.rec_counters;
    w.rec.rec = reinterpret_cast<int4*>(base + o); o += al((size_t)rcap * sizeof(int4));
    w.rec.chunk_fill = reinterpret_cast<int*>(base + o); o += al((size_t)(rcap / kRecChunk) * sizeof(int));
    w.rec.fallback = reinterpret_cast<int*>(base + o); o += al(rcap > 0 ? (size_t)num_tiles * 8 * sizeof(int) : 0);
    if (total) *total = o;
    return w;
}

// log2 of the width of the tiled kernels' pixel blocks for ds_step_config.block_shape
static int block_shape_log2(const ds_step_config& c) {
    return c.block_shape == 1 ? 4 : (c.block_shape == 2 ? 2 : kDefaultBlockShape);
}

// The fused shading kernels a step can run, by MLP shape.
enum ShadeShape {
    kShadeUnsupported = 0,
    kShadeC8Dir16 = 1,     // 8 features + view direction -> 16 -> 3 (the benchmark configurations 1-3)
    kShadeC7Sh2_16x2 = 2,  // 7 features + SH2 -> 16 -> 16 -> 3 (the reference's own model)
    kShadeC16Dir64x2 = 3,  // 16 features + view direction -> 64 -> 64 -> 3 (configurations 4-5)
};

static int shade_shape(const ds_step_config& c) {
    if (c.hidden == 16 && c.n_layers == 1 && c.C == 8 && c.view_enc == 0) return kShadeC8Dir16;
    if (c.hidden == 16 && c.n_layers == 2 && c.C == 7 && c.view_enc == 1) return kShadeC7Sh2_16x2;
    if (c.hidden == 64 && c.n_layers == 2 && c.C == 16 && c.view_enc == 0) return kShadeC16Dir64x2;
    return kShadeUnsupported;
}

}  // namespace dsb

using namespace dsb;

using ShadeC8Dir16 = RegCfg<8, 3, 1, false>;        // 8 features + 3 view dir -> 16 -> 3
using ShadeC8Dir16Split = RegCfg<8, 3, 1, true>;
using ShadeC7Sh2_16x2 = RegCfg<7, 9, 2, false>;     // 7 features + 9 SH2 -> 16 -> 16 -> 3
using ShadeC7Sh2_16x2Split = RegCfg<7, 9, 2, true>;
using ShadeC16H64 = ShadeCfg<16, 32, 64, 2>;        // 16 + 3 -> 64 -> 64 -> 3
using ShadeC16H64Split = ShadeCfg<16, 32, 64, 2, true>;

extern "C" {

size_t ds_train_step_workspace_size(const ds_step_config* cfg, int num_tiles, int64_t num_pixels,
                                    int64_t list_capacity) {
    size_t total = 0;
    carve_step(nullptr, *cfg, num_tiles, num_pixels, list_capacity, &total);
    return total;
}

int ds_train_step_set_events(void* const* events, int n) {
    DS_CHECK_ARG(n >= 0 && n <= kStepEvents && (n == 0 || events != nullptr), "train_step_set_events: bad count");
    for (int i = 0; i < n; ++i) g_step_events[i] = (cudaEvent_t)events[i];
    g_step_nevents = n;
    return DS_OK;
}

int ds_train_step_layout(const ds_step_config* cfg, int num_tiles, int64_t num_pixels, int64_t list_capacity,
                         int64_t* offsets) {
    DS_CHECK_ARG(cfg != nullptr && offsets != nullptr, "train_step_layout: null argument");
    StepWs w = carve_step(nullptr, *cfg, num_tiles, num_pixels, list_capacity, nullptr);
    const void* ptrs[15] = {w.pos, w.alpha_acc, w.feat_acc, w.feat_bf16, w.rast, w.color, w.grad_color, w.l1,
                            w.grad_pos, w.grad_alpha_acc, w.grad_feat_acc, w.rec.rec, w.rec.chunk_fill,
                            w.rec_counters, w.rec.fallback};
    for (int i = 0; i < 15; ++i) offsets[i] = (int64_t)(reinterpret_cast<const char*>(ptrs[i]) - (const char*)nullptr);
    offsets[15] = w.rec.capacity;
    return DS_OK;
}

int ds_project_vertices(int B, int V, const float* verts, const float* mvp, float* pos, ds_stream_t stream) {
    DS_CHECK_ARG(B >= 0 && V >= 0 && (int64_t)B * V <= 0x7fffffff, "project_vertices: bad sizes");
    DS_CHECK_ARG((int64_t)B * V == 0 || (verts && mvp && pos), "project_vertices: null pointer");
    DS_CHECK_ARG(((uintptr_t)pos & 15) == 0, "project_vertices: pos not 16-byte aligned");
    if ((int64_t)B * V == 0) return DS_OK;
    project_kernel<<<blocks_for((int64_t)B * V), kThreads, 0, (cudaStream_t)stream>>>(B, V, verts, mvp, pos);
    return check_launch("project_vertices");
}

int ds_mlp_param_count(int C, int hidden, int n_layers) {
    const int in = C + 3;
    return hidden * in + hidden + (n_layers - 1) * (hidden * hidden + hidden) + 3 * hidden + 3;
}

int ds_step_mlp_param_count(const ds_step_config* cfg) {
    if (cfg == nullptr) return set_error(DS_ERR_ARG, "step_mlp_param_count: null config"), -1;
    // C + 9 inputs with SH2: the count for C + 6 features and a 3-D direction
    return ds_mlp_param_count(cfg->C + (cfg->view_enc ? 6 : 0), cfg->hidden, cfg->n_layers);
}

int ds_train_step(const ds_step_config* cfg, const ds_view_desc* views, int num_tiles, int64_t num_pixels,
                  const float* verts, const int* tri, const float* mvp, const float* inv_mvp, const float* feat_src,
                  const float* alpha_src, const float* mlp_params, const void* target, uint64_t* rng,
                  float* loss, float* grad_verts, float* grad_feat_src, float* grad_alpha_src,
                  float* grad_mlp_params, float* rast_out, float* color_out, void* workspace, size_t workspace_bytes,
                  int64_t list_capacity, int* status, ds_stream_t stream) {
    DS_CHECK_ARG(cfg != nullptr, "train_step: null config");
    const ds_step_config c = *cfg;
    DS_CHECK_ARG(c.B > 0 && c.T >= 0 && c.V >= 0 && num_tiles > 0 && num_pixels > 0, "train_step: bad sizes");
    DS_CHECK_ARG(c.min_level >= 0 && c.max_level >= c.min_level && c.max_level <= 8, "train_step: bad levels");
    DS_CHECK_ARG(c.stochastic == 0 || rng != nullptr, "train_step: stochastic opacity needs the rng state");
    DS_CHECK_ARG(c.precision == 0 || c.precision == 1, "train_step: precision must be 0 (bf16) or 1 (split bf16)");
    DS_CHECK_ARG(c.block_shape >= 0 && c.block_shape <= 2, "train_step: block_shape must be 0 (8x4), 1 (16x2) or 2 (4x8)");
    DS_CHECK_ARG(c.view_enc == 0 || c.view_enc == 1, "train_step: view_enc must be 0 (direction) or 1 (SH2)");
    DS_CHECK_ARG(c.target_u8 == 0 || c.target_u8 == 1, "train_step: target_u8 must be 0 (fp32) or 1 (8-bit)");
    DS_CHECK_ARG(c.shade_mode == 0 || c.shade_mode == 1, "train_step: shade_mode must be 0 (mma.sync) or 1 (tcgen05)");
    const int shape = shade_shape(c);
    DS_CHECK_ARG(shape != kShadeUnsupported,
                 "train_step: unsupported MLP (C=%d, %s, hidden=%d, layers=%d); built: 8+dir->16->3, "
                 "7+SH2->16->16->3, 16+dir->64->64->3", c.C, c.view_enc ? "SH2" : "dir", c.hidden, c.n_layers);
    const int CP = feat_stride(c);
    const int S = (int)total_feats((uint32_t)c.min_level, (uint32_t)c.max_level);
    const int ST = (int)feats_at_level((uint32_t)c.max_level);
    DS_CHECK_ARG(S * c.C <= kMaxSrc, "train_step: %d samples x %d channels exceed the per-triangle limit", S, c.C);
    DS_CHECK_ARG(num_pixels <= 0xffffffffLL, "train_step: more than 2^32 pixels");
    DS_CHECK_ARG(c.frag_records >= 0.f && record_capacity(c, num_tiles, num_pixels) <= 0x7fffffffLL - max_resident_warps() * kRecChunk,
                 "train_step: frag_records %g gives too many records", (double)c.frag_records);
    size_t need = 0;
    StepWs w = carve_step(workspace, c, num_tiles, num_pixels, list_capacity, &need);
    const RecordStore* rs = w.rec.capacity > 0 ? &w.rec : nullptr;
    if (workspace_bytes < need) return set_error(DS_ERR_WORKSPACE, "train_step: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;

    int rc = mark(0, st);
    if (rc) return rc;
    // Side stream for independent parts; the phase events (profiling) time
    // the phases one after another on st instead.
    SideStream* side = g_step_nevents == 0 ? side_stream() : nullptr;
    const cudaStream_t sst = side ? side->s : st;
    if (side && (rc = fork_to(side, 0, st))) return rc;

    // zero the accumulators of this step, beside the level accumulation
    DS_CUDA(cudaMemsetAsync(w.grad_pos, 0,
                            reinterpret_cast<char*>(w.rec_counters + 2) - reinterpret_cast<char*>(w.grad_pos), st));
    DS_CUDA(cudaMemsetAsync(grad_mlp_params, 0, sizeof(float) * ds_step_mlp_param_count(&c), st));

    // prep: opacity and feature accumulation + sigmoid (side), projection (st)
    const unsigned tb = (unsigned)((c.T + kPrepWarps - 1) / kPrepWarps);
    const bool tab = lattice_tab_fits(c.min_level, c.max_level, S, ST, CP);
    // one wave of persistent CTAs, each holding the rows once (EXTRA: the forward's CTA for the adjoint's rows)
#define DSB_TAB(KERNEL, BWD, EXTRA, CC, CPP, STREAM, ...)                                                          \
    do {                                                                                                           \
        const size_t tsm = lattice_tab_smem<CPP>(c.min_level, c.max_level, S, ST, BWD);                            \
        int per_sm = 1, trc = resident_ctas<KERNEL<CC, CPP>>(kMapWarps * 32, tsm, &per_sm);                        \
        if (trc) return trc;                                                                                       \
        const int per = kTabGroup<CPP> * (kMapWarps / kTabGroupWarps<CPP>); /* triangles of a CTA's pass */        \
        const int64_t want = ((int64_t)c.T + per - 1) / per;                                                       \
        const int64_t wave = (int64_t)sm_count() * per_sm - EXTRA;                                                 \
        const dim3 tgrid((unsigned)((want < wave ? want : wave) + EXTRA));                                         \
        if (BWD) /* after the opacity pass; the forward follows an event wait */                                   \
            launch_chained(KERNEL<CC, CPP>, tgrid, kMapWarps * 32, tsm, STREAM, c.T, c.min_level, c.max_level, S, ST, \
                           __VA_ARGS__);                                                                           \
        else                                                                                                       \
            KERNEL<CC, CPP><<<tgrid, kMapWarps * 32, tsm, STREAM>>>(c.T, c.min_level, c.max_level, S, ST,          \
                                                                    __VA_ARGS__);                                  \
    } while (0)
#define DSB_TAB_C(KERNEL, BWD, EXTRA, STREAM, ...)                                                                 \
    do {                                                                                                           \
        if (c.C == 8) DSB_TAB(KERNEL, BWD, EXTRA, 8, 8, STREAM, __VA_ARGS__);                                      \
        else if (c.C == 7) DSB_TAB(KERNEL, BWD, EXTRA, 7, 8, STREAM, __VA_ARGS__);                                 \
        else DSB_TAB(KERNEL, BWD, EXTRA, 16, 16, STREAM, __VA_ARGS__);                                             \
    } while (0)
    if (c.T > 0 && tab) {
        DSB_TAB_C(accum_tab_kernel, false, 1, sst, alpha_src, feat_src, w.alpha_acc, w.feat_acc, w.feat_bf16,
                  w.adj_ent, w.adj_row);
    } else if (c.T > 0) {
        accum_sigmoid_kernel<false><<<tb, kPrepWarps * 32, 0, sst>>>(c.T, c.min_level, c.max_level, c.max_level, S, ST,
                                                                    1, 1, alpha_src, w.alpha_acc, nullptr);
        accum_sigmoid_kernel<true><<<tb, kPrepWarps * 32, 0, sst>>>(c.T, c.min_level, c.max_level, c.max_level, S, ST,
                                                                   c.C, CP, feat_src, w.feat_acc, w.feat_bf16);
    }
    if ((int64_t)c.B * c.V > 0)
        project_kernel<<<blocks_for((int64_t)c.B * c.V), kThreads, 0, st>>>(c.B, c.V, verts, mvp, w.pos);
    rc = check_launch("train_step prep");
    if (rc || (rc = mark(1, st))) return rc;

    // forward rasterization
    float* rast = rast_out ? rast_out : w.rast;
    rc = ds_tiles_bin(c.B, views, num_tiles, c.V, w.pos, c.T, tri, w.tiles, w.tiles_bytes, list_capacity, status,
                      stream);
    if (rc || (rc = mark(2, st))) return rc;
    if (side && (rc = join_from(side, 0, st))) return rc;  // the rasterizer reads the accumulated opacities
    rc = tiles_rasterize_impl(c.B, views, num_tiles, c.T, c.max_level, ST, w.alpha_acc, c.stochastic ? 1 : 0,
                              c.thr_const, rng, rast, w.tiles, list_capacity, rs, st, block_shape_log2(c), side == nullptr);
    if (rc || (rc = mark(3, st))) return rc;

    // fused shading forward + backward
    ShadeArgs a;
    a.B = c.B; a.views = views; a.num_pixels = num_pixels; a.rast = rast; a.feat = w.feat_bf16;
    a.feat_f32 = w.feat_acc;
    a.level = c.max_level; a.S = ST; a.inv_mvp = inv_mvp; a.params = mlp_params;
    a.target = c.target_u8 ? nullptr : reinterpret_cast<const float*>(target);
    a.target_u8 = c.target_u8 ? reinterpret_cast<const uint8_t*>(target) : nullptr;
    a.inv_n = (float)(1.0 / ((double)num_pixels * 3.0));
    a.color = color_out ? color_out : w.color; a.grad_color = w.grad_color; a.l1 = w.l1;
    a.grad_feat = w.grad_feat_acc; a.grad_params = grad_mlp_params; a.loss_sum = w.loss_sum; a.status = status;
    const bool split = c.precision == 1;
    switch (shape) {
        case kShadeC8Dir16:
            rc = split ? launch_shade_reg<ShadeC8Dir16Split>(a, st) : launch_shade_reg<ShadeC8Dir16>(a, st);
            break;
        case kShadeC7Sh2_16x2:
            rc = split ? launch_shade_reg<ShadeC7Sh2_16x2Split>(a, st) : launch_shade_reg<ShadeC7Sh2_16x2>(a, st);
            break;
        default:
            if (split) rc = launch_shade<ShadeC16H64Split>(a, st);
            else rc = c.shade_mode == 1 ? launch_shade_tc(a, st) : launch_shade<ShadeC16H64>(a, st);
    }
    if (rc || (rc = mark(4, st))) return rc;

    // adjoints of sigmoid + level accumulation: they read the opacity and feature gradients, not the
    // vertex gradients, so with a side stream they run there after the opacity pass, beside the edge
    // gradients
    auto accum_backward = [&](cudaStream_t s) -> int {
        if (c.T > 0 && tab) {
            DSB_TAB_C(accum_tab_backward_kernel, true, 0, s, w.alpha_acc, w.grad_alpha_acc, w.feat_acc, w.grad_feat_acc,
                      grad_alpha_src, grad_feat_src, w.adj_ent, w.adj_row);
        } else if (c.T > 0) {
            accum_sigmoid_backward_kernel<<<tb, kPrepWarps * 32, 0, s>>>(c.T, c.min_level, c.max_level, c.max_level,
                                                                         S, ST, 1, 1, w.alpha_acc, w.grad_alpha_acc,
                                                                         grad_alpha_src);
            accum_sigmoid_backward_kernel<<<tb, kPrepWarps * 32, 0, s>>>(c.T, c.min_level, c.max_level, c.max_level,
                                                                         S, ST, c.C, CP, w.feat_acc,
                                                                         w.grad_feat_acc, grad_feat_src);
        }
        return DS_OK;
    };
#undef DSB_TAB_C
#undef DSB_TAB

    // opacity auxiliary gradient (scaled by 1/numel(colour), rasterize.py:183-195), on the side
    // stream beside the edge gradients
    if (side && (rc = fork_to(side, 1, st))) return rc;
    rc = tiles_aux_impl(c.B, views, num_tiles, c.T, c.max_level, ST, w.alpha_acc, w.l1, rast, a.inv_n,
                        w.grad_alpha_acc, w.tiles, list_capacity, rs, sst, block_shape_log2(c), side == nullptr);
    if (rc) return rc;
    if (side && (rc = accum_backward(sst))) return rc;
    if ((rc = mark(5, st))) return rc;

    // edge gradients to clip-space positions
    launch_chained(edge_step_kernel, dim3((unsigned)num_tiles), kEdgeThreads, 0, st, c.B, views, c.V, c.T,
                   tiles_tables(w.tiles, c.B, c.T, num_tiles, list_capacity), tri, a.color, w.grad_color, rast,
                   w.grad_pos);
    if ((rc = mark(6, st))) return rc;
    if (side && (rc = join_from(side, 1, st))) return rc;
    // (one stream: the phases in order, so that the profiling events time each alone)
    if (!side && (rc = accum_backward(st))) return rc;
    // adjoint of the projection
    project_backward_kernel<<<blocks_for(c.V > 0 ? c.V : 1), kThreads, 0, st>>>(
        c.B, c.V, mvp, w.grad_pos, grad_verts, w.loss_sum, a.inv_n, loss, c.stochastic ? rng : nullptr,
        w.rec_counters, status);
    if ((rc = mark(7, st))) return rc;
    return check_launch("train_step");
}

}  // extern "C"
