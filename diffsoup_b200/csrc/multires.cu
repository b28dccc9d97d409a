// diffsoup_b200/csrc/multires.cu -- multi-resolution barycentric features
// (kenji-tojo/diffsoup src/cuda/multires.cu) behind the C ABI.
//
// Forward gathers use 16-byte vector loads when the feature width allows it;
// the scatters use vector atomics (red.global.add.v4.f32, sm_90+) so one
// instruction updates four channels.
#include "lattice_map.cuh"
#include "rows.cuh"

namespace dsb {

// multires.cu:130-156: alpha per fragment.
__global__ void __launch_bounds__(kThreads) alpha_kernel(int n, const float* __restrict__ frag_attrs, uint32_t lo,
                                                         uint32_t hi, uint32_t S, const float* __restrict__ alpha_src,
                                                         float* __restrict__ frag_alpha) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = reinterpret_cast<const float4*>(frag_attrs)[i];
    const int t = (int)a.w - 1;
    if (t < 0) return;
    frag_alpha[i] = interp_scalar(a.x, a.y, lo, hi, alpha_src + (size_t)t * S);
}

// multires.cu:178-202
__global__ void __launch_bounds__(kThreads) alpha_backward_kernel(int n, const float* __restrict__ frag_attrs,
                                                                  uint32_t lo, uint32_t hi, uint32_t S,
                                                                  float* __restrict__ grad_alpha_src,
                                                                  const float* __restrict__ grad_frag_alpha) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = reinterpret_cast<const float4*>(frag_attrs)[i];
    const int t = (int)a.w - 1;
    if (t < 0) return;
    const float g = grad_frag_alpha[i];
    float* dst = grad_alpha_src + (size_t)t * S;
    uint32_t off = 0;
    for (uint32_t l = lo; l <= hi; ++l) {
        uint32_t idx[3]; float w[3];
        lattice_cell(a.x, a.y, l, idx, w);
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(dst + off + idx[k], g * w[k]);
        off += feats_at_level(l);
    }
}

// multires.cu:224-247: features per pixel, accumulated into out.
template <int VEC>
__global__ void __launch_bounds__(kThreads) color_kernel(int64_t n, const float* __restrict__ rast, uint32_t lo,
                                                         uint32_t hi, uint32_t S, int C,
                                                         const float* __restrict__ feat, float* __restrict__ out) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const float4 r = reinterpret_cast<const float4*>(rast)[p];
    const int t = (int)r.w - 1;
    if (t < 0) return;
    const float* tf = feat + (size_t)t * S * C;
    float* o = out + (size_t)p * C;
    uint32_t off = 0;
    for (uint32_t l = lo; l <= hi; ++l) {
        uint32_t idx[3]; float w[3];
        lattice_cell(r.x, r.y, l, idx, w);
        if (VEC == 4) {
            for (int c = 0; c < C; c += 4) {
                float4 acc = *reinterpret_cast<float4*>(o + c);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float4 f = __ldg(reinterpret_cast<const float4*>(tf + (size_t)(off + idx[k]) * C + c));
                    acc.x = madd(acc.x, w[k], f.x); acc.y = madd(acc.y, w[k], f.y);
                    acc.z = madd(acc.z, w[k], f.z); acc.w = madd(acc.w, w[k], f.w);
                }
                *reinterpret_cast<float4*>(o + c) = acc;
            }
        } else {
            for (int c = 0; c < C; ++c) {
                float acc = o[c];
#pragma unroll
                for (int k = 0; k < 3; ++k) acc = madd(acc, w[k], __ldg(tf + (size_t)(off + idx[k]) * C + c));
                o[c] = acc;
            }
        }
        off += feats_at_level(l);
    }
}

// Seven-channel rows (the reference's own model) of a 16-byte aligned table:
// row r starts at float 7 r, so it is one aligned group of four floats, one of
// two and one single, whose places depend on 7 r mod 4 alone:
//   7 r mod 4 = 0: four at 0, two at 4, one at 6      1: one at 0, two at 1, four at 3
//               2: two at 0, four at 2, one at 6      3: one at 0, four at 1, two at 5
struct Row7 {
    int a, four, two, one;
    __device__ explicit Row7(uint32_t r) {
        a = (int)((7u * r) & 3u);
        four = (4 - a) & 3;
        two = a == 0 ? 4 : (a == 1 ? 1 : (a == 2 ? 0 : 5));
        one = (a & 1) ? 0 : 6;
    }
    // v[0..6] of the row at p
    __device__ void load(const float* __restrict__ p, float v[7]) const {
        const float4 f = __ldg(reinterpret_cast<const float4*>(p + four));
        const float2 t = __ldg(reinterpret_cast<const float2*>(p + two));
        const float o = __ldg(p + one);
        v[0] = a == 0 ? f.x : (a == 2 ? t.x : o);
        v[1] = a == 0 ? f.y : (a == 1 ? t.x : (a == 2 ? t.y : f.x));
        v[2] = a == 0 ? f.z : (a == 1 ? t.y : (a == 2 ? f.x : f.y));
        v[3] = a == 0 ? f.w : (a == 1 ? f.x : (a == 2 ? f.y : f.z));
        v[4] = a == 0 ? t.x : (a == 1 ? f.y : (a == 2 ? f.z : f.w));
        v[5] = a == 0 ? t.y : (a == 1 ? f.z : (a == 2 ? f.w : t.x));
        v[6] = a == 0 || a == 2 ? o : (a == 1 ? f.w : t.y);
    }
    // adds w * v[0..6] to the row at p
    __device__ void add(float* __restrict__ p, const float v[7], float w) const {
        const float f0 = a == 0 ? v[0] : (a == 1 ? v[3] : (a == 2 ? v[2] : v[1]));
        const float f1 = a == 0 ? v[1] : (a == 1 ? v[4] : (a == 2 ? v[3] : v[2]));
        const float f2 = a == 0 ? v[2] : (a == 1 ? v[5] : (a == 2 ? v[4] : v[3]));
        const float f3 = a == 0 ? v[3] : (a == 1 ? v[6] : (a == 2 ? v[5] : v[4]));
        const float t0 = a == 0 ? v[4] : (a == 1 ? v[1] : (a == 2 ? v[0] : v[5]));
        const float t1 = a == 0 ? v[5] : (a == 1 ? v[2] : (a == 2 ? v[1] : v[6]));
        const float o = (a & 1) ? v[0] : v[6];
        atomicAdd(reinterpret_cast<float4*>(p + four), make_float4(f0 * w, f1 * w, f2 * w, f3 * w));
        atomicAdd(reinterpret_cast<float2*>(p + two), make_float2(t0 * w, t1 * w));
        atomicAdd(p + one, o * w);
    }
};

// Zeroes the rows (C floats each, from g on) of the lanes in `rows`, by the whole
// warp in runs: a row a lane would be C / 4 stores a row apart.
__device__ __forceinline__ void zero_rows(float* g, uint32_t C, unsigned rows) {
    const uint32_t lane = threadIdx.x & 31;
    if (((uintptr_t)g & 15) == 0 && (C % 4 == 0 || rows == 0xffffffffu)) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t i = lane; i < 8 * C; i += 32)
            if ((rows >> (i * 4 / C)) & 1u) reinterpret_cast<float4*>(g)[i] = z;
    } else {
        for (uint32_t i = lane; i < 32 * C; i += 32)
            if ((rows >> (i / C)) & 1u) g[i] = 0.f;
    }
}

// color_kernel with every pixel written (background pixels zero): no zeroed
// buffer and no read of it.  The covered pixels' rows are stored
//   kLookupNarrow  by their lanes, four channels at a time, background rows by the same stores: rows of four
//                channels are half a sector, and apart from one another the two kinds of rows write it twice;
//   kLookupVec4  by their lanes, four channels at a time;
//   kLookupRow7  (seven channels of an aligned table, read as Row7) and
//   kLookupTile  through shared memory, so that a warp's 32 rows leave as one run of
//                aligned 16-byte stores;
//   kLookupRows  by their lanes, a channel at a time, onto rows zeroed first: the read brings the line that
//                the stores then share (two views of 800x800, 60,000 triangles on nine tenths of the pixels, 33 channels:
//                289 us with a zeroed buffer, 337 stored without the read, 286 so).
// Background pixels are zeroed by whole warps.  Two views of 800x800, 500 triangles on a twentieth of the pixels,
// 32 channels: 43 us with a zeroed buffer, 91 with every lane zeroing its own row, 32 so; 60,000
// triangles on nine tenths: 181, 115 and 105.  4 views of 800x800, 7 channels: 53, 12 of them
// zeroing, -> 39 us.
enum { kLookupNarrow, kLookupVec4, kLookupRow7, kLookupTile, kLookupRows };
// Channels up to which kLookupTile is taken: its shared memory stays below the 48 KB of a plain launch.  31
// channels on nine tenths as above: 267 us with a zeroed buffer, 309 by lanes, 152 through the tile.
constexpr int kColorTile = 32;
// Channels up to which kLookupNarrow is taken.  4 views of 800x800, 15,000 triangles on half of the pixels, 4 / 8
// channels: 18 / 33 us, 25 / 37 as kLookupVec4; 894x670, 5 views, 16: 68, 62.
constexpr int kLookupNarrowest = 8;

template <int MODE>
__global__ void __launch_bounds__(kThreads) color_set_kernel(int64_t n, const float* __restrict__ rast, uint32_t lo,
                                                             uint32_t hi, uint32_t S, int C,
                                                             const float* __restrict__ feat, float* __restrict__ out) {
    extern __shared__ __align__(16) float color_smem[];
    constexpr bool STAGED = MODE == kLookupRow7 || MODE == kLookupTile;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int64_t p0 = p - lane;
    const bool in = p < n;
    if (MODE == kLookupNarrow && !in) return;
    const float4 r = in ? reinterpret_cast<const float4*>(rast)[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int t = (int)r.w - 1;
    if (MODE == kLookupNarrow) {
        uint32_t idx[3]; float w[3];
        lattice_cell(r.x, r.y, lo, idx, w);
        for (int c = 0; c < C; c += 4) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t off = 0;
            for (uint32_t l = lo; t >= 0 && l <= hi; ++l) {
                if (lo < hi) lattice_cell(r.x, r.y, l, idx, w);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float4 f =
                        __ldg(reinterpret_cast<const float4*>(feat + ((size_t)t * S + off + idx[k]) * C + c));
                    acc.x = madd(acc.x, w[k], f.x); acc.y = madd(acc.y, w[k], f.y);
                    acc.z = madd(acc.z, w[k], f.z); acc.w = madd(acc.w, w[k], f.w);
                }
                off += feats_at_level(l);
            }
            *reinterpret_cast<float4*>(out + (size_t)p * C + c) = acc;
        }
        return;
    }
    const unsigned zero = __ballot_sync(0xffffffffu, in && (t < 0 || MODE == kLookupRows));
    if (STAGED ? zero == 0xffffffffu : zero != 0u) zero_rows(out + (size_t)p0 * C, (uint32_t)C, zero);
    if (MODE == kLookupRows) __syncwarp();
    if (STAGED ? zero == 0xffffffffu : t < 0) return;
    float* tile = color_smem + (threadIdx.x >> 5) * 32 * C;
    float* o = STAGED ? tile + lane * C : out + (size_t)p * C;
    if (MODE == kLookupRow7) {
        float acc[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        uint32_t off = 0;
        for (uint32_t l = lo; t >= 0 && l <= hi; ++l) {
            uint32_t idx[3]; float w[3];
            lattice_cell(r.x, r.y, l, idx, w);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const size_t row = (size_t)t * S + off + idx[k];
                float v[7];
                Row7((uint32_t)row).load(feat + row * 7, v);
#pragma unroll
                for (int c = 0; c < 7; ++c) acc[c] = madd(acc[c], w[k], v[c]);
            }
            off += feats_at_level(l);
        }
#pragma unroll
        for (int c = 0; c < 7; ++c) o[c] = acc[c];
    } else if (t < 0) {
        for (int c = 0; c < C; ++c) o[c] = 0.f;
    } else {
        const float* tf = feat + (size_t)t * S * C;
        for (uint32_t l = lo; l <= hi; ++l) {
            uint32_t idx[3]; float w[3];
            lattice_cell(r.x, r.y, l, idx, w);
            if (MODE == kLookupVec4) {
                for (int c = 0; c < C; c += 4) {
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (l > lo) acc = *reinterpret_cast<const float4*>(o + c);
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float4 f = __ldg(reinterpret_cast<const float4*>(tf + (size_t)idx[k] * C + c));
                        acc.x = madd(acc.x, w[k], f.x); acc.y = madd(acc.y, w[k], f.y);
                        acc.z = madd(acc.z, w[k], f.z); acc.w = madd(acc.w, w[k], f.w);
                    }
                    *reinterpret_cast<float4*>(o + c) = acc;
                }
            } else {
                for (int c = 0; c < C; ++c) {
                    float acc = l > lo || MODE == kLookupRows ? o[c] : 0.f;
#pragma unroll
                    for (int k = 0; k < 3; ++k) acc = madd(acc, w[k], __ldg(tf + (size_t)idx[k] * C + c));
                    o[c] = acc;
                }
            }
            tf += (size_t)feats_at_level(l) * C;
        }
    }
    if (!STAGED) return;
    __syncwarp();
    if (p0 < n) warp_rows<true>(tile, out + (size_t)p0 * C, C, n - p0 < 32 ? (int)(n - p0) : 32);
}

// multires.cu:268-292: scatter of per-pixel feature gradients.  VEC 4: one
// vector atomic per four channels; ROW7: three vector atomics a row (Row7)
// instead of seven scalar ones, the gradient's rows through shared memory.  The
// atomics' rate at L2 is the bound.  4 views of 800x800, 7
// channels: 221 -> 103 us.
template <int VEC, bool ROW7>
__global__ void __launch_bounds__(kThreads) color_backward_kernel(int64_t n, const float* __restrict__ rast,
                                                                  uint32_t lo, uint32_t hi, uint32_t S, int C,
                                                                  float* __restrict__ grad_feat,
                                                                  const float* __restrict__ grad_out) {
    __shared__ __align__(16) float s_rows[ROW7 ? kThreads / 32 : 1][ROW7 ? 32 * 7 : 4];
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    float row[7];
    if (ROW7) {
        const int64_t p0 = p - lane;
        if (p0 >= n) return;
        float* tile = s_rows[threadIdx.x >> 5];
        warp_rows<false>(tile, const_cast<float*>(grad_out) + (size_t)p0 * 7, 7, n - p0 < 32 ? (int)(n - p0) : 32);
#pragma unroll
        for (int c = 0; c < 7; ++c) row[c] = tile[lane * 7 + c];
    }
    if (p >= n) return;
    const float4 r = reinterpret_cast<const float4*>(rast)[p];
    const int t = (int)r.w - 1;
    if (t < 0) return;
    float* tg = grad_feat + (size_t)t * S * C;
    const float* g = grad_out + (size_t)p * C;
    uint32_t off = 0;
    for (uint32_t l = lo; l <= hi; ++l) {
        uint32_t idx[3]; float w[3];
        lattice_cell(r.x, r.y, l, idx, w);
        if (ROW7) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const size_t at = (size_t)t * S + off + idx[k];
                Row7((uint32_t)at).add(grad_feat + at * 7, row, w[k]);
            }
        } else if (VEC == 4) {
            for (int c = 0; c < C; c += 4) {
                const float4 gv = __ldg(reinterpret_cast<const float4*>(g + c));
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    atomicAdd(reinterpret_cast<float4*>(tg + (size_t)(off + idx[k]) * C + c),
                              make_float4(gv.x * w[k], gv.y * w[k], gv.z * w[k], gv.w * w[k]));
            }
        } else {
            for (int c = 0; c < C; ++c) {
                const float gv = __ldg(g + c);
#pragma unroll
                for (int k = 0; k < 3; ++k) atomicAdd(tg + (size_t)(off + idx[k]) * C + c, gv * w[k]);
            }
        }
        off += feats_at_level(l);
    }
}

// The scatter at one level with the pixels of a lattice cell summed before the
// atomics, which bound the kernel above: a warp takes 8x4 pixels of a view,
// groups those of one (triangle, cell), and an item (group, sample and, of eight or more
// channels, a group of four) sums its members' weighted rows and issues the atomics of
// one row, its members shared by eight or four lanes where there are up to four or eight items (801x603, one cell a
// triangle of 64 pixels, 7 channels: 21 us, 13 so; sharing by a run-time count at more items cost 10%
// where cells are small).  Where less than a third of the warp's pixels would be merged they go out
// per pixel.  4 views of 800x800, 7 channels: 103 -> 43 us.
constexpr int kMergeRow = 32;  // channels up to which the rows are staged
// Rows of at least this many channels are merged: one vector atomic a sample is as cheap as the merging. 4 channels, a
// thread per pixel / merged: shell of 15,000 triangles, 4 views of 800x800, 29 / 33 us, of 3,000, one view of 801x603 at
// level 1, 15 / 21, boxes of 60,000 and 50,000 64 / 52, 117 / 93; 8 channels, the first, 60 / 49.
constexpr int kMergeFrom = 7;
// Quads of channels from which unmerged pixels go out as items too, the lanes of a row beside one another: triangle IDs
// drawn by pixel, two views of 800x800, 60,000 / 100 triangles, 32 channels: 237 / 414 us a lane per pixel, 207 / 191 as
// items.  Narrower rows are the faster by pixel where a scene's triangles leave few warps unmerged (894x670, 12,000
// triangles, 16 channels at level 3: 60 us, 72 as items).
constexpr int kMergeQuads = 8;

// Floats between the staged rows: the row and its three weights, an odd number of floats, or of
// groups of four, so that the rows of eight lanes fall in different banks (12 channels 88 us with 16 floats,
// 72 with 20).
__host__ __device__ constexpr int merge_stride(int C) { return C == 7 ? 11 : C + 4 + (C & 4); }

// The items (group, sample, quad) of a warp, each by 1 << SHARE lanes.
template <bool ROW7, int SHARE>
__device__ __forceinline__ void merge_items(int items, int Q, int lane, int stride, const float* rows, const int* meta,
                                            uint32_t S, int C, float* __restrict__ grad_feat) {
    constexpr unsigned kPart = SHARE == 0 ? 0xffffffffu : SHARE == 2 ? 0x11111111u : 0x01010101u;
    const int first = lane >> SHARE, own = lane & ((1 << SHARE) - 1);
    for (int n0 = 0; n0 < items; n0 += 32 >> SHARE) {  // warp-uniform
        const int n = n0 + first;
        const bool some = n < items;
        if (SHARE == 0 && !some) break;
        const int gi = n / (3 * Q), rest = n - gi * 3 * Q, k = rest / Q, c = (rest - k * Q) * 4;
        const int* g = meta + gi * 5;
        float v[ROW7 ? 7 : 4];
#pragma unroll
        for (int j = 0; j < (ROW7 ? 7 : 4); ++j) v[j] = 0.f;
        for (unsigned members = some ? (unsigned)g[0] & (kPart << own) : 0u; members != 0; members &= members - 1u) {
            const float* m = rows + (__ffs(members) - 1) * stride;
            const float wk = m[C + k];
#pragma unroll
            for (int j = 0; j < (ROW7 ? 7 : 4); ++j) v[j] = fmaf(wk, m[c + j], v[j]);
        }
#pragma unroll
        for (int d = 1; d < 1 << SHARE; d += d)
#pragma unroll
            for (int j = 0; j < (ROW7 ? 7 : 4); ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], d);
        if (!some || own != 0) continue;
        const size_t at = (size_t)g[1] * S + (size_t)g[2 + k];
        if (ROW7) Row7((uint32_t)at).add(grad_feat + at * 7, v, 1.f);
        else atomicAdd(reinterpret_cast<float4*>(grad_feat + at * C + c), make_float4(v[0], v[1], v[2], v[3]));
    }
}

template <bool ROW7>
__global__ void __launch_bounds__(kThreads) color_backward_merge_kernel(int H, int W, int bx, int64_t blocks, int per_view,
                                                                        const float* __restrict__ rast,
                                                                        uint32_t level, uint32_t S, int C,
                                                                        float* __restrict__ grad_feat,
                                                                        const float* __restrict__ grad_out) {
    extern __shared__ __align__(16) float merge_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t block = (int64_t)blockIdx.x * (kThreads / 32) + warp;
    if (block >= blocks) return;  // warp-uniform
    const int stride = merge_stride(C);
    float* rows = merge_smem + (size_t)warp * (32 * stride + 160);
    int* meta = reinterpret_cast<int*>(rows + 32 * stride);
    const int64_t b = block / per_view;
    const int i = (int)(block - b * per_view), y0 = i / bx * 4, x0 = (i - i / bx * bx) * 8;
    const int y = y0 + (lane >> 3), x = x0 + (lane & 7);
    const bool in = y < H && x < W;
    const int64_t p = (b * H + y) * W + x;
    const float4 r = in ? reinterpret_cast<const float4*>(rast)[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int t = (int)r.w - 1;
    const bool covered = in && t >= 0;
    const unsigned live = __ballot_sync(0xffffffffu, covered);
    if (live == 0u) return;
    uint32_t idx[3];
    float w[3];
    lattice_cell(r.x, r.y, level, idx, w);
    float* mine = rows + lane * stride;
    if (covered) {
        const float* g = grad_out + p * C;
        if (ROW7) {
#pragma unroll
            for (int c = 0; c < 7; ++c) mine[c] = __ldg(g + c);
        } else {
            for (int c = 0; c < C; c += 4)
                *reinterpret_cast<float4*>(mine + c) = __ldg(reinterpret_cast<const float4*>(g + c));
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) mine[C + k] = w[k];
    }
    // a cell is its first two samples and the place of the third among them
    const unsigned long long key =
        covered ? ((unsigned long long)(unsigned)t << 34) | ((unsigned long long)(idx[0] & 0xffffu) << 18) |
                      ((unsigned long long)(idx[1] & 0xffffu) << 2) | (idx[2] == idx[0] ? 2u : (idx[2] > idx[1] ? 1u : 0u))
                : ~0ull;
    // Grouping is tried where it can merge a third of the pixels: as many must share a cell with the pixel beside or
    // above them (by a hash of the key), for a cell's pixels hang together.  It is slow for many different keys
    // (60,000 triangles, one a pixel, two views of 800x800, 8 channels: 47 us without it, 54 with it always, 49 so).
    const unsigned mix = (unsigned)key ^ ((unsigned)(key >> 32) * 0x9e3779b1u);
    const unsigned beside = __shfl_down_sync(0xffffffffu, mix, 1), above = __shfl_down_sync(0xffffffffu, mix, 8);
    const int pairs = __popc(__ballot_sync(0xffffffffu, covered && (lane & 7) != 7 && beside == mix)) +
                      __popc(__ballot_sync(0xffffffffu, covered && lane < 24 && above == mix));
    unsigned peers = 0u, leaders = live;
    bool leader = false;
    if (3 * pairs >= __popc(live)) {
        peers = __match_any_sync(0xffffffffu, key);
        leader = covered && lane == __ffs(peers) - 1;
        leaders = __ballot_sync(0xffffffffu, leader);
    }
    const int Q = ROW7 ? 1 : C / 4;
    int groups = __popc(leaders);
    if (3 * groups > 2 * __popc(live) && Q >= kMergeQuads) {
        peers = 1u << lane;  // each pixel an item's only member
        leader = covered;
        leaders = live;
        groups = __popc(live);
    } else if (3 * groups > 2 * __popc(live)) {
        if (!covered) return;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const size_t at = (size_t)t * S + idx[k];
            if (ROW7) {
                Row7((uint32_t)at).add(grad_feat + at * 7, mine, w[k]);
            } else {
                for (int c = 0; c < C; c += 4) {
                    const float4 g = *reinterpret_cast<const float4*>(mine + c);
                    atomicAdd(reinterpret_cast<float4*>(grad_feat + at * C + c),
                              make_float4(g.x * w[k], g.y * w[k], g.z * w[k], g.w * w[k]));
                }
            }
        }
        return;
    }
    if (leader) {
        int* g = meta + __popc(leaders & ((1u << lane) - 1u)) * 5;
        g[0] = (int)peers; g[1] = t; g[2] = (int)idx[0]; g[3] = (int)idx[1]; g[4] = (int)idx[2];
    }
    __syncwarp();
    const int items = groups * 3 * Q;
    if (items <= 4)
        merge_items<ROW7, 3>(items, Q, lane, stride, rows, meta, S, C, grad_feat);
    else if (items <= 8)
        merge_items<ROW7, 2>(items, Q, lane, stride, rows, meta, S, C, grad_feat);
    else
        merge_items<ROW7, 0>(items, Q, lane, stride, rows, meta, S, C, grad_feat);
}

// The level accumulation through the map's tables (lattice_map.cuh), forward
// or adjoint: in [T, n_in / C, C] -> out [T, rows, C].  SET: out is
// overwritten, else added to atomically (out's other writers are unknown).
//
// 60,000 triangles, levels 0..3, 7 channels (191 MB read and written each way):
// forward 262 -> 73 us, adjoint 1169 (17 of them zeroing) -> 79 us against one thread per target
// sample (accumulate_*_kernel below), whose channel loops read and wrote
// through global memory 4 bytes at a time and whose adjoint issued 21 scalar atomics
// per target sample and level.  Shared-memory latency (short scoreboard) and the loads
// share what is left; two triangles a pass instead of four, or a deeper unrolling of
// the row loop, measured the same within 3%.
template <int I, bool ADJOINT, bool SET>
__global__ void __launch_bounds__(kMapWarps * 32) accumulate_map_kernel(int T, int lo, int hi, int target, int S,
                                                                       int ST, int C, const float* __restrict__ in,
                                                                       float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char map_smem[];
    const int rows = ADJOINT ? S : ST, N = ST * (hi - lo + 1) * 3;
    const MapTables m = map_tables_at(map_smem, N, rows);
    if (ADJOINT) build_adjoint_rows(m, lo, hi, target, ST, S);
    else build_forward_rows(m, lo, hi, target, ST);
    const int n_in = (ADJOINT ? ST : S) * C, n_out = rows * C;
    const int warp = threadIdx.x >> 5;
    float* tile = reinterpret_cast<float*>(map_smem + map_table_bytes(N, rows)) + (size_t)warp * n_in * I;
    const float inv_c = 1.f / (float)C;
    for (int64_t t = ((int64_t)blockIdx.x * kMapWarps + warp) * I; t < T; t += (int64_t)gridDim.x * kMapWarps * I)
        map_triangles<I>(
            m, (int)t, T, n_in, n_out, tile, [&](int q, int e) { return __ldg(in + (size_t)q * n_in + e); },
            [&](int s, int& row, int& base, int& stride) {
                row = (int)(((float)s + 0.5f) * inv_c);  // s / C (s + 1/2 keeps the product off the integers)
                base = s - row * C;
                stride = C;
            },
            [&](int q, int s, float v) {
                float* o = out + (size_t)q * n_out + s;
                if (SET) *o = v; else atomicAdd(o, v);
            });
}

// multires.cu:329-369: evaluate levels [lo, hi] at the target lattice vertices.
__global__ void __launch_bounds__(kThreads) accumulate_forward_kernel(int T, uint32_t lo, uint32_t hi, uint32_t target,
                                                                      uint32_t S, uint32_t ST, int C,
                                                                      const float* __restrict__ feat,
                                                                      float* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)T * ST) return;
    const uint32_t t = (uint32_t)(i / ST), k = (uint32_t)(i % ST);
    uint32_t x, y;
    index_to_xy(k, x, y);
    const float R = (float)(1u << target);
    const float b0 = __fdiv_rn((float)x, R), b1 = __fdiv_rn((float)y, R);
    const float* tf = feat + (size_t)t * S * C;
    float* o = out + (size_t)i * C;
    for (int c = 0; c < C; ++c) o[c] = 0.f;
    uint32_t off = 0;
    for (uint32_t l = lo; l <= hi; ++l) {
        uint32_t idx[3]; float w[3];
        lattice_cell(b0, b1, l, idx, w);
        for (int c = 0; c < C; ++c) {
            float acc = o[c];
#pragma unroll
            for (int q = 0; q < 3; ++q) acc = madd(acc, w[q], __ldg(tf + (size_t)(off + idx[q]) * C + c));
            o[c] = acc;
        }
        off += feats_at_level(l);
    }
}

// Zeroes n floats, a group of four a thread (1.8 MB and the additions of 153,000 samples after it: 10.3 us, with
// a memset 12.2).
__global__ void __launch_bounds__(kThreads) zero_floats_kernel(int64_t n, float* __restrict__ p) {
    const int64_t i = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * 4;
    if (i + 4 <= n && ((uintptr_t)p & 15) == 0) {
        *reinterpret_cast<float4*>(p + i) = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        for (int64_t k = i; k < i + 4 && k < n; ++k) p[k] = 0.f;
    }
}

// multires.cu:393-430
__global__ void __launch_bounds__(kThreads) accumulate_backward_kernel(int T, uint32_t lo, uint32_t hi,
                                                                       uint32_t target, uint32_t S, uint32_t ST, int C,
                                                                       float* __restrict__ grad_feat,
                                                                       const float* __restrict__ grad_out) {
    chain_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)T * ST) return;
    const uint32_t t = (uint32_t)(i / ST), k = (uint32_t)(i % ST);
    uint32_t x, y;
    index_to_xy(k, x, y);
    const float R = (float)(1u << target);
    const float b0 = __fdiv_rn((float)x, R), b1 = __fdiv_rn((float)y, R);
    float* tg = grad_feat + (size_t)t * S * C;
    const float* g = grad_out + (size_t)i * C;
    uint32_t off = 0;
    for (uint32_t l = lo; l <= hi; ++l) {
        uint32_t idx[3]; float w[3];
        lattice_cell(b0, b1, l, idx, w);
        for (int c = 0; c < C; ++c) {
            const float gv = __ldg(g + c);
#pragma unroll
            for (int q = 0; q < 3; ++q) atomicAdd(tg + (size_t)(off + idx[q]) * C + c, gv * w[q]);
        }
        off += feats_at_level(l);
    }
}

static bool levels_ok(int lo, int hi) { return lo >= 0 && hi >= lo && hi <= 12; }
static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// The map's tables and tiles in shared memory, or *interleave = 0 where the
// kernels of one thread per target sample run: lattices whose pairs or samples
// outgrow shared memory (beyond levels 0..4 with 16 channels or so), and calls in which those kernels are
// faster.  The lines were laid between 1,791 forms timed on both sides (22 ranges of levels, 1 to 128 channels, 10 to
// 100,000 triangles); on their side of them, those that take the map lose to the other kernel by at most 2.5 us:
//   * both: the map reads all S samples of a triangle and the other kernel only the N pairs' (levels 0..5 at level 2,
//     30,000 triangles of 7 channels: N = 270, S = 783, forward 270 us against 102);
//   * forward: less than a pass of one CTA an SM leaves SMs idle while the others build the tables (levels 2..2 at level 4,
//     100 triangles of 8 channels: 18.6 against 6.3 us), and a few values a triangle are not worth the tables at all
//     (level 0, 100,000 triangles of 3 channels: 10.4 against 6.7 us);
//   * adjoint: kMapMinProducts atomic additions (of three) end before the tables are built (level 4, 3,000 triangles of 3
//     channels: 19.1 against 16.6 us; of 4 channels 20.6 against 22.7).
constexpr int kMapMaxPairs = 2400;
constexpr int kMapMinValues = 32;
constexpr int64_t kMapMinProducts = 1500000;

static size_t map_smem_bytes(int64_t T, int lo, int hi, int S, int ST, int C, bool adjoint, int* interleave) {
    *interleave = 0;
    const int NL = hi - lo + 1;
    if ((int64_t)ST * NL * 3 > kMapMaxPairs || (int64_t)(S > ST ? S : ST) * C > 6 * 1024) return 0;
    const int N = ST * NL * 3, n_in = (adjoint ? ST : S) * C, I = map_interleave(n_in);
    if (adjoint ? 2 * N < S || T * ST * NL * C < kMapMinProducts
                : 4 * N < 5 * S || T < (int64_t)I * kMapWarps * sm_count() || ST * NL * C < kMapMinValues)
        return 0;
    *interleave = I;
    return map_table_bytes(N, adjoint ? S : ST) + (size_t)kMapWarps * n_in * *interleave * sizeof(float);
}

template <int I, bool ADJOINT, bool SET>
static int launch_map(size_t smem, int T, int lo, int hi, int target, int S, int ST, int C, const float* in,
                      float* out, cudaStream_t st) {
    int per_sm = 1;
    const int rc = resident_ctas<accumulate_map_kernel<I, ADJOINT, SET>>(kMapWarps * 32, smem, &per_sm);
    if (rc) return rc;
    const int64_t want = ((int64_t)T + I * kMapWarps - 1) / (I * kMapWarps);
    const int64_t wave = (int64_t)sm_count() * per_sm;  // the tables are built once per CTA
    accumulate_map_kernel<I, ADJOINT, SET><<<(unsigned)(want < wave ? want : wave), kMapWarps * 32, smem, st>>>(
        T, lo, hi, target, S, ST, C, in, out);
    return check_launch("accumulate_to_level");
}

template <bool ADJOINT, bool SET>
static int launch_map_any(int interleave, size_t smem, int T, int lo, int hi, int target, int S, int ST, int C,
                          const float* in, float* out, cudaStream_t st) {
    if (interleave == 4) return launch_map<4, ADJOINT, SET>(smem, T, lo, hi, target, S, ST, C, in, out, st);
    if (interleave == 2) return launch_map<2, ADJOINT, SET>(smem, T, lo, hi, target, S, ST, C, in, out, st);
    return launch_map<1, ADJOINT, SET>(smem, T, lo, hi, target, S, ST, C, in, out, st);
}

static int accumulate_backward(bool set, int T, int min_level, int max_level, int target_level, int S, int S_target,
                               int C, float* grad_features, const float* grad_out, cudaStream_t st) {
    DS_CHECK_ARG(T >= 0 && C > 0 && levels_ok(min_level, max_level) && target_level >= 0 && target_level <= 12,
                 "accumulate_to_level_backward: bad sizes");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    DS_CHECK_ARG((uint32_t)S_target == feats_at_level(target_level), "Invalid feature size.");
    const int64_t n = (int64_t)T * S_target;
    if (n == 0) return DS_OK;
    int interleave = 0;
    const size_t smem = map_smem_bytes(T, min_level, max_level, S, S_target, C, true, &interleave);
    if (interleave > 0)
        return set ? launch_map_any<true, true>(interleave, smem, T, min_level, max_level, target_level, S, S_target, C,
                                                grad_out, grad_features, st)
                   : launch_map_any<true, false>(interleave, smem, T, min_level, max_level, target_level, S, S_target,
                                                 C, grad_out, grad_features, st);
    const int64_t floats = (int64_t)T * S * C;
    if (set) zero_floats_kernel<<<blocks_for((floats + 3) / 4), kThreads, 0, st>>>(floats, grad_features);
    launch_kernel(set, accumulate_backward_kernel, dim3(blocks_for(n)), kThreads, 0, st, T, min_level, max_level,
                  target_level, S, S_target, C, grad_features, grad_out);
    return check_launch("accumulate_to_level_backward");
}

}  // namespace dsb

using namespace dsb;

extern "C" {

int ds_multires_triangle_alpha(int num_frags, const float* frag_attrs, int min_level, int max_level, int S,
                               const float* alpha_src, float* frag_alpha, ds_stream_t stream) {
    DS_CHECK_ARG(num_frags >= 0 && levels_ok(min_level, max_level), "multires_triangle_alpha: bad levels");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    if (num_frags == 0) return DS_OK;
    DS_CHECK_ARG(aligned16(frag_attrs), "multires_triangle_alpha: frag_attrs not 16-byte aligned");
    alpha_kernel<<<blocks_for(num_frags), kThreads, 0, (cudaStream_t)stream>>>(num_frags, frag_attrs, min_level,
                                                                               max_level, S, alpha_src, frag_alpha);
    return check_launch("multires_triangle_alpha");
}

int ds_backward_multires_triangle_alpha(int num_frags, const float* frag_attrs, int min_level, int max_level, int S,
                                        float* grad_alpha_src, const float* grad_frag_alpha, ds_stream_t stream) {
    DS_CHECK_ARG(num_frags >= 0 && levels_ok(min_level, max_level), "backward_multires_triangle_alpha: bad levels");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    if (num_frags == 0) return DS_OK;
    DS_CHECK_ARG(aligned16(frag_attrs), "backward_multires_triangle_alpha: frag_attrs not 16-byte aligned");
    alpha_backward_kernel<<<blocks_for(num_frags), kThreads, 0, (cudaStream_t)stream>>>(
        num_frags, frag_attrs, min_level, max_level, S, grad_alpha_src, grad_frag_alpha);
    return check_launch("backward_multires_triangle_alpha");
}

int ds_multires_triangle_color(int B, int H, int W, const float* rast, int min_level, int max_level, int S, int C,
                               const float* features, float* out, ds_stream_t stream) {
    DS_CHECK_ARG(B >= 0 && H >= 0 && W >= 0 && C > 0 && levels_ok(min_level, max_level),
                 "multires_triangle_color: bad sizes");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    const int64_t n = (int64_t)B * H * W;
    if (n == 0) return DS_OK;
    DS_CHECK_ARG(aligned16(rast), "multires_triangle_color: rast not 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    if (C % 4 == 0 && aligned16(features) && aligned16(out))
        color_kernel<4><<<blocks_for(n), kThreads, 0, st>>>(n, rast, min_level, max_level, S, C, features, out);
    else
        color_kernel<1><<<blocks_for(n), kThreads, 0, st>>>(n, rast, min_level, max_level, S, C, features, out);
    return check_launch("multires_triangle_color");
}

int ds_multires_triangle_color_set(int B, int H, int W, const float* rast, int min_level, int max_level, int S, int C,
                                   const float* features, float* out, ds_stream_t stream) {
    DS_CHECK_ARG(B >= 0 && H >= 0 && W >= 0 && C > 0 && levels_ok(min_level, max_level),
                 "multires_triangle_color: bad sizes");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    const int64_t n = (int64_t)B * H * W;
    if (n == 0) return DS_OK;
    DS_CHECK_ARG(aligned16(rast), "multires_triangle_color: rast not 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t tile = (size_t)kThreads * C * sizeof(float);
    const bool vec = C % 4 == 0 && aligned16(features) && aligned16(out);
    const auto kernel = vec && C <= kLookupNarrowest    ? color_set_kernel<kLookupNarrow>
                        : vec                           ? color_set_kernel<kLookupVec4>
                        : C == 7 && aligned16(features) ? color_set_kernel<kLookupRow7>
                        : C <= kColorTile               ? color_set_kernel<kLookupTile>
                                                        : color_set_kernel<kLookupRows>;
    const bool staged = kernel == color_set_kernel<kLookupRow7> || kernel == color_set_kernel<kLookupTile>;
    kernel<<<blocks_for(n), kThreads, staged ? tile : 0, st>>>(n, rast, min_level, max_level, S, C, features, out);
    return check_launch("multires_triangle_color");
}

int ds_backward_multires_triangle_color(int B, int H, int W, const float* rast, int min_level, int max_level, int S,
                                        int C, float* grad_features, const float* grad_out, ds_stream_t stream) {
    DS_CHECK_ARG(B >= 0 && H >= 0 && W >= 0 && C > 0 && levels_ok(min_level, max_level),
                 "backward_multires_triangle_color: bad sizes");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    const int64_t n = (int64_t)B * H * W;
    if (n == 0) return DS_OK;
    DS_CHECK_ARG(aligned16(rast), "backward_multires_triangle_color: rast not 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const bool vec = C % 4 == 0 && aligned16(grad_features) && aligned16(grad_out);
    // one level of a lattice whose sample indices fit the merging kernel's keys (16 bits; a triangle has 30, and an
    // ID buffer's floats count to 2^24), and channels that fit its rows
    const int bx = (W + 7) / 8, by = (H + 3) / 4;
    const int64_t nb = (int64_t)B * bx * by;
    if (min_level == max_level && max_level <= 8 && C >= kMergeFrom && C <= kMergeRow &&
        (vec || (C == 7 && aligned16(grad_features))) && (int64_t)bx * by <= 0x7fffffff && nb <= 0x7fffffff) {
        const size_t smem = (size_t)(kThreads / 32) * (32 * merge_stride(C) + 160) * sizeof(float);
        const unsigned grid = (unsigned)((nb + kThreads / 32 - 1) / (kThreads / 32));
        if (C == 7)
            color_backward_merge_kernel<true><<<grid, kThreads, smem, st>>>(H, W, bx, nb, bx * by, rast, max_level, S, C,
                                                                            grad_features, grad_out);
        else
            color_backward_merge_kernel<false><<<grid, kThreads, smem, st>>>(H, W, bx, nb, bx * by, rast, max_level, S, C,
                                                                             grad_features, grad_out);
        return check_launch("backward_multires_triangle_color");
    }
    if (vec)
        color_backward_kernel<4, false><<<blocks_for(n), kThreads, 0, st>>>(n, rast, min_level, max_level, S, C,
                                                                            grad_features, grad_out);
    else if (C == 7 && aligned16(grad_features))
        color_backward_kernel<1, true><<<blocks_for(n), kThreads, 0, st>>>(n, rast, min_level, max_level, S, C,
                                                                           grad_features, grad_out);
    else
        color_backward_kernel<1, false><<<blocks_for(n), kThreads, 0, st>>>(n, rast, min_level, max_level, S, C,
                                                                            grad_features, grad_out);
    return check_launch("backward_multires_triangle_color");
}

int ds_accumulate_to_level_forward(int T, int min_level, int max_level, int target_level, int S, int S_target, int C,
                                   const float* features, float* out, ds_stream_t stream) {
    DS_CHECK_ARG(T >= 0 && C > 0 && levels_ok(min_level, max_level) && target_level >= 0 && target_level <= 12,
                 "accumulate_to_level_forward: bad sizes");
    DS_CHECK_ARG((uint32_t)S == total_feats(min_level, max_level), "Invalid feature size.");
    DS_CHECK_ARG((uint32_t)S_target == feats_at_level(target_level), "Invalid feature size.");
    const int64_t n = (int64_t)T * S_target;
    if (n == 0) return DS_OK;
    int interleave = 0;
    const size_t smem = map_smem_bytes(T, min_level, max_level, S, S_target, C, false, &interleave);
    if (interleave > 0)
        return launch_map_any<false, true>(interleave, smem, T, min_level, max_level, target_level, S, S_target, C,
                                           features, out, (cudaStream_t)stream);
    accumulate_forward_kernel<<<blocks_for(n), kThreads, 0, (cudaStream_t)stream>>>(
        T, min_level, max_level, target_level, S, S_target, C, features, out);
    return check_launch("accumulate_to_level_forward");
}

int ds_accumulate_to_level_backward(int T, int min_level, int max_level, int target_level, int S, int S_target,
                                    int C, float* grad_features, const float* grad_out, ds_stream_t stream) {
    return accumulate_backward(false, T, min_level, max_level, target_level, S, S_target, C, grad_features, grad_out,
                               (cudaStream_t)stream);
}

int ds_accumulate_to_level_backward_set(int T, int min_level, int max_level, int target_level, int S, int S_target,
                                        int C, float* grad_features, const float* grad_out, ds_stream_t stream) {
    return accumulate_backward(true, T, min_level, max_level, target_level, S, S_target, C, grad_features, grad_out,
                               (cudaStream_t)stream);
}

}  // extern "C"
