// diffsoup_b200/csrc/lattice_map.cuh -- the level accumulation (multires.cu:
// 314-450) as a sparse linear map applied to every triangle.
//
// Evaluating levels [lo, hi] at the vertices of the target lattice is the same
// sparse map for every triangle and channel: target sample k reads three
// corners of every level.  A CTA builds the map's rows once in shared memory
// (forward: per target sample its (source, weight) pairs in level-then-corner
// order; adjoint: per source sample its (target, weight) pairs in target
// order), and then each warp takes I triangles at a time:
//   * their input samples are staged in the warp's own tile, interleaved as
//     [element][triangle], so that one 4*I-byte shared load brings the same
//     element of all I triangles and a table entry is read once for them;
//   * lane s takes output element s (row s / C, channel s % C): a gather, so the
//     adjoint has no atomics, and all global loads and stores are coalesced.
// What bounds it: the tile's shared-memory reads, one 128-byte wavefront per 32
// products, against the global reads and writes of each sample once.  Half of
// the pairs have weight zero (a target vertex that is a lattice vertex of a
// level takes one corner there), so a second pair of tables leaves them out;
// the full one serves the triangles that hold an infinity or a NaN, where
// 0 * x is not 0.
#pragma once

#include "geometry.cuh"

namespace dsb {

constexpr int kMapWarps = 8;

// Rows of the map: row r holds ent[row[r] .. row[r + 1]), entries {input
// sample, weight bits}.
struct MapRows {
    int2* ent;
    int* row;
};

struct MapTables {
    MapRows all, nonzero;
};

// Bytes of the tables: N = 3 * levels * target samples pairs, `rows` output rows.
__host__ __device__ inline size_t map_table_bytes(int N, int rows) {
    return ((size_t)N * 16 + (size_t)(rows + 1) * 8 + 127) & ~(size_t)127;
}

__device__ inline MapTables map_tables_at(unsigned char* base, int N, int rows) {
    MapTables m;
    m.all.ent = reinterpret_cast<int2*>(base);
    m.nonzero.ent = m.all.ent + N;
    m.all.row = reinterpret_cast<int*>(m.nonzero.ent + N);
    m.nonzero.row = m.all.row + rows + 1;
    return m;
}

// Exclusive prefix of rows[1..n] into rows[0..n] (rows[0] = 0), one warp.
__device__ inline void map_scan(int* rows, int n) {
    const int lane = threadIdx.x & 31;
    int carry = 0;
    if (lane == 0) rows[0] = 0;
    for (int d0 = 0; d0 < n; d0 += 32) {
        const int d = d0 + lane;
        int v = d < n ? rows[d + 1] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (d < n) rows[d + 1] = carry + v;
        carry += __shfl_sync(0xffffffffu, v, 31);
    }
}

// The three (source, weight) pairs of target sample k at level l, whose
// samples start at `off`.
__device__ __forceinline__ void map_cell(int k, float inv_r, int l, int off, int src[3], float w[3]) {
    uint32_t x, y, idx[3];
    index_to_xy((uint32_t)k, x, y);
    // inv_r is a power of two: x * inv_r == x / 2^target exactly
    lattice_cell(__fmul_rn((float)x, inv_r), __fmul_rn((float)y, inv_r), (uint32_t)l, idx, w);
#pragma unroll
    for (int j = 0; j < 3; ++j) src[j] = off + (int)idx[j];
}

// Rows of the forward map (output rows = the ST target samples).  Called by
// the whole CTA.
__device__ inline void build_forward_rows(const MapTables& m, int lo, int hi, int target, int ST) {
    const int NL = hi - lo + 1, NE = 3 * NL;
    const float inv_r = 1.f / (float)(1u << target);
    for (int k = threadIdx.x; k < ST; k += blockDim.x) {
        int n = 0, off = 0;
        for (int li = 0; li < NL; ++li) {
            int src[3];
            float w[3];
            map_cell(k, inv_r, lo + li, off, src, w);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                m.all.ent[k * NE + li * 3 + j] = make_int2(src[j], __float_as_int(w[j]));
                n += w[j] != 0.f;
            }
            off += (int)feats_at_level((uint32_t)(lo + li));
        }
        m.all.row[k + 1] = (k + 1) * NE;
        m.nonzero.row[k + 1] = n;
    }
    __syncthreads();
    if (threadIdx.x < 32) map_scan(m.nonzero.row, ST);
    if (threadIdx.x == 0) m.all.row[0] = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < ST; k += blockDim.x) {
        int at = m.nonzero.row[k];
        for (int n = 0; n < NE; ++n) {
            const int2 e = m.all.ent[k * NE + n];
            if (__int_as_float(e.y) != 0.f) m.nonzero.ent[at++] = e;
        }
    }
    __syncthreads();
}

// Rows of the adjoint (output rows = the S source samples), each in (target,
// corner) order.  The sources of different levels are different rows, so warp
// l places the pairs of level l: __match_any_sync groups the lanes of one source.
__device__ inline void build_adjoint_rows(const MapTables& m, int lo, int hi, int target, int ST, int S) {
    const int NL = hi - lo + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const float inv_r = 1.f / (float)(1u << target);
    for (int d = threadIdx.x; d < S; d += blockDim.x) m.all.row[d + 1] = m.nonzero.row[d + 1] = 0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
        for (int li = warp; li < NL; li += nw) {
            int off = 0;
            for (int l = lo; l < lo + li; ++l) off += (int)feats_at_level((uint32_t)l);
            for (int k0 = 0; k0 < ST; k0 += 32) {
                const int k = k0 + lane;
                int src[3] = {-1 - lane, -1 - lane, -1 - lane};
                float w[3] = {0.f, 0.f, 0.f};
                if (k < ST) map_cell(k, inv_r, lo + li, off, src, w);
                if (pass == 0) {
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        if (k < ST) {
                            atomicAdd(m.all.row + src[j] + 1, 1);
                            if (w[j] != 0.f) atomicAdd(m.nonzero.row + src[j] + 1, 1);
                        }
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 3; ++j) {
#pragma unroll
                    for (int z = 0; z < 2; ++z) {  // the full rows, then those without zero weights
                        const MapRows& r = z == 0 ? m.all : m.nonzero;
                        const bool in = k < ST && (z == 0 || w[j] != 0.f);
                        const int d = in ? src[j] : -1 - lane;
                        const unsigned peers = __match_any_sync(0xffffffffu, d);
                        int base = 0;
                        if (in) base = r.row[d];  // the next free slot: rows are advanced while filling
                        __syncwarp();
                        if (in) {
                            r.ent[base + __popc(peers & ((1u << lane) - 1u))] = make_int2(k, __float_as_int(w[j]));
                            if (lane == __ffs(peers) - 1) r.row[d] = base + __popc(peers);
                        }
                        __syncwarp();
                    }
                }
            }
        }
        __syncthreads();
        if (pass == 0) {
            if (warp == 0) map_scan(m.all.row, S);
            if (warp == 1 % nw) map_scan(m.nonzero.row, S);
            __syncthreads();
        }
    }
    // filling moved every row's start to its end, the start of the next row: shift back
    if (warp == 0) {
        for (int z = 0; z < 2; ++z) {
            int* row = z == 0 ? m.all.row : m.nonzero.row;
            int carry = 0;
            for (int d0 = 0; d0 <= S; d0 += 32) {
                const int d = d0 + lane;
                const int v = d < S ? row[d] : 0;
                const int prev = __shfl_up_sync(0xffffffffu, v, 1);
                const int last = __shfl_sync(0xffffffffu, v, 31);
                __syncwarp();
                if (d <= S) row[d] = lane == 0 ? carry : prev;
                carry = last;
                __syncwarp();
            }
        }
    }
    __syncthreads();
}

template <int I>
struct MapVec;
template <>
struct MapVec<1> { typedef float type; };
template <>
struct MapVec<2> { typedef float2 type; };
template <>
struct MapVec<4> { typedef float4 type; };

// Applies the map to triangles [t0, t0 + I) with the warp's tile.  Input
// element e of triangle t is src(t, e), e < n_in; output element s < n_out reads
// column (base, stride) of where(s, row, base, stride), input sample d at
// element base + d * stride, and goes to dst(t, s, value).  Triangles at or
// past T stage zeros and are not written.  Triangles holding an infinity or NaN
// use every pair.
template <int I, class Src, class Where, class Dst>
__device__ __forceinline__ void map_triangles(const MapTables& m, int t0, int T, int n_in, int n_out, float* tile,
                                              Src src, Where where, Dst dst) {
    typedef typename MapVec<I>::type Vec;
    const int lane = threadIdx.x & 31;
    bool odd = false;
    constexpr int U = 16 / I;  // 16 loads in flight per lane
    for (int e0 = lane; e0 < n_in; e0 += 32 * U) {
        float v[U][I];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < I; ++i) v[u][i] = e0 + 32 * u < n_in && t0 + i < T ? src(t0 + i, e0 + 32 * u) : 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (e0 + 32 * u >= n_in) break;
            Vec p;
            float* q = reinterpret_cast<float*>(&p);
#pragma unroll
            for (int i = 0; i < I; ++i) {
                q[i] = v[u][i];
                odd = odd || !(fabsf(v[u][i]) <= 3.402823466e38f);
            }
            *reinterpret_cast<Vec*>(tile + (size_t)(e0 + 32 * u) * I) = p;
        }
    }
    __syncwarp();
    const MapRows r = __any_sync(0xffffffffu, odd) ? m.all : m.nonzero;
    for (int s = lane; s < n_out; s += 32) {
        int row, base, stride;
        float acc[I];
#pragma unroll
        for (int i = 0; i < I; ++i) acc[i] = 0.f;
        where(s, row, base, stride);
        const int end = r.row[row + 1];
#pragma unroll 2
        for (int n = r.row[row]; n < end; ++n) {
            const int2 e = r.ent[n];
            const Vec x = *reinterpret_cast<const Vec*>(tile + (size_t)(base + e.x * stride) * I);
            const float* xv = reinterpret_cast<const float*>(&x);
#pragma unroll
            for (int i = 0; i < I; ++i) acc[i] = madd(acc[i], __int_as_float(e.y), xv[i]);
        }
#pragma unroll
        for (int i = 0; i < I; ++i)
            if (t0 + i < T) dst(t0 + i, s, acc[i]);
    }
    __syncwarp();  // the tile is rewritten by the next triangles
}

// Triangles per warp pass: as many of 4, 2, 1 as keep the warp's tile of
// n_in elements at most 12 KB (with 8 warps' tiles of that size and the tables of levels 0..2
// two CTAs share an SM, with those of levels 0..4 one has it alone); 0 when
// one triangle does not fit in 24 KB.
__host__ inline int map_interleave(int n_in) {
    if (n_in * 16 <= 12 * 1024) return 4;
    if (n_in * 8 <= 12 * 1024) return 2;
    return n_in * 4 <= 24 * 1024 ? 1 : 0;
}

}  // namespace dsb
