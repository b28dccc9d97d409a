// diffsoup_b200/csrc/tiled.cu -- screen-tile binning, tiled forward
// rasterizer and tiled opacity auxiliary gradient.
//
// The reference enumerates one fragment per bbox pixel into global memory,
// compacts it, and resolves depth with 64-bit atomics
// (src/cuda/rasterize.cu:139-400).  Here each (view, triangle) is binned into
// the 16x16 screen tiles its rect (rasterize.cu:43-137) overlaps, and each
// tile's list is sorted by the triangles' near-depth bound.  A work item is
// one 8x4 pixel block of a tile, owned by one warp: the warp takes the tile's
// entries 32 at a time (rect overlap, depth bound, pixels that may be covered),
// stages the survivors' vertices in its own shared memory, and every lane walks
// its own pixel's candidates and resolves the depth test in registers.  Warps never wait for each other: no
// fragment list, no CTA barrier, no global atomics, one 16-byte store per
// pixel.
//
// Results equal the reference's: coverage, barycentrics and depth use its
// FP32 arithmetic, the depth key is bits(z+2) with ties broken by the lower
// triangle index (its fragment order), and the opacity test is applied
// before the depth comparison exactly as depth_test_kernel does.
#include "edge_math.cuh"
#include "scan.cuh"
#include "tiled.cuh"

namespace dsb {

constexpr int kWarpsPerCta = 8;
constexpr int kBlocksPerTile = 8;  // 32-pixel blocks of a 16x16 tile, one warp each
static_assert(DS_TILE == 16, "the block decode of block_geometry assumes 16x16 tiles");
constexpr int kSortMax = 512;      // longest tile list sorted by depth
constexpr int kSortWarps = 4;      // warps (tiles) per CTA of the sort pass

// One entry of a tile's list: the (view, triangle) record's pixel rect and
// near depth bound, and the record index -- what the rasterizer's staging
// and the sort by depth read, without a second, dependent load.
struct __align__(16) ListEntry {
    short y0, y1, x0, x1;
    float zlo;
    int ri;
};
static_assert(sizeof(ListEntry) == 16, "ListEntry layout");

struct TileWs {
    TriBox* boxes;
    TriVerts* verts;
    TriNdc* ndc;
    TriEdges* edges;
    int* counts;
    int64_t* offsets;  // [num_tiles + 1] exclusive prefix of counts
    int* cursor;
    int* sorted;       // per tile: 1 when its list is ordered by zlo
    ListEntry* list;
    ListEntry* fill;   // the fill pass's unsorted lists (same offsets)
    int* work;         // persistent-kernel work counters [2], then the status word of ds_tiles_bin_report
    void* scan;
};

static inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

static TileWs carve(void* ws, int B, int T, int num_tiles, int64_t capacity, size_t* total) {
    char* p = reinterpret_cast<char*>(ws);
    TileWs w;
    size_t o = 0;
    w.boxes = reinterpret_cast<TriBox*>(p + o); o += al256((size_t)B * T * sizeof(TriBox));
    w.verts = reinterpret_cast<TriVerts*>(p + o); o += al256((size_t)B * T * sizeof(TriVerts));
    w.ndc = reinterpret_cast<TriNdc*>(p + o); o += al256((size_t)B * T * sizeof(TriNdc));
    w.edges = reinterpret_cast<TriEdges*>(p + o); o += al256((size_t)B * T * sizeof(TriEdges));
    w.counts = reinterpret_cast<int*>(p + o); o += al256((size_t)num_tiles * sizeof(int));
    w.offsets = reinterpret_cast<int64_t*>(p + o); o += al256((size_t)(num_tiles + 1) * sizeof(int64_t));
    w.cursor = reinterpret_cast<int*>(p + o); o += al256((size_t)num_tiles * sizeof(int));
    w.sorted = reinterpret_cast<int*>(p + o); o += al256((size_t)num_tiles * sizeof(int));
    w.work = reinterpret_cast<int*>(p + o); o += 256;
    w.scan = p + o; o += al256(scan_workspace_bytes(num_tiles));
    w.list = reinterpret_cast<ListEntry*>(p + o); o += al256((size_t)capacity * sizeof(ListEntry));
    w.fill = reinterpret_cast<ListEntry*>(p + o); o += al256((size_t)capacity * sizeof(ListEntry));
    if (total) *total = o;
    return w;
}

__device__ __forceinline__ int find_view(const ds_view_desc* __restrict__ views, int B, int tile) {
    int lo = 0, hi = B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&views[mid].tile_base) <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Tile range of a box; false when its rect is empty.
__device__ __forceinline__ bool box_tiles(const TriBox& r, int& tx0, int& tx1, int& ty0, int& ty1) {
    if (r.y1 <= r.y0 || r.x1 <= r.x0) return false;
    tx0 = r.x0 / DS_TILE; tx1 = (r.x1 - 1) / DS_TILE;
    ty0 = r.y0 / DS_TILE; ty1 = (r.y1 - 1) / DS_TILE;
    return true;
}

// False only when no pixel centre of the tile can be covered by the
// triangle (the conservative test of block_surely_outside over the tile's
// 16x16 pixel centres).
__device__ __forceinline__ bool tile_may_cover(const TriVerts& v, const ds_view_desc& vd, int tx, int ty) {
    const int x = tx * DS_TILE, y = ty * DS_TILE;
    return !block_surely_outside(v.p0, v.p1, v.p2, pix_ndc(x, vd.W), pix_ndc(x + DS_TILE - 1, vd.W), pix_ndc(y, vd.H),
                                 pix_ndc(y + DS_TILE - 1, vd.H));
}

// The items of a warp, 32 at a time: lane j owns n_j consecutive items and
// f(valid, owner, k) is called by every lane for one item each pass (k-th
// item of lane `owner`; valid is false for the lanes past the last item).
// Every lane must call this (f may shuffle).
template <class F>
__device__ __forceinline__ void warp_items(int n, F&& f) {
    const int lane = threadIdx.x & 31;
    int excl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, excl, o);
        if (lane >= o) excl += v;
    }
    const int total = __shfl_sync(0xffffffffu, excl, 31);
    excl -= n;  // first item of this lane
    for (int base = 0; base < total; base += 32) {
        const int slot = base + lane;
        int owner = 0;  // the last lane whose first item is at or before slot
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
            const int e = __shfl_sync(0xffffffffu, excl, owner + step);
            if (e <= slot) owner += step;
        }
        const int k = slot - __shfl_sync(0xffffffffu, excl, owner);
        f(slot < total, owner, k);
    }
}

// Triangles per warp of the two binning passes.  A warp's time is a chain of
// items / 32 dependent rounds, so when 32 triangles a warp would leave most of
// the chip without a warp, a warp takes 8 (its first lanes own one each, all
// lanes work on their tiles).  Whole binning with 8 and with 32 a warp, in us: one view of 800x800 of
// 15,000 triangles 35 and 38, of 24,000 40 and 43, of 27,000 47.5 and 47.5, of 45,000 62 and 60, of 60,000 76 and 62;
// one of 1200x1200 of 15,000 40 and 52; 4 views of 300x300 of 20,000 74 and 51; 200,000 triangles in
// full HD 78 and 52.
constexpr int64_t kBinNarrow = 24000;  // (view, triangle) pairs up to which a warp takes 8

// Record index of the calling lane, or n for a lane without one.
template <int TPW>
__device__ __forceinline__ int64_t bin_record(int64_t n) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * TPW + lane;
    return lane < TPW && i < n ? i : n;
}

// Pass 1: boxes, vertices, depth bounds, edge records and per-tile counts.
// The (triangle, tile) pairs of a warp's triangles are tested 32 at a
// time (warp_items), so lanes do not wait on the lane with the largest rect.
template <int TPW>
__global__ void __launch_bounds__(kThreads) bin_setup_kernel(int B, const ds_view_desc* __restrict__ views, int V,
                                                             const float* __restrict__ pos, int T,
                                                             const int* __restrict__ tri, TriBox* __restrict__ boxes,
                                                             TriVerts* __restrict__ verts, TriNdc* __restrict__ ndc,
                                                             TriEdges* __restrict__ edges, int* __restrict__ counts) {
    __shared__ unsigned long long s_mask[kThreads];
    chain_wait();
    const int64_t i = bin_record<TPW>((int64_t)B * T);
    const bool live = i < (int64_t)B * T;
    const int b = live ? (int)(i / T) : 0, t = live ? (int)(i % T) : 0;
    const ds_view_desc vd = views[b];
    TriVerts v;
    TriBox r;
    r.y0 = r.y1 = r.x0 = r.x1 = 0;
    r.zlo = r.zhi = 0.f;
    int tx0 = 0, tx1 = -1, ty0 = 0, ty1 = -1;
    if (live) {
        const float* P = pos + (size_t)b * V * 4;
        v.p0 = load_vertex(P, __ldg(tri + t * 3 + 0));
        v.p1 = load_vertex(P, __ldg(tri + t * 3 + 1));
        v.p2 = load_vertex(P, __ldg(tri + t * 3 + 2));
        int h0, hl, w0, wl;
        triangle_rect(vd.H, vd.W, v.p0, v.p1, v.p2, h0, hl, w0, wl);
        r.y0 = (short)h0; r.y1 = (short)(h0 + hl); r.x0 = (short)w0; r.x1 = (short)(w0 + wl);
        // depth bounds (only used when the rect is non-empty, i.e. every w > 0)
        const float d0 = v.p0.z / v.p0.w, d1 = v.p1.z / v.p1.w, d2 = v.p2.z / v.p2.w;
        const float mz = fmaxf(fmaxf(fabsf(v.p0.z), fabsf(v.p1.z)), fabsf(v.p2.z));
        const float mw = fminf(fminf(v.p0.w, v.p1.w), v.p2.w);
        const float margin = 1e-5f + 4e-6f * (mz / mw + fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fabsf(d2)));
        r.zlo = fminf(fminf(d0, d1), d2) - margin;
        r.zhi = fmaxf(fmaxf(d0, d1), d2) + margin;
        if (!(r.zlo == r.zlo && r.zhi == r.zhi)) { r.zlo = -INFINITY; r.zhi = INFINITY; }  // NaN: no bounds
        boxes[i] = r;
        verts[i] = v;
        if (!box_tiles(r, tx0, tx1, ty0, ty1)) { tx1 = tx0 - 1; ty1 = ty0 - 1; }
    } else {
        v.p0 = v.p1 = v.p2 = make_float4(0.f, 0.f, 0.f, 1.f);
    }
    // tiles the triangle may cover; for rects of at most 64 tiles their bit
    // mask (row-major over the rect) rides in the NDC record's spare lanes
    const int ntx = tx1 - tx0 + 1, nty = ty1 - ty0 + 1;
    const int ntiles = ntx > 0 && nty > 0 ? ntx * nty : 0;
    s_mask[threadIdx.x] = 0ull;
    __syncwarp();
    const int wbase = threadIdx.x & ~31;
    warp_items(ntiles, [&](bool valid, int owner, int k) {
        float4 q[3];
        const float4 mine[3] = {v.p0, v.p1, v.p2};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            q[j].x = __shfl_sync(0xffffffffu, mine[j].x, owner);
            q[j].y = __shfl_sync(0xffffffffu, mine[j].y, owner);
            q[j].z = __shfl_sync(0xffffffffu, mine[j].z, owner);
            q[j].w = __shfl_sync(0xffffffffu, mine[j].w, owner);
        }
        const int otx0 = __shfl_sync(0xffffffffu, tx0, owner), oty0 = __shfl_sync(0xffffffffu, ty0, owner);
        const int ontx = __shfl_sync(0xffffffffu, ntx, owner), ont = __shfl_sync(0xffffffffu, ntiles, owner);
        const int ob = __shfl_sync(0xffffffffu, b, owner);
        if (!valid) return;
        const ds_view_desc ovd = views[ob];
        const int ty = oty0 + k / ontx, tx = otx0 + k % ontx;
        TriVerts ov;
        ov.p0 = q[0]; ov.p1 = q[1]; ov.p2 = q[2];
        if (tile_may_cover(ov, ovd, tx, ty)) {
            atomicAdd(counts + ovd.tile_base + ty * ovd.tiles_x + tx, 1);
            if (ont <= 64) atomicOr(&s_mask[wbase + owner], 1ull << k);
        }
    });
    __syncwarp();
    if (!live) return;
    const uint64_t m = ntiles <= 64 ? s_mask[threadIdx.x] : 0ull;
    TriEdges te;
    te.lo = te.hi = make_float4(0.f, 0.f, 0.f, 0.f);  // not read: the rect is empty
    if (ntiles > 0)
        te = tri_edges_over_rect(v.p0, v.p1, v.p2, pix_ndc(r.x0, vd.W), pix_ndc(r.x1 - 1, vd.W), pix_ndc(r.y0, vd.H),
                                 pix_ndc(r.y1 - 1, vd.H), vd.W);
    TriNdc q;
    q.a = make_float4(v.p0.x / v.p0.w, v.p0.y / v.p0.w, v.p1.x / v.p1.w, v.p1.y / v.p1.w);
    q.b = make_float4(v.p2.x / v.p2.w, v.p2.y / v.p2.w, __uint_as_float((uint32_t)m),
                      __uint_as_float((uint32_t)(m >> 32)));
    ndc[i] = q;
    edges[i] = te;
}

// Bit position of the k-th set bit of m (k < popcount), by halving the word.
__device__ __forceinline__ int select_bit(uint64_t m, int k) {
    const int nlo = __popc((uint32_t)m);
    const bool up = k >= nlo;
    uint32_t w = up ? (uint32_t)(m >> 32) : (uint32_t)m;
    k -= up ? nlo : 0;
    int at = up ? 32 : 0;
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
        const int c = __popc(w & ((1u << h) - 1u));
        const bool hi = k >= c;
        k -= hi ? c : 0;
        at += hi ? h : 0;
        w = hi ? w >> h : w;
    }
    return at;
}

// Pass 2: scatter record indices into the per-tile lists: the tiles of the
// count pass's masks, distributed over the warp, and for rects of more than
// 64 tiles the test itself, one triangle at a time with its tiles over the
// lanes.  An entry is a chain of two dependent global round trips (the list's
// start and the cursor's atomic, then the store), so each lane keeps kFillItems
// of them in flight.  Together with the bit selection
// and the shared large rects: 200,000 triangles in 3 views of 1920x1080
// (5,237 rects of more than 64 tiles) 369 -> 45 us, 360,000 pairs in 6 uneven views
// 101 -> 20 us, one 1200x1200 view 37 -> 9.5 us; 120,000 pairs without a
// large rect stay at 13-15 us.
constexpr int kFillItems = 4;

template <int TPW>
__global__ void __launch_bounds__(kThreads) bin_fill_kernel(int B, const ds_view_desc* __restrict__ views, int T,
                                                            const TriBox* __restrict__ boxes,
                                                            const TriVerts* __restrict__ verts,
                                                            const TriNdc* __restrict__ ndc,
                                                            const int64_t* __restrict__ offsets,
                                                            int* __restrict__ cursor, ListEntry* __restrict__ list,
                                                            int64_t capacity, int* __restrict__ status) {
    chain_wait();
    const int lane = threadIdx.x & 31;
    const int64_t i = bin_record<TPW>((int64_t)B * T);
    const bool live = i < (int64_t)B * T;
    const int b = live ? (int)(i / T) : 0;
    int ntx = 0, nty = 0, org = 0, pitch = 0;  // the rect in tiles; the tile of its corner, tiles per row of its view
    uint64_t m = 0;
    ListEntry le;
    le.y0 = le.y1 = le.x0 = le.x1 = 0;
    le.zlo = 0.f;
    le.ri = (int)i;
    if (live) {
        const TriBox rc = boxes[i];
        le.y0 = rc.y0; le.y1 = rc.y1; le.x0 = rc.x0; le.x1 = rc.x1;
        le.zlo = rc.zlo;
        int tx0, tx1, ty0, ty1;
        if (box_tiles(rc, tx0, tx1, ty0, ty1)) {
            const float4 nb = ndc[i].b;
            m = (uint64_t)__float_as_uint(nb.z) | ((uint64_t)__float_as_uint(nb.w) << 32);
            ntx = tx1 - tx0 + 1;
            nty = ty1 - ty0 + 1;
            pitch = views[b].tiles_x;
            org = views[b].tile_base + ty0 * pitch + tx0;
        }
    }
    const bool small = ntx * nty <= 64;
    bool over = false;
    const int4 lw = *reinterpret_cast<const int4*>(&le);
    const uint32_t mlo = (uint32_t)m, mhi = (uint32_t)(m >> 32);
    int excl = small ? __popcll(m) : 0;
    const int mine = excl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, excl, o);
        if (lane >= o) excl += v;
    }
    const int total = __shfl_sync(0xffffffffu, excl, 31);
    excl -= mine;  // first item of this lane
    for (int base = 0; base < total; base += 32 * kFillItems) {
        int tile[kFillItems];
        int4 ent[kFillItems];
#pragma unroll
        for (int u = 0; u < kFillItems; ++u) {
            const int slot = base + u * 32 + lane;
            int owner = 0;  // the last lane whose first item is at or before slot
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int e = __shfl_sync(0xffffffffu, excl, owner + step);
                if (e <= slot) owner += step;
            }
            const int k = slot - __shfl_sync(0xffffffffu, excl, owner);
            const uint32_t olo = __shfl_sync(0xffffffffu, mlo, owner), ohi = __shfl_sync(0xffffffffu, mhi, owner);
            ent[u] = make_int4(__shfl_sync(0xffffffffu, lw.x, owner), __shfl_sync(0xffffffffu, lw.y, owner),
                               __shfl_sync(0xffffffffu, lw.z, owner), __shfl_sync(0xffffffffu, lw.w, owner));
            const int oorg = __shfl_sync(0xffffffffu, org, owner), opitch = __shfl_sync(0xffffffffu, pitch, owner);
            const int ontx = __shfl_sync(0xffffffffu, ntx, owner);
            tile[u] = -1;
            if (slot < total) {
                const int bit = select_bit((uint64_t)olo | ((uint64_t)ohi << 32), k);
                // bit / ontx, both at most 64: (bit + 1/2) / ontx stays clear of the integers
                const int row = (int)__fdividef((float)bit + 0.5f, (float)ontx);
                tile[u] = oorg + row * opitch + (bit - row * ontx);
            }
        }
        int64_t at[kFillItems];
#pragma unroll
        for (int u = 0; u < kFillItems; ++u)
            if (tile[u] >= 0) at[u] = offsets[tile[u]] + atomicAdd(cursor + tile[u], 1);
#pragma unroll
        for (int u = 0; u < kFillItems; ++u)
            if (tile[u] >= 0) {
                if (at[u] < capacity) *reinterpret_cast<int4*>(list + at[u]) = ent[u];
                else over = true;
            }
    }
    for (unsigned big = __ballot_sync(0xffffffffu, live && !small); big != 0; big &= big - 1u) {
        const int src = __ffs(big) - 1;
        const int64_t oi = __shfl_sync(0xffffffffu, i, src);
        const int ontx = __shfl_sync(0xffffffffu, ntx, src), onty = __shfl_sync(0xffffffffu, nty, src);
        const int4 ent = make_int4(__shfl_sync(0xffffffffu, lw.x, src), __shfl_sync(0xffffffffu, lw.y, src),
                                   __shfl_sync(0xffffffffu, lw.z, src), __shfl_sync(0xffffffffu, lw.w, src));
        const ds_view_desc vd = views[__shfl_sync(0xffffffffu, b, src)];
        const TriVerts v = verts[oi];
        const int tx0 = (short)(ent.y & 0xffff) / DS_TILE, ty0 = (short)(ent.x & 0xffff) / DS_TILE;
        for (int k = lane; k < ontx * onty; k += 32) {
            const int ty = ty0 + k / ontx, tx = tx0 + k % ontx;
            if (!tile_may_cover(v, vd, tx, ty)) continue;
            const int tile = vd.tile_base + ty * vd.tiles_x + tx;
            const int64_t at = offsets[tile] + atomicAdd(cursor + tile, 1);
            if (at < capacity) *reinterpret_cast<int4*>(list + at) = ent;
            else over = true;
        }
    }
    if (over) atomicOr(status, DS_STATUS_LIST_OVERFLOW);
}

// Bitonic network over the R * 32 (key, position) pairs of a warp, element
// e = s * 32 + lane in register slot s, ascending.  Partners 32 or more apart
// sit in the same lane (a compare-exchange between two slots), nearer ones in
// the same slot of another lane (a shuffle).
template <int R>
__device__ __forceinline__ void warp_bitonic(float (&key)[R], int (&pos)[R], int lane) {
#pragma unroll 1
    for (int k = 2; k <= R * 32; k <<= 1) {
#pragma unroll
        for (int h = R / 2; h > 0; h >>= 1) {  // partners h slots apart (register indices are static)
            if (k <= 32 * h) continue;
#pragma unroll
            for (int s = 0; s < R; ++s) {
                const int t = s ^ h;
                if (t > s) {
                    const bool up = ((s * 32 + lane) & k) == 0;  // the lower element keeps the smaller key
                    const float a = key[s], c = key[t];
                    const int pa = pos[s], pc = pos[t];
                    const bool swap = ((a > c) == up) & (a != c);  // selects, no branch
                    key[s] = swap ? c : a; key[t] = swap ? a : c;
                    pos[s] = swap ? pc : pa; pos[t] = swap ? pa : pc;
                }
            }
        }
#pragma unroll 1
        for (int j = k > 32 ? 16 : k >> 1; j > 0; j >>= 1) {
#pragma unroll
            for (int s = 0; s < R; ++s) {
                const float ok = __shfl_xor_sync(0xffffffffu, key[s], j);
                const int op = __shfl_xor_sync(0xffffffffu, pos[s], j);
                const bool up = ((s * 32 + lane) & k) == 0, lower = (lane & j) == 0;
                const bool take = ((ok < key[s]) == (lower == up)) & (ok != key[s]);
                key[s] = take ? ok : key[s];
                pos[s] = take ? op : pos[s];
            }
        }
    }
}

// Sorts the n <= R * 32 entries of F by zlo into L (register network, one
// gather per entry).
template <int R>
__device__ __forceinline__ void sort_in_registers(const int4* __restrict__ F, int4* __restrict__ L, int n, int lane) {
    float key[R];
    int pos[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int e = s * 32 + lane;
        key[s] = e < n ? fminf(__int_as_float(F[e].z), 3.0e38f) : INFINITY;  // real keys stay below the padding
        pos[s] = e;
    }
    warp_bitonic<R>(key, pos, lane);
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int e = s * 32 + lane;
        if (e < n) L[e] = F[pos[s]];
    }
}

// Pass 3: each tile's list ordered by zlo, from the fill pass's lists into
// the rasterizer's (warp per tile): the (key, position) pairs of up to kSortMax
// entries are sorted by a bitonic network in registers, and each entry is then
// gathered once.  Longer lists are copied as they are and marked unsorted; lists
// cut by the capacity are not used.  A warp's own latency is the bound: the
// network's selects have no branches and its stages are loops (with branches and
// two smem words per pair for the long lists, the 282-entry list of 6 uneven
// views alone took 60 us): 75 -> 24 us there, 28 -> 20 us for 8 views of 800x800,
// 13 -> 7.6 us for one view of 1200x1200.
__global__ void __launch_bounds__(kSortWarps * 32) sort_lists_kernel(int num_tiles,
                                                                     const int64_t* __restrict__ offsets,
                                                                     const ListEntry* __restrict__ fill,
                                                                     ListEntry* __restrict__ list, int64_t capacity,
                                                                     int* __restrict__ sorted) {
    chain_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x * kSortWarps + warp;
    if (tile >= num_tiles) return;
    const int64_t begin = offsets[tile], end = offsets[tile + 1];
    const int n = (int)(end - begin);
    if (end > capacity) {  // cut: the tile runs the exhaustive path
        if (lane == 0) sorted[tile] = 0;
        return;
    }
    const int4* F = reinterpret_cast<const int4*>(fill + begin);
    int4* L = reinterpret_cast<int4*>(list + begin);
    if (n > kSortMax) {
        for (int i = lane; i < n; i += 32) L[i] = F[i];
        if (lane == 0) sorted[tile] = 0;
        return;
    }
    if (n <= 32) sort_in_registers<1>(F, L, n, lane);
    else if (n <= 64) sort_in_registers<2>(F, L, n, lane);
    else if (n <= 128) sort_in_registers<4>(F, L, n, lane);
    else if (n <= 256) sort_in_registers<8>(F, L, n, lane);
    else sort_in_registers<16>(F, L, n, lane);
    if (lane == 0) sorted[tile] = 1;
}

// Geometry of one work item (tile, 32-pixel block) for the calling lane.
// Blocks are 2^bwl pixels wide and 32 / 2^bwl high (bwl = 3: 8x4, 4: 16x2,
// 2: 4x8); a tile holds 8 of them, row-major, and lane l takes pixel
// (l mod width, l div width) of its block.
struct BlockGeom {
    int b, px, py, H, W;
    int64_t pix;          // packed pixel index
    bool valid;
    int wx0, wy0;         // block origin
    int bw, bh;           // block width and height
    int64_t begin, end;   // list range, or [b*T, b*T+T) records when exhaustive
    bool exhaustive, ordered;
};

__device__ __forceinline__ BlockGeom block_geometry(int item, int B, const ds_view_desc* __restrict__ views, int T,
                                                    const int64_t* __restrict__ offsets,
                                                    const int* __restrict__ sorted, int64_t capacity, int bwl) {
    BlockGeom g;
    const int tile = item / kBlocksPerTile, blk = item % kBlocksPerTile;
    g.b = find_view(views, B, tile);
    const ds_view_desc vd = views[g.b];
    const int tl = tile - vd.tile_base;
    const int tx = tl % vd.tiles_x, ty = tl / vd.tiles_x;
    const int lane = threadIdx.x & 31;
    g.bw = 1 << bwl;
    g.bh = 32 >> bwl;
    const int rl = 4 - bwl;  // log2 of the blocks per tile row (DS_TILE = 16)
    g.wx0 = tx * DS_TILE + ((blk & ((1 << rl) - 1)) << bwl);
    g.wy0 = ty * DS_TILE + (blk >> rl) * g.bh;
    g.px = g.wx0 + (lane & (g.bw - 1));
    g.py = g.wy0 + (lane >> bwl);
    g.H = vd.H; g.W = vd.W;
    g.valid = g.px < vd.W && g.py < vd.H;
    g.pix = vd.pix_offset + (int64_t)g.py * vd.W + g.px;
    g.begin = offsets[tile];
    g.end = offsets[tile + 1];
    g.exhaustive = g.end > capacity;
    g.ordered = !g.exhaustive && sorted[tile] != 0;
    if (g.exhaustive) { g.begin = (int64_t)g.b * T; g.end = g.begin + T; }
    return g;
}

__device__ __forceinline__ bool box_overlaps(const TriBox& r, const BlockGeom& g) {
    return r.y0 < g.wy0 + g.bh && r.y1 > g.wy0 && r.x0 < g.wx0 + g.bw && r.x1 > g.wx0;
}

// The warp's next item of `items`.  Every warp of the grid ends on one value at or
// past `items`, so the warp that draws the last of them puts the counter back to
// zero for the next kernel (the binning pass cleared it first).
__device__ __forceinline__ int warp_next(int* work, int items) {
    int item = 0;
    if ((threadIdx.x & 31) == 0) {
        item = atomicAdd(work, 1);
        if (item == items + (int)(gridDim.x * (blockDim.x >> 5)) - 1) *work = 0;
    }
    return __shfl_sync(0xffffffffu, item, 0);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Per-warp buffer of the fragment records of one 8x4 block (REC kernels).
constexpr int kRecCap = 192;

struct WarpRecs {
    int t[kRecCap];
    float b0[kRecCap], b1[kRecCap], z[kRecCap];
    unsigned char lane[kRecCap];
};

__device__ __forceinline__ void push_fallback(const RecordStore& rs, int item) {
    if ((threadIdx.x & 31) == 0) rs.fallback[atomicAdd(rs.counters + 1, 1)] = item;
}

// Writes the records of the finished block that lie in front of (or level
// with) each lane's final surface into the warp's chunk.  The chunk must
// hold all nrec of them (the kept count is not known before the pass), so a
// new one is reserved when it does not; `cid` = current chunk (-1: none,
// -2: the store is exhausted), `cfill` = records in it.  Record j's lane
// passes its pixel, surface depth and visible triangle by shuffle.
__device__ __forceinline__ void flush_records(const RecordStore& rs, const WarpRecs& R, int nrec, int item, uint32_t pix,
                                              unsigned long long best, float bz, int& cid, int& cfill) {
    const int lane = threadIdx.x & 31;
    if (nrec > kRecCap) {
        push_fallback(rs, item);
        return;
    }
    // the surface depth (+inf when empty) and the visible triangle as the backward pass reads it back from
    // rast (id + 1 stored as a float; -1 when empty)
    const float fz = best == ~0ull ? INFINITY : bz;
    const int ft = best == ~0ull ? -1 : (int)(float)((uint32_t)(best & 0xffffffffu) + 1u) - 1;
    if (cid == -1 || (cid >= 0 && cfill + nrec > kRecChunk)) {
        if (cid >= 0 && lane == 0) rs.chunk_fill[cid] = cfill;
        int base = 0;
        if (lane == 0) base = atomicAdd(rs.counters, kRecChunk);
        base = __shfl_sync(0xffffffffu, base, 0);
        cid = (int64_t)base + kRecChunk <= rs.capacity ? base / kRecChunk : -2;
        cfill = 0;
    }
    if (cid == -2) {
        push_fallback(rs, item);
        return;
    }
    int4* out = rs.rec + (int64_t)cid * kRecChunk + cfill;
    const unsigned below = (1u << lane) - 1u;
    int at = 0;
    for (int j0 = 0; j0 < nrec; j0 += 32) {
        const int j = j0 + lane;
        const bool in = j < nrec;
        const int src = in ? (int)R.lane[j] : 0;
        const float sz = __shfl_sync(0xffffffffu, fz, src);
        const int stri = __shfl_sync(0xffffffffu, ft, src);
        const uint32_t p = __shfl_sync(0xffffffffu, pix, src);
        const bool keep = in && R.z[j] <= sz;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int t = R.t[j];
            const uint32_t tv = (uint32_t)t | (t == stri ? 0x80000000u : 0u);
            out[at + __popc(m & below)] = make_int4((int)p, (int)tv, __float_as_int(R.b0[j]), __float_as_int(R.b1[j]));
        }
        at += __popc(m);
    }
    cfill += at;
}

// Candidates of one group of 32 list entries, by the entry's place in the group,
// and the NDC y of the block's rows.
struct RasterStage {
    TriVerts v[32];
    float zlo[32];
    int t[32];
    float row_y[8];
};

// Lanes of the block (lane l = pixel (l mod bw, l div bw)) whose pixel centre the
// triangle may cover: its pixel rect, cut row by row to its column bounds.
__device__ __forceinline__ unsigned cover_lanes(const TriBox& r, const TriEdges& te, const BlockGeom& g,
                                                const float* row_y) {
    const float lo0 = (float)max((int)r.x0, g.wx0), hi0 = (float)(min((int)r.x1, g.wx0 + g.bw) - 1);
    const int y0 = max((int)r.y0 - g.wy0, 0), y1 = min((int)r.y1 - g.wy0, g.bh);
    unsigned lanes = 0u;
    for (int y = y0; y < y1; ++y) {
        const float ny = row_y[y];
        const float lo = fmaxf(lo0, fmaxf(fmaf(te.lo.y, ny, te.lo.x), fmaf(te.lo.w, ny, te.lo.z)));
        const float hi = fminf(hi0, fminf(fmaf(te.hi.y, ny, te.hi.x), fmaf(te.hi.w, ny, te.hi.z)));
        // whole columns inside [lo, hi], relative to the block (lo >= its first, hi <= its last column)
        const int a = (int)ceilf(fminf(lo, hi0 + 1.f)) - g.wx0, c = (int)floorf(fmaxf(hi, lo0 - 1.f)) - g.wx0;
        if (a <= c) lanes |= ((2u << c) - (1u << a)) << (y * g.bw);
    }
    return lanes;
}

// Transposes the 32x32 bit matrix held as one row per lane: bit l of lane k's word
// becomes bit k of lane l's.
__device__ __forceinline__ unsigned warp_transpose(unsigned m) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned low = 0xffffffffu / ((1u << o) + 1u);  // the low halves of the 2 o-bit fields
        const unsigned other = __shfl_xor_sync(0xffffffffu, m, o);
        m = (lane & o) ? (m & ~low) | ((other >> o) & low) : (m & low) | ((other << o) & ~low);
    }
    return m;
}

// Loads entries [g0, g0 + 32) of the work item's range, stages those whose box
// meets the block, whose depth bound passes `zcut` and that may cover one of its
// valid pixels, and returns the calling lane's pixel's candidates as a mask over
// the group.  *head_zlo receives the zlo of the group's first entry (the
// smallest, when the list is ordered); *any_large whether a staged triangle's rect
// has `large` pixels or more.
__device__ __forceinline__ unsigned stage_pixels(const BlockGeom& g, int64_t g0, const TriBox* __restrict__ boxes,
                                                 const TriVerts* __restrict__ verts,
                                                 const TriEdges* __restrict__ edges,
                                                 const ListEntry* __restrict__ list, int T, float zcut, unsigned valid,
                                                 RasterStage& st, float* head_zlo, int large = 0x7fffffff,
                                                 bool* any_large = nullptr) {
    const int lane = threadIdx.x & 31;
    const int64_t e = g0 + lane;
    const bool in = e < g.end;
    int ri = 0;
    TriBox bx;
    bx.y0 = bx.y1 = bx.x0 = bx.x1 = 0;
    bx.zlo = INFINITY; bx.zhi = INFINITY;
    if (in) {
        if (g.exhaustive) {
            ri = (int)e;
            bx = boxes[ri];
        } else {
            const int4 le = __ldg(reinterpret_cast<const int4*>(list + e));
            ri = le.w;
            bx.y0 = (short)(le.x & 0xffff); bx.y1 = (short)(le.x >> 16);
            bx.x0 = (short)(le.y & 0xffff); bx.x1 = (short)(le.y >> 16);
            bx.zlo = __int_as_float(le.z);
        }
    }
    *head_zlo = __shfl_sync(0xffffffffu, bx.zlo, 0);
    unsigned lanes = 0u;
    if (in && box_overlaps(bx, g) && bx.zlo <= zcut) lanes = cover_lanes(bx, edges[ri], g, st.row_y) & valid;
    if (lanes != 0u) {
        st.v[lane] = verts[ri];
        st.zlo[lane] = bx.zlo;
        st.t[lane] = ri - g.b * T;
    }
    __syncwarp();
    if (any_large != nullptr)
        *any_large = __any_sync(0xffffffffu, lanes != 0u && (bx.y1 - bx.y0) * (bx.x1 - bx.x0) >= large);
    return warp_transpose(lanes);
}

// Forward: depth test with stochastic opacity.  A warp takes the triangles of
// its block front to back (the tile list is sorted by zlo), 32 list entries at a time:
// staging finds for every entry the pixels it may cover (cover_lanes, one entry a
// lane), and then every lane walks its own pixel's candidates in order, so a pass
// evaluates up to 32 different (pixel, triangle) pairs.  A lane stops once its next
// triangle's depth bound lies behind its winner, and the warp once the next
// group's lies behind every lane's: no later triangle can improve a key (the bound's margin
// keeps bits(z+2) strictly larger).
//
// Issue slots bound the kernel, and a triangle covers 7 of a block's 32 pixels: with the
// warp on one triangle at a time a block took 7.5 passes of coverage, opacity and
// threshold and 10 of edge functions; now its passes are the most candidates of
// one pixel, about 4.  8 views of 800x800 (15,000 triangles, records kept): 367 ->
// 269 us, 6 uneven views 282 -> 227 us, one 1200x1200 view without records
// 74 -> 61 us.  (Four 4x2 sub-blocks of a warp with a candidate each took 6.5
// passes, not worth their staging; 3 or 5 CTAs per SM, 304 and 302 us; drawing the next work
// item ahead, 272 us.)
//
// REC: also keeps every fragment whose depth key does not lie behind the
// lane's current winner.  Winner keys only decrease, and every fragment at
// or in front of a lane's final surface has zlo <= that depth <= the lane's winner's
// at every point of the walk, so the walk meets and keeps all of them;
// at the end of the block those behind the final surface are dropped.
#ifndef DSB_RASTER_MIN_CTAS
#define DSB_RASTER_MIN_CTAS 4  // resident 8-warp CTAs per SM the register budget is sized for (64 registers)
#endif

template <bool REC>
__global__ void __launch_bounds__(kWarpsPerCta * 32, DSB_RASTER_MIN_CTAS) raster_kernel(
    int B, const ds_view_desc* __restrict__ views, int num_tiles, int T, const TriBox* __restrict__ boxes,
    const TriVerts* __restrict__ verts, const TriEdges* __restrict__ edges, const int64_t* __restrict__ offsets,
    const int* __restrict__ sorted, const ListEntry* __restrict__ list, int64_t capacity, int level, int S,
    const float* __restrict__ alpha_src, int thr_mode, float thr_const, const uint64_t* __restrict__ rng, int* work, float* __restrict__ rast,
    RecordStore rs, int bwl) {
    __shared__ RasterStage s_stage[kWarpsPerCta];
    __shared__ WarpRecs s_rec[REC ? kWarpsPerCta : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RasterStage& st = s_stage[warp];
    WarpRecs& R = s_rec[REC ? warp : 0];
    chain_wait();
    uint64_t seed = 0;
    uint32_t iter = 0;
    if (thr_mode == 1) { seed = rng[0]; iter = (uint32_t)rng[1]; }
    int cid = -1, cfill = 0;  // REC: the warp's current record chunk
    const int items = num_tiles * kBlocksPerTile;
    for (int item = warp_next(work, items); item < items; item = warp_next(work, items)) {
        const BlockGeom g = block_geometry(item, B, views, T, offsets, sorted, capacity, bwl);
        if (g.begin >= g.end) {  // no candidate: background (a quarter to a third of the blocks)
            if (g.valid) reinterpret_cast<float4*>(rast)[g.pix] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const float ndc_x = pix_ndc(g.px, g.W), ndc_y = pix_ndc(g.py, g.H);
        if ((lane & (g.bw - 1)) == 0) st.row_y[lane >> bwl] = ndc_y;
        const unsigned valid = __ballot_sync(0xffffffffu, g.valid);
        __syncwarp();
        const PhiloxPixel php = philox_pixel(seed, iter, (uint32_t)g.b, (uint32_t)(g.py * g.W + g.px));
        unsigned long long best = ~0ull;
        float bb0 = 0.f, bb1 = 0.f, bz = 0.f;
        float bz_cut = g.valid ? INFINITY : -INFINITY;  // the winner's depth, +inf while a valid lane has none
        int nrec = 0;
        for (int64_t g0 = g.begin; g0 < g.end; g0 += 32) {
            float head;
            const float warp_far = warp_max(bz_cut);  // the farthest winner
            unsigned todo = stage_pixels(g, g0, boxes, verts, edges, list, T, warp_far, valid, st, &head);
            if (g.ordered && head > warp_far) break;  // this group and all later ones lie behind
            while (__any_sync(0xffffffffu, todo != 0u)) {
                const int k = todo != 0u ? __ffs(todo) - 1 : 0;
                // the winner does not lie in front of the triangle: zlo's margin exceeds the rounding of
                // z + 2, so with zlo > bz every fragment's depth key lies strictly behind the winner's
                // (neither a winner nor a record)
                const bool near = todo != 0u && !(st.zlo[k] > bz_cut);
                todo = !near && g.ordered ? 0u : todo & (todo - 1u);
                if (!__any_sync(0xffffffffu, near)) continue;  // warp-uniform
                bool rec = false;
                float b0 = 0.f, b1 = 0.f, depth = 0.f;
                const uint32_t t = (uint32_t)st.t[k];
                if (near) {
                    const float4 p0 = st.v[k].p0, p1 = st.v[k].p1, p2 = st.v[k].p2;
                    float A0, A1, A2, A;
                    edge_terms(ndc_y, ndc_x, p0, p1, p2, A0, A1, A2, A);
                    float z, w;
                    if (!surely_outside(A0, A1, A2, A) && finish_coverage(A0, A1, A, p0, p1, p2, b0, b1, z, w)) {
                        depth = __fdiv_rn(z, w);
                        if (depth >= -1.f && depth <= 1.f) {
                            const unsigned long long key = depth_key(depth, t);
                            // keep it unless its depth key lies behind the current winner's: the
                            // winner's key only decreases, so nothing at or in front of the final
                            // surface is dropped (the winner's depth itself can grow within one
                            // bits(z+2) step when a lower triangle index takes a tie)
                            if (REC) rec = (key >> 32) <= (best >> 32);
                            if (depth > -1.f && key < best) {
                                const float alpha = interp_level(b0, b1, level, alpha_src + (size_t)t * S);
                                // Philox thresholds lie in [0, 1): an opacity of 1 passes without a draw
                                const bool pass = thr_mode == 1
                                                      ? alpha >= 1.f || !(alpha < philox_uniform_tri(php, seed, t))
                                                      : !(alpha < thr_const);
                                if (pass) {
                                    best = key; bb0 = b0; bb1 = b1; bz = depth; bz_cut = depth;
                                }
                            }
                        }
                    }
                }
                if (REC) {
                    const unsigned m = __ballot_sync(0xffffffffu, rec);
                    if (m) {
                        const int at = nrec + __popc(m & ((1u << lane) - 1u));
                        if (rec && at < kRecCap) {
                            R.t[at] = (int)t; R.b0[at] = b0; R.b1[at] = b1; R.z[at] = depth;
                            R.lane[at] = (unsigned char)lane;
                        }
                        nrec += __popc(m);
                    }
                }
            }
            __syncwarp();  // the stage is rewritten by the next group
        }
        if (g.valid) {
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            if (best != ~0ull) o = make_float4(bb0, bb1, bz, (float)((uint32_t)(best & 0xffffffffu) + 1u));
            reinterpret_cast<float4*>(rast)[g.pix] = o;
        }
        if (REC && nrec > 0) {
            __syncwarp();
            flush_records(rs, R, nrec, item, (uint32_t)g.pix, best, bz, cid, cfill);
            __syncwarp();  // the buffer is rewritten by the next block
        }
    }
    if (REC && cid >= 0 && lane == 0) rs.chunk_fill[cid] = cfill;
}

// Opacity contributions in the re-enumerating pass.  About one fragment a pixel is
// in front of its surface, far below the atomics' rate, so most go straight to
// memory.  The atomics of a large triangle, though, meet on its few samples: 20 ms for
// two triangles over 8 views of 800x800 at level 2.  So where one of the 32 list entries that
// a warp stages is a triangle of kAuxLarge pixels of its rect or more per sample, the warp's fragments are
// summed before the atomics: those on one triangle (kAuxSameTriangle lanes or more) in one lattice
// cell (kAuxSameCell or more).  The two triangles then take 0.30 ms (0.34 with a warp's sums
// in shared memory, for every triangle), 20 nearly transparent layers over one view 10 -> 0.20 ms (0.59), 200
// triangles of 240 pixels' size in two views 20 -> 0.68 ms at level 0 (1.71).  Summed everywhere, two views of
// 803x601 of 15,000 triangles take 71 us and 61 without any sums: 66 so (124).  Between them, 2,000 triangles of 80
// pixels' size at level 4 take 59 us summed, 85 by this line and 109 by one twice as far (88); 12 and 6 lanes
// instead of 8 and 4 take 1,056 us for the 200 triangles' 690.
constexpr int kAuxLarge = 170;
constexpr int kAuxSameTriangle = 8;
constexpr int kAuxSameCell = 4;

// dL/dalpha of one fragment through the lattice adjoint (rasterize.cu:951-970
// followed by multires.cu:130-222): three samples idx and their contributions g.
__device__ __forceinline__ void aux_contributions(float b0, float b1, int level, int S,
                                                  const float* __restrict__ alpha_src, int t, float loss, bool visible,
                                                  float scale, uint32_t idx[3], float g[3]) {
    float w[3];
    lattice_cell(b0, b1, level, idx, w);
    const float* src = alpha_src + (size_t)t * S;  // interp_level (the same sum)
    float alpha = 0.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) alpha = madd(alpha, w[q], __ldg(src + idx[q]));
    const float ga = aux_alpha_grad(loss, alpha, visible) * scale;
#pragma unroll
    for (int q = 0; q < 3; ++q) g[q] = ga * w[q];
}

__device__ __forceinline__ void aux_scatter(float b0, float b1, int level, int S, const float* __restrict__ alpha_src,
                                            int t, float loss, bool visible, float scale,
                                            float* __restrict__ grad_alpha_src) {
    uint32_t idx[3];
    float g[3];
    aux_contributions(b0, b1, level, S, alpha_src, t, loss, visible, scale, idx, g);
    float* dst = grad_alpha_src + (size_t)t * S;
#pragma unroll
    for (int q = 0; q < 3; ++q) atomicAdd(dst + idx[q], g[q]);
}

// The same for the warp's fragments (one a lane, where `hit`; called by the whole
// warp), those of one triangle and lattice cell summed before the atomics.
__device__ __forceinline__ void aux_scatter_merged(bool hit, float b0, float b1, int level, int S,
                                                   const float* __restrict__ alpha_src, int t, float loss,
                                                   bool visible, float scale, float* __restrict__ grad_alpha_src) {
    const int lane = threadIdx.x & 31;
    uint32_t idx[3] = {0u, 0u, 0u};
    float g[3] = {0.f, 0.f, 0.f};
    if (hit) aux_contributions(b0, b1, level, S, alpha_src, t, loss, visible, scale, idx, g);
    const unsigned mates = __match_any_sync(0xffffffffu, hit ? t : -1);  // the lanes on this lane's triangle
    if (__any_sync(0xffffffffu, hit && __popc(mates) >= kAuxSameTriangle)) {
        // a cell is its first sample and where the third lies to the first two
        const uint32_t cell = idx[0] << 2 | (idx[2] == idx[0] ? 2u : (idx[2] > idx[1] ? 1u : 0u));
        const unsigned peers = __match_any_sync(0xffffffffu, cell) & mates;
        const bool merged = hit && __popc(peers) >= kAuxSameCell;
        for (unsigned leaders = __ballot_sync(0xffffffffu, merged && lane == __ffs(peers) - 1); leaders != 0u;
             leaders &= leaders - 1u) {
            const int leader = __ffs(leaders) - 1;
            const bool mine = (__shfl_sync(0xffffffffu, peers, leader) >> lane) & 1u;
            const float v0 = mine ? g[0] : 0.f, v1 = mine ? g[1] : 0.f, v2 = mine ? g[2] : 0.f;
            // sums over the warp, sum q in the lanes of quarter q
            const bool hi = lane & 16, odd = lane & 8;
            const float a = (hi ? v2 : v0) + __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 16);
            const float b = (hi ? 0.f : v1) + __shfl_xor_sync(0xffffffffu, hi ? v1 : 0.f, 16);
            float v = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const uint32_t i0 = __shfl_sync(0xffffffffu, idx[0], leader), i1 = __shfl_sync(0xffffffffu, idx[1], leader),
                           i2 = __shfl_sync(0xffffffffu, idx[2], leader);
            const int lt = __shfl_sync(0xffffffffu, t, leader);
            // three lanes in one instruction: samples of one 32-byte sector are one access
            if ((lane & 7) == 0 && lane < 24)
                atomicAdd(grad_alpha_src + (size_t)lt * S + (hi ? i2 : (odd ? i1 : i0)), v);
        }
        hit = hit && !merged;
    }
    if (!hit) return;
    float* dst = grad_alpha_src + (size_t)t * S;
#pragma unroll
    for (int q = 0; q < 3; ++q) atomicAdd(dst + idx[q], g[q]);
}

// Opacity auxiliary gradient from the fragment records: one thread per
// record, blocks stride over the chunks.  Records follow the rasterizer's
// passes, so neighbours that share a triangle and a lattice cell come from
// neighbouring pixels of one pass: runs of equal (triangle, cell) in a warp are summed with a segmented
// reduction before the global atomics.
__global__ void __launch_bounds__(kRecChunk) aux_records_kernel(RecordStore rs, int level, int S,
                                                               const float* __restrict__ alpha_src,
                                                               const float* __restrict__ l1, float scale,
                                                               float* __restrict__ grad_alpha_src) {
    const int lane = threadIdx.x & 31;
    const int64_t reserved = rs.counters[0];
    const int64_t nchunks = (reserved < rs.capacity ? reserved : rs.capacity) / kRecChunk;
    for (int64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const bool valid = (int)threadIdx.x < rs.chunk_fill[c];
        int t = -1 - lane;
        uint32_t idx[3] = {0u, 0u, 0u};
        float g[3] = {0.f, 0.f, 0.f};
        if (valid) {
            const int4 r = rs.rec[c * kRecChunk + threadIdx.x];
            const uint32_t tv = (uint32_t)r.y;
            t = (int)(tv & 0x7fffffffu);
            const float b0 = __int_as_float(r.z), b1 = __int_as_float(r.w);
            float w[3];
            lattice_cell(b0, b1, (uint32_t)level, idx, w);
            // interp_scalar at one level (the same sum)
            const float* src = alpha_src + (size_t)t * S;
            float alpha = 0.f;
            alpha = madd(alpha, w[0], __ldg(src + idx[0]));
            alpha = madd(alpha, w[1], __ldg(src + idx[1]));
            alpha = madd(alpha, w[2], __ldg(src + idx[2]));
            const float ga = aux_alpha_grad(l1[(uint32_t)r.x], alpha, (tv >> 31) != 0) * scale;
#pragma unroll
            for (int q = 0; q < 3; ++q) g[q] = ga * w[q];
        }
        const int pt = __shfl_up_sync(0xffffffffu, t, 1);
        const uint32_t p0 = __shfl_up_sync(0xffffffffu, idx[0], 1), p1 = __shfl_up_sync(0xffffffffu, idx[1], 1),
                       p2 = __shfl_up_sync(0xffffffffu, idx[2], 1);
        const bool same = lane > 0 && pt == t && p0 == idx[0] && p1 == idx[1] && p2 == idx[2];
        const unsigned heads = __ballot_sync(0xffffffffu, !same);
        const int seg = __popc(heads & ((2u << lane) - 1u));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int oseg = __shfl_down_sync(0xffffffffu, seg, o);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float v = __shfl_down_sync(0xffffffffu, g[q], o);
                if (lane + o < 32 && oseg == seg) g[q] += v;
            }
        }
        if (valid && !same) {
            float* dst = grad_alpha_src + (size_t)t * S;
#pragma unroll
            for (int q = 0; q < 3; ++q) atomicAdd(dst + idx[q], g[q]);
        }
    }
}

// Opacity auxiliary gradient by re-enumeration: each block's fragments are
// recomputed and dL/dalpha is scattered through the lattice adjoint.
// Fragments behind the visible surface contribute nothing
// (rasterize.cu:950), so triangles whose depth bound lies behind every
// lane's surface are never staged.
// With item_list, only the blocks listed there (*item_count of them) are processed.
__global__ void __launch_bounds__(kWarpsPerCta * 32) aux_kernel(
    int B, const ds_view_desc* __restrict__ views, int num_tiles, int T, const TriBox* __restrict__ boxes,
    const TriVerts* __restrict__ verts, const TriEdges* __restrict__ edges, const int64_t* __restrict__ offsets,
    const int* __restrict__ sorted, const ListEntry* __restrict__ list, int64_t capacity, int level, int S,
    const float* __restrict__ alpha_src, int C,
    const float* __restrict__ color, const float* __restrict__ target, const float* __restrict__ rast, float scale,
    const int* __restrict__ item_list, const int* __restrict__ item_count, int* work,
    float* __restrict__ grad_alpha_src, int bwl) {
    __shared__ RasterStage s_stage[kWarpsPerCta];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RasterStage& st = s_stage[warp];
    chain_wait();
    const int items = item_list ? *item_count : num_tiles * kBlocksPerTile;
    for (int n = warp_next(work, items); n < items; n = warp_next(work, items)) {
        const int item = item_list ? item_list[n] : n;
        const BlockGeom g = block_geometry(item, B, views, T, offsets, sorted, capacity, bwl);
        if (g.begin >= g.end) continue;  // no triangle, no fragment
        const float ndc_x = pix_ndc(g.px, g.W), ndc_y = pix_ndc(g.py, g.H);
        if ((lane & (g.bw - 1)) == 0) st.row_y[lane >> bwl] = ndc_y;
        const unsigned valid = __ballot_sync(0xffffffffu, g.valid);
        __syncwarp();
        int tp = -1;
        float zp = 0.f, loss = 0.f;
        if (g.valid) {
            const float4 rp = reinterpret_cast<const float4*>(rast)[g.pix];
            tp = (int)rp.w - 1;
            zp = rp.z;
            if (target != nullptr) {
                for (int c = 0; c < C; ++c) loss += fabsf(color[g.pix * C + c] - target[g.pix * C + c]);
            } else {
                loss = color[g.pix];  // caller passes the per-pixel sum |c - target| directly
            }
        }
        // the surface's depth (+inf where a valid pixel is empty) and the block's farthest
        const float z_cut = !g.valid ? -INFINITY : (tp >= 0 ? zp : INFINITY);
        const float warp_far = warp_max(z_cut);
        const int large = kAuxLarge * S;
        for (int64_t g0 = g.begin; g0 < g.end; g0 += 32) {
            float head;
            bool merge;
            unsigned todo = stage_pixels(g, g0, boxes, verts, edges, list, T, warp_far, valid, st, &head, large, &merge);
            if (g.ordered && head > warp_far) break;
            while (__any_sync(0xffffffffu, todo != 0u)) {
                const int k = todo != 0u ? __ffs(todo) - 1 : 0;
                // the pixel's surface does not lie in front of the triangle
                const bool near = todo != 0u && !(st.zlo[k] > z_cut);
                todo = !near && g.ordered ? 0u : todo & (todo - 1u);
                if (!merge && !near) continue;
                const int t = st.t[k];
                const float4 p0 = st.v[k].p0, p1 = st.v[k].p1, p2 = st.v[k].p2;
                float b0 = 0.f, b1 = 0.f, depth;
                const bool hit = near && fragment_at(ndc_y, ndc_x, p0, p1, p2, b0, b1, depth) && !(tp >= 0 && depth > zp);
                const bool visible = tp >= 0 && t == tp;
                if (!merge) {
                    if (hit) aux_scatter(b0, b1, level, S, alpha_src, t, loss, visible, scale, grad_alpha_src);
                } else if (__any_sync(0xffffffffu, hit)) {
                    aux_scatter_merged(hit, b0, b1, level, S, alpha_src, t, loss, visible, scale, grad_alpha_src);
                }
            }
            __syncwarp();
        }
    }
}

}  // namespace dsb

using namespace dsb;

extern "C" {

size_t ds_tiles_workspace_size(int B, int T, int num_tiles, int64_t list_capacity) {
    size_t total = 0;
    carve(nullptr, B, T, num_tiles, list_capacity, &total);
    return total;
}

static int check_tiles_args(int B, const ds_view_desc* views, int num_tiles, int V, const float* pos, int T,
                            size_t ws_bytes, int64_t capacity) {
    DS_CHECK_ARG(B >= 0 && num_tiles >= 0 && V >= 0 && T >= 0 && capacity >= 0, "tiles: bad sizes");
    DS_CHECK_ARG((int64_t)B * T <= 0x7fffffff, "tiles: B*T exceeds int32");
    DS_CHECK_ARG(capacity <= 0x7fffffff, "tiles: list capacity exceeds int32");
    DS_CHECK_ARG((int64_t)num_tiles * kBlocksPerTile <= 0x7fffffff, "tiles: too many tiles");
    DS_CHECK_ARG(B == 0 || views != nullptr, "tiles: null view table");
    DS_CHECK_ARG(((uintptr_t)pos & 15) == 0, "tiles: pos not 16-byte aligned");
    if (ws_bytes < ds_tiles_workspace_size(B, T, num_tiles, capacity))
        return set_error(DS_ERR_WORKSPACE, "tiles: workspace too small (%zu < %zu)", ws_bytes,
                         ds_tiles_workspace_size(B, T, num_tiles, capacity));
    return DS_OK;
}

int ds_tiles_bin(int B, const ds_view_desc* views, int num_tiles, int V, const float* pos, int T, const int* tri,
                 void* workspace, size_t workspace_bytes, int64_t list_capacity, int* status, ds_stream_t stream) {
    int rc = check_tiles_args(B, views, num_tiles, V, pos, T, workspace_bytes, list_capacity);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    TileWs w = carve(workspace, B, T, num_tiles, list_capacity, nullptr);
    // one memset clears the counts, the fill cursors, the work counters and the workspace's status word
    // (counts .. work; the offsets and flags in between are written below): a launch costs more than their bytes
    DS_CUDA(cudaMemsetAsync(w.counts, 0, reinterpret_cast<char*>(w.work + 3) - reinterpret_cast<char*>(w.counts), st));
    const int64_t n = (int64_t)B * T;
    const bool narrow = n <= kBinNarrow;
    const unsigned grid = blocks_for(narrow ? n * 4 : n);  // 8 or 32 triangles per warp
    if (n > 0) {
        const auto setup = narrow ? bin_setup_kernel<8> : bin_setup_kernel<32>;
        launch_chained(setup, dim3(grid), kThreads, 0, st, B, views, V, pos, T, tri, w.boxes, w.verts, w.ndc, w.edges,
                       w.counts);
    }
    // offsets[num_tiles] = total number of entries; up to kScanOneMax tiles in one launch
    if (num_tiles <= kScanOneMax) {
        launch_chained(scan_one_cta_kernel, dim3(1), kScanOneThreads, 0, st, w.counts, num_tiles, w.offsets);
    } else {
        rc = device_scan<int, int64_t>(w.counts, num_tiles, w.offsets, false, w.scan, st, nullptr,
                                       w.offsets + num_tiles);
        if (rc) return rc;
    }
    if (n > 0) {
        const auto fill = narrow ? bin_fill_kernel<8> : bin_fill_kernel<32>;
        launch_chained(fill, dim3(grid), kThreads, 0, st, B, views, T, w.boxes, w.verts, w.ndc, w.offsets, w.cursor,
                       w.fill, list_capacity, status);
    }
    if (num_tiles > 0)
        launch_chained(sort_lists_kernel, dim3((unsigned)((num_tiles + kSortWarps - 1) / kSortWarps)), kSortWarps * 32, 0,
                       st, num_tiles, w.offsets, w.fill, w.list, list_capacity, w.sorted);
    return check_launch("tiles_bin");
}

size_t ds_tiles_status_offset(int B, int T, int num_tiles, int64_t list_capacity) {
    const TileWs w = carve(nullptr, B, T, num_tiles, list_capacity, nullptr);
    return (size_t)(reinterpret_cast<const char*>(w.work + 2) - (const char*)nullptr);
}

int ds_tiles_bin_report(int B, const ds_view_desc* views, int num_tiles, int V, const float* pos, int T, const int* tri,
                        void* workspace, size_t workspace_bytes, int64_t list_capacity, int* status_host,
                        ds_stream_t stream) {
    const int rc0 = check_tiles_args(B, views, num_tiles, V, pos, T, workspace_bytes, list_capacity);
    if (rc0) return rc0;
    int* status = carve(workspace, B, T, num_tiles, list_capacity, nullptr).work + 2;
    const int rc = ds_tiles_bin(B, views, num_tiles, V, pos, T, tri, workspace, workspace_bytes, list_capacity, status,
                                stream);
    if (rc) return rc;
    // not from a captured call: its replays would write to the word, whoever has it by then
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    DS_CUDA(cudaStreamIsCapturing((cudaStream_t)stream, &capture));
    if (status_host != nullptr && capture == cudaStreamCaptureStatusNone)
        DS_CUDA(cudaMemcpyAsync(status_host, status, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    return DS_OK;
}

}  // extern "C"

namespace dsb {

// Persistent grid: as many 8-warp CTAs as fit on the SMs (queried once per
// kernel), capped by the number of blocks.
static unsigned block_grid(int num_tiles, const void* kernel, int& per_sm, size_t smem = 0) {
    if (per_sm == 0) {
        int n = 0;
        if (smem > 0) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kWarpsPerCta * 32, smem) != cudaSuccess || n < 1)
            n = 1;
        per_sm = n;
    }
    const int64_t warps = (int64_t)num_tiles * kBlocksPerTile;
    const int64_t ctas = (warps + kWarpsPerCta - 1) / kWarpsPerCta;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    return (unsigned)(ctas < 1 ? 1 : (ctas < cap ? ctas : cap));
}

static int g_occ_raster = 0, g_occ_raster_rec = 0, g_occ_aux = 0;

int tiles_rasterize_impl(int B, const ds_view_desc* views, int num_tiles, int T, int level, int S,
                         const float* alpha_src, int thr_mode, float thr_const, const uint64_t* rng, float* rast,
                         void* workspace, int64_t list_capacity, const RecordStore* rs, cudaStream_t st, int bwl,
                         bool chained) {
    if (num_tiles == 0) return DS_OK;
    TileWs w = carve(workspace, B, T, num_tiles, list_capacity, nullptr);
    if (rs != nullptr) {
        const void* k = reinterpret_cast<const void*>(&raster_kernel<true>);
        const dim3 grid(block_grid(num_tiles, k, g_occ_raster_rec));
        launch_kernel(chained, raster_kernel<true>, grid, kWarpsPerCta * 32, 0, st, B, views, num_tiles, T, w.boxes,
                      w.verts, w.edges, w.offsets, w.sorted, w.list, list_capacity, level, S, alpha_src, thr_mode,
                      thr_const, rng, w.work, rast, *rs, bwl);
    } else {
        const void* k = reinterpret_cast<const void*>(&raster_kernel<false>);
        const dim3 grid(block_grid(num_tiles, k, g_occ_raster));
        launch_kernel(chained, raster_kernel<false>, grid, kWarpsPerCta * 32, 0, st, B, views, num_tiles, T, w.boxes,
                      w.verts, w.edges, w.offsets, w.sorted, w.list, list_capacity, level, S, alpha_src, thr_mode,
                      thr_const, rng, w.work, rast, RecordStore{}, bwl);
    }
    return check_launch("tiles_rasterize");
}

static int aux_launch(int B, const ds_view_desc* views, int num_tiles, int T, int level, int S,
                      const float* alpha_src, int C, const float* color, const float* target, const float* rast,
                      float scale, float* grad_alpha_src, void* workspace, int64_t list_capacity,
                      const int* item_list, const int* item_count, cudaStream_t st, int bwl, bool chained) {
    TileWs w = carve(workspace, B, T, num_tiles, list_capacity, nullptr);
    const void* k = reinterpret_cast<const void*>(&aux_kernel);
    launch_kernel(chained, aux_kernel, dim3(block_grid(num_tiles, k, g_occ_aux)), kWarpsPerCta * 32, 0, st, B, views,
                  num_tiles, T, w.boxes, w.verts, w.edges, w.offsets, w.sorted, w.list, list_capacity, level, S, alpha_src,
                  C, color, target, rast, scale, item_list, item_count, w.work + 1, grad_alpha_src, bwl);
    return check_launch("tiles_opacity_aux");
}

TileTables tiles_tables(void* workspace, int B, int T, int num_tiles, int64_t list_capacity) {
    const TileWs w = carve(workspace, B, T, num_tiles, list_capacity, nullptr);
    return TileTables{w.boxes, w.verts, w.ndc, w.offsets};
}

int tiles_aux_impl(int B, const ds_view_desc* views, int num_tiles, int T, int level, int S, const float* alpha_src,
                   const float* l1, const float* rast, float scale, float* grad_alpha_src, void* workspace,
                   int64_t list_capacity, const RecordStore* rs, cudaStream_t st, int bwl, bool chained) {
    if (num_tiles == 0) return DS_OK;
    if (rs == nullptr)
        return aux_launch(B, views, num_tiles, T, level, S, alpha_src, 1, l1, nullptr, rast, scale, grad_alpha_src,
                          workspace, list_capacity, nullptr, nullptr, st, bwl, chained);
    aux_records_kernel<<<sm_count() * 8, kRecChunk, 0, st>>>(*rs, level, S, alpha_src, l1, scale, grad_alpha_src);
    const int rc = check_launch("tiles_opacity_aux records");
    if (rc) return rc;
    return aux_launch(B, views, num_tiles, T, level, S, alpha_src, 1, l1, nullptr, rast, scale, grad_alpha_src,
                      workspace, list_capacity, rs->fallback, rs->counters + 1, st, bwl, true);
}

}  // namespace dsb

extern "C" {

int ds_tiles_rasterize(int B, const ds_view_desc* views, int num_tiles, int V, const float* pos, int T,
                       const int* tri, int level, int S, const float* alpha_src, int thr_mode, float thr_const,
                       const uint64_t* rng, float* rast, void* workspace, size_t workspace_bytes,
                       int64_t list_capacity, ds_stream_t stream) {
    (void)tri;
    int rc = check_tiles_args(B, views, num_tiles, V, pos, T, workspace_bytes, list_capacity);
    if (rc) return rc;
    DS_CHECK_ARG(level >= 0 && level <= 12 && (uint32_t)S == feats_at_level(level), "Invalid feature size.");
    DS_CHECK_ARG(thr_mode == 0 || (thr_mode == 1 && rng != nullptr), "tiles_rasterize: bad threshold mode");
    DS_CHECK_ARG(((uintptr_t)rast & 15) == 0, "tiles_rasterize: rast not 16-byte aligned");
    return tiles_rasterize_impl(B, views, num_tiles, T, level, S, alpha_src, thr_mode, thr_const, rng, rast,
                                workspace, list_capacity, nullptr, (cudaStream_t)stream, kDefaultBlockShape, false);
}

int ds_tiles_opacity_aux(int B, const ds_view_desc* views, int num_tiles, int V, const float* pos, int T,
                         const int* tri, int level, int S, const float* alpha_src, int C, const float* color,
                         const float* target, const float* rast, float scale, float* grad_alpha_src,
                         void* workspace, size_t workspace_bytes, int64_t list_capacity, ds_stream_t stream) {
    (void)tri;
    int rc = check_tiles_args(B, views, num_tiles, V, pos, T, workspace_bytes, list_capacity);
    if (rc) return rc;
    DS_CHECK_ARG(level >= 0 && level <= 12 && (uint32_t)S == feats_at_level(level), "Invalid feature size.");
    DS_CHECK_ARG(C > 0, "tiles_opacity_aux: C must be positive");
    DS_CHECK_ARG(target != nullptr || C == 1, "tiles_opacity_aux: without a target, color holds one value per pixel");
    DS_CHECK_ARG(((uintptr_t)rast & 15) == 0, "tiles_opacity_aux: rast not 16-byte aligned");
    if (num_tiles == 0) return DS_OK;
    return aux_launch(B, views, num_tiles, T, level, S, alpha_src, C, color, target, rast, scale, grad_alpha_src,
                      workspace, list_capacity, nullptr, nullptr, (cudaStream_t)stream, kDefaultBlockShape, false);
}

}  // extern "C"
