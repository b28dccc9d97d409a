// diffsoup_b200/csrc/color_mlp.cu -- the shading MLP of the operator path
// (ColorMLP.forward, python/diffsoup/multires.py:169-207) and its gradients in
// FP32, for hidden width 16, one or two hidden layers and three outputs:
//   y = sigmoid(Wo relu(W1 relu(W0 x + b0) + b1) + bo)
//   out = (1 - x3) x[0:3] + x3 y     where mask, else 0
//
// One thread per pixel holds its activations in registers and reads the
// weights from shared memory (every lane the same 16 bytes: one wavefront for
// four products).  The backward kernel recomputes the forward, so nothing but x
// is kept between them.  A weight gradient is a sum over all pixels of an outer
// product: a warp puts its 32 pixels' layer inputs and deltas into shared memory
// and each lane accumulates its eight entries over them, for all the warp's
// pixels; the CTAs' sums are added in a fixed order by a last kernel, so the
// gradients do not depend on scheduling.
//
// Issue slots bound both kernels (about 700 and 2,400 warp instructions per 32
// pixels).  One 800x800 view, 16 -> 16 -> 16 -> 3, three fifths of the pixels covered: 35 and 86 us;
// as matrix products over gathered rows (nine GEMMs, mask indexing and its scatter) the two took about 1,300 us.
#include "rows.cuh"

namespace dsb {

constexpr int kMlpHidden = 16;
constexpr int kMlpWarps = kThreads / 32;
constexpr int kMlpRow = 20;  // floats per pixel of a warp's tiles: 16-byte rows of 8 lanes fall in 32 banks

struct MlpWeights {
    const float* w[3];  // W0 [16,in], W1 [16,16] (two layers), Wo [3,16]
    const float* b;     // b0 [16], b1 [16] (two layers), bo [3]
};

struct MlpGrads {
    float* w[3];
    float* b;
};

template <int IN4, int L>
struct MlpSmem {
    float w0[kMlpHidden * IN4];
    float w1[L == 2 ? 256 : 4];
    float wo[48];
    float b[36];
};

__host__ __device__ constexpr int mlp_param_floats(int in, int layers) {
    return kMlpHidden * in + (layers - 1) * 256 + 48 + layers * 16 + 3;
}

template <int IN4, int L>
__device__ __forceinline__ void mlp_load(MlpSmem<IN4, L>& s, const MlpWeights& w, int in) {
    for (int i = threadIdx.x; i < kMlpHidden * IN4; i += blockDim.x)
        s.w0[i] = i % IN4 < in ? w.w[0][i / IN4 * in + i % IN4] : 0.f;
    if (L == 2)
        for (int i = threadIdx.x; i < 256; i += blockDim.x) s.w1[i] = w.w[1][i];
    for (int i = threadIdx.x; i < 48; i += blockDim.x) s.wo[i] = w.w[2][i];
    for (int i = threadIdx.x; i < L * 16 + 3; i += blockDim.x) s.b[i] = w.b[i];
    __syncthreads();
}

// NaN stays NaN, as torch's relu keeps it.
__device__ __forceinline__ float relu(float v) { return v <= 0.f ? 0.f : v; }

// out[j] = b[j] + sum_i w[j][i] x[i]
template <int OUT, int IN>
__device__ __forceinline__ void mlp_dense(const float* w, const float* b, const float x[IN], float out[OUT]) {
#pragma unroll
    for (int j = 0; j < OUT; ++j) {
        float v = b[j];
#pragma unroll
        for (int i = 0; i < IN; i += 4) {
            const float4 q = *reinterpret_cast<const float4*>(w + j * IN + i);
            v = fmaf(q.x, x[i], v); v = fmaf(q.y, x[i + 1], v); v = fmaf(q.z, x[i + 2], v); v = fmaf(q.w, x[i + 3], v);
        }
        out[j] = v;
    }
}

// out[i] = sum_j w[j][i] d[j]
template <int OUT, int IN>
__device__ __forceinline__ void mlp_transposed(const float* w, const float d[OUT], float out[IN]) {
#pragma unroll
    for (int i = 0; i < IN; ++i) out[i] = 0.f;
#pragma unroll
    for (int j = 0; j < OUT; ++j)
#pragma unroll
        for (int i = 0; i < IN; i += 4) {
            const float4 q = *reinterpret_cast<const float4*>(w + j * IN + i);
            out[i] = fmaf(q.x, d[j], out[i]); out[i + 1] = fmaf(q.y, d[j], out[i + 1]);
            out[i + 2] = fmaf(q.z, d[j], out[i + 2]); out[i + 3] = fmaf(q.w, d[j], out[i + 3]);
        }
}

template <int IN4, int L>
__device__ __forceinline__ void mlp_forward(const MlpSmem<IN4, L>& s, const float x[IN4], float h1[16], float h2[16],
                                            float y[3]) {
    mlp_dense<16, IN4>(s.w0, s.b, x, h1);
#pragma unroll
    for (int j = 0; j < 16; ++j) h1[j] = relu(h1[j]);
    if (L == 2) {
        mlp_dense<16, 16>(s.w1, s.b + 16, h1, h2);
#pragma unroll
        for (int j = 0; j < 16; ++j) h2[j] = relu(h2[j]);
    }
    mlp_dense<3, 16>(s.wo, s.b + L * 16, L == 2 ? h2 : h1, y);
#pragma unroll
    for (int o = 0; o < 3; ++o) y[o] = 1.f / (1.f + expf(-y[o]));
}

// The calling lane's row of x (zeros when not `in_use`), straight from memory
// when the rows are 16-byte vectors, else through the warp's tile.
template <int IN4>
__device__ __forceinline__ void mlp_row(const float* __restrict__ x, int64_t p0, int live, int in, bool vec, bool in_use,
                                        float* tile, float v[IN4]) {
    const int lane = threadIdx.x & 31;
    if (!vec) warp_rows<false>(tile, const_cast<float*>(x) + p0 * in, in, live);
#pragma unroll
    for (int i = 0; i < IN4; i += 4) {
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in_use) {
            if (vec) {
                q = __ldg(reinterpret_cast<const float4*>(x + (p0 + lane) * IN4 + i));
            } else {
                const float* r = tile + lane * in;
                q.x = i < in ? r[i] : 0.f; q.y = i + 1 < in ? r[i + 1] : 0.f;
                q.z = i + 2 < in ? r[i + 2] : 0.f; q.w = i + 3 < in ? r[i + 3] : 0.f;
            }
        }
        v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
    }
    if (!vec) __syncwarp();
}

template <int IN4, int L>
__global__ void __launch_bounds__(kThreads) color_mlp_kernel(int64_t n, int in, const float* __restrict__ x,
                                                             const unsigned char* __restrict__ mask, MlpWeights w,
                                                             float* __restrict__ out) {
    __shared__ __align__(16) MlpSmem<IN4, L> s;
    __shared__ __align__(16) float s_tile[kMlpWarps][32 * kMlpRow];
    mlp_load<IN4, L>(s, w, in);
    const int lane = threadIdx.x & 31;
    float* tile = s_tile[threadIdx.x >> 5];
    const bool vec = in == IN4 && ((uintptr_t)x & 15) == 0;
    const int64_t stride = (int64_t)gridDim.x * kThreads;
    for (int64_t p0 = ((int64_t)blockIdx.x * kMlpWarps + (threadIdx.x >> 5)) * 32; p0 < n; p0 += stride) {
        const int live = n - p0 < 32 ? (int)(n - p0) : 32;
        const bool covered = lane < live && (mask == nullptr || mask[p0 + lane] != 0);
        float c[3] = {0.f, 0.f, 0.f};
        if (__any_sync(0xffffffffu, covered)) {
            float v[IN4], h1[16], h2[16], y[3];
            mlp_row<IN4>(x, p0, live, in, vec, covered, tile, v);
            mlp_forward<IN4, L>(s, v, h1, h2, y);
            if (covered)
#pragma unroll
                for (int o = 0; o < 3; ++o) c[o] = (1.f - v[3]) * v[o] + v[3] * y[o];
        }
#pragma unroll
        for (int o = 0; o < 3; ++o) tile[lane * 3 + o] = c[o];
        __syncwarp();
        warp_rows<true>(tile, out + p0 * 3, 3, live);
    }
}

// acc[k] += sum over the 32 pixels of d[px][lane / 2] * a[px][half * N + k], half =
// lane mod 2, N = IN / 2, and *bias += sum of d[px][lane / 2].
template <int IN>
__device__ __forceinline__ void mlp_outer(const float* a, const float* d, float acc[IN / 2], float& bias) {
    constexpr int N = IN / 2;
    const int lane = threadIdx.x & 31, j = lane >> 1, half = (lane & 1) * N;
#pragma unroll 4
    for (int px = 0; px < 32; ++px) {
        const float dv = d[px * kMlpRow + j];
        const float* r = a + px * kMlpRow + half;
        bias += dv;
        if (N % 4 == 0) {
#pragma unroll
            for (int k = 0; k < N; k += 4) {
                const float4 q = *reinterpret_cast<const float4*>(r + k);
                acc[k] = fmaf(dv, q.x, acc[k]); acc[k + 1] = fmaf(dv, q.y, acc[k + 1]);
                acc[k + 2] = fmaf(dv, q.z, acc[k + 2]); acc[k + 3] = fmaf(dv, q.w, acc[k + 3]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; k += 2) {
                const float2 q = *reinterpret_cast<const float2*>(r + k);
                acc[k] = fmaf(dv, q.x, acc[k]); acc[k + 1] = fmaf(dv, q.y, acc[k + 1]);
            }
        }
    }
}

template <int N>
__device__ __forceinline__ void mlp_put(float* tile, const float v[N]) {
    float* r = tile + (threadIdx.x & 31) * kMlpRow;
#pragma unroll
    for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(r + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// Gradients: grad_x [n,in] (may be null) and the CTA's sums of the parameters'
// gradients in partial [gridDim.x][mlp_param_floats] (W0 W1 Wo b0 b1 bo).
template <int IN4, int L>
__global__ void __launch_bounds__(kThreads, 2) color_mlp_backward_kernel(
    int64_t n, int in, const float* __restrict__ x, const unsigned char* __restrict__ mask, MlpWeights w,
    const float* __restrict__ grad_out, float* __restrict__ grad_x, float* __restrict__ partial) {
    __shared__ __align__(16) MlpSmem<IN4, L> s;
    __shared__ __align__(16) float s_a[kMlpWarps][32 * kMlpRow], s_d[kMlpWarps][32 * kMlpRow];
    mlp_load<IN4, L>(s, w, in);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *ta = s_a[warp], *td = s_d[warp];
    const bool vec = in == IN4 && (((uintptr_t)x | (uintptr_t)grad_x) & 15) == 0;
    float g0[IN4 / 2], g1[8], go[2] = {0.f, 0.f}, b0 = 0.f, b1 = 0.f, bo = 0.f;
#pragma unroll
    for (int k = 0; k < IN4 / 2; ++k) g0[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) g1[k] = 0.f;
    const int64_t stride = (int64_t)gridDim.x * kThreads;
    for (int64_t p0 = ((int64_t)blockIdx.x * kMlpWarps + warp) * 32; p0 < n; p0 += stride) {
        const int live = n - p0 < 32 ? (int)(n - p0) : 32;
        const bool covered = lane < live && (mask == nullptr || mask[p0 + lane] != 0);
        float dx[IN4];
        if (__any_sync(0xffffffffu, covered)) {
            float v[IN4], h1[16], h2[16], y[3], g[3], dz[4] = {0.f, 0.f, 0.f, 0.f};
            mlp_row<IN4>(x, p0, live, in, vec, covered, ta, v);
            warp_rows<false>(td, const_cast<float*>(grad_out) + p0 * 3, 3, live);
#pragma unroll
            for (int o = 0; o < 3; ++o) g[o] = covered ? td[lane * 3 + o] : 0.f;
            __syncwarp();
            mlp_forward<IN4, L>(s, v, h1, h2, y);
            if (!covered)  // keeps 0 * inf of such lanes out of the sums
#pragma unroll
                for (int j = 0; j < 16; ++j) h1[j] = h2[j] = 0.f;
            float dr = 0.f;
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                dr = fmaf(g[o], y[o] - v[o], dr);
                dz[o] = v[3] * g[o] * y[o] * (1.f - y[o]);
                if (!covered) dz[o] = 0.f;
            }
            // output layer: lane (o, j) of two outputs, the third on the first 16 lanes
            float* hl = L == 2 ? h2 : h1;
            mlp_put<16>(ta, hl);
            mlp_put<4>(td, dz);
            __syncwarp();
#pragma unroll 4
            for (int px = 0; px < 32; ++px) {
                const float a = ta[px * kMlpRow + (lane & 15)];
                const float4 q = *reinterpret_cast<const float4*>(td + px * kMlpRow);
                go[0] = fmaf(a, lane < 16 ? q.x : q.y, go[0]);
                go[1] = fmaf(a, q.z, go[1]);
                bo += lane == 0 ? q.x : (lane == 1 ? q.y : q.z);
            }
            float d[16];
            mlp_transposed<3, 16>(s.wo, dz, d);
#pragma unroll
            for (int j = 0; j < 16; ++j) d[j] = hl[j] <= 0.f ? 0.f : d[j];
            __syncwarp();
            if (L == 2) {
                mlp_put<16>(ta, h1);
                mlp_put<16>(td, d);
                __syncwarp();
                mlp_outer<16>(ta, td, g1, b1);
                float e[16];
                mlp_transposed<16, 16>(s.w1, d, e);
#pragma unroll
                for (int j = 0; j < 16; ++j) d[j] = h1[j] <= 0.f ? 0.f : e[j];
                __syncwarp();
            }
            mlp_put<IN4>(ta, v);
            mlp_put<16>(td, d);
            __syncwarp();
            mlp_outer<IN4>(ta, td, g0, b0);
            mlp_transposed<16, IN4>(s.w0, d, dx);
#pragma unroll
            for (int o = 0; o < 3; ++o) dx[o] = fmaf(1.f - v[3], g[o], dx[o]);
            dx[3] += dr;
            __syncwarp();
        }
        if (grad_x == nullptr) continue;
        if (!covered)
#pragma unroll
            for (int i = 0; i < IN4; ++i) dx[i] = 0.f;
        if (vec) {
            if (lane < live)
#pragma unroll
                for (int i = 0; i < IN4; i += 4)
                    *reinterpret_cast<float4*>(grad_x + (p0 + lane) * IN4 + i) =
                        make_float4(dx[i], dx[i + 1], dx[i + 2], dx[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < IN4; ++i)
                if (i < in) ta[lane * in + i] = dx[i];
            __syncwarp();
            warp_rows<true>(ta, grad_x + p0 * in, in, live);
        }
    }
    // the CTA's sums, its warps in order
    const int P = mlp_param_floats(in, L);
    float* sum = s_a[0];
    __syncthreads();
    for (int i = threadIdx.x; i < P; i += blockDim.x) sum[i] = 0.f;
    __syncthreads();
    float* sw1 = sum + 16 * in;
    float* swo = sw1 + (L - 1) * 256;
    float* sb = swo + 48;
    for (int q = 0; q < kMlpWarps; ++q) {
        if (warp == q) {
            const int j = lane >> 1, h = lane & 1;
#pragma unroll
            for (int k = 0; k < IN4 / 2; ++k)
                if (h * (IN4 / 2) + k < in) sum[j * in + h * (IN4 / 2) + k] += g0[k];
            if (L == 2)
#pragma unroll
                for (int k = 0; k < 8; ++k) sw1[j * 16 + h * 8 + k] += g1[k];
            swo[lane] += go[0];
            if (lane < 16) swo[32 + lane] += go[1];
            if (h == 0) {
                sb[j] += b0;
                if (L == 2) sb[16 + j] += b1;
            }
            if (lane < 3) sb[L * 16 + lane] += bo;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < P; i += blockDim.x) partial[(size_t)blockIdx.x * P + i] = sum[i];
}

// Sums the CTAs' partial gradients in a fixed order (eight interleaved runs,
// then their sum, in double) into the parameters' gradients.
__global__ void __launch_bounds__(kThreads) color_mlp_reduce_kernel(int blocks, int in, int layers,
                                                                    const float* __restrict__ partial, MlpGrads g) {
    __shared__ double s_sum[8][32];
    const int P = mlp_param_floats(in, layers), lane = threadIdx.x & 31, run = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    double v = 0.0;
    if (i < P)
        for (int b = run; b < blocks; b += 8) v += (double)partial[(size_t)b * P + i];
    s_sum[run][lane] = v;
    __syncthreads();
    if (run != 0 || i >= P) return;
    for (int r = 1; r < 8; ++r) v += s_sum[r][lane];
    const int n0 = 16 * in, n1 = n0 + (layers - 1) * 256, n2 = n1 + 48;
    float* dst = i < n0 ? g.w[0] + i : (i < n1 ? g.w[1] + (i - n0) : (i < n2 ? g.w[2] + (i - n1) : g.b + (i - n2)));
    *dst = (float)v;
}

static int mlp_check(int64_t n, int in, int hidden, int layers, int out_dim) {
    DS_CHECK_ARG(n >= 0 && in >= 4 && in <= 20 && hidden == kMlpHidden && (layers == 1 || layers == 2) && out_dim == 3,
                 "color_mlp: %d -> %d x %d -> %d is not built", in, hidden, layers, out_dim);
    return DS_OK;
}

static unsigned mlp_grid(int64_t n, int per_sm) {
    const int64_t want = (n + kThreads - 1) / kThreads, cap = (int64_t)sm_count() * per_sm;
    return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

constexpr int kMlpBackwardPerSm = 2;

}  // namespace dsb

using namespace dsb;

#define DSB_MLP(KERNEL, GRID, ...)                                                          \
    do {                                                                                    \
        const int in4 = in <= 12 ? 12 : (in <= 16 ? 16 : 20);                               \
        if (layers == 1) {                                                                  \
            if (in4 == 12) KERNEL<12, 1><<<GRID, kThreads, 0, st>>>(__VA_ARGS__);           \
            else if (in4 == 16) KERNEL<16, 1><<<GRID, kThreads, 0, st>>>(__VA_ARGS__);      \
            else KERNEL<20, 1><<<GRID, kThreads, 0, st>>>(__VA_ARGS__);                     \
        } else {                                                                            \
            if (in4 == 12) KERNEL<12, 2><<<GRID, kThreads, 0, st>>>(__VA_ARGS__);           \
            else if (in4 == 16) KERNEL<16, 2><<<GRID, kThreads, 0, st>>>(__VA_ARGS__);      \
            else KERNEL<20, 2><<<GRID, kThreads, 0, st>>>(__VA_ARGS__);                     \
        }                                                                                   \
    } while (0)

extern "C" {

int ds_color_mlp_forward(int64_t n, int in, int hidden, int layers, const float* x, const unsigned char* mask,
                         const float* w0, const float* w1, const float* wo, const float* biases, float* out,
                         ds_stream_t stream) {
    const int rc = mlp_check(n, in, hidden, layers, 3);
    if (rc) return rc;
    if (n == 0) return DS_OK;
    DS_CHECK_ARG(x && w0 && (layers == 1 || w1) && wo && biases && out, "color_mlp_forward: null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    const MlpWeights w{{w0, w1, wo}, biases};
    DSB_MLP(color_mlp_kernel, mlp_grid(n, 4), n, in, x, mask, w, out);
    return check_launch("color_mlp_forward");
}

size_t ds_color_mlp_backward_workspace(int64_t n, int in, int layers) {
    return (size_t)mlp_grid(n, kMlpBackwardPerSm) * mlp_param_floats(in, layers) * sizeof(float);
}

int ds_color_mlp_backward(int64_t n, int in, int hidden, int layers, const float* x, const unsigned char* mask,
                          const float* w0, const float* w1, const float* wo, const float* biases,
                          const float* grad_out, float* grad_x, float* grad_w0, float* grad_w1, float* grad_wo,
                          float* grad_biases, void* workspace, size_t workspace_bytes, ds_stream_t stream) {
    const int rc = mlp_check(n, in, hidden, layers, 3);
    if (rc) return rc;
    DS_CHECK_ARG((n == 0 || (x && grad_out)) && w0 && (layers == 1 || (w1 && grad_w1)) && wo && biases && grad_w0 &&
                     grad_wo && grad_biases && workspace,
                 "color_mlp_backward: null pointer");
    if (workspace_bytes < ds_color_mlp_backward_workspace(n, in, layers))
        return set_error(DS_ERR_WORKSPACE, "color_mlp_backward: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    const MlpWeights w{{w0, w1, wo}, biases};
    const MlpGrads g{{grad_w0, grad_w1, grad_wo}, grad_biases};
    float* partial = reinterpret_cast<float*>(workspace);
    const unsigned grid = mlp_grid(n, kMlpBackwardPerSm);
    DSB_MLP(color_mlp_backward_kernel, grid, n, in, x, mask, w, grad_out, grad_x, partial);
    const int P = mlp_param_floats(in, layers);
    color_mlp_reduce_kernel<<<(P + 31) / 32, kThreads, 0, st>>>((int)grid, in, layers, partial, g);
    return check_launch("color_mlp_backward");
}

}  // extern "C"
