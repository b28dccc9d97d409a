// diffsoup_b200/csrc/optim.cu -- the optimiser updates that follow the
// training step: VectorAdam for the soup's vertex positions
// (python/diffsoup/optimize.py:7-68) and Adam for the neural features,
// opacities and MLP (torch.optim.Adam as examples/02_synthetic.py:310-315
// uses it: no weight decay, no amsgrad).  One fused elementwise pass each,
// memory bound: a parameter, its gradient and its moments are read once and
// written once.  The step count lives in device memory and is advanced by the
// call itself, so an update captures into a CUDA graph with the step.
#include <cmath>

#include "common.cuh"

namespace dsb {

struct AdamScale {
    float b1, b2, one_m_b1, one_m_b2, step_size, bc2_sqrt;
};

// The hyperparameters arrive in double, as torch's Python scalars: the
// complements 1 - beta are formed in double and then rounded, like torch's
// alpha / weight arguments.
__device__ __forceinline__ AdamScale adam_betas(double b1, double b2) {
    AdamScale s;
    s.b1 = (float)b1;
    s.b2 = (float)b2;
    s.one_m_b1 = (float)(1.0 - b1);
    s.one_m_b2 = (float)(1.0 - b2);
    return s;
}

// A bias correction of step t (the count after this update's increment): lr / (1 - b1^t), or sqrt(1 - b2^t).
__device__ __forceinline__ float adam_correction(const int* step, double lr, double b, bool second) {
    const double bc = 1.0 - pow(b, (double)(*step + 1));
    return (float)(second ? sqrt(bc) : lr / bc);
}

// torch.optim.Adam, one element: m <- m + (1-b1)(g - m), v <- b2 v + (1-b2) g^2,
// p <- p - lr/bc1 * m / (sqrt(v)/sqrt(bc2) + eps).
__device__ __forceinline__ void adam_one(float& p, float g, float& m, float& v, const AdamScale& s, float eps) {
    m = fmaf(s.one_m_b1, g - m, m);
    v = fmaf(s.one_m_b2 * g, g, s.b2 * v);
    p = p - s.step_size * m / (sqrtf(v) / s.bc2_sqrt + eps);
}

// Parameters of one update, by value in the kernel's arguments.  Parameter i
// takes blocks [first[i], first[i + 1]) of kAdamBlock elements.
constexpr int kAdamMax = 32;
constexpr int kAdamBlock = kThreads * 4;
constexpr int kAdamPerSm = 5;  // resident CTAs (48 registers)
// The grid is one wave of CTAs that stride over the blocks while what a step reads and writes stays in L2
// (ten blocks a CTA: 7.6 M values, 121 MB); beyond that CTAs of four blocks, whose later ones fill the last
// wave's gaps.  One parameter, us, a wave / fours: 5 M values 19 / 21, 7 M 34 / 38, 8 M 43 / 41, 20 M 103 / 91.
constexpr unsigned kAdamWaveBlocks = 10, kAdamCtaBlocks = 4;

struct AdamParams {
    float* p[kAdamMax];
    const float* g[kAdamMax];
    float* m[kAdamMax];
    float* v[kAdamMax];
    int* step[kAdamMax];
    int64_t n[kAdamMax];
    unsigned first[kAdamMax + 1];
    int count;
};

// All parameters of a group in one launch; a CTA strides over the blocks of kAdamBlock elements, one float4 a
// thread.  Bound by memory: 28 bytes an element.  The bias corrections (two double-precision powers) are formed
// by two warps of a CTA, once for each parameter that the CTA comes to, and before the loads, so that no
// value is live across them: formed by every thread they were most of the time of a small parameter, by every
// block (a grid of one block of 2,048 elements a CTA) 27 us for one parameter of 5 M values against 19 here, with the
// loads in flight (spilled at 48 registers) 21.  Unaligned, or a parameter's last block: the same loads four
// bytes wide, all of a thread's in flight (5 M values 39 us in a loop -> 21).
__global__ void __launch_bounds__(kThreads, kAdamPerSm)
    adam_kernel(const __grid_constant__ AdamParams a, double lr, double b1, double b2, float eps) {
    __shared__ float s_scale[2];
    int q = 0, scaled = -1;
    AdamScale s = adam_betas(b1, b2);
    for (unsigned blk = blockIdx.x; blk < a.first[a.count]; blk += gridDim.x) {
        while (blk >= a.first[q + 1]) ++q;  // CTA-uniform
        if (scaled != q) {
            __syncthreads();  // every thread has taken the last parameter's
            if (threadIdx.x == 0 || threadIdx.x == 32) {
                const int k = threadIdx.x >> 5;
                s_scale[k] = adam_correction(a.step[q], lr, k ? b2 : b1, k);
            }
            __syncthreads();
            s.step_size = s_scale[0];
            s.bc2_sqrt = s_scale[1];
            scaled = q;
        }
        const int64_t base = (int64_t)(blk - a.first[q]) * kAdamBlock, left = a.n[q] - base;
        float* __restrict__ p = a.p[q] + base;
        const float* __restrict__ g = a.g[q] + base;
        float* __restrict__ m = a.m[q] + base;
        float* __restrict__ v = a.v[q] + base;
        const bool full = left >= kAdamBlock && (((uintptr_t)p | (uintptr_t)g | (uintptr_t)m | (uintptr_t)v) & 15) == 0;
        const int count = left < kAdamBlock ? (int)left : kAdamBlock;
        float pp[4], gg[4], mm[4], vv[4];
        if (full) {
            *reinterpret_cast<float4*>(pp) = reinterpret_cast<const float4*>(p)[threadIdx.x];
            *reinterpret_cast<float4*>(gg) = reinterpret_cast<const float4*>(g)[threadIdx.x];
            *reinterpret_cast<float4*>(mm) = reinterpret_cast<const float4*>(m)[threadIdx.x];
            *reinterpret_cast<float4*>(vv) = reinterpret_cast<const float4*>(v)[threadIdx.x];
        } else {  // a parameter's last block, or an unaligned one
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = threadIdx.x + k * kThreads;
                pp[k] = i < count ? p[i] : 0.0f;
                gg[k] = i < count ? g[i] : 0.0f;
                mm[k] = i < count ? m[i] : 0.0f;
                vv[k] = i < count ? v[i] : 0.0f;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) adam_one(pp[k], gg[k], mm[k], vv[k], s, eps);
        if (full) {
            reinterpret_cast<float4*>(p)[threadIdx.x] = *reinterpret_cast<float4*>(pp);
            reinterpret_cast<float4*>(m)[threadIdx.x] = *reinterpret_cast<float4*>(mm);
            reinterpret_cast<float4*>(v)[threadIdx.x] = *reinterpret_cast<float4*>(vv);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = threadIdx.x + k * kThreads;
                if (i < count) {
                    p[i] = pp[k];
                    m[i] = mm[k];
                    v[i] = vv[k];
                }
            }
        }
    }
}

__global__ void advance_steps_kernel(const __grid_constant__ AdamParams a) {
    if (threadIdx.x < (unsigned)a.count) *a.step[threadIdx.x] += 1;
}

// VectorAdam, one row of `dim` components sharing one second moment:
// g1 <- b1 g1 + (1-b1) g, g2 <- b2 g2 + (1-b2) |g|^2,
// p <- p - lr * (g1/bc1) / (sqrt(g2/bc2) + 1e-8)   (optimize.py:51-68).
template <int D>
__global__ void __launch_bounds__(kThreads) vector_adam_kernel(int64_t rows, int dim, float* __restrict__ p,
                                                               const float* __restrict__ g, float* __restrict__ g1,
                                                               float* __restrict__ g2, const int* __restrict__ step,
                                                               double lr_d, double b1_d, double b2_d) {
    __shared__ float s_bc[2];
    if (threadIdx.x == 0) {
        const double t = (double)(*step + 1);
        s_bc[0] = (float)(1.0 - pow(b1_d, t));
        s_bc[1] = (float)(1.0 - pow(b2_d, t));
    }
    __syncthreads();
    const float bc1 = s_bc[0], bc2 = s_bc[1];
    const float lr = (float)lr_d, b1 = (float)b1_d, b2 = (float)b2_d;
    const float c1 = (float)(1.0 - b1_d), c2 = (float)(1.0 - b2_d);
    const int n = D > 0 ? D : dim;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
         r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = r * n;
        float sq = 0.f;
        for (int k = 0; k < n; ++k) {
            const float gk = g[o + k];
            sq = fmaf(gk, gk, sq);
            g1[o + k] = b1 * g1[o + k] + c1 * gk;
        }
        const float m2 = b2 * g2[r] + c2 * sq;
        g2[r] = m2;
        const float denom = sqrtf(m2 / bc2) + 1e-8f;
        for (int k = 0; k < n; ++k) p[o + k] -= lr * (g1[o + k] / bc1) / denom;
    }
}

__global__ void advance_step_kernel(int* step) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *step += 1;
}

static unsigned grid_for(int64_t n) {
    const int64_t b = (n + kThreads - 1) / kThreads;
    const int64_t cap = (int64_t)sm_count() * 8;
    return (unsigned)(b < 1 ? 1 : (b < cap ? b : cap));
}

}  // namespace dsb

using namespace dsb;

extern "C" {

int ds_adam_step_multi(int count, float* const* params_host, const float* const* grads_host,
                       float* const* exp_avgs_host, float* const* exp_avg_sqs_host, const int64_t* n_host,
                       int* const* steps_host, double lr, double beta1, double beta2, double eps, ds_stream_t stream) {
    DS_CHECK_ARG(count >= 0 && (count == 0 || (params_host && grads_host && exp_avgs_host && exp_avg_sqs_host &&
                                               n_host && steps_host)),
                 "adam_step: bad arguments");
    DS_CHECK_ARG(beta1 >= 0.0 && beta1 < 1.0 && beta2 >= 0.0 && beta2 < 1.0, "adam_step: betas outside [0, 1)");
    for (int i = 0; i < count; ++i) {
        DS_CHECK_ARG(n_host[i] >= 0, "adam_step: n < 0");
        DS_CHECK_ARG(steps_host[i] != nullptr &&
                         (n_host[i] == 0 || (params_host[i] && grads_host[i] && exp_avgs_host[i] && exp_avg_sqs_host[i])),
                     "adam_step: null pointer");
    }
    cudaStream_t st = (cudaStream_t)stream;
    int i = 0;
    while (i < count) {
        // as many parameters as one launch takes (kAdamMax, and 2^31 - 1 blocks)
        AdamParams a;
        a.count = 0;
        a.first[0] = 0;
        while (i < count && a.count < kAdamMax) {
            const int64_t blocks = (n_host[i] + kAdamBlock - 1) / kAdamBlock;
            if (a.count > 0 && (int64_t)a.first[a.count] + blocks > 0x7fffffff) break;
            DS_CHECK_ARG(blocks <= 0x7fffffff, "adam_step: too many elements");
            const int k = a.count++;
            a.p[k] = params_host[i];
            a.g[k] = grads_host[i];
            a.m[k] = exp_avgs_host[i];
            a.v[k] = exp_avg_sqs_host[i];
            a.step[k] = steps_host[i];
            a.n[k] = n_host[i];
            a.first[k + 1] = a.first[k] + (unsigned)blocks;
            ++i;
        }
        const unsigned all = a.first[a.count], wave = (unsigned)sm_count() * kAdamPerSm;
        const unsigned grid = all <= wave                    ? all
                              : all / kAdamWaveBlocks < wave ? wave
                                                             : (all + kAdamCtaBlocks - 1) / kAdamCtaBlocks;
        if (all > 0) adam_kernel<<<grid, kThreads, 0, st>>>(a, lr, beta1, beta2, (float)eps);
        advance_steps_kernel<<<1, 32, 0, st>>>(a);
    }
    return check_launch("adam_step");
}

int ds_adam_step(float* param, const float* grad, float* exp_avg, float* exp_avg_sq, int64_t n, double lr,
                 double beta1, double beta2, double eps, int* step, ds_stream_t stream) {
    return ds_adam_step_multi(1, &param, &grad, &exp_avg, &exp_avg_sq, &n, &step, lr, beta1, beta2, eps, stream);
}

int ds_vector_adam_step(float* param, const float* grad, float* g1, float* g2, int64_t rows, int dim, double lr,
                        double beta1, double beta2, int* step, ds_stream_t stream) {
    DS_CHECK_ARG(rows >= 0 && dim > 0, "vector_adam_step: bad shape (%lld rows of %d)", (long long)rows, dim);
    DS_CHECK_ARG(step != nullptr && (rows == 0 || (param && grad && g1 && g2)), "vector_adam_step: null pointer");
    DS_CHECK_ARG(beta1 >= 0.0 && beta1 < 1.0 && beta2 >= 0.0 && beta2 < 1.0,
                 "vector_adam_step: betas outside [0, 1)");
    cudaStream_t st = (cudaStream_t)stream;
    if (rows > 0) {
        if (dim == 3)
            vector_adam_kernel<3><<<grid_for(rows), kThreads, 0, st>>>(rows, dim, param, grad, g1, g2, step, lr, beta1,
                                                                       beta2);
        else
            vector_adam_kernel<0><<<grid_for(rows), kThreads, 0, st>>>(rows, dim, param, grad, g1, g2, step, lr, beta1,
                                                                       beta2);
    }
    advance_step_kernel<<<1, 32, 0, st>>>(step);
    return check_launch("vector_adam_step");
}

}  // extern "C"
