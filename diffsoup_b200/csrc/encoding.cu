// diffsoup_b200/csrc/encoding.cu -- per-pixel view-direction encodings
// (kenji-tojo/diffsoup src/cuda/encoding.cu:9-130).
#include "geometry.cuh"

namespace dsb {

// encoding.cu:89-118 (SH2, 9 coefficients) and the raw direction (3).  A warp's
// 32 rows go through shared memory and leave as one run of 16-byte stores: per
// lane a row is K scattered 4-byte stores, 39 us for the SH2 of 4 views of
// 800x800 against 26 us here.  SET: every pixel is written (background pixels
// zero, which also saves the caller's zeroing, 15 us there); else background
// pixels keep what the buffer holds, and a direction's row is stored by its lane (4
// views of 1080x1920, half of them covered: 58.6 us staged, 45.4 so).  grid.y is the view.
template <int K, bool SET>
__global__ void __launch_bounds__(kThreads) encode_view_kernel(int H, int W, const float* __restrict__ rast,
                                                               const float* __restrict__ inv_mvp,
                                                               float* __restrict__ enc) {
    __shared__ __align__(16) float s_rows[kThreads / 32][32 * K];
    const int b = blockIdx.y, lane = threadIdx.x & 31;
    const int64_t hw = (int64_t)H * W, i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, i0 = i - lane;
    if (i0 >= hw) return;
    const int64_t first = (int64_t)b * hw;
    const bool in = i < hw;
    const bool covered = in && (int)__ldg(rast + (first + i) * 4 + 3) - 1 >= 0;
    if (!SET && K == 3) {  // by itself: shared with the code below it needs 37 registers, not 32 (55 us)
        if (!covered) return;
        const int y = hw <= 0x7fffffff ? (int)i / W : (int)(i / W), x = (int)(i - (int64_t)y * W);
        float M[16], d[3];
#pragma unroll
        for (int k = 0; k < 16; ++k) M[k] = __ldg(inv_mvp + (size_t)b * 16 + k);
        view_direction(pix_ndc(x, W), pix_ndc(y, H), M, d);
        float* o = enc + (first + i) * K;
        o[0] = d[0]; o[1] = d[1]; o[2] = d[2];
        return;
    }
    float v[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (covered) {
        const int y = hw <= 0x7fffffff ? (int)i / W : (int)(i / W), x = (int)(i - (int64_t)y * W);
        float M[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) M[k] = __ldg(inv_mvp + (size_t)b * 16 + k);
        float d[3];
        view_direction(pix_ndc(x, W), pix_ndc(y, H), M, d);
        if (K == 9) {
            sh2_basis(d[0], d[1], d[2], v);
        } else {
            v[0] = d[0]; v[1] = d[1]; v[2] = d[2];
        }
    }
    float* o = enc + (first + i0) * K;
    const bool run = hw - i0 >= 32 && ((uintptr_t)o & 15) == 0 &&
                     (SET || __all_sync(0xffffffffu, covered));
    if (!run) {
        if (SET ? in : covered)
#pragma unroll
            for (int k = 0; k < K; ++k) o[lane * K + k] = v[k];
        return;
    }
    float* tile = s_rows[threadIdx.x >> 5];
#pragma unroll
    for (int k = 0; k < K; ++k) tile[lane * K + k] = v[k];
    __syncwarp();
    for (int k = lane; k < 8 * K; k += 32) reinterpret_cast<float4*>(o)[k] = reinterpret_cast<const float4*>(tile)[k];
}

template <int K, bool SET>
static int encode_view(const char* what, int B, int H, int W, const float* rast, const float* inv_mvp, float* enc,
                       cudaStream_t st) {
    DS_CHECK_ARG(B >= 0 && H >= 0 && W >= 0, "%s: bad sizes", what);
    if ((int64_t)B * H * W == 0) return DS_OK;
    DS_CHECK_ARG(((uintptr_t)rast & 15) == 0, "%s: rast not 16-byte aligned", what);
    const int64_t hw = (int64_t)H * W;
    for (int b0 = 0; b0 < B; b0 += 65535) {
        const int nb = B - b0 < 65535 ? B - b0 : 65535;
        encode_view_kernel<K, SET><<<dim3(blocks_for(hw), nb), kThreads, 0, st>>>(
            H, W, rast + (size_t)b0 * hw * 4, inv_mvp + (size_t)b0 * 16, enc + (size_t)b0 * hw * K);
    }
    return check_launch(what);
}

}  // namespace dsb

using namespace dsb;

extern "C" {

int ds_encode_view_dir_sh2(int B, int H, int W, const float* rast, const float* inv_mvp, float* encoding,
                           ds_stream_t stream) {
    return encode_view<9, false>("encode_view_dir_sh2", B, H, W, rast, inv_mvp, encoding, (cudaStream_t)stream);
}

int ds_encode_view_dir(int B, int H, int W, const float* rast, const float* inv_mvp, float* encoding,
                       ds_stream_t stream) {
    return encode_view<3, false>("encode_view_dir", B, H, W, rast, inv_mvp, encoding, (cudaStream_t)stream);
}

int ds_encode_view_dir_sh2_set(int B, int H, int W, const float* rast, const float* inv_mvp, float* encoding,
                               ds_stream_t stream) {
    return encode_view<9, true>("encode_view_dir_sh2", B, H, W, rast, inv_mvp, encoding, (cudaStream_t)stream);
}

int ds_encode_view_dir_set(int B, int H, int W, const float* rast, const float* inv_mvp, float* encoding,
                           ds_stream_t stream) {
    return encode_view<3, true>("encode_view_dir", B, H, W, rast, inv_mvp, encoding, (cudaStream_t)stream);
}

}  // extern "C"
