// LayerNorm of each of `groups` column blocks of a row (groups = 1: over the whole row; groups = heads: the GroupNorm of the
// sLSTM output, whose groups are the heads), affine, in one pass: the block is held in registers as packed 16-byte vectors,
// mean first, then the sum of squared distances from it, fp32 throughout, one rounding on the way out.
//
// HBM-bound (2 elements of traffic per element).  W = 1: a warp per block, no barrier, all loads of a block in flight at
// once.  W = 8: a CTA per block, for the few wide rows of a decode step, where a warp alone would walk 16 vectors a lane.
#include "vec16.cuh"

namespace xl {
namespace {

constexpr int LN_WARPS = 8;

template <int W> __device__ __forceinline__ float block_sum(float v, float *part) {
    v = warp_sum(v);
    if (W == 1) return v;
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < W; ++i) tot += part[i];
    return tot;
}

template <typename T, int NV, int W>
__global__ void __launch_bounds__(LN_WARPS * 32) layer_norm_kernel(const T *__restrict__ x, const T *__restrict__ w,
                                                                   const T *__restrict__ b, T *__restrict__ y, int64_t blocks,
                                                                   int groups, int cols, float eps) {
    constexpr int VN = Vec16<T>::N;
    constexpr int LANES = 32 * W;                     // threads of one block of columns
    __shared__ float s_part[2][W];
    const int lane = threadIdx.x % LANES, nvec = cols / VN;
    const float inv_n = 1.0f / (float)cols;
    for (int64_t blk = (int64_t)blockIdx.x * (LN_WARPS / W) + threadIdx.x / LANES; blk < blocks;
         blk += (int64_t)gridDim.x * (LN_WARPS / W)) {      // W = 8: one block of columns a CTA, so the barriers are uniform
        const uint4 *xr = reinterpret_cast<const uint4 *>(x + (size_t)blk * cols);
        uint4 raw[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + LANES * i < nvec) raw[i] = xr[lane + LANES * i];
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + LANES * i < nvec) {
                float a[VN];
                unpack16<T>(raw[i], a);
#pragma unroll
                for (int e = 0; e < VN; ++e) s += a[e];
            }
        const float mean = block_sum<W>(s, s_part[0]) * inv_n;
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + LANES * i < nvec) {
                float a[VN];
                unpack16<T>(raw[i], a);
#pragma unroll
                for (int e = 0; e < VN; ++e) ss = fmaf(a[e] - mean, a[e] - mean, ss);
            }
        const float inv = rsqrtf(block_sum<W>(ss, s_part[1]) * inv_n + eps);
        const size_t c0 = (size_t)(blk % groups) * cols;
        uint4 *yr = reinterpret_cast<uint4 *>(y + (size_t)blk * cols);
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (lane + LANES * i < nvec) {
                const size_t c = c0 + (size_t)(lane + LANES * i) * VN;
                float a[VN], wv[VN], bv[VN];
                unpack16<T>(raw[i], a);
                ld16<T>(w + c, wv);
                ld16<T>(b + c, bv);
#pragma unroll
                for (int e = 0; e < VN; ++e) a[e] = fmaf((a[e] - mean) * inv, wv[e], bv[e]);
                uint4 o;
                st16<T>(reinterpret_cast<T *>(&o), a);
                yr[lane + LANES * i] = o;
            }
    }
}

template <typename T, int NV, int W>
int ln_run(const void *x, const void *w, const void *b, void *y, int64_t blocks, int groups, int cols, float eps, cudaStream_t st) {
    const int64_t want = (blocks + LN_WARPS / W - 1) / (LN_WARPS / W);
    layer_norm_kernel<T, NV, W><<<(unsigned)(want < 148 * 8 ? want : 148 * 8), LN_WARPS * 32, 0, st>>>(
        static_cast<const T *>(x), static_cast<const T *>(w), static_cast<const T *>(b), static_cast<T *>(y), blocks, groups, cols, eps);
    return launch_status();
}

template <typename T>
int ln_launch(const void *x, const void *w, const void *b, void *y, int64_t blocks, int groups, int cols, float eps, cudaStream_t st) {
    const int nvec = cols / Vec16<T>::N;
    // a warp holds up to 16 vectors a lane; blocks that are wide AND too few to give every SM a CTA of such warps go to whole CTAs
    if (nvec <= 32 * 2) return ln_run<T, 2, 1>(x, w, b, y, blocks, groups, cols, eps, st);
    if (nvec <= 32 * 4) return ln_run<T, 4, 1>(x, w, b, y, blocks, groups, cols, eps, st);
    if (nvec <= 32 * 16 && blocks >= LN_WARPS * 148) {
        if (nvec <= 32 * 8) return ln_run<T, 8, 1>(x, w, b, y, blocks, groups, cols, eps, st);
        return ln_run<T, 16, 1>(x, w, b, y, blocks, groups, cols, eps, st);
    }
    if (nvec <= 256 * 2) return ln_run<T, 2, LN_WARPS>(x, w, b, y, blocks, groups, cols, eps, st);
    if (nvec <= 256 * 8) return ln_run<T, 8, LN_WARPS>(x, w, b, y, blocks, groups, cols, eps, st);
    return XLSTM_ERR_UNSUPPORTED;
}

}  // namespace
}  // namespace xl

extern "C" int xlstm_layer_norm(const void *x, const void *w, const void *b, void *y, int64_t rows, int groups, int cols,
                                float eps, int dtype, void *stream) {
    if (!x || !w || !b || !y || rows < 0 || groups <= 0 || cols <= 0) return XLSTM_ERR_INVALID;
    if (dtype != XLSTM_F32 && dtype != XLSTM_BF16) return XLSTM_ERR_UNSUPPORTED;
    if (cols % (dtype == XLSTM_F32 ? 4 : 8) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) |
                                                 reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(y)) & 15u))
        return XLSTM_ERR_UNSUPPORTED;
    if (cols > (dtype == XLSTM_F32 ? 8192 : 16384)) return XLSTM_ERR_UNSUPPORTED;
    if (rows == 0) return XLSTM_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return dtype == XLSTM_F32 ? xl::ln_launch<float>(x, w, b, y, rows * groups, groups, cols, eps, st)
                              : xl::ln_launch<__nv_bfloat16>(x, w, b, y, rows * groups, groups, cols, eps, st);
}
