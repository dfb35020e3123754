// value * gelu(gate) over rows [value | gate] of 2 cols elements, in one pass: 16-byte accesses, the exact (erf) GELU in
// fp32, rounded where the two separate ops would round.  HBM-bound: reads 2, writes 1 element per output; as a strided GELU
// and a strided product the middle result went through memory once more in each direction (B=32, S=1024, 1368 columns, bf16:
// 450 MB against 270).
#include "vec16.cuh"

namespace xl {
namespace {

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float as_stored(float x, const float *) { return x; }
__device__ __forceinline__ float as_stored(float x, const __nv_bfloat16 *) { return __bfloat162float(__float2bfloat16_rn(x)); }

template <typename T> __global__ void __launch_bounds__(256) geglu_kernel(const T *__restrict__ x, T *__restrict__ y, unsigned total, unsigned cols_v) {
    constexpr int N = Vec16<T>::N;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned row = i / cols_v, c = i - row * cols_v;
        const T *p = x + ((size_t)row * 2 * cols_v + c) * N;
        float a[N], g[N];
        ld16(p, a);
        ld16(p + (size_t)cols_v * N, g);
#pragma unroll
        for (int e = 0; e < N; ++e) a[e] *= as_stored(gelu(g[e]), p);
        st16(y + (size_t)i * N, a);
    }
}

template <typename T> int geglu_launch(const void *x, void *y, int64_t rows, int cols, cudaStream_t st) {
    const int64_t cols_v = cols / Vec16<T>::N, slab = 0x7fffffffLL / cols_v;   // rows per launch: 32-bit indices in the kernel
    for (int64_t r = 0; r < rows; r += slab) {
        const int64_t total = (rows - r < slab ? rows - r : slab) * cols_v, want = (total + 255) / 256;
        geglu_kernel<T><<<(int)(want < 148 * 16 ? want : 148 * 16), 256, 0, st>>>(
            static_cast<const T *>(x) + r * 2 * cols, static_cast<T *>(y) + r * cols, (unsigned)total, (unsigned)cols_v);
        if (cudaGetLastError() != cudaSuccess) return XLSTM_ERR_CUDA;
    }
    return XLSTM_OK;
}

}  // namespace
}  // namespace xl

extern "C" int xlstm_geglu(const void *x, void *y, int64_t rows, int cols, int dtype, void *stream) {
    if (!x || !y || rows < 0 || cols <= 0) return XLSTM_ERR_INVALID;
    if (dtype != XLSTM_F32 && dtype != XLSTM_BF16) return XLSTM_ERR_UNSUPPORTED;
    if (cols % (dtype == XLSTM_F32 ? 4 : 8) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u))
        return XLSTM_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return dtype == XLSTM_F32 ? xl::geglu_launch<float>(x, y, rows, cols, st)
                              : xl::geglu_launch<__nv_bfloat16>(x, y, rows, cols, st);
}
