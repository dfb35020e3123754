// value * gelu(gate) over rows [value | gate] of 2 cols elements, in one pass: 16-byte accesses, the exact (erf) GELU in
// fp32, rounded where the two separate ops would round.  HBM-bound: reads 2, writes 1 element per output; as a strided GELU
// and a strided product the middle result went through memory once more in each direction (B=32, S=1024, 1368 columns, bf16:
// 450 MB against 270).
#include "common.cuh"

namespace xl {
namespace {

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

template <typename T> struct Vec;   // 16 bytes
template <> struct Vec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void ld(const float *p, float (&v)[4]) {
        const float4 f = *reinterpret_cast<const float4 *>(p);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    }
    static __device__ __forceinline__ void st(float *p, const float (&v)[4]) { st4(p, make_float4(v[0], v[1], v[2], v[3])); }
    static __device__ __forceinline__ float round(float x) { return x; }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void ld(const __nv_bfloat16 *p, float (&v)[8]) {
        const uint4 u = *reinterpret_cast<const uint4 *>(p);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
    static __device__ __forceinline__ void st(__nv_bfloat16 *p, const float (&v)[8]) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t *>(&b);
        }
        *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    static __device__ __forceinline__ float round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
};

template <typename T> __global__ void __launch_bounds__(256) geglu_kernel(const T *__restrict__ x, T *__restrict__ y, unsigned total, unsigned cols_v) {
    using V = Vec<T>;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned row = i / cols_v, c = i - row * cols_v;
        const T *p = x + ((size_t)row * 2 * cols_v + c) * V::N;
        float a[V::N], g[V::N];
        V::ld(p, a);
        V::ld(p + (size_t)cols_v * V::N, g);
#pragma unroll
        for (int e = 0; e < V::N; ++e) a[e] *= V::round(gelu(g[e]));
        V::st(y + (size_t)i * V::N, a);
    }
}

template <typename T> int geglu_launch(const void *x, void *y, int64_t rows, int cols, cudaStream_t st) {
    const int64_t total = rows * (cols / Vec<T>::N);
    if (total > 0x7fffffffLL) return XLSTM_ERR_UNSUPPORTED;
    if (!total) return XLSTM_OK;
    const int64_t want = (total + 255) / 256;
    geglu_kernel<T><<<(int)(want < 148 * 16 ? want : 148 * 16), 256, 0, st>>>(static_cast<const T *>(x), static_cast<T *>(y),
                                                                            (unsigned)total, (unsigned)(cols / Vec<T>::N));
    return launch_status();
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
