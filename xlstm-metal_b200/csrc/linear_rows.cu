// Linear layers for 3 to 16 rows of x (one token of a small serving batch): y[m] = epilogue(W . x[m] + bias), bf16.
// Still a weight-streaming pass (every weight is used 16 times at most, HBM-bound up to ~100 rows), but 16 fp32
// multiply-adds per weight on the CUDA cores would bind before HBM does, so the products are mma.sync.m16n8k16 with the
// WEIGHTS as the 16-row operand and the 16 rows of x as two 8-column operands.
//
// A contraction may take its index in any order as long as both operands agree: a lane's 16-byte load (8 consecutive k of
// one row) is used as the fragments of TWO k-steps, so weights go from global memory straight into the MMA's registers, 64
// bytes of a row per quad of lanes, without passing through shared memory.
//
// A CTA owns 2 x 16 weight rows (16 gate and 16 up rows for the SwiGLU pair) and its 8 warps take the 32-wide k blocks in
// turn; the partial sums meet in shared memory, where the epilogue (bias, residual, SwiGLU with the separate layers'
// roundings) runs.  x comes through L2, half a byte per byte of W.  With XLSTM_LINEAR_WEIGHTS_SETTLED the first U blocks
// of weights are loaded BEFORE the wait on the preceding kernel, which the caller promises not to have written them.
// Measured (weights cold, 5 rows): 12304 x 4096 24 us (floor 15.2 at 6.65 TB/s; 385 CTAs in 1.3 waves), 4096 x 10944 23.6
// (13.5), 21888 x 4096 36 (27).
#include "common.cuh"

namespace xl {
namespace {

constexpr int LR_THREADS = 256, LR_WARPS = LR_THREADS / 32;
constexpr int LR_ROWS = 32;      // weight rows per CTA
constexpr int LR_M = 16;         // rows of x
constexpr int LR_U = 4;          // k blocks in flight per warp: 8 KB of weights

__device__ __forceinline__ uint4 ldg_weights(const __nv_bfloat16 *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// EPI: 0 = bias only, 1 = + residual, 2 = SwiGLU pair (W has 2 N rows: gate rows, then up rows)
template <int EPI>
__global__ void __launch_bounds__(LR_THREADS, 2)
linear_rows_kernel(const __nv_bfloat16 *__restrict__ W, const __nv_bfloat16 *x, const __nv_bfloat16 *__restrict__ bias,
                   const __nv_bfloat16 *residual, __nv_bfloat16 *__restrict__ y, int M, int N, int K, int weights_settled) {
    constexpr int STRIDE = EPI == 2 ? 16 : 32;                 // outputs per CTA
    __shared__ float s_part[LR_WARPS][LR_M][LR_ROWS + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int n0 = blockIdx.x * STRIDE;
    const int blocks = K >> 5;
    // rows beyond the end read the last one again; their sums are not stored
    const __nv_bfloat16 *wp[4], *xp[2];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int base = EPI == 2 ? min(n0 + (r & 1) * 8 + g, N - 1) + (r >> 1) * N : min(n0 + r * 8 + g, N - 1);
        wp[r] = W + (size_t)base * K + c * 8;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) xp[r] = x + (size_t)min(r * 8 + g, M - 1) * K + c * 8;

    // a ring of LR_U k blocks: slot u is refilled as soon as its block has been multiplied
    uint4 wr[LR_U][4], xr[LR_U][2];
    // blocks beyond the end are zeros in both operands (0 times an infinite weight would be a NaN)
    auto load_w = [&](int u, int b) {
#pragma unroll
        for (int r = 0; r < 4; ++r) wr[u][r] = b < blocks ? ldg_weights(wp[r] + (size_t)b * 32) : make_uint4(0, 0, 0, 0);
    };
    auto load_x = [&](int u, int b) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
            xr[u][r] = b < blocks ? *reinterpret_cast<const uint4 *>(xp[r] + (size_t)b * 32) : make_uint4(0, 0, 0, 0);
    };
    auto load_first = [&]() {
#pragma unroll
        for (int u = 0; u < LR_U; ++u) load_w(u, warp + u * LR_WARPS);
    };
    if (weights_settled) load_first();
    grid_dependency_wait();
    allow_dependents();
    if (!weights_settled) load_first();

    float acc[2][2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[t][n][e] = 0.f;
#pragma unroll
    for (int u = 0; u < LR_U; ++u) load_x(u, warp + u * LR_WARPS);
    for (int b0 = warp; b0 < blocks; b0 += LR_U * LR_WARPS) {
#pragma unroll
        for (int u = 0; u < LR_U; ++u) {
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    mma_bf16(acc[t][n], wr[u][2 * t].x, wr[u][2 * t + 1].x, wr[u][2 * t].y, wr[u][2 * t + 1].y, xr[u][n].x, xr[u][n].y);
                    mma_bf16(acc[t][n], wr[u][2 * t].z, wr[u][2 * t + 1].z, wr[u][2 * t].w, wr[u][2 * t + 1].w, xr[u][n].z, xr[u][n].w);
                }
            const int b = b0 + (u + LR_U) * LR_WARPS;
            if (b0 + LR_U * LR_WARPS < blocks) { load_w(u, b); load_x(u, b); }
        }
    }
    // element e of a tile: weight row g + 8 (e / 2), x row 2c + (e & 1)
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s_part[warp][n * 8 + 2 * c + (e & 1)][t * 16 + g + 8 * (e >> 1)] = acc[t][n][e];
    __syncthreads();
    auto total = [&](int m, int r) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < LR_WARPS; ++w) s += s_part[w][m][r];
        return s;
    };
    if (EPI == 2) {
        const int m = tid >> 4, r = tid & 15, n = n0 + r;
        if (m < M && n < N) {
            // the two projections are rounded to bf16 before the gate, as separate GEMM outputs would be
            const float gt = __bfloat162float(__float2bfloat16_rn(total(m, r) + (bias ? __bfloat162float(bias[n]) : 0.f)));
            const float up = __bfloat162float(__float2bfloat16_rn(total(m, 16 + r) + (bias ? __bfloat162float(bias[n + N]) : 0.f)));
            y[(size_t)m * N + n] = __float2bfloat16_rn(gt / (1.0f + expf(-gt)) * up);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int m = warp + i * LR_WARPS, n = n0 + lane;
            if (m < M && n < N) {
                float v = total(m, lane) + (bias ? __bfloat162float(bias[n]) : 0.f);
                if (EPI == 1) v = __bfloat162float(__float2bfloat16_rn(v)) + __bfloat162float(residual[(size_t)m * N + n]);
                y[(size_t)m * N + n] = __float2bfloat16_rn(v);
            }
        }
    }
}

template <int EPI>
int linear_rows_launch(const void *W, const void *x, const void *bias, const void *residual, void *y, int M, int N, int K,
                       int settled, cudaStream_t st) {
    const int per = EPI == 2 ? 16 : 32;
    return launch_overlapped(linear_rows_kernel<EPI>, dim3((N + per - 1) / per), dim3(LR_THREADS), 0, st,
                             static_cast<const __nv_bfloat16 *>(W), static_cast<const __nv_bfloat16 *>(x),
                             static_cast<const __nv_bfloat16 *>(bias), static_cast<const __nv_bfloat16 *>(residual),
                             static_cast<__nv_bfloat16 *>(y), M, N, K, settled);
}

}  // namespace
}  // namespace xl

extern "C" int xlstm_linear_rows_ex(const void *W, const void *x, const void *bias, const void *residual, void *y, int M, int N,
                                    int K, int epilogue, int flags, int dtype, void *stream) {
    if (M <= 0 || N <= 0 || K <= 0 || !W || !x || !y) return XLSTM_ERR_INVALID;
    if (epilogue < 0 || epilogue > 2 || (epilogue == 1 && !residual)) return XLSTM_ERR_INVALID;
    if (flags & ~XLSTM_LINEAR_WEIGHTS_SETTLED) return XLSTM_ERR_INVALID;
    if (dtype != XLSTM_BF16 || M > xl::LR_M || K % 32) return XLSTM_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(x)) & 15u) return XLSTM_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int settled = flags & XLSTM_LINEAR_WEIGHTS_SETTLED ? 1 : 0;
    if (epilogue == 2) return xl::linear_rows_launch<2>(W, x, bias, residual, y, M, N, K, settled, st);
    if (epilogue == 1) return xl::linear_rows_launch<1>(W, x, bias, residual, y, M, N, K, settled, st);
    return xl::linear_rows_launch<0>(W, x, bias, residual, y, M, N, K, settled, st);
}

extern "C" int xlstm_linear_rows(const void *W, const void *x, const void *bias, const void *residual, void *y, int M, int N,
                                 int K, int epilogue, int dtype, void *stream) {
    return xlstm_linear_rows_ex(W, x, bias, residual, y, M, N, K, epilogue, 0, dtype, stream);
}
