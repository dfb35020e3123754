// Linear layers for 3 to 16 rows of x (one token of a small serving batch): y[m] = epilogue(W . x[m] + bias), bf16.
// Still a weight-streaming pass (every weight is used 16 times at most, HBM-bound up to ~100 rows), but 16 fp32
// multiply-adds per weight on the CUDA cores would bind before HBM does, so the products are mma.sync.m16n8k16 with the
// WEIGHTS as the 16-row operand and the 16 rows of x as two 8-column operands.
//
// A contraction may take its index in any order as long as both operands agree: a lane's 16-byte load (8 consecutive k of
// one row) is used as the fragments of TWO k-steps, so weights go from global memory straight into the MMA's registers, 64
// bytes of a row per quad of lanes, without passing through shared memory.
//
// A CTA's tile is 2 x 16 weight rows (16 gate and 16 up rows for the SwiGLU pair); its warps take the 32-wide k blocks in turn, and
// their partial sums meet in shared memory for the epilogue (bias, residual, SwiGLU with the separate layers' roundings).  x comes
// through L1 and L2, half a byte per byte of W.  Two forms: a persistent CTA of 16 warps per SM walks the tiles, and a warp's LR_U
// blocks in flight run on into the next one, so the stream of weights does not stop for the epilogue (two buffers, one barrier a
// tile); or a CTA of 8 warps has one tile (which is taken when: linear_rows_form()).
// With XLSTM_LINEAR_WEIGHTS_SETTLED the first weights are loaded BEFORE the wait on the preceding kernel, which the caller
// promises not to have written them; without it they are only asked of L2.  With a norm in front every CTA normalises the rows
// for itself, into shared memory, while its first weights are under way (a launch of its own takes 5.8 us between two of these).
// That is for few rows only: shared memory is taken from the L1, where the weights in flight land.  16 rows of 4096 (132 KB)
// cost 7 us, and a little more of it 25.
// Measured (weights cold, 16 rows; 8 warps and one tile): 12304 x 4096 21.1 us (25.1; floor 15.4), 4096 x 4096 8.0 (10.2; 5.1),
// 21888 x 4096 as a pair 33.3 (38.0; 27.3), 4096 x 10944 16.9 (22.9; 13.7).  LR_U = 2: 4 % more, 12 warps with LR_U = 4 or 8 with 8:
// the same within 2 %.
#include "cp_async.cuh"
#include "mma_sync.cuh"
#include "vec16.cuh"

namespace xl {
namespace {

constexpr int LR_ROWS = 32;      // weight rows per tile
constexpr int LR_M = 16;         // rows of x
constexpr int LR_LD = LR_ROWS + 1;
// the two forms of a CTA: 16 warps that walk tiles, 8 warps with one tile
template <int WARPS> struct Form {
    static constexpr int THREADS = WARPS * 32;
    static constexpr int U = WARPS == 16 ? 3 : 4;            // k blocks in flight per warp: 6 or 8 KB of weights
    static constexpr int BUFFERS = WARPS == 16 ? 2 : 1;      // of partial sums
    static constexpr int PART = WARPS * LR_M * LR_LD;
    static constexpr uint32_t SMEM = BUFFERS * PART * sizeof(float);
};

// bytes between normalised rows of x in shared memory: the eight rows and four 16-byte lanes of a load on different banks
__host__ __device__ __forceinline__ int norm_ld(int K) { return 2 * K + 64; }

__device__ __forceinline__ uint4 ldg_weights(const __nv_bfloat16 *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// EPI: 0 = bias only, 1 = + residual, 2 = SwiGLU pair (W has 2 N rows: gate rows, then up rows)
template <int EPI, bool NORM, int LR_WARPS>
__global__ void __launch_bounds__(LR_WARPS * 32, LR_WARPS == 16 ? 1 : 2)
linear_rows_kernel(const __nv_bfloat16 *__restrict__ W, const __nv_bfloat16 *x, const __nv_bfloat16 *__restrict__ bias,
                   const __nv_bfloat16 *residual, const __nv_bfloat16 *__restrict__ norm_w, float norm_eps,
                   __nv_bfloat16 *__restrict__ y, int M, int N, int K, int weights_settled) {
    constexpr int STRIDE = EPI == 2 ? 16 : 32;                 // outputs per tile
    constexpr int LR_U = Form<LR_WARPS>::U, LR_THREADS = Form<LR_WARPS>::THREADS;
    extern __shared__ __align__(16) float lr_part[];           // [BUFFERS][LR_WARPS][LR_M][LR_LD]; NORM: the rows of x after it
    unsigned char *sx = reinterpret_cast<unsigned char *>(lr_part) + Form<LR_WARPS>::SMEM;
    const int ldx = norm_ld(K);                                // bytes between them
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int blocks = K >> 5, tiles = (N + STRIDE - 1) / STRIDE;
    const int groups = (blocks + LR_WARPS * LR_U - 1) / (LR_WARPS * LR_U);   // of LR_U blocks of this warp, per tile

    // the load stream: weight rows of the tile it is in (rows beyond the end read the last one again; their sums are not
    // stored), and the first block of the group
    const __nv_bfloat16 *wp[4], *xp[2];
    auto rows_of = [&](int tile) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int n0 = tile * STRIDE;
            const int row = EPI == 2 ? min(n0 + (r & 1) * 8 + g, N - 1) + (r >> 1) * N : min(n0 + r * 8 + g, N - 1);
            wp[r] = W + (size_t)row * K + c * 8;
        }
    };
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
        if (NORM) return;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            xr[u][r] = b < blocks ? *reinterpret_cast<const uint4 *>(xp[r] + (size_t)b * 32) : make_uint4(0, 0, 0, 0);
    };
    auto load_first = [&]() {
        rows_of(blockIdx.x);
#pragma unroll
        for (int u = 0; u < LR_U; ++u) load_w(u, warp + u * LR_WARPS);
    };
    if (weights_settled) {
        load_first();
    } else if (c == 0) {   // asked of L2 only: what the preceding kernel writes, it writes there
        rows_of(blockIdx.x);
#pragma unroll
        for (int u = 0; u < LR_U; ++u)
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (warp + u * LR_WARPS < blocks)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(wp[r] + (size_t)(warp + u * LR_WARPS) * 32));
    }
    grid_dependency_wait();
    allow_dependents();
    if (!weights_settled) load_first();
    if (NORM) {   // RMSNorm of the rows, a warp each, summed and rounded as the norm's own launch does; in place
        const int nvec = K >> 3;
        unsigned char *snw = sx + (size_t)M * ldx;
        for (int v = tid; v < nvec; v += LR_THREADS) {
            for (int m = 0; m < M; ++m) cp_async16(sx + (size_t)m * ldx + v * 16, x + (size_t)m * K + v * 8);
            cp_async16(snw + v * 16, norm_w + (size_t)v * 8);
        }
        cp_async_wait_all();
        __syncthreads();
        for (int m = warp; m < M; m += LR_WARPS) {
            uint4 *row = reinterpret_cast<uint4 *>(sx + (size_t)m * ldx);
            float ss[4] = {0.f, 0.f, 0.f, 0.f};
            for (int v = lane; v < nvec; v += 128)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (v + 32 * q < nvec) {
                        float a[8];
                        unpack16<__nv_bfloat16>(row[v + 32 * q], a);
#pragma unroll
                        for (int e = 0; e < 8; ++e) ss[q] += a[e] * a[e];
                    }
            float tot = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) tot += warp_sum(ss[q]);
            const float inv = rsqrtf(tot / (float)K + norm_eps);
            for (int v = lane; v < nvec; v += 32) {
                float a[8], w[8];
                unpack16<__nv_bfloat16>(row[v], a);
                ld16<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16 *>(snw + v * 16), w);
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = a[e] * inv * w[e];
                st16<__nv_bfloat16>(reinterpret_cast<__nv_bfloat16 *>(row + v), a);
            }
        }
        __syncthreads();
    }
    const unsigned char *sxp[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) sxp[r] = sx + min(r * 8 + g, M - 1) * ldx + c * 16;
#pragma unroll
    for (int u = 0; u < LR_U; ++u) load_x(u, warp + u * LR_WARPS);

    int par = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, par ^= Form<LR_WARPS>::BUFFERS - 1) {
        float acc[2][2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[t][n][e] = 0.f;
        for (int gr = 0; gr < groups; ++gr) {
            const bool tile_ends = gr + 1 == groups;
            const int b0 = tile_ends ? warp : warp + (gr + 1) * LR_U * LR_WARPS;   // what the slots are refilled with
            const bool more = !tile_ends || (LR_WARPS == 16 && tile + (int)gridDim.x < tiles);
            if (LR_WARPS == 16 && tile_ends && more) rows_of(tile + gridDim.x);
#pragma unroll
            for (int u = 0; u < LR_U; ++u) {
                if (NORM) {
                    const int b = warp + (gr * LR_U + u) * LR_WARPS;
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        xr[u][r] = b < blocks ? *reinterpret_cast<const uint4 *>(sxp[r] + b * 64) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        mma_m16n8k16(acc[t][n], wr[u][2 * t].x, wr[u][2 * t + 1].x, wr[u][2 * t].y, wr[u][2 * t + 1].y, xr[u][n].x, xr[u][n].y);
                        mma_m16n8k16(acc[t][n], wr[u][2 * t].z, wr[u][2 * t + 1].z, wr[u][2 * t].w, wr[u][2 * t + 1].w, xr[u][n].z, xr[u][n].w);
                    }
                if (more) { load_w(u, b0 + u * LR_WARPS); load_x(u, b0 + u * LR_WARPS); }
            }
        }
        // element e of an MMA tile: weight row g + 8 (e / 2), x row 2c + (e & 1)
        float *part = lr_part + par * Form<LR_WARPS>::PART;
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) part[(warp * LR_M + n * 8 + 2 * c + (e & 1)) * LR_LD + t * 16 + g + 8 * (e >> 1)] = acc[t][n][e];
        __syncthreads();
        auto total = [&](int m, int r) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < LR_WARPS; ++w) s += part[(w * LR_M + m) * LR_LD + r];
            return s;
        };
        const int n0 = tile * STRIDE;
        if (EPI == 2) {
            const int m = tid >> 4, r = tid & 15, n = n0 + r;
            if (m < M && n < N) {   // (16 x 16 threads)
                // the two projections are rounded to bf16 before the gate, as separate GEMM outputs would be
                const float gt = __bfloat162float(__float2bfloat16_rn(total(m, r) + (bias ? __bfloat162float(bias[n]) : 0.f)));
                const float up = __bfloat162float(__float2bfloat16_rn(total(m, 16 + r) + (bias ? __bfloat162float(bias[n + N]) : 0.f)));
                y[(size_t)m * N + n] = __float2bfloat16_rn(gt / (1.0f + expf(-gt)) * up);
            }
        } else {
            const int n = n0 + lane;
            for (int m = warp; m < M; m += LR_WARPS)
                if (n < N) {
                    float v = total(m, lane) + (bias ? __bfloat162float(bias[n]) : 0.f);
                    if (EPI == 1) v = __bfloat162float(__float2bfloat16_rn(v)) + __bfloat162float(residual[(size_t)m * N + n]);
                    y[(size_t)m * N + n] = __float2bfloat16_rn(v);
                }
        }
    }
}

struct Args {
    const void *W, *x, *bias, *residual, *norm_w;
    float norm_eps;
    void *y;
    int M, N, K, settled;
};
template <int EPI, bool NORM, int WARPS> int linear_rows_launch(const Args &a, int tiles, cudaStream_t st) {
    using F = Form<WARPS>;
    using B = const __nv_bfloat16 *;
    const int64_t norm = NORM ? (int64_t)a.M * norm_ld(a.K) + 2 * a.K : 0;   // rows of x, norm weight
    if (norm > XLSTM_LINEAR_NORM_BYTES) return XLSTM_ERR_UNSUPPORTED;
    auto kern = linear_rows_kernel<EPI, NORM, WARPS>;
    if (!allow_smem(kern, F::SMEM + (NORM ? XLSTM_LINEAR_NORM_BYTES : 0))) return XLSTM_ERR_CUDA;
    return launch_overlapped(kern, dim3(WARPS == 16 && tiles > 148 ? 148 : tiles), dim3(F::THREADS), (size_t)(F::SMEM + norm), st,
                             static_cast<B>(a.W), static_cast<B>(a.x), static_cast<B>(a.bias), static_cast<B>(a.residual),
                             static_cast<B>(a.norm_w), a.norm_eps, static_cast<__nv_bfloat16 *>(a.y), a.M, a.N, a.K, a.settled);
}
template <int EPI, bool NORM> int linear_rows_form(const Args &a, cudaStream_t st) {
    const int per = EPI == 2 ? 16 : 32, tiles = (a.N + per - 1) / per;
    // Tiles of short rows are over before a second one pays for the walk, and with one and a bit to two rounds of tiles half the CTAs
    // would be idle in the last one; two small CTAs an SM hold all of them at once.  us, 16 rows of x, one tile a CTA and walking:
    // 1024 x 1024 2.3 / 2.6, 3088 x 1024 as a pair 3.6 / 5.1, 16384 x 1024 8.4 / 10.3; 6160 x 1536 5.7 / 5.5; 8192 x 2048 7.5 / 8.4,
    // 6144 x 4096 12.6 / 13.9; 12288 x 2048 13.8 / 11.6, 4096 x 2048 6.1 / 4.9.
    if (a.K <= 1024 || (a.K >= 2048 && tiles > 148 && tiles <= 2 * 148)) return linear_rows_launch<EPI, NORM, 8>(a, tiles, st);
    return linear_rows_launch<EPI, NORM, 16>(a, tiles, st);
}

}  // namespace
}  // namespace xl

extern "C" int xlstm_linear_rows_norm(const void *W, const void *x, const void *bias, const void *norm_w, float norm_eps,
                                      const void *residual, void *y, int M, int N, int K, int epilogue, int flags, int dtype,
                                      void *stream) {
    if (M <= 0 || N <= 0 || K <= 0 || !W || !x || !y) return XLSTM_ERR_INVALID;
    if (epilogue < 0 || epilogue > 2 || (epilogue == 1 && !residual)) return XLSTM_ERR_INVALID;
    if (flags & ~XLSTM_LINEAR_WEIGHTS_SETTLED) return XLSTM_ERR_INVALID;
    if (dtype != XLSTM_BF16 || M > xl::LR_M || K % 32 || (norm_w && epilogue == 1)) return XLSTM_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(norm_w)) & 15u) return XLSTM_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int settled = flags & XLSTM_LINEAR_WEIGHTS_SETTLED ? 1 : 0;
    const xl::Args a{W, x, bias, residual, norm_w, norm_eps, y, M, N, K, settled};
    if (norm_w) return epilogue == 2 ? xl::linear_rows_form<2, true>(a, st) : xl::linear_rows_form<0, true>(a, st);
    if (epilogue == 2) return xl::linear_rows_form<2, false>(a, st);
    return epilogue == 1 ? xl::linear_rows_form<1, false>(a, st) : xl::linear_rows_form<0, false>(a, st);
}

extern "C" int xlstm_linear_rows_ex(const void *W, const void *x, const void *bias, const void *residual, void *y, int M, int N,
                                    int K, int epilogue, int flags, int dtype, void *stream) {
    return xlstm_linear_rows_norm(W, x, bias, nullptr, 0.f, residual, y, M, N, K, epilogue, flags, dtype, stream);
}

extern "C" int xlstm_linear_rows(const void *W, const void *x, const void *bias, const void *residual, void *y, int M, int N,
                                 int K, int epilogue, int dtype, void *stream) {
    return xlstm_linear_rows_ex(W, x, bias, residual, y, M, N, K, epilogue, 0, dtype, stream);
}
