// Block-diagonal recurrent sLSTM for bf16 weights: the sequential loop over t with the four recurrent matrices resident
// in REGISTERS for the whole sequence, as B operands of mma.sync.m16n8k16.
//
// One cluster of DH / 32 CTAs of 4 warps per (head, 16 batch rows).  A warp owns 8 units: per step it needs
//   pre[b][g][u] = sum_k h_{t-1}[b][k] R_g[u][k]       16 batch rows x (4 gates x 8 units) x DH
// = 4 n-tiles x DH / 16 k-steps of the MMA with A = h_{t-1} (ldmatrix from shared memory, the whole head, all 16 rows)
// and B = its rows of R (2 registers per tile and k-step: 128 registers at DH = 256).  The accumulators of the four
// gates of one (row, unit) cell land in the same thread, so the gating runs on them in place, and the warp sends its
// finished 16 x 8 block of h_t (256 bytes) straight from registers into the h buffer of every CTA of the cluster
// (st.async, completing bytes on the receiver's mbarrier).  A step has ONE wait (all blocks of h_{t-1} have landed) and
// no CTA or cluster barrier.
//
// The step is a latency chain; the tensor-memory form of it (R as the A operand of 32 tcgen05.mma of 128x16x16, cluster
// of 4) took 2.45 us a step at B = 32, 4 heads x 256: 0.85 us to read R from tensor memory, 0.15 us from the last MMA
// through tensor memory and shared memory to the gating threads, two CTA barriers, and 0.45 us until a bulk copy had
// crossed to the peers.  With N = 16 columns the tensor pipe itself is idle in either form.
//
// h is fed back as bf16 at DH = 256 (NS = 1) and unrounded at DH = 64 and 128 (NS = 3: a float is exactly the sum of
// three bf16, and the products with the bf16 R are exact in fp32), with the exact tanh, exponentials and quotients there
// (branch-free rational forms with approximate divisions were slower: 1215 against 1110 us for 512 steps of 32 x 4 x 128).
//
// Buffer reuse without further synchronisation: h_t goes to buffer (t + 1) & 1, which held h_{t-2}.  A block of h_t is
// sent only after all blocks of h_{t-1} have arrived, and a warp sends its block of h_{t-1} after it has read h_{t-2}.
#include "slstm_cluster.cuh"

namespace xl {
namespace {
using namespace rec;

constexpr int RW = 4;             // warps per CTA
constexpr int RROWS = 16;         // batch rows per cluster: M of the MMA
constexpr int RU = 8;             // units per warp: N of the MMA
constexpr int RBLK = RROWS * 16;  // bytes of one block of h: 16 rows x 8 bf16, the unit of exchange
constexpr int GX_STAGES = 4;      // steps of input-side pre-activations in flight (1 KB per warp and step)
constexpr int GX_STEP = 4 * RROWS * 16;

__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// one special-function op (max relative error 2^-11): used where the result is a bounded activation
// (cell input, output gate), not where it feeds an exponent (the soft-capped gates)
__device__ __forceinline__ float tanh_sfu(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&a)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

template <int DH, int NS>
__global__ void __launch_bounds__(RW * 32, 2)
slstm_recurrent_mma_kernel(const __nv_bfloat16 *__restrict__ gx, const __nv_bfloat16 *__restrict__ R,
                           const float *__restrict__ rb, const float *__restrict__ c0, const float *__restrict__ n0,
                           const float *__restrict__ h0, const float *__restrict__ m0, __nv_bfloat16 *__restrict__ hs,
                           float *__restrict__ c1, float *__restrict__ n1, float *__restrict__ h1, float *__restrict__ m1,
                           int B, int S, int NH, float cap, int *timeout) {
    constexpr int CL = DH / (RW * RU);         // CTAs per cluster
    constexpr int KS = DH / 16;                // k-steps
    constexpr uint32_t PART = DH / 8 * RBLK;   // bytes of h (one of its NS parts)
    constexpr uint32_t HBUF = NS * PART;
    __shared__ __align__(128) unsigned char s_h[2 * HBUF];
    __shared__ __align__(16) unsigned char s_gx[RW * GX_STAGES * GX_STEP];
    __shared__ __align__(8) uint64_t hbar[2];  // all blocks of the h in buffer q have landed
    __shared__ int s_abort;
    volatile int *abort_flag = &s_abort;

    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const int hd = blockIdx.y, b0 = blockIdx.z * RROWS, D = NH * DH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int blk = (int)rank * RW + warp;     // this warp's block of 8 units
    const int u0 = hd * DH + blk * RU;         // its first column in [.., D]

    if (tid == 0) {
        s_abort = 0;
        tc::mbar_init(&hbar[0], 1);
        tc::mbar_init(&hbar[1], 1);
        tc::mbar_fence_init();
        tc::mbar_expect_tx(&hbar[0], HBUF);
        tc::mbar_expect_tx(&hbar[1], HBUF);
    }
    // ---- R: n = unit g of the block, k = 16 kk + 2c (+8)
    uint32_t Rr[4][KS][2];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __nv_bfloat16 *row = R + (((size_t)q * NH + hd) * DH + blk * RU + g) * DH + 2 * c;
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            Rr[q][kk][0] = *reinterpret_cast<const uint32_t *>(row + kk * 16);
            Rr[q][kk][1] = *reinterpret_cast<const uint32_t *>(row + kk * 16 + 8);
        }
    }
    // ---- h_{-1} of the whole head into buffer 0 (every CTA loads its own copy)
    for (int e = tid; e < RROWS * DH; e += RW * 32) {
        const int r = e / DH, k = e % DH;
        float hv = (h0 && b0 + r < B) ? h0[(size_t)(b0 + r) * D + hd * DH + k] : 0.f;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const __nv_bfloat16 hi = __float2bfloat16_rn(hv);
            *reinterpret_cast<__nv_bfloat16 *>(s_h + s * PART + (k >> 3) * RBLK + r * 16 + (k & 7) * 2) = hi;
            hv -= __bfloat162float(hi);
        }
    }
    // ---- cells of this thread: e = 0..3 -> batch row g + 8 (e / 2), unit 2c + (e & 1), as the accumulators lie
    float sc[4], sn[4], sm[4], hv[4], bias[4][2];
    auto cell = [&](int e) { return (size_t)(b0 + g + 8 * (e >> 1)) * D + u0 + 2 * c + (e & 1); };
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const bool ok = c0 != nullptr && b0 + g + 8 * (e >> 1) < B;
        // (rows beyond the batch: nonzero, off the slow path of the division)
        sc[e] = ok ? c0[cell(e)] : b0 + g + 8 * (e >> 1) < B ? 0.f : 1.f;
        sn[e] = ok ? n0[cell(e)] : 1.f;
        sm[e] = ok ? m0[cell(e)] : 0.f;
        hv[e] = 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e) bias[q][e] = rb[(size_t)q * D + u0 + 2 * c + e];
    // ---- input-side pre-activations: 4 gates x 16 rows x 16 bytes per warp and step, two copies per lane
    const uint32_t gx_s = smem_u32(s_gx) + warp * (GX_STAGES * GX_STEP);
    const int xr = lane & 15, xq = lane >> 4;   // row, and gates xq and xq + 2
    const bool x_ok = b0 + xr < B;
    const __nv_bfloat16 *gxp = gx + ((size_t)(x_ok ? b0 + xr : 0) * S * 4 + xq) * D + u0;
    auto fetch_gx = [&](int t) {
        if (t < S) {
            const uint32_t dst = gx_s + (t & (GX_STAGES - 1)) * GX_STEP + lane * 16;
            const __nv_bfloat16 *src = gxp + (size_t)t * 4 * D;
            cp_async16(dst, src, x_ok);
            cp_async16(dst + GX_STEP / 2, src + 2 * D, x_ok);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int t = 0; t < GX_STAGES - 1; ++t) fetch_gx(t);
    tc::fence_proxy_async_smem();   // the plain writes to buffer 0 come before the remote ones of h_1
    cluster.sync();   // barriers armed and buffer 0 complete in every CTA before any block of h_0 can land

    const bool capped = cap > 0.f;
    const float inv_cap = capped ? 1.0f / cap : 0.f;
    const uint32_t h_s = smem_u32(s_h), bar_s = smem_u32(hbar);

    for (int t = 0; t < S; ++t) {
        const int p = t & 1;
        fetch_gx(t + GX_STAGES - 1);             // into the slot that step t - 1 has read
        if (t > 0) {
            mbar_wait_cluster(&hbar[p], (uint32_t)((t - 1) >> 1) & 1u, abort_flag);
            if (tid == 0) tc::mbar_expect_tx(&hbar[p], HBUF);   // arm it for step t + 2
        }
        float acc[2][4][4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[x][q][e] = 0.f;
        const uint32_t ha = h_s + p * HBUF + lane * 16;
        if constexpr (NS == 1) {   // two halves of k: eight independent accumulator chains
            uint32_t a[2][2][4];
            ldmatrix4(ha, a[0][0]);
            ldmatrix4(ha + (KS / 2) * 512, a[0][1]);
#pragma unroll
            for (int kk = 0; kk < KS / 2; ++kk) {
                if (kk + 1 < KS / 2) {
                    ldmatrix4(ha + (kk + 1) * 512, a[(kk + 1) & 1][0]);
                    ldmatrix4(ha + (KS / 2 + kk + 1) * 512, a[(kk + 1) & 1][1]);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    mma16816(acc[0][q], a[kk & 1][0], Rr[q][kk][0], Rr[q][kk][1]);
                    mma16816(acc[1][q], a[kk & 1][1], Rr[q][KS / 2 + kk][0], Rr[q][KS / 2 + kk][1]);
                }
            }
        } else {                   // leading part of h, and the two remainders
#pragma unroll
            for (int kk = 0; kk < KS; ++kk) {
                uint32_t a[NS][4];
#pragma unroll
                for (int s = 0; s < NS; ++s) ldmatrix4(ha + s * PART + kk * 512, a[s]);
#pragma unroll
                for (int s = 0; s < NS; ++s)
#pragma unroll
                    for (int q = 0; q < 4; ++q) mma16816(acc[s > 0][q], a[s], Rr[q][kk][0], Rr[q][kk][1]);
            }
        }
        cp_async_wait<GX_STAGES - 1>();
        __syncwarp();
        float pre[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned char *gp = s_gx + warp * (GX_STAGES * GX_STEP) + (t & (GX_STAGES - 1)) * GX_STEP +
                                      ((q & 1) * RROWS + (q >> 1) * 2 * RROWS + g) * 16 + c * 4;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t w = *reinterpret_cast<const uint32_t *>(gp + r * 128);
                pre[q][2 * r] = (acc[0][q][2 * r] + acc[1][q][2 * r]) + bf_lo(w) + bias[q][0];
                pre[q][2 * r + 1] = (acc[0][q][2 * r + 1] + acc[1][q][2 * r + 1]) + bf_hi(w) + bias[q][1];
            }
        }
        __syncwarp();   // every lane has read this slot before a lane refills it in the next step
        // gates i, f, z, o
        if constexpr (NS == 1) {
            // few special-function ops per cell, absolute error ~1e-6, below the bf16 rounding of the h fed back: 2 + 2
            // for the two soft-caps, 1 each for tanh(z) and sigmoid(o) = (1 + tanh(o/2)) / 2, ONE exponential for the
            // pair (e^{i-m'}, e^{f+m-m'}) (one of the two is exactly 1), 1 reciprocal for c / max(n, 1)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float it = pre[0][e], ft = pre[1][e];
                const float itc = cap * (1.0f - 2.0f * rcp_fast(1.0f + __expf(2.0f * it * inv_cap)));
                const float ftc = cap * (1.0f - 2.0f * rcp_fast(1.0f + __expf(2.0f * ft * inv_cap)));
                it = capped ? itc : it;
                ft = capped ? ftc : ft;
                const float zt = tanh_sfu(pre[2][e]), ot = fmaf(0.5f, tanh_sfu(0.5f * pre[3][e]), 0.5f);
                const float a = ft + sm[e];
                const float lo = __expf(-fabsf(a - it));   // the smaller of the two weights; the larger is 1
                const float fe = a >= it ? 1.0f : lo, ie = a >= it ? lo : 1.0f;
                sc[e] = fmaf(fe, sc[e], ie * zt);
                sn[e] = fmaf(fe, sn[e], ie);
                sm[e] = fmaxf(a, it);
                hv[e] = ot * sc[e] * rcp_fast(fmaxf(sn[e], 1.0f));
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float it = pre[0][e], ft = pre[1][e];
                if (capped) { it = cap * tanhf(it / cap); ft = cap * tanhf(ft / cap); }
                const float zt = tanhf(pre[2][e]), ot = sigmoidf(pre[3][e]);
                const float mt = fmaxf(ft + sm[e], it);
                const float ie = expf(it - mt), fe = expf(ft - mt + sm[e]);
                sc[e] = fmaf(fe, sc[e], ie * zt);
                sn[e] = fmaf(fe, sn[e], ie);
                sm[e] = mt;
                hv[e] = ot * (sc[e] / fmaxf(sn[e], 1.0f));
            }
        }
        // the block as 16-byte rows: lane l collects row l & 15 from the four lanes that hold it
        float rem[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) rem[e] = hv[e];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            uint32_t pk[2], w[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const __nv_bfloat162 v = __floats2bfloat162_rn(rem[2 * r], rem[2 * r + 1]);
                pk[r] = *reinterpret_cast<const uint32_t *>(&v);
                rem[2 * r] -= bf_lo(pk[r]);
                rem[2 * r + 1] -= bf_hi(pk[r]);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const uint32_t w0 = __shfl_sync(0xffffffffu, pk[0], (lane & 7) * 4 + x);
                const uint32_t w1 = __shfl_sync(0xffffffffu, pk[1], (lane & 7) * 4 + x);
                w[x] = (lane & 8) ? w1 : w0;
            }
            if (t + 1 < S) {
                const uint32_t dst = h_s + (p ^ 1) * HBUF + s * PART + blk * RBLK + (lane & 15) * 16;
                const uint32_t bar = bar_s + (p ^ 1) * 8;
#pragma unroll
                for (int j = 0; j < CL / 2; ++j) {
                    const uint32_t peer = (uint32_t)((lane >> 4) * (CL / 2) + j);
                    st_async16(mapa_u32(dst, peer), mapa_u32(bar, peer), w);
                }
            }
            if (s == 0 && lane < 16 && x_ok)
                *reinterpret_cast<uint4 *>(hs + ((size_t)(b0 + xr) * S + t) * D + u0) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    const bool failed = *abort_flag != 0;
    if (failed) {
        if (tid == 0) atomicExch(timeout, 1);
        drain_after_abort();
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (b0 + g + 8 * (e >> 1) < B) {
            c1[cell(e)] = sc[e]; n1[cell(e)] = sn[e]; h1[cell(e)] = hv[e];
            m1[cell(e)] = failed ? __int_as_float(0x7fc00000) : sm[e];   // a device-side time-out shows as NaN state
        }
    }
    cluster.sync();   // no CTA leaves while a peer may still write into its shared memory
}

template <int DH, int NS>
int launch_mma(const void *gx, const void *R, const float *rb, const float *c0, const float *n0, const float *h0,
               const float *m0, void *hs, float *c1, float *n1, float *h1, float *m1, int B, int S, int NH, float cap,
               int *timeout, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(DH / (RW * RU), NH, (B + RROWS - 1) / RROWS);
    cfg.blockDim = dim3(RW * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = DH / (RW * RU);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, slstm_recurrent_mma_kernel<DH, NS>, static_cast<const __nv_bfloat16 *>(gx),
                                             static_cast<const __nv_bfloat16 *>(R), rb, c0, n0, h0, m0,
                                             static_cast<__nv_bfloat16 *>(hs), c1, n1, h1, m1, B, S, NH, cap, timeout);
    return e == cudaSuccess ? launch_status() : XLSTM_ERR_CUDA;
}

}  // namespace

bool slstm_recurrent_mma_supported(int dtype, int dh, const void *R, const void *gx, const void *hs) {
    return dtype == XLSTM_BF16 && (dh == 256 || dh == 128 || dh == 64) &&
           ((reinterpret_cast<uintptr_t>(R) | reinterpret_cast<uintptr_t>(gx) | reinterpret_cast<uintptr_t>(hs)) & 15u) == 0;
}

int slstm_recurrent_mma(const void *gx, const void *R, const float *rb, const float *c0, const float *n0, const float *h0,
                        const float *m0, void *hs, float *c1, float *n1, float *h1, float *m1, int B, int S, int NH, int dh,
                        float cap, int *timeout, cudaStream_t st) {
    if (dh == 256) return launch_mma<256, 1>(gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
    if (dh == 128) return launch_mma<128, 3>(gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
    return launch_mma<64, 3>(gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
}

}  // namespace xl
