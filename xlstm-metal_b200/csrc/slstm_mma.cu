// Block-diagonal recurrent sLSTM for bf16 weights: the sequential loop over t with the four recurrent matrices resident
// in REGISTERS for the whole sequence, as A operands of mma.sync.m16n8k16.
//
// One cluster of DH / 32 CTAs of 4 warps per (head, 8 NT batch rows).  A warp owns 8 units: per step it needs
//   pre[b][g][u] = sum_k h_{t-1}[b][k] R_g[u][k]       8 NT batch rows x (4 gates x 8 units) x DH
// = 2 m-tiles (gates i, f and gates z, o of its 8 units) x NT n-tiles (8 batch rows) x DH / 16 k-steps of the MMA with A = its
// rows of R (4 registers per tile and k-step: 128 registers at DH = 256) and B = h_{t-1} (ldmatrix from shared memory, the
// whole head, all rows).  The accumulators of the four gates of one (row, unit) cell land in the same thread, so the gating
// runs on them in place, and the warp sends its finished block of h_t (128 NT bytes, transposed to rows on the way) straight
// from registers into the h buffer of every CTA of the cluster (st.async, completing bytes on the receiver's mbarrier).  A
// step has ONE wait (all blocks of h_{t-1} have landed) and no CTA or cluster barrier; the input side is read before it.
//
// With the batch rows as the 8-wide dimension a cluster can be as small as 8 rows (NT = 1), which halves the MMAs, the cells
// and the bytes of a warp's step against 16 rows.  A step of 4 heads, NT = 1 against 2 against the form with R as the 8-wide
// operand (16 rows a cluster) before it: dh = 256 0.62 / 1.00 / 0.96 us while every CTA has an SM of its own (15 clusters),
// 0.89 / 1.01 / 0.96 at 32 rows (16 clusters: one pair shares its SMs, and the MMAs of two warps on a scheduler add up: 32 of
// them take 0.27 us), 0.94 / 1.31 / 1.63 at 64; dh = 128 1.23 / 2.31 / 2.17; dh = 64 1.10 / 1.92.
//
// The step is a latency chain; the tensor-memory form of it (R as the A operand of 32 tcgen05.mma of 128x16x16, cluster
// of 4) took 2.45 us a step at B = 32, 4 heads x 256: 0.85 us to read R from tensor memory, 0.15 us from the last MMA
// through tensor memory and shared memory to the gating threads, two CTA barriers, and 0.45 us until a bulk copy had
// crossed to the peers.
//
// h is fed back as bf16 at DH = 256 (NS = 1) and unrounded at DH = 64 and 128 (NS = 3: a float is exactly the sum of
// three bf16, and the products with the bf16 R are exact in fp32), with the exact tanh, exponentials and quotients there
// (branch-free rational forms with approximate divisions were slower: 1215 against 1110 us for 512 steps of 32 x 4 x 128).
//
// Buffer reuse without further synchronisation: h_t goes to buffer (t + 1) & 1, which held h_{t-2}.  A block of h_t is
// sent only after all blocks of h_{t-1} have arrived, and a warp sends its block of h_{t-1} after it has read h_{t-2}.
#include "mma_sync.cuh"
#include "slstm_cluster.cuh"

namespace xl {
namespace {
using namespace rec;

constexpr int RW = 4;             // warps per CTA
constexpr int RU = 8;             // units per warp: half an m-tile
constexpr int GX_STAGES = 4;      // steps of input-side pre-activations in flight (512 NT bytes per warp and step)

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
// 8x8 matrix of bf16 in fragment layout (lane (g, c) holds row g, columns 2c and 2c + 1) -> its transpose
__device__ __forceinline__ uint32_t transpose8x8(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

template <int DH, int NS, int NT>
__global__ void __launch_bounds__(RW * 32, 2)
slstm_recurrent_mma_kernel(const __nv_bfloat16 *__restrict__ gx, const __nv_bfloat16 *__restrict__ R,
                           const float *__restrict__ rb, const float *__restrict__ c0, const float *__restrict__ n0,
                           const float *__restrict__ h0, const float *__restrict__ m0, __nv_bfloat16 *__restrict__ hs,
                           float *__restrict__ c1, float *__restrict__ n1, float *__restrict__ h1, float *__restrict__ m1,
                           int B, int S, int NH, float cap, int *timeout) {
    constexpr int CL = DH / (RW * RU);         // CTAs per cluster
    constexpr int KS = DH / 16;                // k-steps
    constexpr int ROWS = 8 * NT;               // batch rows per cluster
    constexpr int CELLS = 2 * NT;              // cells of a thread: unit g, rows 8 nt + 2c and + 1
    constexpr int RBLK = ROWS * 16;            // bytes of one block of h: rows x 8 bf16, the unit of exchange
    constexpr int GX_STEP = 4 * ROWS * 16;
    constexpr int KX = NT == 1 && NS == 1 ? 4 : 2;   // the k-steps go to KX independent accumulator chains
    constexpr uint32_t PART = DH / 8 * RBLK;   // bytes of h (one of its NS parts)
    constexpr uint32_t HBUF = NS * PART;
    __shared__ __align__(128) unsigned char s_h[2 * HBUF];
    __shared__ __align__(16) unsigned char s_gx[RW * GX_STAGES * GX_STEP];
    __shared__ __align__(8) uint64_t hbar[2];  // all blocks of the h in buffer q have landed
    __shared__ int s_abort;
    volatile int *abort_flag = &s_abort;

    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const int hd = blockIdx.y, b0 = blockIdx.z * ROWS, D = NH * DH;
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
    // ---- R: rows g and g + 8 of m-tile mt = unit g of gates 2 mt and 2 mt + 1, k = 16 kk + 2c (+8)
    uint32_t Rr[2][KS][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __nv_bfloat16 *row = R + (((size_t)q * NH + hd) * DH + blk * RU + g) * DH + 2 * c;
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            Rr[q >> 1][kk][q & 1] = *reinterpret_cast<const uint32_t *>(row + kk * 16);
            Rr[q >> 1][kk][2 + (q & 1)] = *reinterpret_cast<const uint32_t *>(row + kk * 16 + 8);
        }
    }
    // ---- h_{-1} of the whole head into buffer 0 (every CTA loads its own copy)
    for (int e = tid; e < ROWS * DH; e += RW * 32) {
        const int r = e / DH, k = e % DH;
        float hv = (h0 && b0 + r < B) ? h0[(size_t)(b0 + r) * D + hd * DH + k] : 0.f;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const __nv_bfloat16 hi = __float2bfloat16_rn(hv);
            *reinterpret_cast<__nv_bfloat16 *>(s_h + s * PART + (k >> 3) * RBLK + r * 16 + (k & 7) * 2) = hi;
            hv -= __bfloat162float(hi);
        }
    }
    // ---- cells of this thread, as the accumulators lie: e -> batch row 8 (e / 2) + 2c + (e & 1), unit g
    float sc[CELLS], sn[CELLS], sm[CELLS], hv[CELLS], bias[4];
    auto row_of = [&](int e) { return b0 + 8 * (e >> 1) + 2 * c + (e & 1); };
    auto cell = [&](int e) { return (size_t)row_of(e) * D + u0 + g; };
#pragma unroll
    for (int e = 0; e < CELLS; ++e) {
        const bool ok = c0 != nullptr && row_of(e) < B;
        // (rows beyond the batch: nonzero, off the slow path of the division)
        sc[e] = ok ? c0[cell(e)] : row_of(e) < B ? 0.f : 1.f;
        sn[e] = ok ? n0[cell(e)] : 1.f;
        sm[e] = ok ? m0[cell(e)] : 0.f;
        hv[e] = 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) bias[q] = rb[(size_t)q * D + u0 + g];
    // ---- input-side pre-activations: 4 gates x ROWS rows x 16 bytes per warp and step, NT copies per lane
    const uint32_t gx_s = smem_u32(s_gx) + warp * (GX_STAGES * GX_STEP);
    const int xr = lane % ROWS, xq = lane / ROWS;   // row, and gates xq (and xq + 2)
    const bool x_ok = b0 + xr < B;
    const __nv_bfloat16 *gxp = gx + ((size_t)(x_ok ? b0 + xr : 0) * S * 4 + xq) * D + u0;
    auto fetch_gx = [&](int t) {
        if (t < S) {
            const uint32_t dst = gx_s + (t & (GX_STAGES - 1)) * GX_STEP + lane * 16;
            const __nv_bfloat16 *src = gxp + (size_t)t * 4 * D;
            cp_async16(dst, src, x_ok);
            if (NT == 2) cp_async16(dst + GX_STEP / 2, src + 2 * D, x_ok);
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
        // input side of the cells, transposed on the way: matrix q = gate q of 8 rows x 8 units
        cp_async_wait<GX_STAGES - 1>();
        __syncwarp();
        float pre[4][CELLS];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            uint32_t w[4];
            ldmatrix4_trans(gx_s + (t & (GX_STAGES - 1)) * GX_STEP + ((lane >> 3) * ROWS + 8 * n + (lane & 7)) * 16, w);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                pre[q][2 * n] = bf_lo(w[q]) + bias[q];
                pre[q][2 * n + 1] = bf_hi(w[q]) + bias[q];
            }
        }
        __syncwarp();   // every lane has read this slot before a lane refills it in the next step
        if (t > 0) {
            mbar_wait_cluster(&hbar[p], (uint32_t)((t - 1) >> 1) & 1u, abort_flag);
            if (tid == 0) tc::mbar_expect_tx(&hbar[p], HBUF);   // arm it for step t + 2
        }
        float acc[NS][KX][2][NT][4];
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int x = 0; x < KX; ++x)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[s][x][m][n][e] = 0.f;
        const uint32_t ha = h_s + p * HBUF + lane * 16;
        // a load brings 512 bytes of a part: two k-steps of 8 rows, or one of 16
#pragma unroll
        for (int ld = 0; ld < KS * NT / 2; ++ld) {
            uint32_t b[NS][4];
#pragma unroll
            for (int s = 0; s < NS; ++s) ldmatrix4(ha + s * PART + ld * 512, b[s]);
#pragma unroll
            for (int s = 0; s < NS; ++s)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int kk = NT == 1 ? 2 * ld + half : ld, n = NT == 1 ? 0 : half;
#pragma unroll
                    for (int m = 0; m < 2; ++m)
                        mma_m16n8k16(acc[s][kk % KX][m][n], Rr[m][kk], b[s][NT == 1 ? 2 * half : half], b[s][NT == 1 ? 2 * half + 1 : half + 2]);
                }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int e = 0; e < CELLS; ++e) {
                float part[NS];   // k in pairs of chains; then the leading part of h, and the two remainders
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    auto a = [&](int x) { return acc[s][x][q >> 1][e >> 1][2 * (q & 1) + (e & 1)]; };
                    part[s] = a(0) + a(1);
                    if (KX == 4) part[s] += a(KX - 2) + a(KX - 1);
                }
                pre[q][e] += NS == 3 ? part[0] + (part[NS - 2] + part[NS - 1]) : part[0];
            }
        // gates i, f, z, o
        if constexpr (NS == 1) {
            // few special-function ops per cell, absolute error ~1e-6, below the bf16 rounding of the h fed back: 2 + 2
            // for the two soft-caps, 1 each for tanh(z) and sigmoid(o) = (1 + tanh(o/2)) / 2, ONE exponential for the
            // pair (e^{i-m'}, e^{f+m-m'}) (one of the two is exactly 1), 1 reciprocal for c / max(n, 1)
#pragma unroll
            for (int e = 0; e < CELLS; ++e) {
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
            for (int e = 0; e < CELLS; ++e) {
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
        // the block as 16-byte rows: after the transpose lane l collects row l % ROWS from the four lanes that hold it
        float rem[CELLS];
#pragma unroll
        for (int e = 0; e < CELLS; ++e) rem[e] = hv[e];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            uint32_t pk[NT], w[4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const __nv_bfloat162 v = __floats2bfloat162_rn(rem[2 * n], rem[2 * n + 1]);
                const uint32_t u = *reinterpret_cast<const uint32_t *>(&v);
                rem[2 * n] -= bf_lo(u);
                rem[2 * n + 1] -= bf_hi(u);
                pk[n] = transpose8x8(u);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                w[x] = __shfl_sync(0xffffffffu, pk[0], (lane & 7) * 4 + x);
                if (NT == 2) {
                    const uint32_t w1 = __shfl_sync(0xffffffffu, pk[NT - 1], (lane & 7) * 4 + x);
                    w[x] = (lane & 8) ? w1 : w[x];
                }
            }
            if (t + 1 < S) {
                const uint32_t dst = h_s + (p ^ 1) * HBUF + s * PART + blk * RBLK + xr * 16;
                const uint32_t bar = bar_s + (p ^ 1) * 8;
#pragma unroll
                for (int j = 0; j < CL; j += 32 / ROWS) {
                    const uint32_t peer = (uint32_t)(j + xq);
                    if (CL >= 32 / ROWS || peer < CL) st_async16(mapa_u32(dst, peer), mapa_u32(bar, peer), w);
                }
            }
            if (s == 0 && lane < ROWS && x_ok)
                *reinterpret_cast<uint4 *>(hs + ((size_t)(b0 + xr) * S + t) * D + u0) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    const bool failed = *abort_flag != 0;
    if (failed) {
        if (tid == 0) atomicExch(timeout, 1);
        drain_after_abort();
    }
#pragma unroll
    for (int e = 0; e < CELLS; ++e) {
        if (row_of(e) < B) {
            c1[cell(e)] = sc[e]; n1[cell(e)] = sn[e]; h1[cell(e)] = hv[e];
            m1[cell(e)] = failed ? __int_as_float(0x7fc00000) : sm[e];   // a device-side time-out shows as NaN state
        }
    }
    cluster.sync();   // no CTA leaves while a peer may still write into its shared memory
}

template <int DH, int NS, int NT>
int launch_mma(const void *gx, const void *R, const float *rb, const float *c0, const float *n0, const float *h0,
               const float *m0, void *hs, float *c1, float *n1, float *h1, float *m1, int B, int S, int NH, float cap,
               int *timeout, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(DH / (RW * RU), NH, (B + 8 * NT - 1) / (8 * NT));
    cfg.blockDim = dim3(RW * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = DH / (RW * RU);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, slstm_recurrent_mma_kernel<DH, NS, NT>, static_cast<const __nv_bfloat16 *>(gx),
                                             static_cast<const __nv_bfloat16 *>(R), rb, c0, n0, h0, m0,
                                             static_cast<__nv_bfloat16 *>(hs), c1, n1, h1, m1, B, S, NH, cap, timeout);
    return e == cudaSuccess ? launch_status() : XLSTM_ERR_CUDA;
}

template <int DH, int NS, typename... Args> int launch_rows(int B, int NH, Args... args) {
    // 8 rows a cluster while all clusters are resident at once (two CTAs an SM: 33 clusters of 8 CTAs, 71 of 4): beyond that a
    // second wave of them costs more than 16 rows a cluster (96 rows of 4 x 256: 1.83 us a step against 1.40)
    if ((int64_t)((B + 7) / 8) * NH * (DH / (RW * RU)) <= 264) return launch_mma<DH, NS, 1>(args...);
    return launch_mma<DH, NS, 2>(args...);
}

}  // namespace

bool slstm_recurrent_mma_supported(int dtype, int dh, const void *R, const void *gx, const void *hs) {
    return dtype == XLSTM_BF16 && (dh == 256 || dh == 128 || dh == 64) &&
           ((reinterpret_cast<uintptr_t>(R) | reinterpret_cast<uintptr_t>(gx) | reinterpret_cast<uintptr_t>(hs)) & 15u) == 0;
}

int slstm_recurrent_mma(const void *gx, const void *R, const float *rb, const float *c0, const float *n0, const float *h0,
                        const float *m0, void *hs, float *c1, float *n1, float *h1, float *m1, int B, int S, int NH, int dh,
                        float cap, int *timeout, cudaStream_t st) {
    if (dh == 256) return launch_rows<256, 1>(B, NH, gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
    if (dh == 128) return launch_rows<128, 3>(B, NH, gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
    return launch_rows<64, 3>(B, NH, gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
}

}  // namespace xl
