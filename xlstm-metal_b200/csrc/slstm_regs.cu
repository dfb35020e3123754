// Block-diagonal recurrent sLSTM in fp32: the sequential loop over t with the four recurrent matrices resident in
// REGISTERS for the whole sequence.
//
// One cluster of DH / 32 CTAs per (head, BG batch rows); a CTA owns 32 units = 128 gate columns, a thread two of its
// columns and 64 of the DH k's (128 registers of R).  Per step a thread multiplies them with h_{t-1}[k] of all BG rows,
// which a warp reads as broadcasts, four k's per 16-byte load for 2 x 2 packed multiply-adds; the DH / 64 partial sums of
// a column meet in shared memory, one thread per (row, unit) gates them, and the CTA's 32 values of h_t per row go to
// every CTA of the cluster as remote stores that complete bytes on the receiver's mbarrier.  One CTA barrier per step
// (partial sums) and one wait (h_{t-1} complete); buffers alternate as in slstm_mma.cu.
//
// R in shared memory (slstm.cu, kept for other head sizes) costs a shared-memory load per multiply-add group and has two
// barriers per step, one of them across the cluster; half of its threads have no column at DH = 256.
#include "packed_f32.cuh"
#include "slstm_cluster.cuh"

namespace xl {
namespace {
using namespace rec;

constexpr int GU = 32;                 // units per CTA
constexpr int GCOL = 4 * GU;           // gate columns per CTA
constexpr int GK = 64;                 // k's per thread
constexpr int BG = 4;                  // batch rows per cluster (8 doubled the step and saved no wave of clusters)

__device__ __forceinline__ float sum2(u64 v) {
    const float2 f = unpack2(v);
    return f.x + f.y;
}

template <int DH>
__global__ void __launch_bounds__(DH, 1)
slstm_recurrent_regs_kernel(const float *__restrict__ gx, const float *__restrict__ R, const float *__restrict__ rb,
                            const float *__restrict__ c0, const float *__restrict__ n0, const float *__restrict__ h0,
                            const float *__restrict__ m0, float *__restrict__ hs, float *__restrict__ c1,
                            float *__restrict__ n1, float *__restrict__ h1, float *__restrict__ m1, int B, int S, int NH,
                            float cap, int *timeout) {
    constexpr int CL = DH / GU, PARTS = DH / GK, WARPS = DH / 32;
    constexpr int CPT = BG / WARPS > 0 ? BG / WARPS : 1;     // cells per thread: rows warp, warp + WARPS, ...
    constexpr uint32_t HBYTES = BG * DH * 4;
    __shared__ __align__(16) float s_h[2][BG][DH];
    __shared__ __align__(16) float s_pre[PARTS][BG][GCOL];
    __shared__ __align__(8) uint64_t hbar[2];
    __shared__ int s_abort;
    volatile int *abort_flag = &s_abort;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int hd = blockIdx.y, b0 = blockIdx.z * BG, D = NH * DH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int u0 = rank * GU;

    if (tid == 0) {
        s_abort = 0;
        tc::mbar_init(&hbar[0], 1);
        tc::mbar_init(&hbar[1], 1);
        tc::mbar_fence_init();
        tc::mbar_expect_tx(&hbar[0], HBYTES);
        tc::mbar_expect_tx(&hbar[1], HBYTES);
    }
    // columns col and col + 64 (gates col / 32 and col / 32 + 2, unit col % 32), k's [k0, k0 + 64)
    const int col = tid & 63, k0 = (tid >> 6) * GK;
    ulonglong2 Rr[2][GK / 4];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(
            R + (((size_t)(col / GU + 2 * x) * NH + hd) * DH + u0 + col % GU) * DH + k0);
#pragma unroll
        for (int k4 = 0; k4 < GK / 4; ++k4) Rr[x][k4] = src[k4];
    }
    for (int e = tid; e < BG * DH; e += DH) {
        const int r = e / DH, k = e % DH;
        s_h[0][r][k] = (h0 && b0 + r < B) ? h0[(size_t)(b0 + r) * D + hd * DH + k] : 0.f;
    }
    // cells: unit `lane`, rows warp + i * WARPS (warps beyond the rows gate nothing)
    const bool gating = warp < BG;
    float sc[CPT], sn[CPT], sm[CPT], hv[CPT], gn[CPT][4], bias[4];
    auto row_ok = [&](int i) { return gating && b0 + warp + i * WARPS < B; };
    auto cell = [&](int i) { return (size_t)(b0 + warp + i * WARPS) * D + hd * DH + u0 + lane; };
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
        const bool ok = c0 != nullptr && row_ok(i);
        sc[i] = ok ? c0[cell(i)] : row_ok(i) ? 0.f : 1.f;   // rows beyond the batch: nonzero, off the slow path of the division
        sn[i] = ok ? n0[cell(i)] : 1.f;
        sm[i] = ok ? m0[cell(i)] : 0.f;
        hv[i] = 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) bias[q] = rb[(size_t)q * D + hd * DH + u0 + lane];
    auto load_gx = [&](int t) {
#pragma unroll
        for (int i = 0; i < CPT; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                gn[i][q] = row_ok(i) ? gx[(((size_t)(b0 + warp + i * WARPS) * S + t) * 4 + q) * D + hd * DH + u0 + lane] : 0.f;
    };
    tc::fence_proxy_async_smem();   // the plain writes to buffer 0 come before the remote ones of h_1
    cluster.sync();                 // barriers armed and buffer 0 complete in every CTA before any of h_0 can land
    load_gx(0);

    const bool capped = cap > 0.f;
    const uint32_t h_s = smem_u32(s_h), bar_s = smem_u32(hbar);
    for (int t = 0; t < S; ++t) {
        const int p = t & 1;
        if (t > 0) {
            mbar_wait_cluster(&hbar[p], (uint32_t)((t - 1) >> 1) & 1u, abort_flag);
            if (tid == 0) tc::mbar_expect_tx(&hbar[p], HBYTES);   // arm it for step t + 2
        }
        u64 acc[2][BG];
#pragma unroll
        for (int r = 0; r < BG; ++r) acc[0][r] = acc[1][r] = 0ull;
        const float *hp = &s_h[p][0][k0];
#pragma unroll
        for (int k4 = 0; k4 < GK / 4; ++k4)
#pragma unroll
            for (int r = 0; r < BG; ++r) {
                const ulonglong2 h4 = *reinterpret_cast<const ulonglong2 *>(hp + r * DH + k4 * 4);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    acc[x][r] = ffma2(Rr[x][k4].x, h4.x, acc[x][r]);
                    acc[x][r] = ffma2(Rr[x][k4].y, h4.y, acc[x][r]);
                }
            }
#pragma unroll
        for (int r = 0; r < BG; ++r) {
            s_pre[tid >> 6][r][col] = sum2(acc[0][r]);
            s_pre[tid >> 6][r][col + 64] = sum2(acc[1][r]);
        }
        __syncthreads();
        if (gating) {
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
                const int r = warp + i * WARPS;
                float pre[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float s = s_pre[0][r][q * GU + lane];
#pragma unroll
                    for (int x = 1; x < PARTS; ++x) s += s_pre[x][r][q * GU + lane];
                    pre[q] = gn[i][q] + (s + bias[q]);
                }
                float it = pre[0], ft = pre[1];
                if (capped) { it = cap * tanhf(it / cap); ft = cap * tanhf(ft / cap); }
                const float zt = tanhf(pre[2]), ot = sigmoidf(pre[3]);
                const float mt = fmaxf(ft + sm[i], it);
                const float ie = expf(it - mt), fe = expf(ft - mt + sm[i]);
                sc[i] = fmaf(fe, sc[i], ie * zt);
                sn[i] = fmaf(fe, sn[i], ie);
                sm[i] = mt;
                hv[i] = ot * (sc[i] / fmaxf(sn[i], 1.0f));
                if (t + 1 < S) {
                    // 16 bytes per lane: lane l sends units 4 (l % 8) .. + 3 to the CTAs l / 8, l / 8 + 4
                    uint32_t w[4];
#pragma unroll
                    for (int x = 0; x < 4; ++x) w[x] = __float_as_uint(__shfl_sync(0xffffffffu, hv[i], (lane & 7) * 4 + x));
                    const uint32_t dst = h_s + (uint32_t)((((p ^ 1) * BG + r) * DH + u0 + (lane & 7) * 4) * 4);
#pragma unroll
                    for (int j = 0; j < CL; j += 4) {
                        const uint32_t peer = (uint32_t)(j + (lane >> 3));
                        if (peer < (uint32_t)CL) st_async16(mapa_u32(dst, peer), mapa_u32(bar_s + (p ^ 1) * 8, peer), w);
                    }
                }
                if (row_ok(i)) hs[((size_t)(b0 + r) * S + t) * D + hd * DH + u0 + lane] = hv[i];
            }
            if (t + 1 < S) load_gx(t + 1);
        }
        // the partial sums are overwritten in the next step only after all of h_t has arrived, hence after the gating
        // warps of this CTA (which send a part of it) have read them
    }
    const bool failed = *abort_flag != 0;
    if (failed) {
        if (tid == 0) atomicExch(timeout, 1);
        drain_after_abort();
    }
#pragma unroll
    for (int i = 0; i < CPT; ++i)
        if (row_ok(i)) {
            c1[cell(i)] = sc[i]; n1[cell(i)] = sn[i]; h1[cell(i)] = hv[i];
            m1[cell(i)] = failed ? __int_as_float(0x7fc00000) : sm[i];   // a device-side time-out shows as NaN state
        }
    cluster.sync();   // no CTA leaves while a peer may still write into its shared memory
}

template <int DH>
int launch_regs(const void *gx, const void *R, const float *rb, const float *c0, const float *n0, const float *h0,
                const float *m0, void *hs, float *c1, float *n1, float *h1, float *m1, int B, int S, int NH, float cap,
                int *timeout, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(DH / GU, NH, (B + BG - 1) / BG);
    cfg.blockDim = dim3(DH);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = DH / GU;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, slstm_recurrent_regs_kernel<DH>, static_cast<const float *>(gx),
                                             static_cast<const float *>(R), rb, c0, n0, h0, m0, static_cast<float *>(hs), c1,
                                             n1, h1, m1, B, S, NH, cap, timeout);
    return e == cudaSuccess ? launch_status() : XLSTM_ERR_CUDA;
}

}  // namespace

bool slstm_recurrent_regs_supported(int dtype, int dh, const void *R) {
    return dtype == XLSTM_F32 && (dh == 256 || dh == 128 || dh == 64) && (reinterpret_cast<uintptr_t>(R) & 15u) == 0;
}

int slstm_recurrent_regs(const void *gx, const void *R, const float *rb, const float *c0, const float *n0, const float *h0,
                         const float *m0, void *hs, float *c1, float *n1, float *h1, float *m1, int B, int S, int NH, int dh,
                         float cap, int *timeout, cudaStream_t st) {
    if (dh == 256) return launch_regs<256>(gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
    if (dh == 128) return launch_regs<128>(gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
    return launch_regs<64>(gx, R, rb, c0, n0, h0, m0, hs, c1, n1, h1, m1, B, S, NH, cap, timeout, st);
}

}  // namespace xl
