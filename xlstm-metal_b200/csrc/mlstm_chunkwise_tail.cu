// Up to 128 bf16 tokens with a carried fp32 state in one launch, to fp32 accuracy: the tokens after the last whole 128-token
// tile of the tensor-core kernels, and sequences that are shorter than one tile.
//
// The operands that are bf16 (Q, K, V) are exact; the fp32 ones (C, the gate matrix P, the weighted V) are cut into three
// bf16 parts whose sum is the float, so mma.sync forms exact products and adds them in fp32:
//   S = Q K^T                                         1 product
//   H^T = (C^T Q^T) diag(w_in) + V^T P^T              3 products each (parts of C, of P)
//   C^T = decay C^T + (w V)^T K                       4 products (parts of w V; K in two for the leading one, see below);
//                                                     few tokens: fp32 multiply-adds
// One CTA per (head, 32 columns of dv), for all tokens at once or for 64 in turn, C, n and m staying with it.  Its 8 warps share
// the dqk dimension: a warp keeps its rows of C in registers, as accumulators of the update and, in the same places, as A
// fragments of the read-out; it takes its share of the keys s for S, P and P V.  The read-outs of the 8 warps meet in shared
// memory, 32 tokens at a time.  Everything that does not need the state (loads, S, gate sums) is done before the wait on the
// tensor-core kernel.
//
// Latency-bound while a CTA has an SM to itself: a few microseconds of products behind a chain of loads, two barriers a 32 tokens
// and the state's way through registers.  As fp32 multiply-adds on CUDA cores a tail of 64 tokens took 52 us (8 heads of 256/512)
// in one launch, of 127 tokens 66 us in two; here 15 and 25 us.
//
// The tensor cores cut off what does not fit 24 bits of a sum, they do not round: with plain parts C was 5.5e-8 from float64 where
// gates forget within a few tokens (fp32 multiply-adds 3.0e-8).  So the leading parts of w V and of K are multiples of one power of
// two each, for the whole sum: their products and all partial sums of up to 128 of them fit 22 bits, nothing is cut off, and the
// other three products are 2^-6 of it.  The two sums and the state meet with one rounding.  C of 1 to 127 tokens is 1.5e-8 to 5.7e-8
// from float64 where fp32 multiply-adds are 1.6e-8 to 9.4e-8 (2-norms; never more than 2 % further, which is the spread of the
// samples).  That is 1 to 2.5 us of 7 to 25 more than plain parts.
//
// Up to FEW_TOKENS the update is fp32 multiply-adds on the CUDA cores instead, as exact and without the splits: us at 256/512, that /
// tensor cores, 1 head, 1 / 17 / 24 / 32 tokens 6.8 8.1 / 8.7 9.4 / 9.1 9.4 / 9.7 9.6; 16 heads 8.3 10.4 / 11.3 12.1 / 12.3 12.2 /
// 13.4 12.5; 64 heads 28.5 35.8 / 38.7 42.2 / 42.0 42.6 / 45.8 43.2.
#include "cp_async.cuh"
#include "mlstm_gate_tile.cuh"
#include "mma_sync.cuh"
#include "packed_f32.cuh"

namespace xl {
namespace {

constexpr int TW = 8;               // warps
constexpr int TC_COLS = 32;         // columns of dv per CTA
constexpr int TG = 32;              // tokens per read-out pass
constexpr int FEW_TOKENS = 24;      // up to so many the update of C is fp32 multiply-adds
constexpr int V_LD = 40;            // bf16 elements between rows of V: 80 bytes, eight rows on different banks
constexpr int PART_LD = 36;         // floats between tokens of a partial read-out

// Two floats as three packed pairs of bf16 whose sums are the floats: 8 significant bits each, cut off (a rounded leading
// part could overflow).  An infinity is its leading part alone.
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint32_t ux = __float_as_uint(x), uy = __float_as_uint(y);
        p[i] = __byte_perm(ux, uy, 0x7632);
        x = fabsf(x) < INFINITY ? x - __uint_as_float(ux & 0xffff0000u) : 0.f;
        y = fabsf(y) < INFINITY ? y - __uint_as_float(uy & 0xffff0000u) : 0.f;
    }
}

// The same with the leading part on a grid, the multiples of 2^-7 of the power of two of `largest`, the largest magnitude there
// is: adding and subtracting 1.5 * 2^23 of that rounds to it.  No grid near the end of the range, or beside an infinity.
__device__ __forceinline__ float grid_of(uint32_t largest) {
    const uint32_t e = largest >> 23;
    return e < 235u ? __uint_as_float(((e + 16u) << 23) | 0x400000u) : 0.f;
}
__device__ __forceinline__ void split3_on_grid(float x, float y, float gx, float gy, uint32_t (&p)[3]) {
    const uint32_t hx = __float_as_uint(__fsub_rn(__fadd_rn(x, gx), gx)) & 0xffff0000u;
    const uint32_t hy = __float_as_uint(__fsub_rn(__fadd_rn(y, gy), gy)) & 0xffff0000u;
    p[0] = __byte_perm(hx, hy, 0x7632);
    x = fabsf(x) < INFINITY ? x - __uint_as_float(hx) : 0.f;
    y = fabsf(y) < INFINITY ? y - __uint_as_float(hy) : 0.f;
#pragma unroll
    for (int i = 1; i < 3; ++i) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const uint32_t *>(&v);
        x -= __uint_as_float(p[i] << 16);
        y -= __uint_as_float(p[i] & 0xffff0000u);
    }
}
// K on the multiples of 2^-5 of its largest magnitude's power of two, and the rest: in bf16 itself, 1.5 * 2^7 of that added and
// subtracted (g: bf16 bits, 0: no grid).
__device__ __forceinline__ uint32_t k_grid_of(uint32_t largest) { return largest < (250u << 7) ? ((largest >> 7) + 2u) << 7 | 0x40u : 0u; }
__device__ __forceinline__ void k_on_grid(uint32_t k, __nv_bfloat162 g, uint32_t &lead, uint32_t &rest) {
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162 *>(&k), h = __hsub2(__hadd2(v, g), g), r = __hsub2(v, h);
    lead = *reinterpret_cast<const uint32_t *>(&h);
    rest = *reinterpret_cast<const uint32_t *>(&r);
}
// c d + a + b for |b| far below |a|, with one rounding that counts: the sum of c d and a with what its rounding leaves.  nd: -d
__device__ __forceinline__ float2 scaled_sum(u64 c, u64 d, u64 nd, u64 a, u64 b) {
    const u64 np = fmul2(c, nd), ep = ffma2(c, d, np);
    const u64 s = fsub2(a, np), t = fsub2(s, a), left = fsub2(fsub2(a, fsub2(s, t)), fadd2(np, t));
    const float2 r = unpack2(fadd2(s, fadd2(left, fadd2(ep, b)))), plain = unpack2(s);
    return make_float2(fabsf(plain.x) < INFINITY ? r.x : plain.x, fabsf(plain.y) < INFINITY ? r.y : plain.y);
}

template <int DQK, int TMAX> struct TailSmem {
    static constexpr uint32_t QK_LD = DQK + 8;                                // elements between rows of Q and K
    static constexpr uint32_t Q = 0;
    static constexpr uint32_t K = Q + TMAX * QK_LD * 2;
    static constexpr uint32_t V = K + TMAX * QK_LD * 2;
    static constexpr uint32_t PART = V + TMAX * V_LD * 2;                     // float [TW][TG][PART_LD]
    static constexpr uint32_t WV = PART;                                      // bf16 [3][TMAX][V_LD], few: float [T][TC_COLS]; after the read-outs
    static constexpr uint32_t PART_BYTES = TW * TG * PART_LD * 4;
    static constexpr uint32_t U = PART + PART_BYTES;                          // double [3][TMAX]: u, b, running maximum of u / x
    static constexpr uint32_t F = U + 3 * TMAX * 8;                           // float [4][TMAX]: w_in, e^{-m_t}, w, q.n
    static constexpr uint32_t RS = F + 4 * TMAX * 4;                          // float [TW][TMAX] row sums of P
    static constexpr uint32_t N = RS + TW * TMAX * 4;                         // float [DQK]
    static constexpr uint32_t KMAX = N + DQK * 4;                             // uint32 [TW]: largest |K|, bf16 bits, by warps
    static constexpr uint32_t TOTAL = KMAX + TW * 4;
    static_assert(3 * TMAX * V_LD * 2 <= PART_BYTES, "weighted V fits the buffer it replaces");
};

template <int DQK, int TMAX, bool FEW>
__global__ void __launch_bounds__(TW * 32, TMAX == 64 ? 2 : 1) mlstm_tail_kernel(const ChunkwiseParams p, int inputs_settled) {
    using SM = TailSmem<DQK, TMAX>;
    constexpr int JW = DQK / TW, KSJ = JW / 16, NTJ = JW / 8;                 // rows of C per warp; k-steps; n-tiles
    constexpr int SW = TMAX / TW, NS = SW / 8;                                // keys per warp; n-tiles
    constexpr int TB = TMAX / 16;
    extern __shared__ __align__(16) unsigned char smem[];
    double *sU = reinterpret_cast<double *>(smem + SM::U), *sB = sU + TMAX, *sX = sB + TMAX;
    float *sWin = reinterpret_cast<float *>(smem + SM::F), *sEmt = sWin + TMAX, *sW = sEmt + TMAX, *sQn = sW + TMAX;
    float *sRs = reinterpret_cast<float *>(smem + SM::RS), *sN = reinterpret_cast<float *>(smem + SM::N);
    float *sPart = reinterpret_cast<float *>(smem + SM::PART);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int col0 = blockIdx.x * TC_COLS, bh = blockIdx.y, b = bh / p.NH, hd = bh % p.NH;
    const int s0 = warp * SW, j0 = warp * JW;
    using bf16 = __nv_bfloat16;
    // the state: this warp's rows j of C^T, element e of tile (mt, nj): column 16 mt + g + 8 (e / 2), row 8 nj + 2c + (e & 1)
    float Ct[2][NTJ][4];
    const size_t c_off = ((size_t)bh * DQK + j0 + 2 * c) * p.dv + col0 + g;
    bool has_C = p.C0 != nullptr;
    double m = 0.0;

    if (!inputs_settled) grid_dependency_wait();
    for (int t0 = 0;; t0 += TMAX) {
        const int T = min(p.S - t0, TMAX), nb = (T + 15) >> 4;                // tokens; blocks of 16 (the rest is zeros)
        const bool last = FEW || TMAX == 128 || t0 + TMAX >= p.S;
        // ---- loads
        const bf16 *qb = static_cast<const bf16 *>(p.q) + b * p.sq[0] + hd * p.sq[1] + t0 * p.sq[2];
        const bf16 *kb = static_cast<const bf16 *>(p.k) + b * p.sk[0] + hd * p.sk[1] + t0 * p.sk[2];
        const bf16 *vb = static_cast<const bf16 *>(p.v) + b * p.sv[0] + hd * p.sv[1] + t0 * p.sv[2] + col0;
        for (int e = tid; e < nb * 16 * (DQK / 8); e += TW * 32) {
            const int t = e / (DQK / 8), x = (e % (DQK / 8)) * 8;
            const bool ok = t < T;
            cp_async16(base + SM::Q + (t * SM::QK_LD + x) * 2, qb + (ok ? (int64_t)t * p.sq[2] + x : 0), ok);
            cp_async16(base + SM::K + (t * SM::QK_LD + x) * 2, kb + (ok ? (int64_t)t * p.sk[2] + x : 0), ok);
        }
        for (int e = tid; e < nb * 16 * 4; e += TW * 32) {
            const int t = e >> 2, x = (e & 3) * 8;
            const bool ok = t < T;
            cp_async16(base + SM::V + (t * V_LD + x) * 2, vb + (ok ? (int64_t)t * p.sv[2] + x : 0), ok);
        }
        if (warp == TW - 1) {                                                 // the warp with the fewest rows of P
            double bsum = 0.0, mx = -INFINITY;
#pragma unroll 1
            for (int h = 0; h < TMAX; h += 32) {
                const GateTile gt = gate_tile(gate_load<bf16>(p, b, hd, t0 + h + lane), p.gate_cap, lane, bsum);
                const double x = fmax(mx, gt.mx);
                sU[h + lane] = gt.u;
                sB[h + lane] = gt.b;
                sX[h + lane] = x;
                bsum = __shfl_sync(0xffffffffu, gt.b, 31);
                mx = __shfl_sync(0xffffffffu, x, 31);
            }
        }
        cp_async_wait_all();
        __syncthreads();
        if constexpr (!FEW) {
            uint32_t k2 = 0u;
#pragma unroll 2
            for (int e = tid; e < nb * 16 * (DQK / 8); e += TW * 32) {
                const uint4 k = *reinterpret_cast<const uint4 *>(smem + SM::K + ((e / (DQK / 8)) * SM::QK_LD + (e % (DQK / 8)) * 8) * 2);
                const uint32_t kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
                for (int x = 0; x < 4; ++x) k2 = __vmaxu2(k2, kk[x] & 0x7fff7fffu);
            }
            k2 = __reduce_max_sync(0xffffffffu, max(k2 & 0xffffu, k2 >> 16));
            if (lane == 0) *reinterpret_cast<uint32_t *>(smem + SM::KMAX + warp * 4) = k2;   // read after the barriers below
        }

        // ---- S = Q K^T: rows t of block tb (16), this warp's keys
        float P[TB][NS][4];
#pragma unroll
        for (int tb = 0; tb < TB; ++tb)
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) P[tb][n][e] = 0.f;
        const uint32_t a_row = base + SM::Q + ((lane & 15) * SM::QK_LD + (lane >> 4) * 8) * 2;
        if (s0 < nb * 16) {
#pragma unroll 1
            for (int kk = 0; kk < DQK / 32; ++kk) {                           // two k-steps
                uint32_t kf[NS][4];                                           // keys of n-tile n: registers 0, 1 and 2, 3
#pragma unroll
                for (int n = 0; n < NS; ++n)
                    ldmatrix4(base + SM::K + ((s0 + n * 8 + (lane & 7)) * SM::QK_LD + kk * 32 + (lane >> 3) * 8) * 2, kf[n]);
#pragma unroll
                for (int tb = 0; tb < TB; ++tb)
                    if (tb < nb && tb * 16 + 15 >= s0) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t a[4];
                            ldmatrix4(a_row + (tb * 16 * SM::QK_LD + kk * 32 + h * 16) * 2, a);
#pragma unroll
                            for (int n = 0; n < NS; ++n) mma_m16n8k16(P[tb][n], a, kf[n][2 * h], kf[n][2 * h + 1]);
                        }
                    }
            }
        }

        if (t0 == 0) {   // ---- the state
            if (inputs_settled) grid_dependency_wait();
            allow_dependents();
            if (p.status && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) *p.status = 0;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nj = 0; nj < NTJ; ++nj)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        Ct[mt][nj][e] = has_C ? p.C0[c_off + (size_t)(nj * 8 + (e & 1)) * p.dv + mt * 16 + (e >> 1) * 8] : 0.f;
            if (tid < DQK) sN[tid] = has_C ? p.n0[(size_t)bh * DQK + tid] : 0.f;
            if (has_C) m = (double)p.m0[bh];
        }
        const double x_last = fmax(m, sX[TMAX - 1]);
        const float decay = expf((float)(m - x_last));
        __syncthreads();                                                      // n; everyone has read the last maximum
        if (tid < TMAX) {
            const double x = fmax(m, sX[tid]);
            sX[tid] = x;
            sWin[tid] = expf((float)(m - x)) * p.qscale;
            sEmt[tid] = expf(-(float)(sB[tid] + x));
            sW[tid] = expf((float)(sU[tid] - x_last));                        // 0 beyond the last token
        }
        {   // q . n: TW * 32 / TMAX threads a token
            constexpr int PT = TW * 32 / TMAX;
            const int t = tid / PT;
            float a = 0.f;
            if (t < T) {
                const bf16 *qrow = reinterpret_cast<const bf16 *>(smem + SM::Q) + t * SM::QK_LD;
#pragma unroll 2
                for (int x = (tid % PT) * 8; x < DQK; x += PT * 8) {
                    const uint4 w = *reinterpret_cast<const uint4 *>(qrow + x);
                    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        a = fmaf(__uint_as_float(ww[e] << 16), sN[x + 2 * e], a);
                        a = fmaf(__uint_as_float(ww[e] & 0xffff0000u), sN[x + 2 * e + 1], a);
                    }
                }
            }
#pragma unroll
            for (int o = 1; o < PT; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (tid % PT == 0) sQn[t] = a;
        }
        __syncthreads();
        // ---- P = tril(S) e^{u_s - x_t}, row sums
#pragma unroll
        for (int tb = 0; tb < TB; ++tb)
            if (tb < nb)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int t = tb * 16 + r * 8 + g;
                    const double xt = sX[t];
                    float rs = 0.f;
#pragma unroll
                    for (int n = 0; n < NS; ++n)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int s = s0 + n * 8 + 2 * c + e;
                            float &v = P[tb][n][2 * r + e];
                            v = s <= t ? v * p.qscale * expf((float)(sU[s] - xt)) : 0.f;
                            rs += v;
                        }
                    rs += __shfl_xor_sync(0xffffffffu, rs, 1);
                    rs += __shfl_xor_sync(0xffffffffu, rs, 2);
                    if (c == 0) sRs[warp * TMAX + t] = rs;
                }

        // ---- read-out, TG tokens at a time
        uint32_t Cp[3][2][KSJ][4];                                            // parts of C^T as A fragments (rows: columns of dv)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int ks = 0; ks < KSJ; ++ks)
#pragma unroll
                for (int r = 0; r < 4; ++r) {                                 // register r: rows + 8 (r & 1), k + 8 (r / 2)
                    const float *src = Ct[mt][2 * ks + (r >> 1)] + 2 * (r & 1);
                    uint32_t w[3];
                    split3(src[0], src[1], w);
#pragma unroll
                    for (int x = 0; x < 3; ++x) Cp[x][mt][ks][r] = w[x];
                }
        bf16 *hb = static_cast<bf16 *>(p.h) + b * p.sh[0] + hd * p.sh[1] + t0 * p.sh[2] + col0;
#pragma unroll
        for (int th = 0; th < TMAX / TG; ++th) {
            if (th * TG >= T) break;
            float acc[2][TG / 8][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < TG / 8; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.f;
            if (has_C) {
#pragma unroll
                for (int ks = 0; ks < KSJ; ++ks)
#pragma unroll
                    for (int np = 0; np < TG / 16; ++np) {
                        if (th * 2 + np >= nb) continue;
                        uint32_t q[4];                                        // tokens of n-tiles 2 np (registers 0, 1), 2 np + 1
                        ldmatrix4(base + SM::Q + ((th * TG + np * 16 + (lane & 7) + ((lane >> 4) << 3)) * SM::QK_LD + j0 + ks * 16 +
                                              ((lane >> 3) & 1) * 8) * 2, q);
#pragma unroll
                        for (int x = 2; x >= 0; --x)
#pragma unroll
                            for (int mt = 0; mt < 2; ++mt) {
                                mma_m16n8k16(acc[mt][2 * np], Cp[x][mt][ks], q[0], q[1]);
                                mma_m16n8k16(acc[mt][2 * np + 1], Cp[x][mt][ks], q[2], q[3]);
                            }
                    }
#pragma unroll
                for (int nt = 0; nt < TG / 8; ++nt) {
                    const float2 w = *reinterpret_cast<const float2 *>(sWin + th * TG + nt * 8 + 2 * c);
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        acc[mt][nt][0] *= w.x; acc[mt][nt][1] *= w.y;
                        acc[mt][nt][2] *= w.x; acc[mt][nt][3] *= w.y;
                    }
                }
            }
            if (s0 < nb * 16 && th * TG + TG > s0) {
                uint32_t vf[2][4];                                            // V^T of this warp's keys
                if (NS == 1) {
                    ldmatrix4_trans(base + SM::V + ((s0 + (lane & 7)) * V_LD + (lane >> 3) * 8) * 2, vf[0]);
                } else {
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt)
                        ldmatrix4_trans(base + SM::V + ((s0 + (lane & 7) + ((lane >> 4) << 3)) * V_LD + mt * 16 + ((lane >> 3) & 1) * 8) * 2, vf[mt]);
                }
#pragma unroll
                for (int nt = 0; nt < TG / 8; ++nt) {
                    const int tb = th * 2 + (nt >> 1), r = nt & 1;
                    if (th * TG + nt * 8 + 8 <= s0) continue;                 // all earlier than the keys: P is 0, V may be infinite
                    uint32_t w[NS][3];
#pragma unroll
                    for (int n = 0; n < NS; ++n) split3(P[tb][n][2 * r], P[tb][n][2 * r + 1], w[n]);
#pragma unroll
                    for (int x = 2; x >= 0; --x)
#pragma unroll
                        for (int mt = 0; mt < 2; ++mt) {
                            if (NS == 1) mma_m16n8k8(acc[mt][nt], vf[0][2 * mt], vf[0][2 * mt + 1], w[0][x]);
                            else mma_m16n8k16(acc[mt][nt], vf[mt], w[0][x], w[NS - 1][x]);
                        }
                }
            }
            if (th > 0) __syncthreads();                                      // the previous pass has been read
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < TG / 8; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        sPart[(warp * TG + nt * 8 + 2 * c + (e & 1)) * PART_LD + mt * 16 + g + (e >> 1) * 8] = acc[mt][nt][e];
            __syncthreads();
            const int tl = tid >> 3, x4 = (tid & 7) * 4, t = th * TG + tl;    // a token's 32 columns in 8 threads
            if (t < T) {
                float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
                float rs = 0.f;
#pragma unroll
                for (int w = 0; w < TW; ++w) {
                    const float4 v = *reinterpret_cast<const float4 *>(sPart + (w * TG + tl) * PART_LD + x4);
                    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
                    rs += sRs[w * TMAX + t];
                }
                const float den = sWin[t] * sQn[t] + rs;
                const float inv = 1.0f / (fmaxf(fabsf(den), sEmt[t]) + p.eps);
                st4(hb + (int64_t)t * p.sh[2] + x4, make_float4(s.x * inv, s.y * inv, s.z * inv, s.w * inv));
            }
        }
        __syncthreads();

        // ---- C^T = decay C^T + (w V)^T K
        const u64 decay2 = pack2(decay, decay);
        if constexpr (FEW) {   // token after token on the CUDA cores: a pair is two rows of a column
            float *sWV = reinterpret_cast<float *>(smem + SM::WV);            // [T][TC_COLS]
            for (int e = tid; e < T * TC_COLS; e += TW * 32)
                sWV[e] = sW[e / TC_COLS] * __bfloat162float(*reinterpret_cast<const bf16 *>(smem + SM::V + (e / TC_COLS * V_LD + e % TC_COLS) * 2));
            __syncthreads();
            u64 acc[4][NTJ];                                                  // column 8 x + g, rows 8 nj + 2c and + 1
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int nj = 0; nj < NTJ; ++nj)
                    acc[x][nj] = fmul2(pack2(Ct[x >> 1][nj][2 * (x & 1)], Ct[x >> 1][nj][2 * (x & 1) + 1]), decay2);
            const unsigned char *krow = smem + SM::K + (j0 + 2 * c) * 2;
#pragma unroll 4
            for (int t = 0; t < T; ++t) {
                u64 kk[NTJ];
#pragma unroll
                for (int nj = 0; nj < NTJ; ++nj) {
                    const uint32_t k2 = *reinterpret_cast<const uint32_t *>(krow + t * SM::QK_LD * 2 + nj * 16);
                    kk[nj] = pack2(__uint_as_float(k2 << 16), __uint_as_float(k2 & 0xffff0000u));
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float wv = sWV[t * TC_COLS + x * 8 + g];
#pragma unroll
                    for (int nj = 0; nj < NTJ; ++nj) acc[x][nj] = ffma2(kk[nj], pack2(wv, wv), acc[x][nj]);
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int nj = 0; nj < NTJ; ++nj) {
                    const float2 v = unpack2(acc[x][nj]);
                    float *dst = p.C1 + c_off + (size_t)(nj * 8) * p.dv + x * 8;
                    dst[0] = v.x;
                    dst[p.dv] = v.y;
                }
        } else {
            bf16 *sWV = reinterpret_cast<bf16 *>(smem + SM::WV);
            static_assert(TW * 32 == 16 * (TC_COLS / 2), "a thread has two columns, of the tokens tid / 16 + 16 i");
            const int vx = (tid % (TC_COLS / 2)) * 2, vt = tid / (TC_COLS / 2);
            auto weighted = [&](int t) {
                const uint32_t v = *reinterpret_cast<const uint32_t *>(smem + SM::V + (t * V_LD + vx) * 2);
                const float w = sW[t];
                return make_float2(w * __uint_as_float(v << 16), w * __uint_as_float(v & 0xffff0000u));
            };
            uint32_t ex = 0u, ey = 0u, kmax = 0u;
#pragma unroll 2
            for (int i = 0; i < nb; ++i) {
                const float2 wv = weighted(vt + 16 * i);
                ex = max(ex, __float_as_uint(fabsf(wv.x)));
                ey = max(ey, __float_as_uint(fabsf(wv.y)));
            }
            ex = max(ex, __shfl_xor_sync(0xffffffffu, ex, 16));
            ey = max(ey, __shfl_xor_sync(0xffffffffu, ey, 16));
            uint2 *sMax = reinterpret_cast<uint2 *>(sRs);                         // [TW][TC_COLS / 2], after the last row sums
            if (lane < 16) sMax[warp * (TC_COLS / 2) + lane] = make_uint2(ex, ey);
            __syncthreads();
#pragma unroll
            for (int w = 0; w < TW; ++w) {
                const uint2 o = sMax[w * (TC_COLS / 2) + (lane & 15)];
                ex = max(ex, o.x);
                ey = max(ey, o.y);
                kmax = max(kmax, *reinterpret_cast<const uint32_t *>(smem + SM::KMAX + w * 4));
            }
            // an infinity keeps its products with all of the other factor: no grids then
            const bool finite = __all_sync(0xffffffffu, max(ex, ey) < 0x7f800000u) && kmax < 0x7f80u;
            const float gx = finite ? grid_of(ex) : 0.f, gy = finite ? grid_of(ey) : 0.f;
            const uint32_t kg = finite ? k_grid_of(kmax) * 0x10001u : 0u;
            const __nv_bfloat162 kgrid = *reinterpret_cast<const __nv_bfloat162 *>(&kg);
#pragma unroll 2
            for (int i = 0; i < nb; ++i) {
                const float2 wv = weighted(vt + 16 * i);
                uint32_t pr[3];
                split3_on_grid(wv.x, wv.y, gx, gy, pr);
#pragma unroll
                for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t *>(sWV + (k * TMAX + vt + 16 * i) * V_LD + vx) = pr[k];
            }
            __syncthreads();
            const u64 minus_decay2 = pack2(-decay, -decay);
            // The sum over the tokens has accumulators of its own, that of the leading parts (exact) and that of the rest
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                float sum[2][NTJ][4];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int nj = 0; nj < NTJ; ++nj)
#pragma unroll
                        for (int e = 0; e < 4; ++e) sum[h][nj][e] = 0.f;
#pragma unroll 1
                for (int ks = 0; ks < nb; ++ks) {
                    uint32_t wp[3][4], kf[NTJ / 2][4];
                    const int trow = ks * 16 + (lane & 7);
#pragma unroll
                    for (int x = 0; x < 3; ++x)
                        ldmatrix4_trans(base + SM::WV + ((x * TMAX + trow + ((lane >> 4) << 3)) * V_LD + mt * 16 + ((lane >> 3) & 1) * 8) * 2, wp[x]);
#pragma unroll
                    for (int np = 0; np < NTJ / 2; ++np)
                        ldmatrix4_trans(base + SM::K + ((trow + (((lane >> 3) & 1) << 3)) * SM::QK_LD + j0 + np * 16 + ((lane >> 4) << 3)) * 2, kf[np]);
#pragma unroll
                    for (int np = 0; np < NTJ / 2; ++np)
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            const int nj = 2 * np + half;
                            const uint32_t k0 = kf[np][2 * half], k1 = kf[np][2 * half + 1];
                            uint32_t l0, l1, r0, r1;
                            k_on_grid(k0, kgrid, l0, r0);
                            k_on_grid(k1, kgrid, l1, r1);
                            mma_m16n8k16(sum[1][nj], wp[2], k0, k1);
                            mma_m16n8k16(sum[0][nj], wp[0], l0, l1);
                            mma_m16n8k16(sum[1][nj], wp[1], k0, k1);
                            mma_m16n8k16(sum[1][nj], wp[0], r0, r1);
                        }
                }
#pragma unroll
                for (int nj = 0; nj < NTJ; ++nj)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float *C = Ct[mt][nj] + 2 * h;
                        const float *s0 = sum[0][nj] + 2 * h, *s1 = sum[1][nj] + 2 * h;
                        const float2 v = scaled_sum(pack2(C[0], C[1]), decay2, minus_decay2, pack2(s0[0], s0[1]), pack2(s1[0], s1[1]));
                        C[0] = v.x;
                        C[1] = v.y;
                        if (last) {
                            float *dst = p.C1 + c_off + (size_t)(nj * 8) * p.dv + mt * 16 + h * 8;
                            dst[0] = v.x;
                            dst[p.dv] = v.y;
                        }
                    }
            }
        }
        static_assert(DQK <= TW * 32, "a thread per element of n");
        m = sB[TMAX - 1] + x_last;
        if ((!last || blockIdx.x == 0) && tid < DQK) {
            const bf16 *sK = reinterpret_cast<const bf16 *>(smem + SM::K);
            float a = decay * sN[tid];
            for (int t = 0; t < T; ++t) a = fmaf(sW[t], __bfloat162float(sK[t * SM::QK_LD + tid]), a);
            if (last) p.n1[(size_t)bh * DQK + tid] = a;
            else sN[tid] = a;                                                 // every CTA of the head has its own
        }
        if (last) {
            if (blockIdx.x == 0 && tid == 0) p.m1[bh] = (float)m;
            break;
        }
        has_C = true;
        __syncthreads();                                                      // Q, K, V and the gates have been read
    }
}

template <int DQK, int TMAX, bool FEW = false> int tail_launch(const ChunkwiseParams &p, bool inputs_settled, cudaStream_t st) {
    auto kern = mlstm_tail_kernel<DQK, TMAX, FEW>;
    constexpr int bytes = (int)TailSmem<DQK, TMAX>::TOTAL;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return XLSTM_ERR_CUDA;
    return launch_overlapped(kern, dim3(p.dv / TC_COLS, p.B * p.NH), dim3(TW * 32), bytes, st, p, inputs_settled ? 1 : 0);
}

}  // namespace

bool mlstm_chunkwise_tail_supported(const ChunkwiseParams &p, int dtype) {
    if (dtype != XLSTM_BF16 || p.S > 128 || (p.dqk != 256 && p.dqk != 128) || p.dv % TC_COLS || p.n_peer) return false;
    for (int d = 0; d < 3; ++d)
        if (p.sq[d] % 8 || p.sk[d] % 8 || p.sv[d] % 8 || p.sh[d] % 4) return false;
    if ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15u) return false;
    return !(reinterpret_cast<uintptr_t>(p.h) & 7u) && (int64_t)p.B * p.NH <= 65535;
}

int mlstm_chunkwise_tail(const ChunkwiseParams &p, bool inputs_settled, cudaStream_t st) {
    // 64 tokens at a time fit an SM twice, 128 once: in turn while every CTA has an SM it takes longer, beyond that it is the faster (127
    // tokens, at once and 64 at a time: 8 heads of 256/512 24.8 / 28.5 us, 16 heads 48.0 / 40.0; 64 of 128/256 75.2 / 51.3)
    const bool in_turn = p.S <= 64 || (int64_t)(p.dv / TC_COLS) * p.B * p.NH > 148;
    if (p.S <= FEW_TOKENS) return p.dqk == 256 ? tail_launch<256, 64, true>(p, inputs_settled, st) : tail_launch<128, 64, true>(p, inputs_settled, st);
    if (p.dqk == 256) return in_turn ? tail_launch<256, 64>(p, inputs_settled, st) : tail_launch<256, 128>(p, inputs_settled, st);
    return in_turn ? tail_launch<128, 64>(p, inputs_settled, st) : tail_launch<128, 128>(p, inputs_settled, st);
}

}  // namespace xl
