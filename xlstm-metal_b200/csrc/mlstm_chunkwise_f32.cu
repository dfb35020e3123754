// Chunkwise mLSTM forward with all arithmetic in fp32 (fp32 inputs, and the bf16 shapes the tensor-core kernels do not
// take), as two launches per group of chunks:
//
//   state   one CTA per (head, 64 rows x 64/128 columns of C): keeps its piece of C in registers, walks the sequence in
//           tiles of 32 tokens, C <- decay C + (w K)^T V, and leaves the state at the start of every 64-token chunk in
//           scratch (the only sequential part, and only 64x128x32 multiply-adds long per step);
//   output  one CTA per (head, chunk, 64/128 columns of h): S = Q K^T, gates, H = w_in Q C_start + P V, normaliser.
//           All chunks at once.
//
// The one-kernel form (mlstm_chunkwise_simt.cu, kept for callers without scratch) does all of it per chunk in sequence
// on a grid of (head, 64 columns): 54 us a chunk at 256/512 because four dependent phases, each between barriers, run
// from shared memory with 4x4 register tiles, and S is recomputed for every 64 columns.
// Both kernels are bound by FMA issue.  Register tiles are 8x8 (8x4 for S) of packed fp32 pairs (fma.rn.f32x2: two
// IEEE multiply-adds per instruction); the operand that is broadcast is kept in shared memory as (a, a) pairs so that
// no instruction is spent on packing.  Global loads of the next piece are in registers while the current one is used.
// The chunk states go through L2: a group is as many chunks as fit SLOT_BYTES of scratch.
//
// Exponents are differences u_s - x_t <= 0 with u = i - b, x = max(m, running max of u) and b the summed log forget
// gates of the chunk, kept in double until the difference is taken (b reaches 1e3 in a chunk of closed gates).
#include "cp_async.cuh"
#include "mlstm_chunkwise.cuh"
#include "mlstm_gate_tile.cuh"
#include "packed_f32.cuh"

namespace xl {
namespace {

constexpr int CH = 64;          // tokens per chunk: distance of the stored states
constexpr int TT = 32;          // tokens per tile of the state kernel: one lane of the gate warp each
constexpr int JT = 64;          // rows of C per CTA of the state kernel
constexpr int KP = 16;          // rows of dqk per piece of the output kernel
constexpr int MAIN = 128;       // threads of the products: 8 row groups x 16 column groups
constexpr size_t SLOT_BYTES = (size_t)192 << 20;

struct F32Params {
    ChunkwiseParams p;
    const float *C0, *n0, *m0;       // state at the start of the group (C0 == NULL: zero); m only for the first group
    float *C1, *n1, *m1;             // state at its end
    float *slot_C, *slot_n, *m_all;  // [BH][g][dqk][dv], [BH][g][dqk], [BH][NC + 1]
    int NC, c_begin, c_end, slots;   // chunks of the sequence, of the group, slots per head
    int slot0;                       // the first chunk's state is in slot 0 too (C1 may overwrite C0)
};

template <typename T> __device__ __forceinline__ float4 ld4_or_zero(const T *ptr, bool ok) {
    return ok ? ld4(ptr) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// ---------------------------------------------------------------------------------------------------------------
// Two CTAs per SM: a scheduler's 16 K registers hold three of the ten warps only up to 168 registers a thread (with 182 it
// was one CTA, 1.25 warps per scheduler, 30 % of the FMA issue slots).
template <typename T, int CT>
__global__ void __launch_bounds__(MAIN + 32, 2) mlstm_f32_state_kernel(const F32Params P) {
    constexpr int NG = CT / 64;                       // groups of 4 columns per thread
    constexpr int KV = TT * JT / 4 / MAIN, VV = TT * CT / 4 / MAIN;
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *sK = reinterpret_cast<float2 *>(smem);                     // [2][TT][JT] (w k, w k)
    float *sV = reinterpret_cast<float *>(sK + 2 * TT * JT);           // [2][TT][CT]
    __shared__ float s_w[4][TT], s_decay[4];
    const ChunkwiseParams &p = P.p;
    const int tid = threadIdx.x, lane = tid & 31;
    const int bh = blockIdx.x, b = bh / p.NH, hd = bh % p.NH;
    const int j0 = blockIdx.y * JT, col0 = blockIdx.z * CT;
    const int t_begin = P.c_begin * CH, t_end = min(p.S, P.c_end * CH);
    const int tiles = (t_end - t_begin + TT - 1) / TT;
    grid_dependency_wait();
    allow_dependents();
    if (p.status && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0) *p.status = 0;

    if (tid >= MAIN) {
        // ---- gate warp: weights two tiles ahead, stabiliser chain, normaliser (first column tile only)
        float m = P.c_begin > 0 ? P.m_all[(size_t)bh * (P.NC + 1) + P.c_begin] : (P.m0 ? P.m0[bh] : 0.f);
        const bool own_m = blockIdx.y == 0 && blockIdx.z == 0, own_n = blockIdx.z == 0;
        const int j = j0 + 2 * lane;
        float n0 = 0.f, n1 = 0.f;
        if (own_n && P.C0) {
            if (j < p.dqk) n0 = P.n0[(size_t)bh * p.dqk + j];
            if (j + 1 < p.dqk) n1 = P.n0[(size_t)bh * p.dqk + j + 1];
        }
        GateRaw raw = gate_load<T>(p, b, hd, t_begin + lane);
        auto gates = [&](int k) {
            if (k >= tiles) return;
            if (own_m && lane == 0 && (k & 1) == 0 && P.m_all) P.m_all[(size_t)bh * (P.NC + 1) + P.c_begin + (k >> 1)] = m;
            const GateTile g = gate_tile(raw, p.gate_cap, lane, 0.0);
            raw = gate_load<T>(p, b, hd, t_begin + (k + 1) * TT + lane);
            const double xl = fmax((double)m, __shfl_sync(0xffffffffu, g.mx, 31));
            s_w[k & 3][lane] = expf((float)(g.u - xl));
            if (lane == 0) s_decay[k & 3] = expf((float)((double)m - xl));
            m = (float)(__shfl_sync(0xffffffffu, g.b, 31) + xl);
        };
        gates(0);
        gates(1);
        __syncthreads();                                     // weights of tile 0
        __syncthreads();                                     // tile 0 in shared memory
        for (int k = 0; k < tiles; ++k) {
            if (own_n) {
                const int c = k >> 1;
                if ((k & 1) == 0 && P.slot_n && (c > 0 || P.slot0)) {
                    float *dst = P.slot_n + ((size_t)bh * P.slots + c) * p.dqk;
                    if (j < p.dqk) dst[j] = n0;
                    if (j + 1 < p.dqk) dst[j + 1] = n1;
                }
                const float4 *row = reinterpret_cast<const float4 *>(sK + (k & 1) * TT * JT) + lane;
                float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
                for (int t = 0; t < TT; ++t) {
                    const float4 v = row[t * (JT / 2)];
                    a0 += v.x;
                    a1 += v.z;
                }
                n0 = fmaf(s_decay[k & 3], n0, a0);
                n1 = fmaf(s_decay[k & 3], n1, a1);
            }
            gates(k + 2);
            __syncthreads();
        }
        if (own_n) {
            if (j < p.dqk) P.n1[(size_t)bh * p.dqk + j] = n0;
            if (j + 1 < p.dqk) P.n1[(size_t)bh * p.dqk + j + 1] = n1;
        }
        if (own_m && lane == 0) {
            if (P.m_all) P.m_all[(size_t)bh * (P.NC + 1) + P.c_end] = m;
            if (P.m1) P.m1[bh] = m;
        }
        return;
    }

    // ---- products
    const int ty = tid >> 4, tx = tid & 15;
    const T *kb = static_cast<const T *>(p.k) + b * p.sk[0] + hd * p.sk[1] + j0;
    const T *vb = static_cast<const T *>(p.v) + b * p.sv[0] + hd * p.sv[1] + col0;
    u64 acc[8][2 * NG];
    auto c_piece = [&](const float *base, int r, int g) {    // row r, column group g of this thread in a [dqk][dv] state
        return base + ((size_t)(j0 + ty * 8 + r)) * p.dv + col0 + g * 64 + tx * 4;
    };
    auto c_ok = [&](int r, int g) { return j0 + ty * 8 + r < p.dqk && col0 + g * 64 + tx * 4 < p.dv; };
    const size_t CE = (size_t)p.dqk * p.dv;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const float4 c4 = ld4_or_zero(P.C0 ? c_piece(P.C0 + bh * CE, r, g) : nullptr, P.C0 && c_ok(r, g));
            acc[r][2 * g] = pack2(c4.x, c4.y);
            acc[r][2 * g + 1] = pack2(c4.z, c4.w);
        }
    float4 kr[KV], vr[VV];
    auto load = [&](int k) {
#pragma unroll
        for (int i = 0; i < KV; ++i) {
            const int e = tid + i * MAIN, t = t_begin + k * TT + e / (JT / 4), c = (e % (JT / 4)) * 4;
            kr[i] = ld4_or_zero(kb + (int64_t)t * p.sk[2] + c, t < t_end && j0 + c < p.dqk);
        }
#pragma unroll
        for (int i = 0; i < VV; ++i) {
            const int e = tid + i * MAIN, t = t_begin + k * TT + e / (CT / 4), c = (e % (CT / 4)) * 4;
            vr[i] = ld4_or_zero(vb + (int64_t)t * p.sv[2] + c, t < t_end && col0 + c < p.dv);
        }
    };
    auto store = [&](int k) {
        float4 *dk = reinterpret_cast<float4 *>(sK + (k & 1) * TT * JT);
        float4 *dvv = reinterpret_cast<float4 *>(sV + (k & 1) * TT * CT);
#pragma unroll
        for (int i = 0; i < KV; ++i) {
            const int e = tid + i * MAIN;
            const float w = s_w[k & 3][e / (JT / 4)];
            const float4 x = kr[i];
            dk[2 * e] = make_float4(w * x.x, w * x.x, w * x.y, w * x.y);
            dk[2 * e + 1] = make_float4(w * x.z, w * x.z, w * x.w, w * x.w);
        }
#pragma unroll
        for (int i = 0; i < VV; ++i) dvv[tid + i * MAIN] = vr[i];
    };
    auto put = [&](float *base) {
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int g = 0; g < NG; ++g)
                if (c_ok(r, g)) {
                    const float2 x = unpack2(acc[r][2 * g]), y = unpack2(acc[r][2 * g + 1]);
                    *reinterpret_cast<float4 *>(const_cast<float *>(c_piece(base, r, g))) = make_float4(x.x, x.y, y.x, y.y);
                }
    };
    load(0);
    __syncthreads();
    store(0);
    cp_async_wait_all();
    __syncthreads();
    for (int k = 0; k < tiles; ++k) {
        if (k + 1 < tiles) load(k + 1);
        if ((k & 1) == 0 && P.slot_C && (k > 0 || P.slot0)) put(P.slot_C + ((size_t)bh * P.slots + (k >> 1)) * CE);
        const u64 d2 = pack2(s_decay[k & 3], s_decay[k & 3]);
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int g = 0; g < 2 * NG; ++g) acc[r][g] = fmul2(acc[r][g], d2);
        const float2 *ka = sK + (k & 1) * TT * JT + ty * 8;
        const float *va = sV + (k & 1) * TT * CT + tx * 4;
#pragma unroll 4
        for (int t = 0; t < TT; ++t) {
            u64 a[8], bv[2 * NG];
#pragma unroll
            for (int r = 0; r < 8; r += 2) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(ka + t * JT + r);
                a[r] = q.x;
                a[r + 1] = q.y;
            }
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(va + t * CT + g * 64);
                bv[2 * g] = q.x;
                bv[2 * g + 1] = q.y;
            }
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int g = 0; g < 2 * NG; ++g) acc[r][g] = ffma2(a[r], bv[g], acc[r][g]);
        }
        if (k + 1 < tiles) store(k + 1);   // the other buffer: last read before the previous barrier
        __syncthreads();
    }
    put(P.C1 + bh * CE);
}

// ---------------------------------------------------------------------------------------------------------------
template <int DVT> struct OutSmem {
    static constexpr uint32_t Q = 0;                                   // float2 [2][KP][CH]  (q, q), transposed
    static constexpr uint32_t K = Q + 2 * KP * CH * 8;                 // float  [2][KP][CH]  transposed
    static constexpr uint32_t C = K + 2 * KP * CH * 4;                 // float  [2][KP][DVT]
    static constexpr uint32_t V = C + 2 * KP * DVT * 4;                // float  [CH][DVT]
    static constexpr uint32_t PM = Q;                                  // float2 [CH s][CH t] (P, P), 16-byte units swizzled:
                                                                       // over Q, K and C, which the last piece leaves free
    static constexpr uint32_t U = V + CH * DVT * 4;                    // double [CH] u, [CH] x
    static constexpr uint32_t WIN = U + 2 * CH * 8;                    // float [CH] e^{m - x_t}, [CH] e^{-m_t}, [2][CH] q.n, [CH] row sums
    static constexpr uint32_t NV = WIN + 5 * CH * 4;                   // float [2][KP] n of the piece
    static constexpr uint32_t TOTAL = NV + 2 * KP * 4;
    static_assert(CH * CH * 8 <= V, "P fits the buffers it replaces");
};

// Two CTAs per SM by registers; a third (168 registers, a few spilled) measured the same, so it is latency inside the
// warps and the shared-memory return path (an LDS.128 takes 2.4 to 4 clocks of it, 7 for 48 packed multiply-adds of 2.3)
// that bind, not their number.
template <typename T, int DVT>
__global__ void __launch_bounds__(MAIN, 2) mlstm_f32_output_kernel(const F32Params P) {
    using SM = OutSmem<DVT>;
    constexpr int NG = DVT / 64;
    constexpr int QV = KP * CH / 4 / MAIN, CV = KP * DVT / 4 / MAIN;
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *sQ = reinterpret_cast<float2 *>(smem + SM::Q);
    float *sK = reinterpret_cast<float *>(smem + SM::K), *sC = reinterpret_cast<float *>(smem + SM::C);
    float *sV = reinterpret_cast<float *>(smem + SM::V);
    float2 *sP = reinterpret_cast<float2 *>(smem + SM::PM);
    double *sU = reinterpret_cast<double *>(smem + SM::U), *sX = sU + CH;
    float *sWin = reinterpret_cast<float *>(smem + SM::WIN), *sEmt = sWin + CH, *sQn = sEmt + CH, *sRow = sQn + 2 * CH;
    float *sN = reinterpret_cast<float *>(smem + SM::NV);
    const ChunkwiseParams &p = P.p;
    const int tid = threadIdx.x, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
    const int ci = blockIdx.x, c = P.c_begin + ci, t0 = c * CH, col0 = blockIdx.y * DVT;
    const int bh = blockIdx.z, b = bh / p.NH, hd = bh % p.NH;
    const bool from_slot = ci > 0 || P.slot0, has_C = from_slot || P.C0 != nullptr;
    const size_t CE = (size_t)p.dqk * p.dv;
    const float *Cs = from_slot ? P.slot_C + ((size_t)bh * P.slots + ci) * CE : P.C0 + bh * CE;
    const float *ns = from_slot ? P.slot_n + ((size_t)bh * P.slots + ci) * p.dqk : P.n0 + (size_t)bh * p.dqk;
    const T *qb = static_cast<const T *>(p.q) + b * p.sq[0] + hd * p.sq[1] + (int64_t)t0 * p.sq[2];
    const T *kb = static_cast<const T *>(p.k) + b * p.sk[0] + hd * p.sk[1] + (int64_t)t0 * p.sk[2];
    const T *vb = static_cast<const T *>(p.v) + b * p.sv[0] + hd * p.sv[1] + (int64_t)t0 * p.sv[2] + col0;

    float4 qr[QV], kr[QV];
    float nr = 0.f;
    auto load_qk = [&](int j0) {
#pragma unroll
        for (int i = 0; i < QV; ++i) {                       // lane = token: the transposed stores are conflict-free
            const int e = tid + i * MAIN, t = e % CH, j = j0 + (e / CH) * 4;
            const bool ok = t0 + t < p.S && j < p.dqk;
            qr[i] = ld4_or_zero(qb + (int64_t)t * p.sq[2] + j, ok);
            kr[i] = ld4_or_zero(kb + (int64_t)t * p.sk[2] + j, ok);
        }
    };
    auto load_c = [&](int j0, int buf) {                     // straight into shared memory
        if (has_C) {
            if (tid < KP) nr = j0 + tid < p.dqk ? ns[j0 + tid] : 0.f;
#pragma unroll
            for (int i = 0; i < CV; ++i) {
                const int e = tid + i * MAIN, j = j0 + e / (DVT / 4), cc = (e % (DVT / 4)) * 4;
                const bool ok = j < p.dqk && col0 + cc < p.dv;
                cp_async16((uint32_t)__cvta_generic_to_shared(reinterpret_cast<float4 *>(sC + buf * KP * DVT) + e), Cs + (ok ? (size_t)j * p.dv + col0 + cc : 0), ok);
            }
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < QV; ++i) {
            const int e = tid + i * MAIN, t = e % CH, j = (e / CH) * 4;
            float2 *dq = sQ + (buf * KP + j) * CH + t;
            float *dk = sK + (buf * KP + j) * CH + t;
            dq[0] = make_float2(qr[i].x, qr[i].x); dq[CH] = make_float2(qr[i].y, qr[i].y);
            dq[2 * CH] = make_float2(qr[i].z, qr[i].z); dq[3 * CH] = make_float2(qr[i].w, qr[i].w);
            dk[0] = kr[i].x; dk[CH] = kr[i].y; dk[2 * CH] = kr[i].z; dk[3 * CH] = kr[i].w;
        }
        if (tid < KP) sN[buf * KP + tid] = nr;
    };
    // The kernel before this one (state) has waited for its own predecessor before it let this one start, so the inputs are
    // there; what it writes itself (C, n, m) is read after the wait.  A single chunk starts from the caller's state and
    // needs nothing of it: the two kernels then run side by side, and one CTA waits at the end, so that this launch is
    // complete only when that one is.
    const bool single = P.m_all == nullptr;
    const GateRaw raw[2] = {gate_load<T>(p, b, hd, t0 + lane), gate_load<T>(p, b, hd, t0 + 32 + lane)};
    load_qk(0);
    // V of the chunk: needed after the last piece
#pragma unroll 4
    for (int e = tid; e < CH * DVT / 4; e += MAIN) {
        const int t = e / (DVT / 4), cc = (e % (DVT / 4)) * 4;
        reinterpret_cast<float4 *>(sV)[e] = ld4_or_zero(vb + (int64_t)t * p.sv[2] + cc, t0 + t < p.S && col0 + cc < p.dv);
    }
    if (!single) {
        grid_dependency_wait();
        allow_dependents();
    }
    load_c(0, 0);
    if (tid < 32) {
        const float m = P.m_all ? P.m_all[(size_t)bh * (P.NC + 1) + c] : (P.m0 ? P.m0[bh] : 0.f);
        double bsum = 0.0, mx = (double)m;
#pragma unroll 1
        for (int h = 0; h < CH; h += 32) {
            const GateTile g = gate_tile(h == 0 ? raw[0] : raw[1], p.gate_cap, lane, bsum);
            const double x = fmax(mx, g.mx);
            sU[h + lane] = g.u;
            sX[h + lane] = x;
            sWin[h + lane] = expf((float)((double)m - x));
            sEmt[h + lane] = expf(-(float)(g.b + x));
            bsum = __shfl_sync(0xffffffffu, g.b, 31);
            mx = __shfl_sync(0xffffffffu, x, 31);
        }
    }
    store(0);
    cp_async_wait_all();
    __syncthreads();

    u64 accS[8][2], accH[8][2 * NG];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        accS[r][0] = accS[r][1] = 0ull;
#pragma unroll
        for (int g = 0; g < 2 * NG; ++g) accH[r][g] = 0ull;
    }
    float qn = 0.f;
    const int nt = tid % CH, nh = tid / CH;                  // q.n: one token, half of each piece
    const int pieces = (p.dqk + KP - 1) / KP;
    for (int pc = 0; pc < pieces; ++pc) {
        const int buf = pc & 1;
        if (pc + 1 < pieces) { load_qk((pc + 1) * KP); load_c((pc + 1) * KP, buf ^ 1); }
        const float2 *qa = sQ + buf * KP * CH + ty * 8;
        const float *ka = sK + buf * KP * CH + tx * 4;
        const float *ca = sC + buf * KP * DVT + tx * 4;
        if (has_C) {
#pragma unroll 4
            for (int j = 0; j < KP; ++j) {
                u64 a[8], bc[2 * NG];
#pragma unroll
                for (int r = 0; r < 8; r += 2) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(qa + j * CH + r);
                    a[r] = q.x;
                    a[r + 1] = q.y;
                }
                const ulonglong2 bk = *reinterpret_cast<const ulonglong2 *>(ka + j * CH);
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(ca + j * DVT + g * 64);
                    bc[2 * g] = q.x;
                    bc[2 * g + 1] = q.y;
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    accS[r][0] = ffma2(a[r], bk.x, accS[r][0]);
                    accS[r][1] = ffma2(a[r], bk.y, accS[r][1]);
#pragma unroll
                    for (int g = 0; g < 2 * NG; ++g) accH[r][g] = ffma2(a[r], bc[g], accH[r][g]);
                }
            }
#pragma unroll
            for (int j = 0; j < KP / 2; ++j) {
                const int jj = nh * (KP / 2) + j;
                qn = fmaf(sQ[(buf * KP + jj) * CH + nt].x, sN[buf * KP + jj], qn);
            }
        } else {
#pragma unroll 4
            for (int j = 0; j < KP; ++j) {
                const ulonglong2 bk = *reinterpret_cast<const ulonglong2 *>(ka + j * CH);
#pragma unroll
                for (int r = 0; r < 8; r += 2) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(qa + j * CH + r);
                    accS[r][0] = ffma2(q.x, bk.x, accS[r][0]);
                    accS[r][1] = ffma2(q.x, bk.y, accS[r][1]);
                    accS[r + 1][0] = ffma2(q.y, bk.x, accS[r + 1][0]);
                    accS[r + 1][1] = ffma2(q.y, bk.y, accS[r + 1][1]);
                }
            }
        }
        if (pc + 1 < pieces) store(buf ^ 1);
        cp_async_wait_all();
        __syncthreads();
    }
    sQn[nh * CH + nt] = qn;

    // ---- P = tril(S) e^{u_s - x_t}, row sums; H scaled to the chunk's frame
    const float qs = p.qscale;
#pragma unroll
    for (int r = 0; r < 8; r += 2) {
        float pv[2][4], rs[2] = {0.f, 0.f};
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int t = ty * 8 + r + rr;
            const double xt = sX[t];
            const float2 s01 = unpack2(accS[r + rr][0]), s23 = unpack2(accS[r + rr][1]);
            const float sv[4] = {s01.x, s01.y, s23.x, s23.y};
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int s = tx * 4 + x;
                pv[rr][x] = s <= t ? sv[x] * qs * expf((float)(sU[s] - xt)) : 0.f;
                rs[rr] += pv[rr][x];
            }
            rs[rr] += __shfl_xor_sync(0xffffffffu, rs[rr], 8);
            rs[rr] += __shfl_xor_sync(0xffffffffu, rs[rr], 4);
            rs[rr] += __shfl_xor_sync(0xffffffffu, rs[rr], 2);
            rs[rr] += __shfl_xor_sync(0xffffffffu, rs[rr], 1);
            if (tx == 0) sRow[t] = rs[rr];
            const u64 w2 = pack2(sWin[t] * qs, sWin[t] * qs);
#pragma unroll
            for (int g = 0; g < 2 * NG; ++g) accH[r + rr][g] = fmul2(accH[r + rr][g], w2);
        }
        // 16-byte unit (two tokens) of row s, at unit ^ (s / 4 % 8): the 16 lanes of a store hit different banks
        const int unit = (ty * 8 + r) >> 1;
#pragma unroll
        for (int x = 0; x < 4; ++x)
            *reinterpret_cast<float4 *>(sP + (tx * 4 + x) * CH + ((unit ^ (tx & 7)) << 1)) =
                make_float4(pv[0][x], pv[0][x], pv[1][x], pv[1][x]);
    }
    __syncthreads();
    const float *va = sV + tx * 4;
    const int s_end = min(CH, ((tid >> 5) + 1) * 16);        // no later token of the chunk contributes to this warp's rows
#pragma unroll 4
    for (int s = 0; s < s_end; ++s) {
        const int sw = (s >> 2) & 7;
        u64 a[8], bv[2 * NG];
#pragma unroll
        for (int r = 0; r < 8; r += 2) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(sP + s * CH + ((((ty * 8 + r) >> 1) ^ sw) << 1));
            a[r] = q.x;
            a[r + 1] = q.y;
        }
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(va + s * DVT + g * 64);
            bv[2 * g] = q.x;
            bv[2 * g + 1] = q.y;
        }
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int g = 0; g < 2 * NG; ++g) accH[r][g] = ffma2(a[r], bv[g], accH[r][g]);
    }
    T *hb = static_cast<T *>(p.h) + b * p.sh[0] + hd * p.sh[1] + (int64_t)t0 * p.sh[2] + col0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int t = ty * 8 + r;
        if (t0 + t >= p.S) break;   // the later rows are beyond the end too
        const float den = sWin[t] * qs * (sQn[t] + sQn[CH + t]) + sRow[t];
        const float inv = 1.0f / (fmaxf(fabsf(den), sEmt[t]) + p.eps);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const int cc = g * 64 + tx * 4;
            if (col0 + cc < p.dv) {
                const float2 x = unpack2(accH[r][2 * g]), y = unpack2(accH[r][2 * g + 1]);
                st4(hb + (int64_t)t * p.sh[2] + cc, make_float4(x.x * inv, x.y * inv, y.x * inv, y.y * inv));
            }
        }
    }
    if (single && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) grid_dependency_wait();
}

template <typename T> int run_group(const F32Params &P, cudaStream_t st) {
    const ChunkwiseParams &p = P.p;
    const int BH = p.B * p.NH, jt = (p.dqk + JT - 1) / JT, chunks = P.c_end - P.c_begin;
    // 128 columns per CTA once that still gives every SM a CTA: half the passes over K (Q and K, and S, in the output)
    const bool wide_s = p.dv > 64 && (int64_t)BH * jt * ((p.dv + 127) / 128) >= 148;
    const bool wide_o = p.dv > 64 && (int64_t)BH * chunks * ((p.dv + 127) / 128) >= 148;
    const int cs = wide_s ? 128 : 64, co = wide_o ? 128 : 64;
    const uint32_t sm_s = 2 * TT * JT * 8 + 2 * TT * cs * 4, sm_o = wide_o ? OutSmem<128>::TOTAL : OutSmem<64>::TOTAL;
    auto ks = wide_s ? mlstm_f32_state_kernel<T, 128> : mlstm_f32_state_kernel<T, 64>;
    auto ko = wide_o ? mlstm_f32_output_kernel<T, 128> : mlstm_f32_output_kernel<T, 64>;
    if (cudaFuncSetAttribute(ks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_s) != cudaSuccess ||
        cudaFuncSetAttribute(ko, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_o) != cudaSuccess)
        return XLSTM_ERR_CUDA;
    const int rc = launch_overlapped(ks, dim3(BH, jt, (p.dv + cs - 1) / cs), dim3(MAIN + 32), sm_s, st, P);
    if (rc != XLSTM_OK) return rc;
    return launch_overlapped(ko, dim3(chunks, (p.dv + co - 1) / co, BH), dim3(MAIN), sm_o, st, P);
}

int group_chunks(int BH, int S, int dqk, int dv) {
    const int NC = (S + CH - 1) / CH;
    const size_t per = (size_t)BH * ((size_t)dqk * dv + dqk) * sizeof(float);
    size_t g = SLOT_BYTES / per;
    if (g < 1) g = 1;
    return g < (size_t)NC ? (int)g : NC;
}

}  // namespace

size_t mlstm_chunkwise_f32_workspace(int B, int NH, int S, int dqk, int dv) {
    const int NC = (S + CH - 1) / CH, BH = B * NH;
    if (NC < 2) return 0;
    const int g = group_chunks(BH, S, dqk, dv);
    return WS_HEADER + (((size_t)BH * (NC + 1) * sizeof(float) + 255) & ~(size_t)255) +
           (size_t)BH * g * ((size_t)dqk * dv + dqk) * sizeof(float);
}

bool mlstm_chunkwise_f32_supported(const ChunkwiseParams &p, int dtype) {
    if (p.dqk % 4 || p.dv % 4) return false;
    for (int d = 0; d < 3; ++d)
        if (p.sq[d] % 4 || p.sk[d] % 4 || p.sv[d] % 4 || p.sh[d] % 4) return false;
    const uintptr_t mask = 4 * (dtype == XLSTM_F32 ? 4 : 2) - 1;
    if ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) |
         reinterpret_cast<uintptr_t>(p.h)) & mask)
        return false;
    if ((reinterpret_cast<uintptr_t>(p.C0) | reinterpret_cast<uintptr_t>(p.C1)) & 15u) return false;
    return (int64_t)p.B * p.NH <= 65535 && (p.dqk + JT - 1) / JT <= 65535 && (p.dv + 63) / 64 <= 65535;
}

int mlstm_chunkwise_f32(const ChunkwiseParams &p, int dtype, void *workspace, cudaStream_t st) {
    const int NC = (p.S + CH - 1) / CH, BH = p.B * p.NH;
    const int g = group_chunks(BH, p.S, p.dqk, p.dv);
    F32Params P{};
    P.p = p;
    P.NC = NC;
    P.slots = g;
    if (NC > 1) {
        unsigned char *ws = static_cast<unsigned char *>(workspace) + WS_HEADER;
        P.m_all = reinterpret_cast<float *>(ws);
        P.slot_C = reinterpret_cast<float *>(ws + (((size_t)BH * (NC + 1) * sizeof(float) + 255) & ~(size_t)255));
        P.slot_n = P.slot_C + (size_t)BH * g * p.dqk * p.dv;
    }
    P.C1 = p.C1; P.n1 = p.n1;
    for (int c = 0; c < NC; c += g) {
        P.c_begin = c;
        P.c_end = c + g < NC ? c + g : NC;
        // later groups continue from the state the previous one left in C1, n1 (and m_all)
        P.slot0 = c > 0;
        P.C0 = c > 0 ? p.C1 : p.C0; P.n0 = c > 0 ? p.n1 : p.n0;
        P.m0 = c == 0 && p.C0 ? p.m0 : nullptr;
        P.m1 = P.c_end == NC ? p.m1 : nullptr;
        const int rc = dtype == XLSTM_F32 ? run_group<float>(P, st) : run_group<__nv_bfloat16>(P, st);
        if (rc != XLSTM_OK) return rc;
    }
    return XLSTM_OK;
}

}  // namespace xl
