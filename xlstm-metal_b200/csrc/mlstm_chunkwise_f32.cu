// Chunkwise mLSTM forward with all arithmetic in fp32 (fp32 inputs, and the bf16 shapes the tensor-core kernels do not
// take), as launches over groups of chunks:
//
//   chain   one CTA per head: the stabiliser m at the start of every 64-token chunk (sums and maxima of the gates by warps,
//           then a scan over the chunks; whole sequence, first group only);
//   state   one CTA per (head, 64 rows x 64 or 128 columns of C): keeps its piece of C in registers, walks the sequence in
//           tiles of 32 tokens, C <- decay C + (w K)^T V, and leaves the state at the start of every chunk in scratch (the
//           only sequential part).  The weights of the chunks ahead and the normaliser are the work of two further warps;
//   matrix  one CTA per (head, chunk): S = Q K^T, P = tril(S) with its gates, beside the state kernel;
//   output  one CTA per (head, chunk, 64 or 128 columns of h): H = w_in Q C_start + P V as one contraction over dqk and the 64
//           keys, normaliser.  All chunks at once.
// A single chunk needs no scratch: its state and its output, which forms P itself, are two launches side by side.
//
// Both products are bound by FMA issue: a thread's tile is 8 rows x 4 NG columns (NG = 1, 2) of packed fp32 pairs (fma.rn.f32x2:
// two IEEE multiply-adds per instruction), the pairs lie along the columns as they are stored, the row operand is doubled in
// registers.  The loops alone reach 98 multiply-adds a clock and SM of 128 (with the doubled operand in shared memory 91).  16 heads of
// 256/512, 1024 tokens: 267 us (378 with the output kernel forming S for every 128 columns and doubled operands in shared memory);
// pieces of 256 columns, one CTA an SM, 279; 4 heads of 64/64, 256 tokens: 26 us (32).
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
constexpr int TT = 32;          // tokens per tile of the state kernel
constexpr int JT = 64;          // rows of C per CTA of the state kernel
constexpr int KP = 16;          // k per piece of the output kernel
constexpr int MAIN = 128;       // threads of the products: 8 row groups x 16 column groups
constexpr int LOAD = 64;        // threads of the state kernel that bring and scale the tiles, and of the normaliser; a warp of weights after them
constexpr int CHAIN_WARPS = 32;
constexpr int PM_WIN = CH * CH, PM_EMT = PM_WIN + CH, PM_ROW = PM_EMT + CH, CHUNK_PM = PM_ROW + CH;   // P[s][t], then per token
constexpr size_t SLOT_BYTES = (size_t)192 << 20;

struct F32Params {
    ChunkwiseParams p;
    const float *C0, *n0, *m0;       // state at the start of the group (C0 == NULL: zero); m of the sequence's start
    float *C1, *n1, *m1;             // state at its end
    float *slot_C, *slot_n;          // [BH][g][dqk][dv], [BH][g][dqk]
    double *m_all;                   // [BH][NC + 1], NULL: a single chunk, which starts at m0
    float *pm;                       // [BH][g][CHUNK_PM]: gate matrix and scalars of every chunk (NULL with m_all)
    int NC, c_begin, c_end, slots;   // chunks of the sequence, of the group, slots per head
    int early;                       // the output kernel may become resident while this group's states are worked on
    int slot0;                       // the first chunk's state is in slot 0 too (C1 may overwrite C0)
};

// One chunk's gates by a warp: tokens lane and lane + 32
struct ChunkGates {
    double u[2], b[2], x[2];         // i - b, summed log forget gates, running maximum of u (without m)
};
template <typename T> __device__ __forceinline__ void chunk_load(const ChunkwiseParams &p, int b, int hd, int t0, int lane, GateRaw (&r)[2]) {
    r[0] = gate_load<T>(p, b, hd, t0 + lane);
    r[1] = gate_load<T>(p, b, hd, t0 + 32 + lane);
}
__device__ __forceinline__ ChunkGates chunk_gates(const GateRaw (&r)[2], float cap, int lane) {
    ChunkGates c;
    double bsum = 0.0, mx = -INFINITY;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const GateTile g = gate_tile(r[h], cap, lane, bsum);
        c.u[h] = g.u;
        c.b[h] = g.b;
        c.x[h] = fmax(mx, g.mx);
        bsum = __shfl_sync(0xffffffffu, g.b, 31);
        mx = __shfl_sync(0xffffffffu, c.x[h], 31);
    }
    return c;
}
__device__ __forceinline__ double last_of(double v) { return __shfl_sync(0xffffffffu, v, 31); }

template <typename T> __device__ __forceinline__ float4 ld4_or_zero(const T *ptr, bool ok) {
    return ok ? ld4(ptr) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ uint32_t smem_addr(const void *q) { return (uint32_t)__cvta_generic_to_shared(q); }

// ---------------------------------------------------------------------------------------------------------------
// m at the start of every chunk: a chunk maps m to max(G + m, G + U) with G its summed log forget gates and U its largest u,
// which composes associatively.  A round is one chunk per warp.
template <typename T> __global__ void __launch_bounds__(CHAIN_WARPS * 32) mlstm_f32_chain_kernel(const F32Params P) {
    __shared__ double s_g[CHAIN_WARPS], s_v[CHAIN_WARPS];
    const ChunkwiseParams &p = P.p;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bh = blockIdx.x, b = bh / p.NH, hd = bh % p.NH;
    grid_dependency_wait();
    allow_dependents();
    if (p.status && bh == 0 && threadIdx.x == 0) *p.status = 0;
    double m = P.m0 ? (double)P.m0[bh] : 0.0;
    double *out = P.m_all + (size_t)bh * (P.NC + 1);
    for (int c0 = 0; c0 < P.NC; c0 += CHAIN_WARPS) {
        const int c = c0 + warp;
        if (c < P.NC) {
            GateRaw raw[2];
            chunk_load<T>(p, b, hd, c * CH, lane, raw);
            const ChunkGates g = chunk_gates(raw, p.gate_cap, lane);
            if (lane == 31) {
                s_g[warp] = g.b[1];
                s_v[warp] = g.b[1] + g.x[1];
            }
        }
        __syncthreads();
        if (warp == 0) {
            const int k = c0 + lane;
            double G = k < P.NC ? s_g[lane] : 0.0, V = k < P.NC ? s_v[lane] : -INFINITY;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {     // (G1, V1) then (G2, V2): (G1 + G2, max(G2 + V1, V2))
                const double Gp = __shfl_up_sync(0xffffffffu, G, o), Vp = __shfl_up_sync(0xffffffffu, V, o);
                if (lane >= o) {
                    V = fmax(G + Vp, V);
                    G += Gp;
                }
            }
            const double after = fmax(G + m, V);
            const double up = __shfl_up_sync(0xffffffffu, after, 1);
            if (k < P.NC) out[k] = lane == 0 ? m : up;
            m = __shfl_sync(0xffffffffu, after, min(31, P.NC - 1 - c0));
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[P.NC] = m;
        if (P.m1) P.m1[bh] = (float)m;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// acc[r][2 g], acc[r][2 g + 1]: row r, columns 64 g + 4 tx .. + 3 of a thread's tile, += sum_k a[k][r] b[k][column]
template <int NG> __device__ __forceinline__ void multiply_step(u64 (&acc)[8][2 * NG], const float4 &a0, const float4 &a1, const float *b) {
    const u64 av[8] = {pack2(a0.x, a0.x), pack2(a0.y, a0.y), pack2(a0.z, a0.z), pack2(a0.w, a0.w),
                       pack2(a1.x, a1.x), pack2(a1.y, a1.y), pack2(a1.z, a1.z), pack2(a1.w, a1.w)};
    u64 bv[2 * NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(b + g * 64);
        bv[2 * g] = q.x;
        bv[2 * g + 1] = q.y;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int g = 0; g < 2 * NG; ++g) acc[r][g] = ffma2(av[r], bv[g], acc[r][g]);
}
template <int NG, int K> __device__ __forceinline__ void multiply(u64 (&acc)[8][2 * NG], const float *a, int lda, const float *b, int ldb) {
#pragma unroll 4
    for (int k = 0; k < K; ++k)
        multiply_step<NG>(acc, *reinterpret_cast<const float4 *>(a + k * lda), *reinterpret_cast<const float4 *>(a + k * lda + 4), b + k * ldb);
}

// ROWS x COLS block of a row-major fp32 or bf16 matrix into shared memory as fp32 by THREADS threads: by asynchronous copies,
// or (bf16) through registers, `fetch` first and `put` once the buffer is free.  A thread stays on one group of four columns.
// Rows from `rows` on, and all of them where the thread's columns are not `in`, are zeros.
template <typename T, int ROWS, int COLS, int THREADS> struct BlockStage {
    static constexpr int STEP = THREADS / (COLS / 4), V = ROWS / STEP;
    static_assert(STEP >= 1 && ROWS % STEP == 0, "whole rows");
    uint2 raw[sizeof(T) == 2 ? V : 1];
    static __device__ __forceinline__ int column(int tid) { return (tid % (COLS / 4)) * 4; }
    __device__ __forceinline__ void fetch(const T *src, int64_t ld, float *dst, int tid, int rows, bool in) {
        const int r0 = tid / (COLS / 4);
        const T *s = src + (in ? r0 * ld + column(tid) : 0);
        const uint32_t d = smem_addr(dst + tid * 4);
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const bool ok = in && r0 + i * STEP < rows;
            if constexpr (sizeof(T) == 4) cp_async16(d + i * THREADS * 16, ok ? s : src, ok);
            else raw[i] = ok ? *reinterpret_cast<const uint2 *>(s) : make_uint2(0u, 0u);
            s += STEP * ld;
        }
    }
    __device__ __forceinline__ void put(float *dst, int tid) {
        if constexpr (sizeof(T) == 2) {
#pragma unroll
            for (int i = 0; i < V; ++i)
                *reinterpret_cast<float4 *>(dst + (tid + i * THREADS) * 4) =
                    make_float4(__uint_as_float(raw[i].x << 16), __uint_as_float(raw[i].x & 0xffff0000u),
                                __uint_as_float(raw[i].y << 16), __uint_as_float(raw[i].y & 0xffff0000u));
        }
    }
};

// K and V tiles
template <int NG> constexpr uint32_t state_smem() { return 2 * TT * JT * 4 + 2 * TT * 64 * NG * 4; }

// The products are two warps per scheduler at most, so whatever else those warps did would stand beside the multiply-adds, not
// behind them: two warps bring K and V of the next tile and scale K, a third turns gates into weights a chunk ahead.
template <typename T, int NG>
__global__ void __launch_bounds__(MAIN + LOAD + 32, 2) mlstm_f32_state_kernel(const F32Params P) {
    constexpr int CT = 64 * NG;
    extern __shared__ __align__(16) unsigned char smem[];
    float *sK = reinterpret_cast<float *>(smem);                       // [2][TT][JT] w k
    float *sV = sK + 2 * TT * JT;                                      // [2][TT][CT]
    __shared__ float s_w[2][CH], s_decay[2];                           // weights of the even and the odd chunks
    const ChunkwiseParams &p = P.p;
    const int tid = threadIdx.x, lane = tid & 31;
    const int bh = blockIdx.x, b = bh / p.NH, hd = bh % p.NH;
    const int j0 = blockIdx.y * JT, col0 = blockIdx.z * CT;
    const int t_begin = P.c_begin * CH, t_end = min(p.S, P.c_end * CH);
    const int tiles = (t_end - t_begin + TT - 1) / TT, chunks = P.c_end - P.c_begin;
    const bool own_n = blockIdx.z == 0;
    // this launch may run beside the end of the one before it: in a group after the first that is the output kernel, which
    // still reads the slots and the state, in the first one the chain kernel, which writes m
    grid_dependency_wait();
    allow_dependents();
    if (p.status && !P.m_all && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0) *p.status = 0;

    if (tid >= MAIN + LOAD) {
        // ---- weights, a chunk ahead
        GateRaw raw[2];
        chunk_load<T>(p, b, hd, t_begin, lane, raw);
        auto weights = [&](int c) {
            if (c >= chunks) return;
            const double m = P.m_all ? P.m_all[(size_t)bh * (P.NC + 1) + P.c_begin + c] : (P.m0 ? (double)P.m0[bh] : 0.0);
            const ChunkGates g = chunk_gates(raw, p.gate_cap, lane);
            chunk_load<T>(p, b, hd, t_begin + (c + 1) * CH, lane, raw);
            const double xl = fmax(m, last_of(g.x[1]));
            s_w[c & 1][lane] = expf((float)(g.u[0] - xl));
            s_w[c & 1][lane + 32] = expf((float)(g.u[1] - xl));
            const double m_new = last_of(g.b[1]) + xl;
            if (lane == 0) {
                s_decay[c & 1] = expf((float)(m - xl));
                if (!P.m_all && blockIdx.y == 0 && own_n && P.m1) P.m1[bh] = (float)m_new;
            }
        };
        weights(0);
        __syncthreads();                                     // weights of chunk 0
        __syncthreads();                                     // tile 0 in shared memory
        for (int k = 0; k < tiles; ++k) {
            // tile k + 1 is scaled during tile k: an even tile's is of the same chunk, so the weights of the next chunk may be
            // written during even tiles, into the buffer that the chunk before has left
            if ((k & 1) == 0) weights((k >> 1) + 1);
            __syncthreads();
        }
        return;
    }
    if (tid >= MAIN) {
        // ---- tiles: K through registers (a tile ahead) and scaled, V straight into shared memory; the normaliser
        constexpr int KV = TT * JT / 4 / LOAD;
        const int lt = tid - MAIN;
        const T *kb = static_cast<const T *>(p.k) + b * p.sk[0] + hd * p.sk[1] + j0;
        const T *vb = static_cast<const T *>(p.v) + b * p.sv[0] + hd * p.sv[1] + col0;
        const int kr0 = lt / (JT / 4), kc = (lt % (JT / 4)) * 4;           // rows kr0 + 4 i of a tile of K, four columns
        using Stage = BlockStage<T, TT / 2, CT, LOAD>;                     // V in two halves: registers, in bf16
        Stage vs;
        const bool k_in = j0 + kc < p.dqk, v_in = col0 + Stage::column(lt) < p.dv;
        float4 kr[KV];
        auto load_k = [&](int k) {
            if (k >= tiles) return;
            const int t0 = t_begin + k * TT, rows = t_end - t0;
            const T *s = kb + (k_in ? (t0 + kr0) * p.sk[2] + kc : 0);
#pragma unroll
            for (int i = 0; i < KV; ++i) {
                const bool ok = k_in && kr0 + i * (TT / KV) < rows;
                kr[i] = ld4_or_zero(ok ? s : kb, ok);
                s += (TT / KV) * p.sk[2];
            }
        };
        auto stage = [&](int k) {
            const int t0 = t_begin + k * TT, rows = t_end - t0;
            float *dv = sV + (k & 1) * TT * CT;
            vs.fetch(vb + t0 * p.sv[2], p.sv[2], dv, lt, rows, v_in);
            float4 *dk = reinterpret_cast<float4 *>(sK + (k & 1) * TT * JT) + lt;
            const float *w32 = s_w[(k >> 1) & 1] + (k & 1) * TT + kr0;
#pragma unroll
            for (int i = 0; i < KV; ++i) {
                const float w = w32[i * (TT / KV)];
                const float4 x = kr[i];
                dk[i * LOAD] = make_float4(w * x.x, w * x.y, w * x.z, w * x.w);
            }
            vs.put(dv, lt);
            vs.fetch(vb + (t0 + TT / 2) * p.sv[2], p.sv[2], dv + TT / 2 * CT, lt, rows - TT / 2, v_in);
            load_k(k + 1);
            vs.put(dv + TT / 2 * CT, lt);
        };
        const int j = j0 + 2 * lane;
        float n0 = 0.f, n1 = 0.f;
        const bool my_n = own_n && lt < 32;
        if (my_n && P.C0) {
            if (j < p.dqk) n0 = P.n0[(size_t)bh * p.dqk + j];
            if (j + 1 < p.dqk) n1 = P.n0[(size_t)bh * p.dqk + j + 1];
        }
        load_k(0);
        __syncthreads();
        stage(0);
        cp_async_wait_all();
        __syncthreads();
        for (int k = 0; k < tiles; ++k) {
            if (k + 1 < tiles) stage(k + 1);   // into the other buffer: last read before the previous barrier
            if (my_n) {
                const int c = k >> 1;
                float decay = 1.f;
                if ((k & 1) == 0) {
                    if (P.slot_n && (c > 0 || P.slot0)) {
                        float *dst = P.slot_n + ((size_t)bh * P.slots + c) * p.dqk;
                        if (j < p.dqk) dst[j] = n0;
                        if (j + 1 < p.dqk) dst[j + 1] = n1;
                    }
                    decay = s_decay[c & 1];
                }
                const float2 *row = reinterpret_cast<const float2 *>(sK + (k & 1) * TT * JT) + lane;
                float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
                for (int t = 0; t < TT; ++t) {
                    const float2 v = row[t * (JT / 2)];
                    a0 += v.x;
                    a1 += v.y;
                }
                n0 = fmaf(n0, decay, a0);
                n1 = fmaf(n1, decay, a1);
            }
            cp_async_wait_all();
            __syncthreads();
        }
        if (my_n) {
            if (j < p.dqk) P.n1[(size_t)bh * p.dqk + j] = n0;
            if (j + 1 < p.dqk) P.n1[(size_t)bh * p.dqk + j + 1] = n1;
        }
        return;
    }

    // ---- products
    const int ty = tid >> 4, tx = tid & 15;
    u64 acc[8][2 * NG];
    const size_t CE = (size_t)p.dqk * p.dv;
    const size_t c_off = (size_t)(j0 + ty * 8) * p.dv + col0 + tx * 4;    // row r, column group g: + r dv + 64 g
    auto c_ok = [&](int r, int g) { return j0 + ty * 8 + r < p.dqk && col0 + g * 64 + tx * 4 < p.dv; };
    const bool full = j0 + JT <= p.dqk && col0 + CT <= p.dv;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const bool ok = P.C0 && c_ok(r, g);
            const float4 c4 = ld4_or_zero(P.C0 + (ok ? bh * CE + c_off + (size_t)r * p.dv + g * 64 : 0), ok);
            acc[r][2 * g] = pack2(c4.x, c4.y);
            acc[r][2 * g + 1] = pack2(c4.z, c4.w);
        }
    auto put = [&](float *base) {
        float *d = base + c_off;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
#pragma unroll
            for (int g = 0; g < NG; ++g)
                if (full || c_ok(r, g)) {
                    const float2 x = unpack2(acc[r][2 * g]), y = unpack2(acc[r][2 * g + 1]);
                    *reinterpret_cast<float4 *>(d + g * 64) = make_float4(x.x, x.y, y.x, y.y);
                }
            d += p.dv;
        }
    };
    __syncthreads();
    __syncthreads();
    for (int k = 0; k < tiles; ++k) {
        if ((k & 1) == 0) {
            const int c = k >> 1;
            if (P.slot_C && (c > 0 || P.slot0)) put(P.slot_C + ((size_t)bh * P.slots + c) * CE);
            const u64 d2 = pack2(s_decay[c & 1], s_decay[c & 1]);
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int g = 0; g < 2 * NG; ++g) acc[r][g] = fmul2(acc[r][g], d2);
        }
        multiply<NG, TT>(acc, sK + (k & 1) * TT * JT + ty * 8, JT, sV + (k & 1) * TT * CT + tx * 4, CT);
        __syncthreads();
    }
    put(P.C1 + bh * CE);
}

// ---------------------------------------------------------------------------------------------------------------
// One chunk's S = Q K^T (8 rows x 4 columns a thread); sQ, sK: [2][KP][CH] each
template <typename T> struct ChunkQK {
    static constexpr int QV = KP * CH / 4 / MAIN;
    const T *qrow, *krow;
    int lt, lj, dqk;
    bool in;
    __device__ __forceinline__ ChunkQK(const ChunkwiseParams &p, int b, int hd, int t0, int tid) {
        lt = tid % CH;                                       // lane = token: the transposed stores are conflict-free
        lj = (tid / CH) * 4;                                 // columns lj + 8 i
        in = t0 + lt < p.S;
        dqk = p.dqk;
        qrow = static_cast<const T *>(p.q) + b * p.sq[0] + hd * p.sq[1] + (in ? (t0 + lt) * p.sq[2] : 0);
        krow = static_cast<const T *>(p.k) + b * p.sk[0] + hd * p.sk[1] + (in ? (t0 + lt) * p.sk[2] : 0);
    }
    __device__ __forceinline__ void load(const T *row, int j0, float4 (&r)[QV]) const {
#pragma unroll
        for (int i = 0; i < QV; ++i) {
            const int j = j0 + lj + i * (KP / QV);
            const bool ok = in && j < dqk;
            r[i] = ld4_or_zero(row + (ok ? j : 0), ok);
        }
    }
    __device__ __forceinline__ void store(float *dst, const float4 (&r)[QV]) const {
        float *d = dst + lj * CH + lt;
#pragma unroll
        for (int i = 0; i < QV; ++i) {
            d[0] = r[i].x; d[CH] = r[i].y; d[2 * CH] = r[i].z; d[3 * CH] = r[i].w;
            d += (KP / QV) * CH;
        }
    }
    __device__ __forceinline__ void scores(float *sQ, float *sK, int ty, int tx, u64 (&acc)[8][2]) const {
        const int pieces = (dqk + KP - 1) / KP;
        float4 qr[QV], kr[QV];
        load(qrow, 0, qr);
        load(krow, 0, kr);
        store(sQ, qr);
        store(sK, kr);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = 0ull;
        for (int pc = 0; pc < pieces; ++pc) {
            const int buf = pc & 1;
            if (pc + 1 < pieces) { load(qrow, (pc + 1) * KP, qr); load(krow, (pc + 1) * KP, kr); }
            multiply<1, KP>(acc, sQ + buf * KP * CH + ty * 8, CH, sK + buf * KP * CH + tx * 4, CH);
            if (pc + 1 < pieces) { store(sQ + (buf ^ 1) * KP * CH, qr); store(sK + (buf ^ 1) * KP * CH, kr); }
            __syncthreads();
        }
    }
};
// Gate scalars of a chunk by one warp
struct ChunkScalars {
    double *u, *x;
    float *win, *emt;                                        // e^{m - x_t} dqk^-1/2, e^{-m_t}
    __device__ __forceinline__ void fill(const ChunkwiseParams &p, const GateRaw (&raw)[2], double m, int lane) const {
        const ChunkGates g = chunk_gates(raw, p.gate_cap, lane);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double xt = fmax(m, g.x[h]);
            u[h * 32 + lane] = g.u[h];
            x[h * 32 + lane] = xt;
            win[h * 32 + lane] = expf((float)(m - xt)) * p.qscale;
            emt[h * 32 + lane] = expf(-(float)(g.b[h] + xt));
        }
    }
};
// P = tril(S) e^{u_s - x_t} dqk^-1/2 as [s][t] rows, and the row sums; unit(s, q): where the four tokens 4 q .. of key s go
template <typename Unit>
__device__ __forceinline__ void gate_matrix(const u64 (&S)[8][2], const ChunkScalars &cs, float qscale, int ty, int tx, float *row_sums, Unit &&unit) {
#pragma unroll
    for (int r = 0; r < 8; r += 4) {
        float pv[4][4];
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) {
            const int t = ty * 8 + r + rr;
            const double xt = cs.x[t];
            const float2 s01 = unpack2(S[r + rr][0]), s23 = unpack2(S[r + rr][1]);
            const float sv[4] = {s01.x, s01.y, s23.x, s23.y};
            float rs = 0.f;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int s = tx * 4 + x;
                pv[rr][x] = s <= t ? sv[x] * qscale * expf((float)(cs.u[s] - xt)) : 0.f;
                rs += pv[rr][x];
            }
            rs += __shfl_xor_sync(0xffffffffu, rs, 8);
            rs += __shfl_xor_sync(0xffffffffu, rs, 4);
            rs += __shfl_xor_sync(0xffffffffu, rs, 2);
            rs += __shfl_xor_sync(0xffffffffu, rs, 1);
            if (tx == 0) row_sums[t] = rs;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
            *reinterpret_cast<float4 *>(unit(tx * 4 + x, (ty * 8 + r) >> 2)) = make_float4(pv[0][x], pv[1][x], pv[2][x], pv[3][x]);
    }
}

// The gate matrix of every chunk: nothing of it needs the states, so this launch runs beside the state kernel (on the SMs that
// one leaves, and behind its CTAs), and the output kernel, whose CTAs of one chunk would each form it again, does not.
template <typename T> __global__ void __launch_bounds__(MAIN, 3) mlstm_f32_gate_matrix_kernel(const F32Params P) {
    __shared__ __align__(16) float sQ[2 * KP * CH], sK[2 * KP * CH];
    __shared__ double sU[CH], sX[CH];
    const ChunkwiseParams &p = P.p;
    const int tid = threadIdx.x, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
    const int ci = blockIdx.x, c = P.c_begin + ci, bh = blockIdx.y, b = bh / p.NH, hd = bh % p.NH;
    // the state kernel has waited for the chain kernel before it let this one start
    if (P.early) allow_dependents();
    GateRaw raw[2];
    chunk_load<T>(p, b, hd, c * CH, lane, raw);
    const ChunkQK<T> qk(p, b, hd, c * CH, tid);
    u64 S[8][2];
    qk.scores(sQ, sK, ty, tx, S);
    float *out = P.pm + ((size_t)bh * P.slots + ci) * CHUNK_PM;
    const ChunkScalars cs{sU, sX, out + PM_WIN, out + PM_EMT};
    if (tid < 32) cs.fill(p, raw, __ldcg(P.m_all + (size_t)bh * (P.NC + 1) + c), lane);
    __syncthreads();
    gate_matrix(S, cs, p.qscale, ty, tx, out + PM_ROW, [&](int s, int q) { return out + s * CH + q * 4; });
    // this launch is complete only when the state kernel is: what follows waits for this one
    if (blockIdx.x == 0 && blockIdx.y == 0) grid_dependency_wait();
}

// ---------------------------------------------------------------------------------------------------------------
template <int NG> struct OutSmem {
    static constexpr int DVT = 64 * NG;
    static constexpr uint32_t Q = 0;                                   // float [2][KP][CH] transposed
    static constexpr uint32_t B = Q + 2 * KP * CH * 4;                 // float [2][KP][CH] K transposed, then [2][KP][DVT] C, V
    static constexpr uint32_t PM = B + 2 * KP * DVT * 4;               // float [CH s][CH t] P, 16-byte units swizzled
    static constexpr uint32_t U = PM + CH * CH * 4;                    // double [CH] u, [CH] x
    static constexpr uint32_t WIN = U + 2 * CH * 8;                    // float [CH] win, [CH] e^{-m_t}, [CH] row sums, [2][CH] q.n
    static constexpr uint32_t NV = WIN + 5 * CH * 4;                   // float [2][KP] n of the piece
    static constexpr uint32_t TOTAL = NV + 2 * KP * 4;
};

template <typename T, int NG>
__global__ void __launch_bounds__(MAIN, 3) mlstm_f32_output_kernel(const F32Params P) {
    using SM = OutSmem<NG>;
    constexpr int DVT = SM::DVT;
    extern __shared__ __align__(16) unsigned char smem[];
    float *sQ = reinterpret_cast<float *>(smem + SM::Q);
    float *sB = reinterpret_cast<float *>(smem + SM::B);
    float *sP = reinterpret_cast<float *>(smem + SM::PM);
    float *sWin = reinterpret_cast<float *>(smem + SM::WIN), *sEmt = sWin + CH, *sRow = sEmt + CH, *sQn = sRow + CH;
    float *sN = reinterpret_cast<float *>(smem + SM::NV);
    const ChunkwiseParams &p = P.p;
    const int tid = threadIdx.x, lane = tid & 31, ty = tid >> 4, tx = tid & 15;
    const int ci = blockIdx.x, c = P.c_begin + ci, t0 = c * CH, col0 = blockIdx.y * DVT;
    const int bh = blockIdx.z, b = bh / p.NH, hd = bh % p.NH;
    const bool from_slot = ci > 0 || P.slot0, has_C = from_slot || P.C0 != nullptr;
    const size_t CE = (size_t)p.dqk * p.dv;
    const float *Cs = from_slot ? P.slot_C + ((size_t)bh * P.slots + ci) * CE : P.C0 + bh * CE;
    const float *ns = from_slot ? P.slot_n + ((size_t)bh * P.slots + ci) * p.dqk : P.n0 + (size_t)bh * p.dqk;
    const T *vb = static_cast<const T *>(p.v) + b * p.sv[0] + hd * p.sv[1] + (int64_t)t0 * p.sv[2] + col0;
    const int pieces = (p.dqk + KP - 1) / KP;
    const ChunkQK<T> qk(p, b, hd, t0, tid);
    // 16-byte unit q (four tokens) of row s of P, at unit q ^ (s / 4): the lanes of a store hit different banks
    auto p_unit = [&](int s, int q) { return sP + s * CH + ((q ^ (s >> 2)) << 2); };

    // ---- pieces of the contraction: Q and C (the first `pieces`, if there is a state), then P and V (CH / KP)
    const int first = has_C ? 0 : pieces, last = pieces + CH / KP;
    float nr = 0.f;
    float4 qr[ChunkQK<T>::QV];
    using StageC = BlockStage<float, KP, DVT, MAIN>;
    StageC cs;
    BlockStage<T, KP, DVT, MAIN> vs;
    const bool col_in = col0 + StageC::column(tid) < p.dv;
    auto load_piece = [&](int pc) {
        float *dst = sB + (pc & 1) * KP * DVT;
        if (pc < pieces) {
            const int j0 = pc * KP;
            qk.load(qk.qrow, j0, qr);
            if (tid < KP) nr = j0 + tid < p.dqk ? ns[j0 + tid] : 0.f;
            cs.fetch(Cs + (size_t)j0 * p.dv + col0, p.dv, dst, tid, p.dqk - j0, col_in);
        } else {
            const int s0 = (pc - pieces) * KP;
            vs.fetch(vb + s0 * p.sv[2], p.sv[2], dst, tid, p.S - t0 - s0, col_in);
        }
    };
    auto store_piece = [&](int pc) {
        if (pc < pieces) {
            qk.store(sQ + (pc & 1) * KP * CH, qr);
            if (tid < KP) sN[(pc & 1) * KP + tid] = nr;
        } else {
            vs.put(sB + (pc & 1) * KP * DVT, tid);
        }
        cp_async_wait_all();
    };
    if (P.m_all) {
        // what the state and gate matrix kernels write (C, n, P and the scalars) is read after the wait
        grid_dependency_wait();
        allow_dependents();
        const float *pm = P.pm + ((size_t)bh * P.slots + ci) * CHUNK_PM;
#pragma unroll
        for (int i = 0; i < CH * CH / 4 / MAIN; ++i) {
            const int e = tid + i * MAIN;
            cp_async16(smem_addr(p_unit(e / (CH / 4), e % (CH / 4))), pm + e * 4, true);
        }
        if (tid < 3 * CH / 4) cp_async16(smem_addr(sWin + tid * 4), pm + PM_WIN + tid * 4, true);
        load_piece(first);
        store_piece(first);
    } else {
        // A single chunk has no scratch and needs nothing of the state kernel, which waited for the inputs before it let this
        // one start: the two run side by side, and one CTA waits at the end, so that this launch is complete only when that
        // one is.
        double *sU = reinterpret_cast<double *>(smem + SM::U), *sX = sU + CH;
        GateRaw raw[2];
        chunk_load<T>(p, b, hd, t0, lane, raw);
        u64 S[8][2];
        qk.scores(sQ, sB, ty, tx, S);
        load_piece(first);
        const ChunkScalars sc{sU, sX, sWin, sEmt};
        if (tid < 32) sc.fill(p, raw, P.m0 ? (double)P.m0[bh] : 0.0, lane);
        store_piece(first);
        __syncthreads();
        gate_matrix(S, sc, p.qscale, ty, tx, sRow, p_unit);
    }
    __syncthreads();
    u64 acc[8][2 * NG];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int g = 0; g < 2 * NG; ++g) acc[r][g] = 0ull;
    float qn = 0.f;
    const int nt = tid % CH, nh = tid / CH;                  // q.n: one token, half of each piece
    for (int pc = first; pc < pieces; ++pc) {
        const int buf = pc & 1;
        load_piece(pc + 1);
        multiply<NG, KP>(acc, sQ + buf * KP * CH + ty * 8, CH, sB + buf * KP * DVT + tx * 4, DVT);
#pragma unroll
        for (int j = 0; j < KP / 2; ++j) {
            const int jj = nh * (KP / 2) + j;
            qn = fmaf(sQ[(buf * KP + jj) * CH + nt], sN[buf * KP + jj], qn);
        }
        store_piece(pc + 1);
        __syncthreads();
    }
    sQn[nh * CH + nt] = qn;
    // H to the chunk's frame, then the chunk's own keys
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float w = sWin[ty * 8 + r];
        const u64 w2 = pack2(w, w);
#pragma unroll
        for (int g = 0; g < 2 * NG; ++g) acc[r][g] = fmul2(acc[r][g], w2);
    }
    const int s_end = min(CH, ((tid >> 5) + 1) * 16);        // no later token of the chunk contributes to this warp's rows
    for (int pc = pieces; pc < last; ++pc) {
        const int buf = pc & 1, s0 = (pc - pieces) * KP;
        if (pc + 1 < last) load_piece(pc + 1);
        if (s0 < s_end) {
            const float *vp = sB + buf * KP * DVT + tx * 4;
#pragma unroll 4
            for (int s = 0; s < KP; ++s)
                multiply_step<NG>(acc, *reinterpret_cast<const float4 *>(p_unit(s0 + s, 2 * ty)),
                                  *reinterpret_cast<const float4 *>(p_unit(s0 + s, 2 * ty + 1)), vp + s * DVT);
        }
        if (pc + 1 < last) {
            store_piece(pc + 1);
            __syncthreads();
        }
    }
    __syncthreads();                                         // q.n of every token
    T *hb = static_cast<T *>(p.h) + b * p.sh[0] + hd * p.sh[1] + (int64_t)t0 * p.sh[2] + col0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int t = ty * 8 + r;
        if (t0 + t >= p.S) break;   // the later rows are beyond the end too
        const float den = sWin[t] * (sQn[t] + sQn[CH + t]) + sRow[t];
        const float inv = 1.0f / (fmaxf(fabsf(den), sEmt[t]) + p.eps);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const int cc = g * 64 + tx * 4;
            if (col0 + cc < p.dv) {
                const float2 x = unpack2(acc[r][2 * g]), y = unpack2(acc[r][2 * g + 1]);
                st4(hb + (int64_t)t * p.sh[2] + cc, make_float4(x.x * inv, x.y * inv, y.x * inv, y.y * inv));
            }
        }
    }
    if (!P.m_all && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) grid_dependency_wait();
}

template <typename T, int NG> int launch_state(const F32Params &P, cudaStream_t st) {
    auto kern = mlstm_f32_state_kernel<T, NG>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)state_smem<NG>()) != cudaSuccess) return XLSTM_ERR_CUDA;
    return launch_overlapped(kern, dim3(P.p.B * P.p.NH, (P.p.dqk + JT - 1) / JT, (P.p.dv + 64 * NG - 1) / (64 * NG)), dim3(MAIN + LOAD + 32),
                             state_smem<NG>(), st, P);
}
template <typename T, int NG> int launch_output(const F32Params &P, cudaStream_t st) {
    auto kern = mlstm_f32_output_kernel<T, NG>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OutSmem<NG>::TOTAL) != cudaSuccess) return XLSTM_ERR_CUDA;
    return launch_overlapped(kern, dim3(P.c_end - P.c_begin, (P.p.dv + 64 * NG - 1) / (64 * NG), P.p.B * P.p.NH), dim3(MAIN),
                             OutSmem<NG>::TOTAL, st, P);
}

template <typename T> int run_group(const F32Params &P, cudaStream_t st) {
    const ChunkwiseParams &p = P.p;
    if (P.m_all && P.c_begin == 0) {
        const int rc = launch_overlapped(mlstm_f32_chain_kernel<T>, dim3(p.B * p.NH), dim3(CHAIN_WARPS * 32), 0, st, P);
        if (rc != XLSTM_OK) return rc;
    }
    const int chunks = P.c_end - P.c_begin;
    auto state_ctas = [&](int ng) { return (int64_t)p.B * p.NH * ((p.dqk + JT - 1) / JT) * ((p.dv + 64 * ng - 1) / (64 * ng)); };
    auto output_ctas = [&](int ng) { return (int64_t)p.B * p.NH * chunks * ((p.dv + 64 * ng - 1) / (64 * ng)); };
    // 128 columns a CTA or 64.  States: 64 make the shorter tile and twice the CTAs, each of which starts, leaves its slots and ends,
    // so the more chunks, the more CTAs are worth it (us with 64 and 128 columns: 16 heads of 256/512, 65 tokens 63 and 58; 8 of 128/256
    // 256 tokens 29 and 40; 24 of 128/256 256 tokens 49 and 47, 512 tokens 79 and 84).  Outputs: 128 where 64 would be more than fit at
    // once, three an SM (24 of 256/512, 256 tokens 123 and 117; 12 heads 74 and 77).  A single chunk's two kernels share the SMs: 32
    // of 256/512, 64 tokens 58 and 42 with 128 output CTAs of 128 columns, 12 heads 27.4 and 28.7 with 48.
    const int ns = p.dv > 64 && state_ctas(2) >= (chunks == 1 ? 111 : chunks < 10 ? 24 * chunks : 222) ? 2 : 1;
    const int no = p.dv > 64 && (chunks == 1 ? output_ctas(2) >= 80 : output_ctas(1) > 444) ? 2 : 1;
    // Output CTAs that become resident beside the state kernel crowd the SMs it leaves free, up to three on one, and stay there: with
    // one wave of them that lasts longer than their start costs (16 heads of 256/512, 128 tokens 85 us, 56 when they start after the
    // states; 24 of 128/256, 192 tokens 60 and 39).  They come early where every CTA of the group has an SM, where several waves
    // even it out (32 of 128/256, 512 tokens: 115 and 119), or where they are short and half the SMs are free (64 of 64/64, 320
    // tokens: 38 and 41).
    F32Params G = P;
    G.early = state_ctas(ns) + (int64_t)p.B * p.NH * chunks + output_ctas(no) <= 148 || output_ctas(no) >= 370 ||
              (p.dqk <= 64 && state_ctas(ns) <= 74);
    int rc = ns == 2 ? launch_state<T, 2>(G, st) : launch_state<T, 1>(G, st);
    if (rc != XLSTM_OK) return rc;
    if (P.m_all) {
        rc = launch_overlapped(mlstm_f32_gate_matrix_kernel<T>, dim3(chunks, p.B * p.NH), dim3(MAIN), 0, st, G);
        if (rc != XLSTM_OK) return rc;
    }
    return no == 2 ? launch_output<T, 2>(G, st) : launch_output<T, 1>(G, st);
}

// scratch of one chunk of a head: its state and its gate matrix (a multiple of 16 bytes, as each of the three arrays is)
size_t slot_floats(int dqk, int dv) { return (size_t)dqk * dv + dqk + CHUNK_PM; }

int group_chunks(int BH, int S, int dqk, int dv) {
    const int NC = (S + CH - 1) / CH;
    const size_t per = (size_t)BH * slot_floats(dqk, dv) * sizeof(float);
    size_t g = SLOT_BYTES / per;
    if (g < 1) g = 1;
    return g < (size_t)NC ? (int)g : NC;
}

}  // namespace

size_t mlstm_chunkwise_f32_workspace(int B, int NH, int S, int dqk, int dv) {
    const int NC = (S + CH - 1) / CH, BH = B * NH;
    if (NC < 2) return 0;
    const int g = group_chunks(BH, S, dqk, dv);
    return WS_HEADER + (((size_t)BH * (NC + 1) * sizeof(double) + 255) & ~(size_t)255) +
           (size_t)BH * g * slot_floats(dqk, dv) * sizeof(float);
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
        P.m_all = reinterpret_cast<double *>(ws);
        P.slot_C = reinterpret_cast<float *>(ws + (((size_t)BH * (NC + 1) * sizeof(double) + 255) & ~(size_t)255));
        P.slot_n = P.slot_C + (size_t)BH * g * p.dqk * p.dv;
        P.pm = P.slot_n + (size_t)BH * g * p.dqk;
    }
    P.C1 = p.C1; P.n1 = p.n1; P.m1 = p.m1;
    for (int c = 0; c < NC; c += g) {
        P.c_begin = c;
        P.c_end = c + g < NC ? c + g : NC;
        // later groups continue from the state the previous one left in C1, n1 (and m_all)
        P.slot0 = c > 0;
        P.C0 = c > 0 ? p.C1 : p.C0; P.n0 = c > 0 ? p.n1 : p.n0;
        P.m0 = c == 0 && p.C0 ? p.m0 : nullptr;
        const int rc = dtype == XLSTM_F32 ? run_group<float>(P, st) : run_group<__nv_bfloat16>(P, st);
        if (rc != XLSTM_OK) return rc;
    }
    return XLSTM_OK;
}

}  // namespace xl
