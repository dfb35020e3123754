// Packaged sLSTM cell (scalar gates per head, no recurrent weights) over S timesteps.
//
//   m_t = max(m_{t-1} + lf_t, i_t)      c_t = e^{m_{t-1}+lf_t-m_t} c_{t-1} + e^{i_t-m_t} tanh(z_t)      (n_t likewise)
//   h_t = sigmoid(o_t) c_t / (|n_t| + eps)
//
// Nothing depends on h_{t-1}, so both recurrences are associative: (A, B) -> m' = max(m + A, B) for the stabiliser
// and (f, i) -> x' = f x + i for c and n.  The floor is one read of z and one write of h (134 MB at B=4, S=2048, 4 x
// 1024 units in bf16: 21 us); a CTA per (batch, head) walking all S steps, which this replaces, left 132 SMs idle and
// paid the sequential stabiliser and two barriers per 32 steps (1912 us; the two launches below 82, with a state 113).
//
// One WARP is one work item: (batch, head) x 32*VEC adjacent units x a segment of the sequence.  Lane = timestep while
// the gates of 32 steps are worked out (transcendentals and both scans by warp shuffles, no shared memory, no
// barrier), lane = VEC adjacent units (one 16-byte vector) while the state walks those steps.  Without an initial n the
// normaliser is one scalar per step, and so is the whole factor of c.  The state is fp32 whatever the activations are, so
// tanh and the quotients are the exact ones in both types (in bf16 the special-function forms took 69 and 79 us, but left two
// digits of a z of 1e-5 in c).
// Few (batch, head) pairs: the sequence is cut into segments of whole 32-step tiles.  A first launch leaves each
// segment's end state from an empty start (reads z once), the second one chains those of the earlier segments (at
// most 31 independent loads per unit) into its own start state and does the full walk.  z is read twice; that costs
// less than the idle SMs as long as the single pass has under a third of the warps that fill the GPU (see plan()).
#include "common.cuh"
#include "vec16.cuh"

namespace xl {
namespace {

constexpr int SC_TILE = 32;         // timesteps per gate tile: one lane each
constexpr int SC_BATCH = 8;         // z vectors in flight per lane
constexpr int SC_MAX_SEG = 32;      // one lane per earlier segment in the chaining step
constexpr int SC_FULL = 148 * 16;   // warps that fill the GPU (16 per SM at 124 registers)

struct ScanParams {
    const void *z, *ig, *fg, *og;
    const float *c0, *n0, *m0;
    void *h;
    float *c1, *n1, *m1;
    float *loc_c, *loc_s;           // [BH][nseg][H] and [BH][nseg][4]: end state of every segment from an empty start
    int S, NH, H, nseg, seg_len;
    float eps, cap;
};

template <typename T, int VEC> struct Units {   // VEC adjacent units of one timestep
    uint4 raw;
    __device__ __forceinline__ void one() {
        const uint32_t w = sizeof(T) == 2 ? 0x3f803f80u : 0x3f800000u;
        raw = make_uint4(w, w, w, w);
    }
    __device__ __forceinline__ void load(const T *p) { raw = *reinterpret_cast<const uint4 *>(p); }
    __device__ __forceinline__ void get(float *f) const { unpack16<T>(raw, f); }
    static __device__ __forceinline__ void put(T *p, const float *f) { st16<T>(p, f); }
};
template <typename T> struct Units<T, 1> {      // widths or addresses that do not allow 16-byte accesses
    float v;
    __device__ __forceinline__ void one() { v = 1.f; }
    __device__ __forceinline__ void load(const T *p) { v = Elem<T>::ld(p); }
    __device__ __forceinline__ void get(float *f) const { f[0] = v; }
    static __device__ __forceinline__ void put(T *p, const float *f) { Elem<T>::st(p, f[0]); }
};

template <typename T, int VEC, bool FINAL>
__global__ void __launch_bounds__(32) slstm_scan_kernel(const ScanParams p) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x;
    const int seg = blockIdx.x % p.nseg, bh = blockIdx.x / p.nseg, b = bh / p.NH, hd = bh % p.NH;
    const int j0 = (blockIdx.y * 32 + lane) * VEC;
    const bool active = j0 < p.H;
    const int t0 = seg * p.seg_len, t1 = min(p.S, t0 + p.seg_len);
    const size_t tstride = (size_t)p.NH * p.H;
    const T *zp = static_cast<const T *>(p.z) + ((size_t)b * p.S * p.NH + hd) * p.H + j0;
    T *hp = static_cast<T *>(p.h) + ((size_t)b * p.S * p.NH + hd) * p.H + j0;
    const T *ig = static_cast<const T *>(p.ig), *fg = static_cast<const T *>(p.fg), *og = static_cast<const T *>(p.og);

    // ---- state at the start of the segment: c and n per unit (N: n without an initial one), m
    float c[VEC], m = -INFINITY, N = 0.f, Asum = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e) c[e] = 0.f;
    const bool has_state = FINAL && p.c0 != nullptr;
    float n[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) n[e] = 0.f;
    if (FINAL) {
        m = has_state ? p.m0[bh] : 0.f;
        if (has_state && active) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                c[e] = p.c0[(size_t)bh * p.H + j0 + e];
                n[e] = p.n0[(size_t)bh * p.H + j0 + e];
            }
        }
        if (seg > 0) {
            // lane l < seg holds segment l; suf = summed log forget gates of the segments between it and this one
            const float4 s4 = lane < seg ? reinterpret_cast<const float4 *>(p.loc_s)[(size_t)bh * p.nseg + lane]
                                         : make_float4(0.f, -INFINITY, 0.f, 0.f);
            float incl = s4.x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_down_sync(FULL, incl, o);
                if (lane + o < 32) incl += up;
            }
            const float total = __shfl_sync(FULL, incl, 0);
            // the EXCLUSIVE suffix as the neighbour's sum: taken as incl - s4.x, one large term (a gate closed for good)
            // would swallow the later ones, and an infinite one make it NaN
            float suf = __shfl_down_sync(FULL, incl, 1);
            if (lane == 31) suf = 0.f;
            const float ms = fmaxf(m + total, warp_max(s4.y + suf));
            const float w = lane < seg ? expf(s4.y + suf - ms) : 0.f;
            const float P = expf(m + total - ms);
            N = warp_sum(w * s4.z);
            m = ms;
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                c[e] *= P;
                n[e] = fmaf(P, n[e], N);
            }
            const float *lc = p.loc_c + (size_t)bh * p.nseg * p.H + j0;
#pragma unroll 8
            for (int l = 0; l < seg; ++l) {
                const float wl = __shfl_sync(FULL, w, l);
                if (active) {
                    float v[VEC];
                    if constexpr (VEC == 1) {
                        v[0] = lc[(size_t)l * p.H];
                    } else {
#pragma unroll
                        for (int e = 0; e < VEC; e += 4) {
                            const float4 q = *reinterpret_cast<const float4 *>(lc + (size_t)l * p.H + e);
                            v[e] = q.x; v[e + 1] = q.y; v[e + 2] = q.z; v[e + 3] = q.w;
                        }
                    }
#pragma unroll
                    for (int e = 0; e < VEC; ++e) c[e] = fmaf(wl, v[e], c[e]);
                }
            }
        }
    }

    Units<T, VEC> zb[SC_BATCH];
#pragma unroll
    for (int s = 0; s < SC_BATCH; ++s)
        if (!active) zb[s].one();           // lanes without a unit: a nonzero c keeps them off the slow path of the division
        else if (t0 + s < t1) zb[s].load(zp + (size_t)(t0 + s) * tstride);

    for (int tt = t0; tt < t1; tt += SC_TILE) {
        const int nt = min(SC_TILE, t1 - tt);
        // ---- lane = timestep: gates, stabiliser and normaliser scans
        const bool valid = lane < nt;
        const size_t g = ((size_t)b * p.S + tt + lane) * p.NH + hd;
        const float lf = valid ? logsigmoid(gate_softcap(Elem<T>::ld(fg + g), p.cap)) : 0.f;
        const float it = valid ? gate_softcap(Elem<T>::ld(ig + g), p.cap) : -INFINITY;
        const float ot = FINAL && valid ? sigmoidf(gate_softcap(Elem<T>::ld(og + g), p.cap)) : 0.f;
        float A = lf, Bm = it;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float Ap = __shfl_up_sync(FULL, A, o), Bp = __shfl_up_sync(FULL, Bm, o);
            if (lane >= o) { Bm = fmaxf(Bp + A, Bm); A += Ap; }
        }
        const float mt = fmaxf(m + A, Bm);
        float mp = __shfl_up_sync(FULL, mt, 1);
        if (lane == 0) mp = m;
        const bool none = mt == -INFINITY;          // no input yet (empty start): nothing to carry
        const float fe = none ? 1.f : expf(mp + lf - mt), ie = none ? 0.f : expf(it - mt);
        float pt = fe, nn = ie;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float pp = __shfl_up_sync(FULL, pt, o), np = __shfl_up_sync(FULL, nn, o);
            if (lane >= o) { nn = fmaf(pt, np, nn); pt *= pp; }
        }
        const float Nt = fmaf(pt, N, nn);
        const float rt = has_state ? ot : ot / (fabsf(Nt) + p.eps);
        // ---- lane = units: walk the tile, the next batch of z in flight
        for (int s0 = 0; s0 < nt; s0 += SC_BATCH) {
            Units<T, VEC> zc[SC_BATCH];
#pragma unroll
            for (int s = 0; s < SC_BATCH; ++s) {
                zc[s] = zb[s];
                const int tn = tt + s0 + SC_BATCH + s;
                if (active && tn < t1) zb[s].load(zp + (size_t)tn * tstride);
            }
#pragma unroll
            for (int s = 0; s < SC_BATCH; ++s) {
                if (s0 + s < nt) {                  // uniform over the warp
                    const float f = __shfl_sync(FULL, fe, s0 + s), i = __shfl_sync(FULL, ie, s0 + s);
                    float zf[VEC];
                    zc[s].get(zf);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) c[e] = fmaf(f, c[e], i * tanhf(zf[e]));
                    if (FINAL) {
                        const float r = __shfl_sync(FULL, rt, s0 + s);
                        float hv[VEC];
                        if (has_state) {
#pragma unroll
                            for (int e = 0; e < VEC; ++e) {
                                n[e] = fmaf(f, n[e], i);
                                hv[e] = r * c[e] / (fabsf(n[e]) + p.eps);
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < VEC; ++e) hv[e] = r * c[e];
                        }
                        if (active) Units<T, VEC>::put(hp + (size_t)(tt + s0 + s) * tstride, hv);
                    }
                }
            }
        }
        m = __shfl_sync(FULL, mt, 31);              // lanes past the end carry the last valid step on unchanged
        N = __shfl_sync(FULL, Nt, 31);
        Asum += __shfl_sync(FULL, A, 31);
    }

    if (!FINAL) {
        if (active) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) p.loc_c[((size_t)bh * p.nseg + seg) * p.H + j0 + e] = c[e];
        }
        if (blockIdx.y == 0 && lane == 0)
            reinterpret_cast<float4 *>(p.loc_s)[(size_t)bh * p.nseg + seg] = make_float4(Asum, m, N, 0.f);
    } else if (seg == p.nseg - 1) {
        if (active) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                p.c1[(size_t)bh * p.H + j0 + e] = c[e];
                p.n1[(size_t)bh * p.H + j0 + e] = has_state ? n[e] : N;
            }
        }
        if (blockIdx.y == 0 && lane == 0) p.m1[bh] = m;
    }
}

// Segments of the sequence.  One pass while it has a third of the warps that fill the GPU: two segments would double
// the warps but read z twice.  Below that as many as fill it, each at least one gate tile long.
int plan(int64_t bh, int S, int H, int dtype, int &seg_len) {
    const int64_t slices = (H * (dtype == XLSTM_BF16 ? 2 : 4) + 511) / 512;
    int64_t nseg = SC_FULL / (bh * slices);
    if (nseg > SC_MAX_SEG) nseg = SC_MAX_SEG;
    if (nseg > S / SC_TILE) nseg = S / SC_TILE;
    if (nseg < 3) nseg = 1;
    seg_len = (int)(((S + nseg - 1) / nseg + SC_TILE - 1) / SC_TILE * SC_TILE);
    return (S + seg_len - 1) / seg_len;
}

size_t scan_workspace(int64_t bh, int H, int nseg) { return nseg > 1 ? (size_t)bh * nseg * (4 + (size_t)H) * sizeof(float) : 0; }

template <typename T, int VEC> int launch(ScanParams p, int64_t bh, cudaStream_t st) {
    const unsigned slices = (unsigned)((p.H + 32 * VEC - 1) / (32 * VEC));
    const dim3 grid((unsigned)(bh * p.nseg), slices);
    if (p.nseg > 1) {
        slstm_scan_kernel<T, VEC, false><<<grid, 32, 0, st>>>(p);
        if (cudaGetLastError() != cudaSuccess) return XLSTM_ERR_CUDA;
    }
    slstm_scan_kernel<T, VEC, true><<<grid, 32, 0, st>>>(p);
    return launch_status();
}

int scan(const void *z, const void *ig, const void *fg, const void *og, const float *c0, const float *n0, const float *m0,
         void *h, float *c1, float *n1, float *m1, int B, int S, int NH, int H, float eps, float cap, int dtype, void *ws,
         size_t ws_bytes, cudaStream_t st) {
    if (!z || !ig || !fg || !og || !h || !c1 || !n1 || !m1) return XLSTM_ERR_INVALID;
    if (B <= 0 || S <= 0 || NH <= 0 || H <= 0) return XLSTM_ERR_INVALID;
    if (c0 && (!n0 || !m0)) return XLSTM_ERR_INVALID;
    if (dtype != XLSTM_F32 && dtype != XLSTM_BF16) return XLSTM_ERR_UNSUPPORTED;
    const int64_t bh = (int64_t)B * NH;
    ScanParams p{z, ig, fg, og, c0, n0, m0, h, c1, n1, m1, nullptr, nullptr, S, NH, H, 1, S, eps, cap};
    p.nseg = plan(bh, S, H, dtype, p.seg_len);
    // an in-place state is read by every segment and written by the last one: one pass then, as without scratch
    const bool alias = c0 && (c1 == c0 || n1 == n0);
    if (alias || !ws || ws_bytes < scan_workspace(bh, H, p.nseg) || (reinterpret_cast<uintptr_t>(ws) & 15u)) {
        p.nseg = 1;
        p.seg_len = S;
    }
    p.loc_s = static_cast<float *>(ws);
    p.loc_c = p.loc_s ? p.loc_s + (size_t)bh * p.nseg * 4 : nullptr;
    if (bh * p.nseg > 2147483647LL || (H + 31) / 32 > 65535) return XLSTM_ERR_UNSUPPORTED;
    // One pass of few warps is bound by the instructions of a step in a warp: one unit a lane then, in place of 4 or 8.  Without a
    // state (no quotient per unit) that pays up to about one warp per SM (bf16, 128 warps of 256 units: 310 -> 259 us, 512: 310
    // -> 352), with one as long as the narrow warps do not fill the GPU several times over (128: 629 -> 302, 512: 630 -> 423).
    const int64_t warps = bh * (((int64_t)H * (dtype == XLSTM_BF16 ? 2 : 4) + 511) / 512);
    const bool narrow = p.nseg == 1 && warps < (c0 ? SC_FULL / 3 : SC_FULL / 16);
    const bool al = !narrow && ((reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(h)) & 15u) == 0;
    if (dtype == XLSTM_F32) return al && H % 4 == 0 ? launch<float, 4>(p, bh, st) : launch<float, 1>(p, bh, st);
    return al && H % 8 == 0 ? launch<__nv_bfloat16, 8>(p, bh, st) : launch<__nv_bfloat16, 1>(p, bh, st);
}

}  // namespace
}  // namespace xl

extern "C" size_t xlstm_slstm_scan_workspace_bytes(int B, int S, int NH, int H, int dtype) {
    if (B <= 0 || S <= 0 || NH <= 0 || H <= 0) return 0;
    int seg_len;
    const int64_t bh = (int64_t)B * NH;
    return xl::scan_workspace(bh, H, xl::plan(bh, S, H, dtype, seg_len));
}

extern "C" int xlstm_slstm_scan(const void *z, const void *ig, const void *fg, const void *og, const float *c0,
                                const float *n0, const float *m0, void *h, float *c1, float *n1, float *m1, int B,
                                int S, int NH, int H, float eps, int dtype, void *stream) {
    return xl::scan(z, ig, fg, og, c0, n0, m0, h, c1, n1, m1, B, S, NH, H, eps, 0.f, dtype, nullptr, 0,
                    static_cast<cudaStream_t>(stream));
}

extern "C" int xlstm_slstm_scan_ex(const void *z, const void *ig, const void *fg, const void *og, const float *c0,
                                   const float *n0, const float *m0, void *h, float *c1, float *n1, float *m1, int B,
                                   int S, int NH, int H, float eps, float gate_cap, int dtype, void *workspace,
                                   size_t workspace_bytes, void *stream) {
    return xl::scan(z, ig, fg, og, c0, n0, m0, h, c1, n1, m1, B, S, NH, H, eps, gate_cap, dtype, workspace, workspace_bytes,
                    static_cast<cudaStream_t>(stream));
}
