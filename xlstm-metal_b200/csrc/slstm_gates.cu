// The three gate projections of the packaged sLSTM in one pass over x (bf16):
//   xc[t] = silu(bias + sum_j w[., j] x[t - 3 + j])            causal depthwise convolution, 4 taps, rounded to bf16
//   i, f  = softcap(W_{i,f} xc[t] + b)     o = softcap(W_o x[t] + b)      NH <= 4 scalars a token each
// As separate launches (convolution, three GEMMs of 4 columns, three soft-caps) the gates of 8192 tokens of 4096 channels took
// 137 us: the convolution's result was written and read back twice for 12 numbers a token.  Here it exists only as MMA operands.
//
// One CTA per 16 J tokens; its 12 warps take the 32-channel blocks in turn and meet in shared memory.  A contraction may take
// its index in any order as long as both operands agree, and so may the rows: lane (g, c) of mma.sync.m16n8k16 owns the 2 J
// CONSECUTIVE tokens 2 J g .. and the 8 consecutive channels 8 c .. of the block, so the convolution runs down a window in
// registers, every row arrives by 16-byte loads, and its results are the A fragments as they stand.  The columns are the
// heads: one product with (i, f) of xc, one with o of x.
// Bound by issue (about 35 instructions per 4 elements, the window and the SiLU) and by the latency of 2 J + 3 loads a block;
// HBM would allow 10 us at the size above, it takes 36.  J = 1 gives the SMs more CTAs where there are few tokens.
#include "mma_sync.cuh"
#include "vec16.cuh"

namespace xl {
namespace {

constexpr int SG_WARPS = 12, SG_NH = 4;

struct GateArgs {
    const __nv_bfloat16 *x, *cw, *cb, *w[3], *b[3];   // i, f, o
    __nv_bfloat16 *out[3];
    int S, C, NH;
    float cap;
};

// SiLU rounded to bf16: the sigmoid from one tanh.approx, as the convolution kernel takes it
__device__ __forceinline__ float silu_bf16(float x) {
    float t;
    const float hx = 0.5f * x;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(hx));
    return fmaf(hx, t, hx);
}

template <int J> __global__ void __launch_bounds__(SG_WARPS * 32, 1) slstm_gates_kernel(const GateArgs p) {
    constexpr int RUN = 2 * J, TOK = 16 * J;
    __shared__ float s_part[SG_WARPS / 2][TOK][17];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int t0 = blockIdx.x * TOK, b = blockIdx.y, C = p.C;
    const int blocks = C >> 5;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const __nv_bfloat16 *xb = p.x + (size_t)b * p.S * C;
    // columns of the two products: 0..3 = i and 4..7 = f of head n & 3; o of head n
    const bool if_ok = (g & 3) < p.NH, o_ok = g < p.NH;
    const __nv_bfloat16 *wif = (g < 4 ? p.w[0] : p.w[1]) + (size_t)(if_ok ? g & 3 : 0) * C;
    const __nv_bfloat16 *wo = p.w[2] + (size_t)(o_ok ? g : 0) * C;
    const int tf = t0 + RUN * g;                                  // first token of this lane

    float aif[J][4], ao[J][4];
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) aif[j][e] = ao[j][e] = 0.f;

    for (int blk = warp; blk < blocks; blk += SG_WARPS) {
        const int c0 = blk * 32 + c * 8;
        uint4 raw[RUN + 3];                                       // tokens tf - 3 .. tf + RUN - 1
#pragma unroll
        for (int r = 0; r < RUN + 3; ++r) {
            const int t = tf - 3 + r;
            raw[r] = t >= 0 && t < p.S ? *reinterpret_cast<const uint4 *>(xb + (size_t)t * C + c0) : zero;
        }
        const uint4 bif = if_ok ? *reinterpret_cast<const uint4 *>(wif + c0) : zero;
        const uint4 bo = o_ok ? *reinterpret_cast<const uint4 *>(wo + c0) : zero;
        uint4 taps[4];                                            // [8 channels][4 taps]: a register holds 2 taps of a channel
#pragma unroll
        for (int j = 0; j < 4; ++j) taps[j] = *reinterpret_cast<const uint4 *>(p.cw + (size_t)c0 * 4 + j * 8);
        float wt[4][8], bias[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {                             // channels 2 j and 2 j + 1
            float v[8];
            unpack16<__nv_bfloat16>(taps[j], v);
#pragma unroll
            for (int k = 0; k < 4; ++k) { wt[k][2 * j] = v[k]; wt[k][2 * j + 1] = v[4 + k]; }
        }
        if (p.cb) ld16<__nv_bfloat16>(p.cb + c0, bias);
        else
#pragma unroll
            for (int e = 0; e < 8; ++e) bias[e] = 0.f;
        float win[4][8];                                          // the row of token tf - 3 + r is in slot r & 3
#pragma unroll
        for (int r = 0; r < 3; ++r) unpack16<__nv_bfloat16>(raw[r], win[r]);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            uint4 xc[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {                         // token tf + 2 j + h: rows 2 j + h .. + 3
                const int r0 = 2 * j + h;
                unpack16<__nv_bfloat16>(raw[r0 + 3], win[(r0 + 3) & 3]);
                float acc[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] = bias[e];
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[e] = fmaf(wt[k][e], win[(r0 + k) & 3][e], acc[e]);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] = silu_bf16(acc[e]);
                st16<__nv_bfloat16>(reinterpret_cast<__nv_bfloat16 *>(&xc[h]), acc);
            }
            // rows g and g + 8 of the tile: tokens tf + 2 j and tf + 2 j + 1
            const uint4 x0 = raw[2 * j + 3], x1 = raw[2 * j + 4];
            mma_m16n8k16(aif[j], xc[0].x, xc[1].x, xc[0].y, xc[1].y, bif.x, bif.y);
            mma_m16n8k16(aif[j], xc[0].z, xc[1].z, xc[0].w, xc[1].w, bif.z, bif.w);
            mma_m16n8k16(ao[j], x0.x, x1.x, x0.y, x1.y, bo.x, bo.y);
            mma_m16n8k16(ao[j], x0.z, x1.z, x0.w, x1.w, bo.z, bo.w);
        }
    }
    // the upper half of the warps hands its sums to the lower half, whose parts are added in order below
    auto part = [&](auto &&op) {
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float *row = s_part[warp % (SG_WARPS / 2)][RUN * g + 2 * j + (e >> 1)] + 2 * c + (e & 1);
                op(row[0], aif[j][e]);
                op(row[8], ao[j][e]);
            }
    };
    if (warp >= SG_WARPS / 2) part([](float &s, float v) { s = v; });
    __syncthreads();
    if (warp < SG_WARPS / 2) part([](float &s, float v) { s += v; });
    __syncthreads();
    for (int e = tid; e < TOK * 12; e += SG_WARPS * 32) {
        const int t = e / 12, n = e % 12, head = n & 3;
        if (t0 + t >= p.S || head >= p.NH) continue;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < SG_WARPS / 2; ++w) s += s_part[w][t][n];
        const int gate = n >> 2;
        // rounded as a Linear's output, then capped
        s = __bfloat162float(__float2bfloat16_rn(s + __bfloat162float((gate == 0 ? p.b[0] : gate == 1 ? p.b[1] : p.b[2])[head])));
        if (p.cap > 0.f) s = p.cap * tanhf(s * (1.0f / p.cap));
        (gate == 0 ? p.out[0] : gate == 1 ? p.out[1] : p.out[2])[((size_t)b * p.S + t0 + t) * p.NH + head] = __float2bfloat16_rn(s);
    }
}

}  // namespace
}  // namespace xl

extern "C" int xlstm_slstm_gates(const void *x, const void *conv_w, const void *conv_b, const void *const *w, const void *const *b,
                                 void *const *gates, int B, int S, int C, int K, int NH, float gate_cap, int dtype, void *stream) {
    if (B < 0 || S < 0 || C <= 0 || NH <= 0 || !w || !b || !gates) return XLSTM_ERR_INVALID;
    if (dtype != XLSTM_BF16 || K != 4 || NH > xl::SG_NH || C % 32 || B > 65535) return XLSTM_ERR_UNSUPPORTED;
    if (B == 0 || S == 0) return XLSTM_OK;
    if (!x || !conv_w) return XLSTM_ERR_INVALID;
    uintptr_t al = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(conv_w) | reinterpret_cast<uintptr_t>(conv_b);
    xl::GateArgs p;
    p.x = static_cast<const __nv_bfloat16 *>(x);
    p.cw = static_cast<const __nv_bfloat16 *>(conv_w);
    p.cb = static_cast<const __nv_bfloat16 *>(conv_b);
    for (int k = 0; k < 3; ++k) {
        if (!w[k] || !b[k] || !gates[k]) return XLSTM_ERR_INVALID;
        al |= reinterpret_cast<uintptr_t>(w[k]);
        p.w[k] = static_cast<const __nv_bfloat16 *>(w[k]);
        p.b[k] = static_cast<const __nv_bfloat16 *>(b[k]);
        p.out[k] = static_cast<__nv_bfloat16 *>(gates[k]);
    }
    if (al & 15u) return XLSTM_ERR_UNSUPPORTED;
    p.S = S; p.C = C; p.NH = NH; p.cap = gate_cap;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // 64 tokens a CTA (11 rows read for 8) once that fills three quarters of the SMs, else 16 (5 rows for 2)
    if ((int64_t)B * ((S + 63) / 64) >= 111) xl::slstm_gates_kernel<4><<<dim3((S + 63) / 64, B), xl::SG_WARPS * 32, 0, st>>>(p);
    else xl::slstm_gates_kernel<1><<<dim3((S + 15) / 16, B), xl::SG_WARPS * 32, 0, st>>>(p);
    return xl::launch_status();
}
