// Gate scalars of 32 consecutive tokens, one lane each, for the kernels that work in fp32.
#pragma once
#include "mlstm_chunkwise.cuh"

namespace xl {

// Gate scalars of 32 tokens, lane = token: inclusive sums b (double), u = i - b, running maximum of u
struct GateTile {
    double b, u, mx;
};
// the raw gates of one token: loaded ahead of their use, the scan below is latency enough
struct GateRaw {
    float i, f;
    bool valid;
};
template <typename T> __device__ __forceinline__ GateRaw gate_load(const ChunkwiseParams &p, int bb, int hd, int t) {
    GateRaw r{0.f, 0.f, t < p.S};
    if (r.valid) {
        const int64_t off = bb * p.sg[0] + hd * p.sg[1] + (int64_t)t * p.sg[2];
        r.i = Elem<T>::ld(static_cast<const T *>(p.ig) + off);
        r.f = Elem<T>::ld(static_cast<const T *>(p.fg) + off);
    }
    return r;
}
__device__ __forceinline__ GateTile gate_tile(const GateRaw &r, float cap, int lane, double b_in) {
    const float lf = r.valid ? logsigmoid(gate_softcap(r.f, cap)) : 0.f;
    const float it = r.valid ? gate_softcap(r.i, cap) : -INFINITY;
    GateTile g;
    g.b = (double)lf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, g.b, o);
        if (lane >= o) g.b += up;
    }
    g.b += b_in;
    g.u = (double)it - g.b;
    g.mx = g.u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, g.mx, o);
        if (lane >= o) g.mx = fmax(g.mx, up);
    }
    return g;
}

}  // namespace xl
