// Pieces shared by the kernels of the block-diagonal recurrent sLSTM whose CTAs exchange h_t through the shared memory of
// their cluster: remote stores that complete bytes on the receiver's mbarrier, the bounded wait for them.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "cp_async.cuh"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace xl {
namespace rec {
using tc::smem_u32;

// shared::cta address of this CTA -> shared::cluster address of the same offset in CTA `rank`
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// 16 bytes from registers into a CTA of the cluster, counted on that CTA's mbarrier
__device__ __forceinline__ void st_async16(uint32_t dst, uint32_t bar, const uint32_t (&w)[4]) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];"
                 ::"r"(dst), "r"(bar), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// bounded wait for bytes that other CTAs of the cluster write (hence the cluster-scope acquire); see tc::mbar_wait
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.b32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(ns) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_wait_cluster(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
    if (mbar_try_wait_cluster(bar, parity, 20000u)) return;
    const long long t0 = clock64();
    while (!mbar_try_wait_cluster(bar, parity, 20000u)) {
        if (*abort_flag) return;
        if (clock64() - t0 > XL_TC_WAIT_CLOCKS) { *abort_flag = 1; return; }
    }
}

// after a wait that gave up: time for stores still under way to land before the CTA may leave (normally every one has
// been waited for)
__device__ __forceinline__ void drain_after_abort() {
    for (int x = 0; x < 200; ++x) __nanosleep(1000);
}

}  // namespace rec
}  // namespace xl
