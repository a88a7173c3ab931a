// tc_cluster.cuh -- helpers of the SM-pair (cta_group::2) tensor-core
// kernels: cluster rank and barrier, remote mbarrier arrivals, and the
// pair MMAs of one stage and their multicast commit.
#pragma once

#include "tc_common.cuh"

namespace chx {
namespace tc {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
}
// Shared-memory address of the same variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// One lane of a converged warp (the same one each time).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p;
}

// The four MMAs of one stage, issued by the lane with lead = 1 of a converged
// warp.  acc = 0 starts new sums.  Re and Im MMAs alternate, so that an MMA does not wait
// for the previous one's update of its accumulator.
//   Re (d0) = R X + I Y,   Im (d1) = I X + N Y
__device__ __forceinline__ void mma_stage_pair(uint32_t lead, uint32_t d0, uint32_t d1, uint64_t r,
                                               uint64_t i, uint64_t n, uint64_t x, uint64_t y,
                                               uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "setp.ne.b32 p, %9, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::i8 [%1], %3, %6, %8, p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::i8 [%2], %4, %6, %8, p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::i8 [%1], %4, %7, %8, t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::i8 [%2], %5, %7, %8, t;\n\t}" ::"r"(lead),
        "r"(d0), "r"(d1), "l"(r), "l"(i), "l"(n), "l"(x), "l"(y), "r"(idesc), "r"(acc)
        : "memory");
}
// Commit of the lead lane's MMAs, arriving on the barrier at `bar` in both CTAs.
__device__ __forceinline__ void mma_commit_pair(uint32_t lead, uint32_t bar) {
    const uint16_t mask = 0x3;
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster"
        ".multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar),
        "h"(mask), "r"(lead)
        : "memory");
}

}  // namespace tc
}  // namespace chx
