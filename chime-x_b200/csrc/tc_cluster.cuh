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
// The loads of one step (packed y tile, the x tiles of lanes 0 and 1 where
// act0 / act1 are set, channel fc, sample t) and the byte count its barrier
// expects, issued by the lead lane.
__device__ __forceinline__ void tma_load_step(uint32_t lead, uint32_t bar, uint32_t bytes,
                                              uint32_t ydst, const CUtensorMap *ymap, int y,
                                              uint32_t xdst0, uint32_t xdst1,
                                              const CUtensorMap *xmap, int x0, int x1,
                                              uint32_t act0, uint32_t act1, int fc, int t) {
    asm volatile(
        "{\n\t.reg .pred q, a, b;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "setp.ne.and.b32 a, %11, 0, q;\n\t"
        "setp.ne.and.b32 b, %12, 0, q;\n\t"
        "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n\t"
        "@q cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%3], [%4, {%5, %13, %14}], [%1];\n\t"
        "@a cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%6], [%8, {%9, %13, %14}], [%1];\n\t"
        "@b cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%7], [%8, {%10, %13, %14}], [%1];\n\t}" ::"r"(lead),
        "r"(bar), "r"(bytes), "r"(ydst), "l"(reinterpret_cast<uint64_t>(ymap)), "r"(y), "r"(xdst0),
        "r"(xdst1), "l"(reinterpret_cast<uint64_t>(xmap)), "r"(x0), "r"(x1), "r"(act0), "r"(act1),
        "r"(fc), "r"(t)
        : "memory");
}

// The MMAs of one step, issued by the lead lane of a converged warp.  A y row
// used more than once stays in the tensor core's A collector from its fill to its
// last use; MMAs into the same accumulator never follow each other.  acc = 0
// starts new sums.
//   Re (d) = R X + I Y,   Im (d + 128) = I X + N Y
#define CHX_MMA "tcgen05.mma.cta_group::2.kind::i8"
#define CHX_FILL ".collector::a::fill"
#define CHX_USE ".collector::a::use"
#define CHX_LAST ".collector::a::lastuse"
__device__ __forceinline__ void mma_step_one(uint32_t lead, uint32_t d, uint64_t r, uint64_t i,
                                             uint64_t n, uint64_t x, uint64_t y, uint32_t idesc,
                                             uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred q, p, t;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "setp.ne.b32 p, %9, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q " CHX_MMA " [%1], %3, %6, %8, p;\n\t"
        "@q " CHX_MMA CHX_FILL " [%2], %4, %6, %8, p;\n\t"
        "@q " CHX_MMA CHX_LAST " [%1], %4, %7, %8, t;\n\t"
        "@q " CHX_MMA " [%2], %5, %7, %8, t;\n\t}" ::"r"(lead),
        "r"(d), "r"(d + 128), "l"(r), "l"(i), "l"(n), "l"(x), "l"(y), "r"(idesc), "r"(acc)
        : "memory");
}
// Both lanes: lane 1's accumulators at d + 256, its x rows dx (descriptor
// units) after lane 0's.
__device__ __forceinline__ void mma_step_two(uint32_t lead, uint32_t d, uint64_t r, uint64_t i,
                                             uint64_t n, uint64_t x, uint64_t y, uint32_t dx,
                                             uint32_t idesc, uint32_t acc0, uint32_t acc1) {
    asm volatile(
        "{\n\t.reg .pred q, p, u, t;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "setp.ne.b32 p, %13, 0;\n\t"
        "setp.ne.b32 u, %14, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q " CHX_MMA CHX_FILL " [%1], %5, %8, %12, p;\n\t"
        "@q " CHX_MMA CHX_LAST " [%3], %5, %10, %12, u;\n\t"
        "@q " CHX_MMA CHX_FILL " [%2], %6, %8, %12, p;\n\t"
        "@q " CHX_MMA CHX_USE " [%1], %6, %9, %12, t;\n\t"
        "@q " CHX_MMA CHX_USE " [%4], %6, %10, %12, u;\n\t"
        "@q " CHX_MMA CHX_LAST " [%3], %6, %11, %12, t;\n\t"
        "@q " CHX_MMA CHX_FILL " [%2], %7, %9, %12, t;\n\t"
        "@q " CHX_MMA CHX_LAST " [%4], %7, %11, %12, t;\n\t}" ::"r"(lead),
        "r"(d), "r"(d + 128), "r"(d + 256), "r"(d + 384), "l"(r), "l"(i), "l"(n), "l"(x), "l"(y),
        "l"(x + dx), "l"(y + dx), "r"(idesc), "r"(acc0), "r"(acc1)
        : "memory");
}
#undef CHX_MMA
#undef CHX_FILL
#undef CHX_USE
#undef CHX_LAST
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
