// tc_small_correlator.cu -- tcgen05 kind::i8 correlator for channels of at
// most 128 elements (cta_group::1).
//
// Such a channel is one tile against itself: the y and the x tile are the same
// 128 bytes per sample, so every packed tile is loaded and converted once and
// the rows R = yr, I = yi serve as the y and the x operand (both scaled by 4, so
// that R R + I I and I R + N I with N = -yr are 16 times the visibility, as in
// the other kernels; tc_correlator.cu).  MAP_PACKED, whose y and x imaginary
// rows differ, stores a fourth row.  N is the element count (a multiple of 32):
// no columns are computed in vain, and lanes whose 16 elements lie outside the
// channel neither load nor store.
//
// Two rows (TWO).  N I is the transpose of -I R, so launches of long units neither
// store N nor multiply by it: K = I R is accumulated, and the epilogue writes
// K - K^T, taking the transposed blocks through shared memory.  A step has three
// MMAs and two thirds of the operand stores and reads; the epilogue reads K twice
// and meets at two barriers.  Per call (us, three rows / two): E = 128, F = 148,
// T = 4096 32.1 / 27.3, E = 96, F = 64, T = 4096 16.3 / 14.7, E = 64, F = 148, T = 4096
// 25.9 / 22.2, E = 96, F = 400, T = 768 (24 steps a unit) 19.6 / 18.8, E = 128,
// F = 160, T = 768 15.6 / 14.4; but E = 96, F = 400, T = 128 (4 steps) 7.9 / 9.8, where
// the drain sets the pace.  Chosen per launch: choosing per unit in one kernel lost
// most of the gain (E = 96, F = 64, T = 4096 16.8).
//
// Roles and hand-over are those of the SM-pair kernel (tc_pair_correlator.cu):
// warps 0-15 unpack in four groups, step s in group s % kGroups; 16 TMA
// producer; 17 MMA issuer; 18-25 epilogue.  TMEM holds two accumulator buffers, so
// a unit's drain overlaps the next unit's MMAs.
//
// What bounds it: shared memory, whose operand stores and reads take about 400
// cycles per step at N = 128 with three rows (430 measured; the step's four M128
// MMAs need 2 N) and 290 with two, and at small N the unpack warps' latency.
// Before, the 1-SM kernel of tc_correlator.cu converted the tile twice (y and x),
// handed its operands over from a lane == 0 branch and drained with its unpack
// warps: about 1000 cycles per step.  Per call (us, before / now): E = 96, F = 64,
// T = 4096 43.1 / 14.7, E = 128, F = 148, T = 4096 72.1 / 27.3, E = 32, F = 148,
// T = 4096 70.0 / 19.3, E = 96, F = 1, T = 64 6.9 / 3.9.
#include "tc_common.cuh"

#include <string.h>

namespace chx {

namespace {

using namespace tc;

constexpr int kStageSamples = kUnitStageSamples;
constexpr int kOpSlots = 6;
constexpr int kUnpackWarps = 16;
constexpr int kGroups = 4;
constexpr int kGroupWarps = kUnpackWarps / kGroups;
constexpr int kPkSlots = 10;  // see tc_pair_correlator.cu
static_assert(kPkSlots >= kGroups + kOpSlots && kOpSlots >= kGroups, "parity of the rings");
constexpr int kTileBytes = kStageSamples * 128;
constexpr int kRowsMax = 4;
constexpr int kOpBytesMax = kRowsMax * kTileBytes;
constexpr int kProducerWarp = 16;
constexpr int kMmaWarp = 17;
constexpr int kEpiWarp0 = 18;
constexpr int kEpiWarps = 8;
constexpr int kEpiTiles = 2;
constexpr int kThreads = (kEpiWarp0 + kEpiWarps) * 32;
constexpr int kTmemCols = 512;  // two buffers of 128 Re and 128 Im columns
constexpr uint32_t kScale = 2;  // rows scaled by 2^kScale

constexpr int kOffOp = 0;
constexpr int kOffPk = kOffOp + kOpSlots * kOpBytesMax;
constexpr int kOffStage = kOffPk + kPkSlots * kTileBytes;
constexpr int kOffBars = kOffStage + kEpiWarps * kEpiTiles * 4096;
constexpr int kSmemBytes = kOffBars + 512 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory per CTA");
// Two-row operands leave half of their area to the transposed blocks of K: ten of
// 32 rows of 33 words (no bank conflicts by rows or by columns).
constexpr int kOffSwap = kOffOp + kOpSlots * 2 * kTileBytes;
constexpr int kSwapPitch = 33;
constexpr int kSwapWords = 32 * kSwapPitch;
static_assert(kOffSwap + 10 * kSwapWords * 4 <= kOffPk, "transposed blocks");

constexpr int kBarFullPk = 0;
constexpr int kBarEmptyPk = kBarFullPk + kPkSlots;
constexpr int kBarFullOp = kBarEmptyPk + kPkSlots;
constexpr int kBarEmptyOp = kBarFullOp + kOpSlots;
constexpr int kBarAccFull = kBarEmptyOp + kOpSlots;  // per buffer
constexpr int kBarAccEmpty = kBarAccFull + 2;        // per buffer
constexpr int kBarDrain = kBarAccEmpty + 2;
constexpr int kBarCount = kBarDrain + 1;
static_assert(kBarCount * 8 + 8 <= 512, "barrier block");

struct KParams {
    const ChanDesc *chans;
    const Unit *units;
    const int *cta_offsets;  // CTA b takes units [cta_offsets[b], cta_offsets[b+1])
    int use_param_map;
    int static_tables;  // the tables were complete before the launch
    int after_zero;     // the previous launch is the one zeroing the output
    int ut;
    int accumulate;
    uint32_t one;  // 1 (YScale)
    int *err;
};

// One packed tile and the byte count its barrier expects, by the lead lane.
__device__ __forceinline__ void tma_load_tile(uint32_t lead, uint32_t bar, uint32_t dst,
                                              const CUtensorMap *map, int fc, int t) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n\t"
        "@q cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%3], [%4, {%5, %6, %7}], [%1];\n\t}" ::"r"(lead),
        "r"(bar), "r"(kTileBytes), "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(fc),
        "r"(t)
        : "memory");
}
// The MMAs of one step, by the lead lane of a converged warp; Re and Im
// alternate, I stays in the A collector for its second use.
//   Re (d) = R X + I Y,   Im (d + 128) = I X + N Y
__device__ __forceinline__ void mma_step(uint32_t lead, uint32_t d, uint64_t r, uint64_t i,
                                         uint64_t n, uint64_t x, uint64_t y, uint32_t idesc,
                                         uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred q, p, t;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "setp.ne.b32 p, %9, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%1], %3, %6, %8, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8.collector::a::fill [%2], %4, %6, %8, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8.collector::a::lastuse [%1], %4, %7, %8, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%2], %5, %7, %8, t;\n\t}" ::"r"(lead),
        "r"(d), "r"(d + 128), "l"(r), "l"(i), "l"(n), "l"(x), "l"(y), "r"(idesc), "r"(acc)
        : "memory");
}
// The same for one operand set of two rows:
//   Re (d) = R R + I I,   K (d + 128) = I R
__device__ __forceinline__ void mma_step_self(uint32_t lead, uint32_t d, uint64_t r, uint64_t i,
                                              uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred q, p, t;\n\t"
        "setp.ne.b32 q, %0, 0;\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%1], %3, %3, %5, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8.collector::a::fill [%2], %4, %3, %5, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8.collector::a::lastuse [%1], %4, %4, %5, t;\n\t}" ::"r"(
            lead),
        "r"(d), "r"(d + 128), "l"(r), "l"(i), "r"(idesc), "r"(acc)
        : "memory");
}
// Barrier of the epilogue warps; true if every thread passed true.
__device__ __forceinline__ bool epi_barrier(bool ok) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, a;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred a, 1, %2, p;\n\t"
        "selp.b32 %0, 1, 0, a;\n\t}"
        : "=r"(all)
        : "r"(ok ? 1u : 0u), "n"(kEpiWarps * 32)
        : "memory");
    __syncwarp();
    return all != 0;
}
__device__ __forceinline__ void mma_commit_lead(uint32_t lead, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(
            bar),
        "r"(lead)
        : "memory");
}

template <int MAP, bool TWO>
__global__ void __launch_bounds__(kThreads, 1)
tc_small_kernel(const __grid_constant__ CUtensorMap pmap, const __grid_constant__ CUtensorMap pomap,
                const KParams P) {
    static_assert(!TWO || MAP != MAP_PACKED, "two rows need equal y and x rows");
    constexpr int kRows = TWO ? 2 : MAP == MAP_PACKED ? 4 : 3;  // R, I, N, the x imaginary row
    constexpr int kOpBytes = kRows * kTileBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = smem_u32(smem);
    const uint32_t op = sbase + kOffOp, pk = sbase + kOffPk, bars = sbase + kOffBars;
    auto bar = [&](int i) { return bars + 8 * i; };
    volatile uint32_t *tmem_slot =
        reinterpret_cast<volatile uint32_t *>(smem + kOffBars + 8 * kBarCount);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // warp-uniform
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPkSlots; s++) {
            mbar_init(bar(kBarFullPk + s), 1);
            mbar_init(bar(kBarEmptyPk + s), kGroupWarps);
        }
        for (int s = 0; s < kOpSlots; s++) {
            mbar_init(bar(kBarFullOp + s), kGroupWarps);
            mbar_init(bar(kBarEmptyOp + s), 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(bar(kBarAccFull + a), 1);
            mbar_init(bar(kBarAccEmpty + a), kEpiWarps);
        }
        mbar_init(bar(kBarDrain), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Set-up overlaps the previous kernel of the stream; tables that the stream
    // itself writes are read only after that kernel.
    if (!P.static_tables) pdl_wait();
    const int first = P.cta_offsets[blockIdx.x], last = P.cta_offsets[blockIdx.x + 1];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // The zeroing kernel started after all earlier work had ended: only the
    // output waits for it.
    if (!P.after_zero || warp >= kEpiWarp0) pdl_wait();

    // Stages of a unit, the same for the whole warp.
    auto stages = [&](int u) {
        return __shfl_sync(0xffffffffu,
                           (P.units[u].t1 - P.units[u].t0 + kStageSamples - 1) / kStageSamples, 0);
    };

    if (warp == kProducerWarp) {
        // ------------------------------------------------------ TMA producer
        const uint32_t lead = elect_one();
        uint32_t g = 0, s = 0, ph = 0;  // steps issued, packed slot, its phase
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const Unit U = P.units[u];
            const ChanDesc *cd = P.chans + U.chan;
            const CUtensorMap *map = P.use_param_map ? &pmap : &cd->map;
            const int fc = cd->fcoord, nst = stages(u);
            for (int k = 0; k < nst; k++) {
                ok = mbar_wait_warp(bar(kBarEmptyPk) + 8 * s, ph ^ 1, abort_flag);
                if (!ok) break;
                tma_load_tile(lead, bar(kBarFullPk) + 8 * s, pk + s * kTileBytes, map, fc,
                              U.t0 + k * kStageSamples);
                g++;
                s = s + 1 == kPkSlots ? 0 : s + 1;
                ph ^= s == 0 ? 1u : 0u;
            }
        }
        pdl_launch_dependents();  // the last steps and drain are left: enough for a set-up
        if (lead) {
            if (!ok) {
                atomicOr(P.err, 0x10);
                *abort_flag = 1;
            }
            // Wait (bounded) for the last loads issued on every slot, so that
            // no TMA write lands after the CTA retires.
            for (uint32_t k = g > kPkSlots ? g - kPkSlots : 0; k < g; k++)
                mbar_wait_drain(bar(kBarFullPk) + 8 * (k % kPkSlots), (k / kPkSlots) & 1);
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------ MMA issuer
        const uint32_t lead = elect_one();
        const uint64_t dR = sdesc(op, 1024, 1024);
        const uint64_t dI = dR + (kTileBytes >> 4), dN = dR + 2 * (kTileBytes >> 4);
        const uint64_t dY = MAP == MAP_PACKED ? dR + 3 * (kTileBytes >> 4) : dI;
        uint32_t g = 0, s = 0, ph = 0, a = 0, aph = 0;  // steps, slot, buffer and their phases
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const int E = __shfl_sync(0xffffffffu, P.chans[P.units[u].chan].E, 0);
            const int nst = stages(u);
            // M = 128, N = E, both operands signed and MN-major
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                   ((uint32_t)(E >> 3) << 17) | ((128u >> 4) << 24);
            ok = mbar_wait_warp(bar(kBarAccEmpty) + 8 * a, aph ^ 1, abort_flag);
            for (int k = 0; ok && k < nst; k++) {
                ok = mbar_wait_warp(bar(kBarFullOp) + 8 * s, ph, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t so = s * (kOpBytes >> 4);
                if (TWO)
                    mma_step_self(lead, tmem_base + 256 * a, dR + so, dI + so, idesc, k > 0 ? 1u : 0u);
                else
                    mma_step(lead, tmem_base + 256 * a, dR + so, dI + so, dN + so, dR + so, dY + so,
                             idesc, k > 0 ? 1u : 0u);
                mma_commit_lead(lead, bar(kBarEmptyOp) + 8 * s);
                g++;
                s = s + 1 == kOpSlots ? 0 : s + 1;
                ph ^= s == 0 ? 1u : 0u;
            }
            if (!ok) break;
            mma_commit_lead(lead, bar(kBarAccFull) + 8 * a);
            a ^= 1;
            aph ^= a == 0 ? 1u : 0u;
        }
        if (lead) {
            if (!ok) {
                atomicOr(P.err, 0x20);
                *abort_flag = 1;
                mma_commit_lead(1, bar(kBarDrain));
                mbar_wait_drain(bar(kBarDrain), 0);
            }
            // No arrival may be pending when the CTA retires: wait for the
            // last phase committed on each operand slot.
            for (uint32_t k = 0; k < kOpSlots; k++)
                if (g > k)
                    mbar_wait_drain(bar(kBarEmptyOp) + 8 * k, ((g - 1 - k) / kOpSlots) & 1);
        }
        __syncwarp();
    } else if (warp < kUnpackWarps) {
        // ------------------------------------------------------ unpack
        // Warp gw of a group converts samples 8 gw .. 8 gw + 7 (one atom):
        // each thread chunk lane & 7 of the samples lane >> 3 and (lane >> 3) + 4.
        const int grp = warp / kGroupWarps, gw = warp % kGroupWarps;
        const int r0 = lane >> 3, chunk = lane & 7;
        const uint32_t ld = (uint32_t)(gw * 1024 + lane * 16);
        const uint32_t st0 = (uint32_t)gw * 1024 + swz(r0, chunk);
        const uint32_t st1 = (uint32_t)gw * 1024 + swz(r0 + 4, chunk);
        const YScale ys(kScale, P.one);
        uint32_t g = 0;  // steps of the units before this one
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const Unit U = P.units[u];
            const int nst = stages(u);
            const bool act = 16 * chunk < P.chans[U.chan].E;
            for (int k = (int)(((uint32_t)grp - g) % kGroups); k < nst; k += kGroups) {
                const uint32_t gs = g + (uint32_t)k;
                const uint32_t ps = gs % kPkSlots;
                ok = mbar_wait_warp(bar(kBarFullPk) + 8 * ps, (gs / kPkSlots) & 1, abort_flag);
                if (!ok) break;
                uint4 w[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
                if (act) {
                    w[0] = lds128(pk + ps * kTileBytes + ld);
                    w[1] = lds128(pk + ps * kTileBytes + ld + 512);
                }
                uint32_t v[2][kRowsMax][4];  // [chunk][row][word]
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint32_t b[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        yconv_scaled<MAP>(ys, b[q], v[j][0][q], v[j][1][q], v[j][2][q]);
                        v[j][3][q] = ys.low(b[q]);  // x'i (MAP_PACKED)
                    }
                }
                // The slot's release must not overtake the loads of any lane: the
                // arriving lane is picked by a vote over the loaded words (see
                // tc_pair_correlator.cu).
                const uint32_t seen = w[0].x ^ w[1].y;
                const int who = __any_sync(0xffffffffu, seen == 0x9E3779B9u) ? 1 : 0;
                if (lane == who) mbar_arrive(bar(kBarEmptyPk) + 8 * ps);
                const int t = U.t0 + k * kStageSamples + 8 * gw;
                if (t + 8 > U.t1) {  // samples past the unit are zero
#pragma unroll
                    for (int q = 0; q < 4; q++)
#pragma unroll
                        for (int j = 0; j < 2; j++)
                            if (t + r0 + 4 * j >= U.t1)
                                v[j][0][q] = v[j][1][q] = v[j][2][q] = v[j][3][q] = 0u;
                }
                const uint32_t os = gs % kOpSlots;
                ok = mbar_wait_warp(bar(kBarEmptyOp) + 8 * os, ((gs / kOpSlots) & 1) ^ 1, abort_flag);
                if (!ok) break;
                if (act) {
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const uint32_t st = op + os * kOpBytes + (j ? st1 : st0);
#pragma unroll
                        for (int r = 0; r < kRows; r++)
                            sts128(st + r * kTileBytes, v[j][r][0], v[j][r][1], v[j][r][2],
                                   v[j][r][3]);
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kBarFullOp) + 8 * os);
            }
            g += (uint32_t)nst;
        }
        if (!ok && lane == 0) {
            atomicOr(P.err, 0x40);
            *abort_flag = 1;
        }
    } else {
        // ------------------------------------------------------ epilogue
        // Epilogue warp w drains TMEM lanes 32 * (w % 4) .. +31 (block row
        // w % 4) over two of the four block columns.
        const int q = warp & 3;
        const int j0 = ((warp - kEpiWarp0) >> 2) * 2;
        const uint32_t stage = sbase + kOffStage + (uint32_t)(warp - kEpiWarp0) * kEpiTiles * 4096u;
        const uint32_t lead = elect_one();
        uint32_t *swap = reinterpret_cast<uint32_t *>(smem + kOffSwap);
        uint32_t a = 0, aph = 0, nchunk = 0;
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const Unit U = P.units[u];
            const ChanDesc *cd = P.chans + U.chan;
            const int nb1 = cd->nb1;
            // Split units add like accumulate mode (see tc_pair_correlator.cu).
            const uint32_t add = U.split || P.accumulate ? 1u : 0u;
            const CUtensorMap *omap = P.use_param_map ? &pomap : &cd->omap;
            const int row0 = cd->orow + (int)(U.out_off >> 6);
            ok = mbar_wait_warp(bar(kBarAccFull) + 8 * a, aph, abort_flag);
            if (TWO) ok = epi_barrier(ok);  // all go on, or none; the last unit's blocks are read
            if (!ok) break;
            tc_fence_after();
            if (TWO) {
                // Im = K - K^T: the blocks of K at or below the diagonal go to
                // shared memory, row x of the block a column, those of the warps'
                // own parity.
#pragma unroll 1
                for (int c = (warp - kEpiWarp0) >> 2; c <= q && q < nb1; c += 2) {
                    uint32_t *dst = swap + (q * (q + 1) / 2 + c) * kSwapWords + lane;
                    const uint32_t taddr =
                        tmem_base + ((uint32_t)(32 * q) << 16) + 256 * a + 128 + 32 * c;
#pragma unroll
                    for (int part = 0; part < 4; part++) {
                        uint32_t k[8];
                        tmem_ld8(taddr + 8 * part, k);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; i++) dst[(8 * part + i) * kSwapPitch] = k[i];
                    }
                }
                epi_barrier(true);
            }
#pragma unroll 1
            for (int j = j0; j < j0 + 2; j++) {
                if (q >= nb1 || j >= nb1 || j < q) continue;  // warp-uniform
                const int b = q * nb1 - q * (q - 1) / 2 + (j - q);
                const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + 256 * a + 32 * j;
                const uint32_t *kt = swap + (j * (j + 1) / 2 + q) * kSwapWords + lane * kSwapPitch;
#pragma unroll 1
                for (int half = 0; half < 2; half++) {
                    // Stage the 32 x 32-word tile (rows = lanes) in two
                    // 8-column parts, then hand it to TMA.
                    const uint32_t tile = stage + (nchunk % (uint32_t)kEpiTiles) * 4096u;
                    bulk_wait_read_lead<kEpiTiles - 1>(lead);
                    __syncwarp();
#pragma unroll
                    for (int part = 0; part < 2; part++) {
                        uint32_t re[8], im[8];
                        tmem_ld8(taddr + 16 * half + 8 * part, re);
                        tmem_ld8(taddr + 128 + 16 * half + 8 * part, im);
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 8; c++) {
                            if (TWO) im[c] -= kt[16 * half + 8 * part + c];
                            re[c] = (uint32_t)((int32_t)re[c] >> (2 * kScale));
                            im[c] = (uint32_t)((int32_t)im[c] >> (2 * kScale));
                            if (!P.ut) im[c] = 0u - im[c];
                        }
                        stage_row_half(tile, lane, part, re, im);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    tma_out_2d(lead, add, omap, tile, 32 * half, row0 + b * 32);
                    nchunk++;
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kBarAccEmpty) + 8 * a);
            a ^= 1;
            aph ^= a == 0 ? 1u : 0u;
        }
        if (!ok && lane == 0) {
            atomicOr(P.err, 0x80);
            *abort_flag = 1;
        }
        bulk_wait_read_lead<0>(lead);  // the staging tiles may go
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(kTmemCols)
                     : "memory");
    }
}

template <int MAP, bool TWO>
cudaError_t launch_small_map(const TcLaunch &L, const TcMaps *maps, cudaStream_t st) {
    static bool attr_done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_done[dev]) {
        e = cudaFuncSetAttribute(tc_small_kernel<MAP, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kSmemBytes);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    KParams P;
    P.chans = L.chans;
    P.units = L.units;
    P.cta_offsets = L.cta_offsets;
    P.use_param_map = L.use_param_map;
    P.static_tables = L.static_tables;
    P.after_zero = L.after_zero;
    P.ut = L.ut;
    P.accumulate = L.accumulate;
    P.one = 1;
    P.err = L.err;
    TcMaps none;
    memset(&none, 0, sizeof(none));
    const TcMaps &m = maps ? *maps : none;
    return launch_pdl(tc_small_kernel<MAP, TWO>, dim3(L.grid), dim3(kThreads), kSmemBytes, st, m.in, m.out,
                      P);
}

}  // namespace

cudaError_t tc_small_launch(const TcLaunch &L, const TcMaps *maps, cudaStream_t st) {
    if (L.nunits <= 0) return cudaSuccess;
    if (L.grid <= 0) return cudaErrorInvalidValue;
    if (L.use_param_map && !maps) return cudaErrorInvalidValue;
    const bool two = small_two_rows(L.max_samples);
    switch (L.map) {
    case MAP_EXACT:
        return two ? launch_small_map<MAP_EXACT, true>(L, maps, st)
                   : launch_small_map<MAP_EXACT, false>(L, maps, st);
    case MAP_CONF:
        return two ? launch_small_map<MAP_CONF, true>(L, maps, st)
                   : launch_small_map<MAP_CONF, false>(L, maps, st);
    default: return launch_small_map<MAP_PACKED, false>(L, maps, st);
    }
}

}  // namespace chx
