// tc_pair_correlator.cu -- 2-SM (cta_group::2) variant of the tcgen05
// kind::i8 correlator.
//
// A cluster of two CTAs computes a 256 x 256-element unit: CTA r holds y tile
// 2*ty2 + r (its 128 rows of A, M = 256 over the pair).  The unit's x range is
// two lanes of 128 elements, x tiles tx and tx + 1; CTA r holds 64
// elements of each (its columns of B, N = 128 per lane over the pair).  One
// elected thread of CTA 0 issues tcgen05.mma.cta_group::2; each SM's tensor core
// reads only its own A rows and B columns from its own shared memory.  Lane h
// accumulates in TMEM columns 256 h: 128 of Re, then 128 of Im.
//
// Operands (per CTA, one 32-sample step): y rows [R | I | N] (12 KiB, atoms of
// 8 samples x 128 elements, 128-byte swizzle) and per lane x rows [X | Y]
// (4 KiB, atoms of 8 samples x 64 elements, 64-byte swizzle); formulation and
// value maps are the 1-SM kernel's (tc_correlator.cu).  A y row used by several
// MMAs of a step is read from shared memory once (A collector).
//
// Skewed lanes.  A unit's 256 KiB of accumulators per SM leave at about 30
// bytes per cycle (the SM's egress), 8,700 cycles in which the tensor pipe used to
// wait: the whole TMEM belongs to one unit.  So lane 1 runs kSkewStages steps
// behind lane 0 and wraps around the sample range (the sums' order is free):
// step k takes stage k mod nst, lane 0 is active in steps [0, nst), lane 1 in
// [skew, nst + skew).  Lane 0 drains while lane 1 finishes alone, lane 1 drains
// while lane 0 of the next unit runs alone.  The price is skew more steps of y
// conversion per unit, and that a step of one lane takes 400-480 cycles (the latency
// of the operand ring, and shared memory while a drain runs) for half the work of
// a 512-cycle step of two.  Measured
// against both lanes in step (E = 2048, F = 37, unsplit; sustained): T = 1024
// 284 -> 272 us, T = 256 141 -> 130 us, T = 16384 unchanged.  Two full units of
// half the width, with an accumulator buffer each, were bound by shared memory
// (360-400 cycles per step instead of 256) and no faster at T = 1024.  A unit
// whose second x tile lies outside the matrix (odd tile counts) has one lane
// only, and so have the narrow units of launches that leave SM pairs idle.
//
// Warps: 0-15 unpack, 16 TMA producer, 17 MMA issuer (CTA 0), 18-25 epilogue.
// The epilogue warps drain each lane's accumulators when its last step is
// done; each 32 x 32-word output tile goes from TMEM through a swizzled staging
// tile in shared memory to a TMA store (or reduce-add) into the block buffer.
//
// What bounds the main loop: the tensor pipe.  A step of two lanes takes 510
// cycles (clock64 around the MMA loop) of the 512 that its MMAs need (M256 N256
// K32 four times over); under a long load the power cap lowers the clock below
// 1965 MHz and that, not the pipeline, sets the time.  What got it there from
// 740-770 cycles (E = 2048, F = 8, T = 16384):
//   * The unpack warps work in kGroups groups, step s in group s % kGroups, so
//     that four steps are in different phases (load, convert, store, fence) at
//     a time.  All 16 warps on one step moved through the phases in step and
//     took 676 cycles even without any MMA.
//   * The MMA and producer warps stay converged and issue with an elected lane's
//     predicate.  Issued from a lane == 0 branch, the MMAs and the waits between
//     them queued up one behind the other and left the tensor pipe idle for about
//     300 cycles at every commit (670 cycles a step), and the producer could
//     not load a step in less than 490 cycles.
//
// Why the y rows are scaled (YScale).  Under the power cap the toggling of the
// operand bits sets the clock: x = 16 xr instead of xr (no sign extension below
// the value) is worth 7 % of the time of a sustained load, y = 8 yr instead of
// yr another 3 % (687 vs 710 us); the negated row on the x side instead (y times
// 16, x times 8) costs 1 %.  8 is the largest factor that leaves -yr in int8;
// |acc| <= 8 * 16 * 128 T then fits int32 for T < 2^17 (the offset-domain maps:
// 8 * 16 * 450 T, T <= 37282), so launches whose longest unit exceeds
// kScaledMaxSamples keep y unscaled.
//
// Synchronisation across the pair:
//   full_op[s]    in CTA 0; the kGroupWarps unpack warps of the step's group
//                 arrive in both CTAs (one lane each, after its lanes' proxy
//                 fences) -> the MMA warp waits.
//   empty_op[s]   in both CTAs; CTA 0's commit arrives on both (multicast).
//   acc_full[h]   in both CTAs; CTA 0's commit arrives on both (multicast).
//   acc_empty[h]  in CTA 0; every epilogue warp of both CTAs arrives.
// TMA loads, the packed ring and its barriers are local to each CTA.  Both
// CTAs meet at cluster barriers after set-up and before exit, so no remote
// arrival can land after a CTA retires.  Every wait is bounded.
#include "tc_cluster.cuh"

#include <cudaTypedefs.h>
#include <string.h>

#include <algorithm>

namespace chx {

namespace {

using namespace tc;

constexpr int kStageSamples = kUnitStageSamples;
constexpr int kOpSlots = 4;     // operand slots, one step each
constexpr int kUnpackWarps = 16;
constexpr int kGroups = 4;      // unpack groups: step s belongs to group s % kGroups
constexpr int kGroupWarps = kUnpackWarps / kGroups;
// Packed slots.  A group may run ahead of another group's late TMA load, and
// the parity wait on a packed slot must not mistake its previous phase for the
// wanted one.  Before step s a group has finished step s - kGroups, whose
// operand slot was free only once the MMAs had consumed step
// s - kGroups - kOpSlots: with kPkSlots >= kGroups + kOpSlots that includes
// the slot's previous step.
constexpr int kPkSlots = 8;
static_assert(kPkSlots >= kGroups + kOpSlots, "parity of the packed ring");
constexpr int kScaledMaxSamples = 1 << 15;  // longest unit with y scaled by 8
constexpr int kYTileBytes = kStageSamples * 128;  // packed y tile of a step
constexpr int kXTileBytes = kStageSamples * 64;   // packed x tile of a lane
constexpr int kYOpBytes = 3 * kYTileBytes;        // rows R, I, N
constexpr int kXOpBytes = 2 * kXTileBytes;        // rows X, Y of a lane
constexpr int kProducerWarp = 16;
constexpr int kMmaWarp = 17;
constexpr int kEpiWarp0 = 18;   // epilogue warps from here on, lane quarter = warp % 4
constexpr int kEpiWarps = 8;    // two per lane quarter, two of a lane's four column blocks each
constexpr int kEpiTiles = 2;    // 4 KiB output staging tiles per epilogue warp
constexpr int kEpiStageBytes = kEpiTiles * 4096;
constexpr int kThreads = (kEpiWarp0 + kEpiWarps) * 32;
constexpr int kTmemCols = 512;

constexpr int kOffOpY = 0;
constexpr int kOffOpX = kOffOpY + kOpSlots * kYOpBytes;  // per slot: lane 0, lane 1
constexpr int kOffPkY = kOffOpX + kOpSlots * 2 * kXOpBytes;
constexpr int kOffPkX = kOffPkY + kPkSlots * kYTileBytes;
constexpr int kOffStage = kOffPkX + kPkSlots * 2 * kXTileBytes;
constexpr int kOffBars = kOffStage + kEpiWarps * kEpiStageBytes;
constexpr int kSmemBytes = kOffBars + 256 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory per CTA");

// Barrier indexes inside the barrier block (8 bytes each).
constexpr int kBarFullPk = 0;
constexpr int kBarEmptyPk = kBarFullPk + kPkSlots;
constexpr int kBarFullOp = kBarEmptyPk + kPkSlots;
constexpr int kBarEmptyOp = kBarFullOp + kOpSlots;
constexpr int kBarAccFull = kBarEmptyOp + kOpSlots;  // per lane
constexpr int kBarAccEmpty = kBarAccFull + 2;        // per lane
constexpr int kBarDrain = kBarAccEmpty + 2;
constexpr int kBarCount = kBarDrain + 1;
static_assert(kBarCount * 8 + 8 <= 256, "barrier block");

struct KParams {
    const ChanDesc *chans;
    const Unit *units;
    const int *cluster_offsets;  // cluster c takes units [off[c], off[c+1])
    int use_param_map;
    int ut;
    int accumulate;
    int static_tables;  // the tables were complete before the launch
    int after_zero;     // the previous launch is the one zeroing the output
    uint32_t yscale;  // y rows are scaled by 2^yscale
    uint32_t one;  // 1 (YScale)
    int *err;
};

// The steps of a unit (see "Skewed lanes" above).
struct Steps {
    int nst, skew, total;  // stages, lane 1's delay, steps (one lane: all nst)
    __device__ __forceinline__ explicit Steps(const Unit &u) {
        // The shuffles tell the compiler that these are the same for the whole
        // warp, so that loops and MMA operands stay in the uniform datapath.
        nst = __shfl_sync(0xffffffffu, (u.t1 - u.t0 + kStageSamples - 1) / kStageSamples, 0);
        const bool pair = __shfl_sync(0xffffffffu, (u.tyx >> 20) & 3, 0) > 1;
        skew = pair ? min(nst, kSkewStages) : nst;
        total = pair ? nst + skew : nst;
    }
    __device__ __forceinline__ bool two() const { return total > nst; }
    __device__ __forceinline__ bool lane0(int k) const { return k < nst; }
    __device__ __forceinline__ bool lane1(int k) const { return k >= skew; }
    __device__ __forceinline__ int stage(int k) const { return k < nst ? k : k - nst; }
};

template <int MAP>
__global__ void __launch_bounds__(kThreads, 1)
tc_pair_kernel(const __grid_constant__ CUtensorMap pmap, const __grid_constant__ CUtensorMap pxmap,
               const __grid_constant__ CUtensorMap pomap, const KParams P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = smem_u32(smem);
    const uint32_t op_y = sbase + kOffOpY, op_x = sbase + kOffOpX;
    const uint32_t pk_y = sbase + kOffPkY, pk_x = sbase + kOffPkX;
    const uint32_t bars = sbase + kOffBars;
    auto bar = [&](int i) { return bars + 8 * i; };
    volatile uint32_t *tmem_slot =
        reinterpret_cast<volatile uint32_t *>(smem + kOffBars + 8 * kBarCount);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // warp-uniform
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cluster = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPkSlots; s++) {
            mbar_init(bar(kBarFullPk + s), 1);
            mbar_init(bar(kBarEmptyPk + s), kGroupWarps);
        }
        for (int s = 0; s < kOpSlots; s++) {
            mbar_init(bar(kBarFullOp + s), 2 * kGroupWarps);
            mbar_init(bar(kBarEmptyOp + s), 1);
        }
        for (int h = 0; h < 2; h++) {
            mbar_init(bar(kBarAccFull + h), 1);
            mbar_init(bar(kBarAccEmpty + h), 2 * kEpiWarps);
        }
        mbar_init(bar(kBarDrain), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    // Set-up overlaps the previous kernel of the stream; tables that the stream
    // itself writes are read only after that kernel.
    if (!P.static_tables) pdl_wait();
    const int first = P.cluster_offsets[cluster], last = P.cluster_offsets[cluster + 1];
    if (warp == 0) {  // the first unit's records are on their way to L1 meanwhile
        const int chan = first < last ? P.units[first].chan : 0;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(&P.chans[chan].E));
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // barriers of both CTAs initialised, TMEM allocated
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // The zeroing kernel started after all earlier work had ended: only the
    // output waits for it.
    if (!P.after_zero || warp >= kEpiWarp0) pdl_wait();

    if (warp == kProducerWarp) {
        // ------------------------------------------------- TMA producer (both CTAs)
        // Converged, the elected lane issues.
        const uint32_t lead = elect_one();
        uint32_t g = 0, s = 0, ph = 0;  // steps issued, packed slot, its phase
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const Unit U = P.units[u];
            const Steps S(U);
            const ChanDesc *cd = P.chans + U.chan;
            const CUtensorMap *map = P.use_param_map ? &pmap : &cd->map;
            const CUtensorMap *xmap = P.use_param_map ? &pxmap : &cd->xmap;
            const int fc = cd->fcoord;
            const int y = (2 * (U.tyx & 1023) + (int)rank) * 128;
            const int x = ((U.tyx >> 10) & 1023) * 128 + (int)rank * 64;
            for (int k = 0; k < S.total; k++) {
                ok = mbar_wait_warp(bar(kBarEmptyPk) + 8 * s, ph ^ 1, abort_flag);
                if (!ok) break;
                const uint32_t a0 = S.lane0(k), a1 = S.lane1(k);
                const uint32_t xdst = pk_x + s * 2 * kXTileBytes;
                tma_load_step(lead, bar(kBarFullPk) + 8 * s, kYTileBytes + (a0 + a1) * kXTileBytes,
                              pk_y + s * kYTileBytes, map, y, xdst, xdst + kXTileBytes, xmap, x,
                              x + 128, a0, a1, fc, U.t0 + S.stage(k) * kStageSamples);
                g++;
                s = (s + 1) % kPkSlots;
                ph ^= s == 0 ? 1u : 0u;
            }
        }
        pdl_launch_dependents();  // the last steps and drain are left: enough for a set-up
        if (lead) {
            if (!ok) {
                atomicOr(P.err, 0x100);
                *abort_flag = 1;
            }
            // Wait (bounded) for the last loads issued on every slot, so that
            // no TMA write lands after the CTA retires.
            for (uint32_t k = g > kPkSlots ? g - kPkSlots : 0; k < g; k++)
                mbar_wait_drain(bar(kBarFullPk) + 8 * (k % kPkSlots), (k / kPkSlots) & 1);
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------- MMA issuer (CTA 0 only)
        // The whole warp runs the loop; the elected lane issues.
        if (rank == 0) {
            const uint32_t lead = elect_one();
            // M = 256 and N = 128 over the pair; x unsigned in the offset-domain
            // maps, y always signed.
            const uint32_t idesc = (2u << 4) | (1u << 7) | ((MAP == MAP_EXACT ? 1u : 0u) << 10) |
                                   (1u << 15) | (1u << 16) | ((128u >> 3) << 17) |
                                   ((256u >> 4) << 24);
            const uint64_t dR = sdesc(op_y, 1024, 1024);
            const uint64_t dI = dR + (kYTileBytes >> 4), dN = dR + 2 * (kYTileBytes >> 4);
            const uint64_t dX = sdesc64(op_x, 512, 512);
            const uint64_t dY = dX + (kXTileBytes >> 4);
            uint32_t s = 0, ph = 0;           // operand slot, its phase
            uint32_t aph0 = 0, aph1 = 0;      // accumulator phases of the lanes
            bool ok = true;
            // Waits for the operands of the next step, unless the look ahead
            // during the one before found them: that look's latency passes behind
            // the MMAs.  Units of one lane only, whose steps take 400 instead of 425
            // cycles; at the power cap units of two lanes lose 0.5 % to it.
            bool look = false, ready = false, ahead = false;
            auto step_ready = [&]() {
                const bool full =
                    ready || mbar_wait_warp<true>(bar(kBarFullOp) + 8 * s, ph, abort_flag);
                tc_fence_after();
                const uint32_t s1 = (s + 1) % kOpSlots;
                ahead = look && mbar_test_cluster(bar(kBarFullOp) + 8 * s1, s1 == 0 ? ph ^ 1 : ph);
                return full;
            };
            // Hands the step's slot back and moves on.
            auto step_done = [&]() {
                mma_commit_pair(lead, bar(kBarEmptyOp) + 8 * s);
                ready = look && __all_sync(0xffffffffu, ahead);
                s = (s + 1) % kOpSlots;
                ph ^= s == 0 ? 1u : 0u;
            };
            // One loop per phase of the unit, so that no step branches.
            for (int u = first; u < last && ok; u++) {
                const Steps S(P.units[u]);
                look = !S.two();
                ok = mbar_wait_warp<true>(bar(kBarAccEmpty), aph0 ^ 1, abort_flag);  // drained
                aph0 ^= 1;
                for (int k = 0; ok && k < S.skew; k++) {
                    ok = step_ready();
                    if (!ok) break;
                    const uint32_t so_y = s * (kYOpBytes >> 4), so_x = s * (2 * kXOpBytes >> 4);
                    mma_step_one(lead, tmem_base, dR + so_y, dI + so_y, dN + so_y, dX + so_x,
                                 dY + so_x, idesc, k > 0 ? 1u : 0u);
                    step_done();
                }
                if (ok && S.two()) {
                    ok = mbar_wait_warp<true>(bar(kBarAccEmpty + 1), aph1 ^ 1, abort_flag);
                    aph1 ^= 1;
                }
                for (int k = S.skew; ok && k < S.nst; k++) {
                    ok = step_ready();
                    if (!ok) break;
                    const uint32_t so_y = s * (kYOpBytes >> 4), so_x = s * (2 * kXOpBytes >> 4);
                    mma_step_two(lead, tmem_base, dR + so_y, dI + so_y, dN + so_y, dX + so_x,
                                 dY + so_x, kXOpBytes >> 4, idesc, 1u, k > S.skew ? 1u : 0u);
                    step_done();
                }
                if (!ok) break;
                mma_commit_pair(lead, bar(kBarAccFull));
                if (!S.two()) continue;
                for (int k = S.nst; k < S.total; k++) {
                    ok = step_ready();
                    if (!ok) break;
                    const uint32_t so_y = s * (kYOpBytes >> 4), so_x = (2 * s + 1) * (kXOpBytes >> 4);
                    mma_step_one(lead, tmem_base + 256, dR + so_y, dI + so_y, dN + so_y, dX + so_x,
                                 dY + so_x, idesc, k > S.skew ? 1u : 0u);
                    step_done();
                }
                if (!ok) break;
                mma_commit_pair(lead, bar(kBarAccFull + 1));
            }
            if (!ok && lead) {
                atomicOr(P.err, 0x200);
                *abort_flag = 1;
                asm volatile(
                    "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64"
                    " [%0];" ::"r"(bar(kBarDrain))
                    : "memory");
                mbar_wait_drain(bar(kBarDrain), 0);
            }
        }
        __syncwarp();
    } else if (warp < kUnpackWarps) {
        // ------------------------------------------------- unpack (both CTAs)
        // Warp gw of a group converts samples 8 gw .. 8 gw + 7 (one atom) of the
        // step's tiles: each thread two 16-byte chunks of the y tile (chunk
        // lane & 7 of the samples lane >> 3 and (lane >> 3) + 4) and one of each
        // active x tile (chunk lane & 3 of sample lane >> 2).
        const int grp = warp / kGroupWarps, gw = warp % kGroupWarps;
        const int yr = lane >> 3, xr = lane >> 2;
        const uint32_t yld = (uint32_t)(gw * 1024 + lane * 16);
        const uint32_t xld = (uint32_t)(gw * 512 + lane * 16);
        const uint32_t yst0 = (uint32_t)gw * 1024 + swz(yr, lane & 7);
        const uint32_t yst1 = (uint32_t)gw * 1024 + swz(yr + 4, lane & 7);
        const uint32_t xst = (uint32_t)gw * 512 + swz64(xr, lane & 3);
        // The n-th step of this group is step kGroups n + grp: always operand slot
        // grp, and packed slots grp and grp + kGroups in turn.
        static_assert(kOpSlots == kGroups && kPkSlots == 2 * kGroups, "slots of a group");
        const uint32_t full_op = bar(kBarFullOp + grp), empty_op = bar(kBarEmptyOp + grp);
        const uint32_t full_op_leader = mapa(full_op, 0);
        const uint32_t ya0 = op_y + grp * kYOpBytes + yst0, ya1 = op_y + grp * kYOpBytes + yst1;
        const uint32_t xa = op_x + grp * 2 * kXOpBytes + xst;
        const YScale ys(P.yscale, P.one);
        uint32_t n = 0, g = 0;  // this group's steps, all steps of the units before this one
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const Unit U = P.units[u];
            const Steps S(U);
            for (int k = (int)(((uint32_t)grp - g) % kGroups); k < S.total; k += kGroups, n++) {
                const uint32_t ps = grp + kGroups * (n & 1);
                ok = mbar_wait_warp(bar(kBarFullPk) + 8 * ps, (n >> 1) & 1, abort_flag);
                if (!ok) break;
                const bool act[2] = {S.lane0(k), S.lane1(k)};
                uint4 wy[2], wx[2];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    wy[j] = lds128(pk_y + ps * kYTileBytes + yld + 512 * j);
                    wx[j] = make_uint4(0, 0, 0, 0);
                    if (act[j]) wx[j] = lds128(pk_x + (2 * ps + j) * kXTileBytes + xld);
                }
                uint32_t y[2][3][4], x[2][2][4];  // [chunk][R I N][word], [lane][X Y][word]
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint32_t a[4] = {wy[j].x, wy[j].y, wy[j].z, wy[j].w};
                    const uint32_t b[4] = {wx[j].x, wx[j].y, wx[j].z, wx[j].w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        yconv_scaled<MAP>(ys, a[q], y[j][0][q], y[j][1][q], y[j][2][q]);
                        if (act[j]) xconv<MAP>(b[q], x[j][0][q], x[j][1][q]);
                    }
                }
                // One arrival per warp frees the slot.  It must not overtake the
                // loads of any lane, so the arriving lane is picked by a vote over
                // the loaded words: with a __syncwarp alone the loads were seen to
                // run after the arrive and read the slot's next tile.
                const uint32_t seen = wy[0].x ^ wy[1].x ^ wx[0].x ^ wx[1].y;
                const int who = __any_sync(0xffffffffu, seen == 0x9E3779B9u) ? 1 : 0;
                if (lane == who) mbar_arrive(bar(kBarEmptyPk) + 8 * ps);
                const int t = U.t0 + S.stage(k) * kStageSamples + 8 * gw;
                if (t + 8 > U.t1) {  // samples past the unit are zero
#pragma unroll
                    for (int q = 0; q < 4; q++) {
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            if (t + yr + 4 * j >= U.t1) y[j][0][q] = y[j][1][q] = y[j][2][q] = 0u;
                            if (t + xr >= U.t1) x[j][0][q] = x[j][1][q] = 0u;
                        }
                    }
                }
                ok = mbar_wait_warp(empty_op, (n & 1) ^ 1, abort_flag);
                if (!ok) break;
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const uint32_t st = j ? ya1 : ya0;
#pragma unroll
                    for (int r = 0; r < 3; r++)
                        sts128(st + r * kYTileBytes, y[j][r][0], y[j][r][1], y[j][r][2], y[j][r][3]);
                }
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (act[h]) {
#pragma unroll
                        for (int r = 0; r < 2; r++)
                            sts128(xa + h * kXOpBytes + r * kXTileBytes, x[h][r][0], x[h][r][1],
                                   x[h][r][2], x[h][r][3]);
                    }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (rank == 0)
                        mbar_arrive(full_op);
                    else
                        mbar_arrive_cluster(full_op_leader);
                }
            }
            g += (uint32_t)S.total;
        }
        if (!ok && lane == 0) {
            atomicOr(P.err, 0x400);
            *abort_flag = 1;
        }
        // No multicast arrival may still be on its way to this CTA's operand
        // barriers when it retires: thread 0 waits for the last phase of each.
        if (threadIdx.x == 0)
            for (uint32_t k = 0; k < kOpSlots; k++)
                if (g > k)  // steps < g in slot k: their last phase
                    mbar_wait_drain(bar(kBarEmptyOp) + 8 * k, ((g - 1 - k) / kOpSlots) & 1);
    } else {
        // ------------------------------------------------- epilogue (both CTAs)
        // Epilogue warp w drains TMEM lanes 32 * (w % 4) .. +31 (its quarter of
        // the CTA's 128 y rows) over two of a lane's four 32-column blocks of Re
        // and Im, hands the cells to TMA through its staging tiles, and releases
        // the accumulators as soon as its last TMEM load completes.
        const int q = warp & 3;
        const int j0 = ((warp - kEpiWarp0) >> 2) * 2;
        const uint32_t acc_empty_leader = mapa(bar(kBarAccEmpty), 0);
        const uint32_t stage = sbase + kOffStage + (uint32_t)(warp - kEpiWarp0) * kEpiStageBytes;
        const uint32_t lead = elect_one();
        const uint32_t shift = 4 + P.yscale;  // x rows are scaled by 16
        uint32_t phases = 0, nchunk = 0;      // bit h: phase of lane h's accumulators
        bool ok = true;
        for (int u = first; u < last && ok; u++) {
            const Unit U = P.units[u];
            const ChanDesc *cd = P.chans + U.chan;
            const int nl = (U.tyx >> 20) & 3;
            const int bx0 = ((U.tyx >> 10) & 1023) * 4;
            const int nb1 = cd->nb1;
            const int by = (2 * (U.tyx & 1023) + (int)rank) * 4 + q;
            // Split units (other units cover the same cells' other sample ranges)
            // add like accumulate mode: every element of a TMA reduce-add is an
            // individual relaxed reduction at gpu scope, so concurrent units meet
            // exactly in the zeroed (or accumulating) output.
            const uint32_t add = U.split || P.accumulate ? 1u : 0u;
            const CUtensorMap *omap = P.use_param_map ? &pomap : &cd->omap;
            const int row0 = cd->orow + (int)(U.out_off >> 6);
            for (int h = 0; h < nl; h++) {
                ok = mbar_wait_warp(bar(kBarAccFull) + 8 * h, (phases >> h) & 1, abort_flag);
                if (!ok) break;
                phases ^= 1u << h;
                tc_fence_after();
#pragma unroll 1
                for (int j = j0; j < j0 + 2; j++) {  // 32-column block of the lane
                    const int bx = bx0 + 4 * h + j;
                    if (by >= nb1 || bx >= nb1 || bx < by) continue;  // warp-uniform
                    const int64_t b = (int64_t)by * nb1 - (int64_t)by * (by - 1) / 2 + (bx - by);
                    const uint32_t taddr =
                        tmem_base + ((uint32_t)(32 * q) << 16) + 256 * h + 32 * j;
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
                                re[c] = (uint32_t)((int32_t)re[c] >> shift);
                                im[c] = (uint32_t)((int32_t)im[c] >> shift);
                                if (!P.ut) im[c] = 0u - im[c];
                            }
                            stage_row_half(tile, lane, part, re, im);
                        }
                        fence_proxy_async();
                        __syncwarp();
                        tma_out_2d(lead, add, omap, tile, 32 * half, row0 + (int)b * 32);
                        nchunk++;
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(acc_empty_leader + 8 * h);
            }
        }
        if (!ok && lane == 0) {
            atomicOr(P.err, 0x800);
            *abort_flag = 1;
        }
        bulk_wait_read_lead<0>(lead);  // the staging tiles may go; the grid's end completes the writes
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();  // no remote arrivals after this point
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(kTmemCols)
                     : "memory");
    }
}

template <int MAP>
cudaError_t launch_pair_map(const TcLaunch &L, const TcMaps *maps, cudaStream_t st) {
    static bool attr_done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_done[dev]) {
        e = cudaFuncSetAttribute(tc_pair_kernel<MAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kSmemBytes);
        if (e != cudaSuccess) return e;
        attr_done[dev] = true;
    }
    KParams P;
    P.chans = L.chans;
    P.units = L.units;
    P.cluster_offsets = L.cta_offsets;
    P.use_param_map = L.use_param_map;
    P.ut = L.ut;
    P.accumulate = L.accumulate;
    P.static_tables = L.static_tables;
    P.after_zero = L.after_zero;
    P.yscale = L.max_samples <= kScaledMaxSamples ? 3 : 0;
    P.one = 1;
    P.err = L.err;
    TcMaps none;
    memset(&none, 0, sizeof(none));
    const TcMaps &m = maps ? *maps : none;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * L.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = cudaLaunchKernelEx(&cfg, tc_pair_kernel<MAP>, m.in, m.in_half, m.out, P);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace

void tc_append_pair_units(std::vector<Unit> &out, bool narrow, int chan, int E, int t_begin,
                          int t_end, int tsplit, long long out_off) {
    const int nt = (E + 127) / 128, lanes = narrow ? 1 : 2;
    const int span = t_end - t_begin;
    if (span <= 0) return;
    int splits = tsplit < 1 ? 1 : tsplit;
    int chunk = (span + splits - 1) / splits;
    chunk = (chunk + kStageSamples - 1) / kStageSamples * kStageSamples;
    if (chunk > kUnitMaxSamples) chunk = kUnitMaxSamples;
    splits = (span + chunk - 1) / chunk;
    for (int ty2 = 0; 2 * ty2 < nt; ty2++)
        for (int tx = 2 * ty2; tx < nt; tx += lanes)
            for (int s = 0; s < splits; s++) {
                const int nl = std::min(lanes, nt - tx);
                Unit u;
                u.chan = chan;
                u.tyx = ty2 | (tx << 10) | (nl << 20);
                u.t0 = t_begin + s * chunk;
                u.t1 = std::min(t_end, u.t0 + chunk);
                u.out_off = out_off;
                u.split = splits > 1 ? 1 : 0;
                u.cost = unit_cost(narrow ? kTileNarrow : kTile2Sm, u.t0, u.t1, nl);
                out.push_back(u);
            }
}

cudaError_t tc_pair_launch(const TcLaunch &L, const TcMaps *maps, cudaStream_t st) {
    if (L.nunits <= 0) return cudaSuccess;
    if (L.grid <= 0) return cudaErrorInvalidValue;
    if (L.use_param_map && !maps) return cudaErrorInvalidValue;
    switch (L.map) {
    case MAP_EXACT: return launch_pair_map<MAP_EXACT>(L, maps, st);
    case MAP_CONF: return launch_pair_map<MAP_CONF>(L, maps, st);
    default: return launch_pair_map<MAP_PACKED>(L, maps, st);
    }
}

}  // namespace chx
