// chimex_internal.h -- shared declarations of libchimex (not installed).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>

#include <algorithm>
#include <functional>
#include <string>
#include <vector>

#include "../../include/chimex.h"

namespace chx {

// Value maps: how a packed byte becomes the int8 operands of the correlator.
// For a row element y the operand pair is (a0, a1); for a column element x
// the Re column is (b0, b1) and the Im column is (b2, b3), so that per sample
//   Re += a0*b0 + a1*b1,   Im += a0*b2 + a1*b3.
// MAP_EXACT   signed values s = nibble - 8: a = (yr, yi), Re = (xr, xi),
//             Im = (-xi, xr); exact visibilities, no corrections needed.
// MAP_CONF    offset nibbles n = s + 8: the partials of the conference corr
//             kernel (pairwise_correlator_UT.cl:107-201).
// MAP_PACKED  offset nibbles with the y imaginary nibble inverted (15 - n):
//             the partials of the packed corr kernel
//             (packed_correlator_overflow_protected_to_2272_iter_UT.cl:91-285):
//             a = (y'r, 15 - y'i), Re = (x'r, -x'i), Im = (-x'i, -x'r).
// The non-UT conventions negate Im in the epilogue.
enum ValueMap : int { MAP_EXACT = 0, MAP_CONF = 1, MAP_PACKED = 2 };

struct Shape {
    int E, F, T;
    int64_t NB1, NB;
};

}  // namespace chx

struct chx_plan {
    int E, F, T, TA, ut, kernel_batch, device;
    int64_t NB1, NB;
    int algo;     // CHX_ALGO_*
    int tsplit;   // 0 = auto
    int tile;     // 0 = auto
    int *d_err;   // device error word (bounded-wait timeouts)
    int sm_count;
    void *d_chans;  // tensor-core channel table (ChanDesc[F]), then both unit tables
    // Work units of a launch that overwrites its output (0) or adds to it (1).
    struct {
        size_t first;   // bytes from d_chans to Unit[nunits], then grid + 1 offsets
        int nunits;
        int grid;       // persistent CTAs (or CTA pairs)
        int tile;       // tile variant
        int max_unit;   // samples of the longest unit
        bool has_split_units;  // some output cells receive several units (TMA reduce-add)
    } tc[2];
};

namespace chx {

// Error helpers: set the thread-local message and return the code.
int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);
void clear_error();

#define CHX_CUDA(call)                                      \
    do {                                                    \
        cudaError_t e_ = (call);                            \
        if (e_ != cudaSuccess) return chx::cuda_fail(e_, #call); \
    } while (0)

// RAII: make `dev` current for the scope, restore the previous device.
struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) ok = (cudaSetDevice(dev) == cudaSuccess);
    }
    ~DeviceGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev)
            cudaSetDevice(prev);
    }
};

// NVTX range around a public entry point: profilers (nsys, ncu) show each
// call by name; without a tool attached a push/pop is a cheap no-op.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// Launches a kernel that may start its set-up before the stream's previous
// kernel has ended (programmatic dependent launch).  Such a kernel calls pdl_wait
// before it touches memory (behind launch_zero: before it touches the output).  Between
// ordinary launches, which the one-SM tile's kernel and the dp4a kernel keep, this GPU
// spends up to 2 us per kernel boundary.
template <class... Params, class... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                       cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}
// Device side of it: the next kernel of the stream may start its set-up once
// every CTA of this one has called pdl_launch_dependents.  A launch that has
// started waits on SMs that other streams could use, so kernels whose CTAs live
// long call it when a CTA has issued its last loads, not at their start (two calls
// of E = 256, F = 18, T = 65536 on 72 SMs, 856 us: a call of E = 256, F = 16,
// T = 512 on another stream ended after 220 us, 70 now).  pdl_wait returns when
// the previous kernel has completed and its writes are visible (at once when the
// launch did not ask for overlap).  What the kernel loads may be written until
// then, within its own lifetime: such loads have to be coherent ones, so no
// __ldg and no const __restrict__ parameters in these kernels.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

inline int64_t num_blocks_of(int E) {
    int64_t n = E / 32;
    return n * (n + 1) / 2;
}

// ---- SIMT kernels (simt_kernels.cu) ----
// Correlates samples [t_begin, t_end) of every channel with the CUDA-core
// dp4a kernel.  mode: 0 store, 1 add (plain RMW), 2 atomic add.
cudaError_t launch_correlate_simt(const uint8_t *packed, int32_t *blocks, int E, int F,
                                  int T, int map, int ut, int mode, int splits,
                                  cudaStream_t st);
// How the offset sums are split: `ctas` CTAs of `warps` warps take equal shares of
// vblocks vector blocks (512 (f, e) bytes of every sample) x ngroups groups of 16
// samples.
struct OffsetSplit {
    int warps;
    int64_t ctas;
};
constexpr int kOaWarps = 16;      // warps per SM
constexpr int kOaShortWarps = 4;  // warps per CTA when T is short
constexpr int kOaMinGroups = 8;   // groups per CTA below which a vector block is not cut:
                                  // the cuts' atomic adds cost more than their loads (E = 128,
                                  // F = 5, T = 2968: 17.6 us with 1, 6.3 with 8)
inline OffsetSplit offset_split(int64_t vblocks, int64_t ngroups, int sms) {
    // One CTA per SM streams best while every warp has groups of a vector block to
    // load.  With fewer groups most warps of it would idle, and its vector blocks, about
    // 2 us each, follow one another: four CTAs per SM then.
    const int warps = ngroups < kOaWarps ? kOaShortWarps : kOaWarps;
    // Vector blocks are independent: they always spread over all CTAs.
    const int64_t work = std::max(vblocks, vblocks * ngroups / kOaMinGroups);
    return {warps, std::min<int64_t>((int64_t)sms * (kOaWarps / warps), work)};
}
// zeroed: launch_zero(sums) was the stream's previous launch.
cudaError_t launch_offset_accumulate(const uint8_t *packed, uint32_t *sums, int E, int F,
                                     int T, bool zeroed, cudaStream_t st);
// Zeroes bytes (a multiple of 16) at a 16-byte aligned address.
cudaError_t launch_zero(void *out, int64_t bytes, cudaStream_t st);
cudaError_t launch_preseed(const uint32_t *sums, int32_t *blocks, int E, int F, int T,
                           int packed_variant, int ut, cudaStream_t st);
cudaError_t launch_blocks_to_triangle(const int32_t *blocks, int32_t *tri, int E, int F,
                                      cudaStream_t st);
cudaError_t launch_blocks_to_full(const int32_t *blocks, int32_t *full, int E, int F,
                                  cudaStream_t st);

// ---- tensor-core kernel (tc_correlator.cu) ----
// A channel as the tensor-core kernel sees it: the TMA map of its packed
// samples (dims {E, channels, samples}), that of its block buffer, and its shape.
struct __align__(64) ChanDesc {
    CUtensorMap map;   // samples (128-element tiles); used unless the launch passes one map for all channels
    CUtensorMap xmap;  // samples in 64-element tiles (x of the SM-pair kernel); same rule
    CUtensorMap omap;  // block output as rows of 64 words (tc_encode_out_map); same rule
    int E;             // elements
    int nb1;           // E / 32
    int fcoord;        // channel coordinate inside the TMA map
    int orow;          // first row of this channel's blocks inside omap
    int pad[12];
};
static_assert(sizeof(ChanDesc) == 448, "ChanDesc layout");

// One work unit: a 128-element y tile against one or two 128-element x tiles
// of one channel over samples [t0, t1).  tyx = ty | x0 << 10 | nx << 20.
struct Unit {
    int chan;
    int tyx;
    int t0, t1;
    long long out_off;  // int32 words added to the channel's block buffer
    int split;          // 1: other units add to the same cells (TMA reduce-add)
    int cost;           // unit_cost, for scheduling
};
static_assert(sizeof(Unit) == 32, "Unit layout");

constexpr int kUnitMaxSamples = 1 << 18;  // int32-exact bound per unit
constexpr int kUnitStageSamples = 32;      // samples per pipeline stage of the kernels

// Steps by which the SM-pair kernel's second x lane trails the first: about
// one lane's accumulator drain.  8 to 14 measured within 1 % of each other
// (E = 2048, T = 256 to 16384); below that the drains show again.
constexpr int kSkewStages = 12;

// Tensor-core tile variants (CHX_OPT_TILE).
constexpr int kTile1Sm = 1;  // 128 x 256 elements per CTA
constexpr int kTile2Sm = 2;  // 256 x 256 elements per CTA pair
constexpr int kTileMax = kTile2Sm;  // last one that a caller can choose
constexpr int kTileNarrow = 3;      // SM pair with narrow units (tc_choose_shape)
constexpr int kTileSmall = 4;       // one SM, for launches of channels of one tile only
constexpr int kSmallElements = 128;  // the largest of these channels
__host__ __device__ inline bool tile_is_pair(int tile) {
    return tile == kTile2Sm || tile == kTileNarrow;
}
// The variant by which a launch of `tile` runs when its largest channel has
// max_elements.  Asked once for the whole launch, before its units are made, so
// that their costs are those of the kernel that runs them.
inline int tc_launch_tile(int tile, int max_elements) {
    return tile == kTile1Sm && max_elements <= kSmallElements ? kTileSmall : tile;
}

// Scheduling cost of a unit over samples [t0, t1), in cycles as measured with
// clock64: nx x tiles of 128 elements against one y tile (one SM) or two (SM
// pair).  SM pair: 512 per step of two lanes, 470 per step of one, at least the
// lanes' drains of 4,700 each, and 1,500 of pipeline latency.  One SM: 910 per stage
// of two x tiles, but 890 of one (the unpack warps' passes set the pace, not the bytes),
// and 6,000 for each x tile's accumulator hand-off (one unit per SM, T = 512 / 16384: 18.7
// / 249.7 us with two x tiles, 14.4 / 242.0 with one, 29.0 / 482.7 one of each).  With 2 : 3
// for them, cut plans gave some SMs half as much again as others (E = 640, F = 8,
// T = 16384 169 us, 135 now; E = 1920 977, 900).  Channels of one tile by themselves
// (tc_small_correlator.cu): 400 per step (250-430 by elements and rows), and the
// drains overlap the next unit's steps.  Plans, batches, streams and the
// allocation-free entry point share it so that their schedules agree.
__host__ __device__ inline int unit_cost(int tile, int t0, int t1, int nx) {
    const int stages = (t1 - t0 + kUnitStageSamples - 1) / kUnitStageSamples;
    if (tile == kTileSmall) return 400 * stages + 2000;
    if (tile == kTile1Sm) return (870 + 20 * nx) * stages + 6000 * nx;
    const int skew = stages < kSkewStages ? stages : kSkewStages;
    const int steps = nx < 2 ? 470 * stages : 512 * (stages - skew) + 2 * 470 * skew;
    const int drain = 4700 * nx;
    return (steps > drain ? steps : drain) + 1500;
}
// Its inverse: the most stages whose cost is at most `budget` cycles (0: none).
// tc_balance asks for it once per piece and trial; a search over unit_cost took
// half of a plan's table building.
inline int unit_stages(int tile, long long budget, int nx) {
    if (tile == kTileSmall) return (int)std::max(0LL, (budget - 2000) / 400);
    if (tile == kTile1Sm) return (int)std::max(0LL, (budget - 6000 * nx) / (870 + 20 * nx));
    const long long steps = budget - 1500;
    if (steps < 4700 * nx) return 0;
    if (nx < 2) return (int)(steps / 470);
    const long long skewed = 2 * 470 * kSkewStages;  // both lanes alone for kSkewStages steps
    return (int)(steps < skewed ? steps / (2 * 470) : kSkewStages + (steps - skewed) / 512);
}

// The TMA maps of a launch whose channels share them (TcLaunch::use_param_map).
struct TcMaps {
    CUtensorMap in;       // samples, 128-element tiles
    CUtensorMap in_half;  // samples, 64-element tiles (x of the SM-pair kernel)
    CUtensorMap out;      // blocks
};

struct TcLaunch {
    const ChanDesc *chans;  // device
    const Unit *units;      // device, grouped by CTA
    int nunits;
    int max_samples;        // samples of the longest unit
    const int *cta_offsets; // device, grid + 1 entries
    int after_zero = 0;     // 1: launch_zero(blocks) was the stream's previous launch
    int static_tables = 0;  // 1: no work of the stream writes the tables
    int use_param_map;      // 1: every channel uses the kernel-parameter map
    int map;                // value map (MAP_*)
    int ut;
    int accumulate;
    int *err;
    int grid;               // persistent CTAs (<= SMs)
};

bool tc_supported(int E, int T);
// Assigns units to `grid` persistent CTAs (longest first, to the least
// loaded CTA) and reorders them CTA by CTA; offsets gets grid + 1 entries.
void tc_schedule(std::vector<Unit> &u, int grid, std::vector<int> &offsets);
// Samples of the longest unit.
int tc_max_samples(const std::vector<Unit> &u);
// Makespan of that assignment, in cycles, from the units' costs (reordered here).
long long tc_estimate_makespan(std::vector<int> &costs, int grid);
// Cycles by which zeroing `out_bytes` of output first delays a launch.
long long tc_zeroing_cost(int64_t out_bytes);
// A tile variant, a number of sample-range splits and their makespan (0: not
// estimated).
struct TcShape {
    int tile, split;
    long long span;
};
// Shape whose units have the shortest estimated makespan: splits 1-32 (split = 0)
// or the given one, wide or narrow units for the SM pair.  costs_of appends the
// unit costs of a shape; zeroing: cycles that a split costs besides
// (tc_zeroing_cost of an output that has to be zeroed first).
TcShape tc_choose_shape(int tile, int split, int sm_count, long long zeroing,
                        const std::function<void(TcShape, std::vector<int> &)> &costs_of);
// Cuts `units` (a whole launch's, unsplit, of `tile`) into pieces so
// that every one of at most `slots` CTAs or clusters gets the same cost, and
// groups them by CTA (offsets: CTAs + 1), if that beats `best` by 5 %.
bool tc_balance(const TcShape &best, int tile, long long zeroing, std::vector<Unit> &units, int slots,
                std::vector<int> &offsets);
// Appends the unit costs of `count` integrations of E elements and T samples.
void tc_append_costs(TcShape shape, int E, int T, int count, std::vector<int> &costs);
// Encodes the TMA map of packed samples: dims {E, channels, samples}.
// box_elements elements x 32 samples per tile.
int tc_encode_map(CUtensorMap *m, const void *base, int E, int channels, int64_t samples,
                  int64_t chan_stride, int64_t sample_stride, int box_elements = 128);
// Encodes the TMA map of a block buffer seen as `rows` rows of 64 int32 words
// (one 32-cell block row of Re/Im pairs), tile {32 words, 32 rows}, 128-byte
// swizzle.  The epilogues store (or add) their tiles through it.  rows must
// stay below 2^31 (tc_out_rows_ok).
int tc_encode_out_map(CUtensorMap *m, void *base, int64_t rows);
inline bool tc_out_rows_ok(int64_t rows) { return rows > 0 && rows < (1LL << 31); }
// maps: the maps every channel uses when L.use_param_map.
cudaError_t tc_launch(const TcLaunch &L, const TcMaps *maps, cudaStream_t st);

// ---- kernel for channels of at most 128 elements (tc_small_correlator.cu) ----
// Whether a launch whose longest unit has max_samples multiplies two operand rows
// instead of three (tc_small_correlator.cu's top): from 24 steps on.  One unit per
// SM gains there at every E (us, three rows / two: F = 148, T = 768 E = 32 6.9 / 6.3,
// E = 96 8.3 / 7.9; pieces of at most 28 steps, E = 64, F = 8, T = 16384 9.7 / 9.2); at 4
// steps two rows lose, between it is even.  Only the longest unit counts, so launches
// whose other units are short lose: E = 96, F = 100, T = 1000 adding, cut into pieces of
// mostly 21 steps and fewer, 8.6 / 9.3; a batch of 1000 x (96, 64) beside one
// (96, 1024) 14.4 / 18.6.
inline bool small_two_rows(int max_samples) {
    return (max_samples + kUnitStageSamples - 1) / kUnitStageSamples >= 24;
}
cudaError_t tc_small_launch(const TcLaunch &L, const TcMaps *maps, cudaStream_t st);

// ---- 2-SM tensor-core kernel (tc_pair_correlator.cu) ----
// Units of 256 y x (128 nl) x elements (tyx = ty2 | tx << 10 | nl << 20: a pair of
// 128-element y tiles, the first of nl x tiles), computed by a cluster of two
// CTAs with tcgen05.mma.cta_group::2; nl = 2, or 1 where the second x tile lies
// outside the matrix and in narrow units.  In the launch, grid counts clusters
// and cta_offsets is indexed by cluster.
void tc_append_pair_units(std::vector<Unit> &out, bool narrow, int chan, int E, int t_begin,
                          int t_end, int tsplit, long long out_off);
cudaError_t tc_pair_launch(const TcLaunch &L, const TcMaps *maps, cudaStream_t st);

int tc_default_tile(int E);
// Dispatch by tile variant: units of one channel's sample range, persistent
// CTAs (or clusters) for `sm_count` SMs, and the launch.
void tc_append_tile_units(int tile, std::vector<Unit> &out, int chan, int E, int t_begin,
                          int t_end, int tsplit, long long out_off);
int tc_tile_slots(int tile, int sm_count);
cudaError_t tc_tile_launch(int tile, const TcLaunch &L, const TcMaps *maps, cudaStream_t st);
// Encodes a launch's shared maps for F channels of E elements and T samples
// with blocks at d_blocks; 0 or an error code.
int tc_encode_maps(TcMaps *m, const void *d_packed, int E, int F, int T, void *d_blocks);
// Device address of the error word of chx_correlate_noalloc on the current
// device (noalloc.cu); the bounded-wait self-test writes it in mode 2.
cudaError_t noalloc_error_word(int **out);
// The autotuner's cached choice for (device, E, T) (batch.cu): true and the
// tile variant when an entry with the same E and a T within a factor 2 exists.
bool tc_tune_lookup(int device, int E, int T, int *tile);

}  // namespace chx
