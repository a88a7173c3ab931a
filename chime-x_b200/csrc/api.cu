// api.cu -- C ABI of libchimex: plans and the plain-path entry points.
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>

#include "chimex_internal.h"

namespace chx {

static thread_local char g_err[512] = "";

int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int cuda_fail(cudaError_t e, const char *what) {
    return fail(e == cudaErrorMemoryAllocation ? CHX_E_NOMEM : CHX_E_CUDA, "%s: %s (%s)",
                what, cudaGetErrorString(e), cudaGetErrorName(e));
}

void clear_error() { g_err[0] = 0; }

}  // namespace chx

using namespace chx;

namespace {

// Device buffers passed to the plan entry points must be 16-byte aligned: the
// tensor-core kernels move them with TMA and the CUDA-core kernels with 8-
// and 16-byte vector accesses.  (Allocations from cudaMalloc and torch are
// 256-byte aligned.)
bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

void free_plan_device(chx_plan *p) {
    if (p->d_err) cudaFree(p->d_err);
    if (p->d_chans) cudaFree(p->d_chans);
    p->d_err = nullptr;
    p->d_chans = nullptr;
}

// Channel table and work units of the tensor-core kernel for the plan's
// shape: F channels sharing one TMA map (passed per launch), and the units of a
// launch that stores and of one that adds, grouped by CTA: longest first, or, where
// they are balanced, end to end in channel order.
cudaError_t build_tc_tables(chx_plan *p) {
    std::vector<ChanDesc> chans(p->F);
    memset(chans.data(), 0, chans.size() * sizeof(ChanDesc));
    for (int f = 0; f < p->F; f++) {
        chans[f].E = p->E;
        chans[f].nb1 = (int)p->NB1;
        chans[f].fcoord = f;
        chans[f].orow = (int)((int64_t)f * p->NB * 32);
    }
    // Unset options: the tile is the autotuner's cached choice for this shape,
    // if any, else the default; the split comes from the makespan estimate,
    // which sees how many units this plan has (the tuner times a workload that
    // fills the GPU, where splitting only adds hand-offs).
    int default_tile = p->tile;
    if (!default_tile && !tc_tune_lookup(p->device, p->E, p->T, &default_tile))
        default_tile = tc_default_tile(p->E);
    default_tile = tc_launch_tile(default_tile, p->E);
    const int slots = std::max(1, tc_tile_slots(default_tile, p->sm_count));
    std::vector<Unit> units[2];
    std::vector<int> offsets[2];
    size_t bytes = chans.size() * sizeof(ChanDesc);
    // Launches that add to their output zero nothing, so cutting units costs
    // them less, and their table may be another one.
    TcShape uncut{0, 0, 0};  // the first table's shape if its units are not balanced
    for (int add = 0; add < 2; add++) {
        const long long zeroing = add ? 0 : tc_zeroing_cost(p->F * p->NB * 8192);
        const TcShape shape = tc_choose_shape(default_tile, p->tsplit, p->sm_count, zeroing,
                                              [&](TcShape s, std::vector<int> &costs) {
                                                  tc_append_costs(s, p->E, p->T, p->F, costs);
                                              });
        auto append_units = [&](int tile, int split) {
            units[add].clear();
            for (int f = 0; f < p->F; f++)
                tc_append_tile_units(tile, units[add], f, p->E, 0, p->T, split, 0);
        };
        int tile = default_tile;
        bool balanced = false;
        if (!p->tsplit && shape.span > 0) {
            append_units(tile, 1);
            balanced = tc_balance(shape, tile, zeroing, units[add], slots, offsets[add]);
        }
        if (!balanced && shape.tile == uncut.tile && shape.split == uncut.split) {
            units[add].clear();
            p->tc[add] = p->tc[0];
            continue;
        }
        if (!balanced) {
            uncut = shape;
            tile = shape.tile;
            append_units(tile, shape.split);
            tc_schedule(units[add], (int)std::min<size_t>(units[add].size(), (size_t)slots),
                        offsets[add]);
        }
        auto &t = p->tc[add];
        t.first = bytes;
        t.nunits = (int)units[add].size();
        t.grid = (int)offsets[add].size() - 1;
        t.tile = tile;
        t.max_unit = tc_max_samples(units[add]);
        t.has_split_units = false;
        for (const Unit &u : units[add]) t.has_split_units |= (u.split != 0);
        bytes += units[add].size() * sizeof(Unit) + (offsets[add].size() * sizeof(int) + 31) / 32 * 32;
    }
    // One allocation and one copy for all tables.
    std::vector<char> tables(bytes);
    memcpy(tables.data(), chans.data(), chans.size() * sizeof(ChanDesc));
    for (int add = 0; add < 2; add++) {
        if (units[add].empty()) continue;  // shares the other table
        char *h = tables.data() + p->tc[add].first;
        const size_t ubytes = units[add].size() * sizeof(Unit);
        memcpy(h, units[add].data(), ubytes);
        memcpy(h + ubytes, offsets[add].data(), offsets[add].size() * sizeof(int));
    }
    if (p->d_chans) cudaFree(p->d_chans);
    p->d_chans = nullptr;
    cudaError_t e = cudaMalloc(&p->d_chans, bytes);
    if (e == cudaSuccess) e = cudaMemcpy(p->d_chans, tables.data(), bytes, cudaMemcpyHostToDevice);
    return e;
}

// The tensor-core path addresses the plan's blocks as F*NB*32 rows of a TMA map.
bool plan_tc_ok(const chx_plan *p) {
    return tc_supported(p->E, p->T) && tc_out_rows_ok((int64_t)p->F * p->NB * 32);
}

// Launches the tensor-core kernel on the plan's tables with `map`.
int run_tc(chx_plan *p, const uint8_t *d_packed, int32_t *d_blocks, int map, int accumulate,
           cudaStream_t st) {
    if ((reinterpret_cast<uintptr_t>(d_packed) & 15) != 0)
        return fail(CHX_E_INVALID, "packed input must be 16-byte aligned for TMA");
    if ((reinterpret_cast<uintptr_t>(d_blocks) & 15) != 0)
        return fail(CHX_E_INVALID, "block buffer must be 16-byte aligned for TMA");
    TcMaps maps;
    const int r = tc_encode_maps(&maps, d_packed, p->E, p->F, p->T, d_blocks);
    if (r != 0) return fail(CHX_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", r);
    TcLaunch L;
    const auto &t = p->tc[accumulate ? 1 : 0];
    if (t.has_split_units && !accumulate) {
        CHX_CUDA(launch_zero(d_blocks, chx_plan_block_words(p) * 4, st));
        L.after_zero = 1;
    }
    L.chans = (const ChanDesc *)p->d_chans;
    L.units = (const Unit *)((const char *)p->d_chans + t.first);
    L.nunits = t.nunits;
    L.max_samples = t.max_unit;
    L.static_tables = 1;
    L.cta_offsets = (const int *)(L.units + t.nunits);
    L.use_param_map = 1;
    L.map = map;
    L.ut = p->ut;
    L.accumulate = accumulate;
    L.err = p->d_err;
    L.grid = t.grid;
    CHX_CUDA(tc_tile_launch(t.tile, L, &maps, st));
    return CHX_OK;
}

}  // namespace

extern "C" {

const char *chx_version(void) { return "chimex-b200 0.1"; }

const char *chx_last_error(void) { return g_err; }

int chx_plan_create(chx_plan **plan, int E, int F, int T, int TA, int ut, int kernel_batch,
                    int device) {
    clear_error();
    NvtxRange nvtx_("chx_plan_create");
    if (!plan) return fail(CHX_E_INVALID, "plan pointer is NULL");
    *plan = nullptr;
    if (E < 32 || E % 32 != 0)
        return fail(CHX_E_INVALID, "num_elements=%d must be a positive multiple of 32", E);
    if (E > 65536) return fail(CHX_E_UNSUPPORTED, "num_elements=%d exceeds 65536", E);
    if (F < 1) return fail(CHX_E_INVALID, "num_frequencies=%d must be >= 1", F);
    if (T < 1 || T > 16777215)
        return fail(CHX_E_INVALID, "num_timesamples=%d outside [1, 16777215]", T);
    if (TA < 1) return fail(CHX_E_INVALID, "time_accum=%d must be >= 1", TA);
    if (ut != 0 && ut != 1)
        return fail(CHX_E_INVALID, "upper_triangle_convention=%d not in {0,1}", ut);
    if (kernel_batch != 0 && kernel_batch != 1)
        return fail(CHX_E_INVALID, "kernel_batch=%d not in {0,1}", kernel_batch);
    int ndev = 0;
    CHX_CUDA(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev)
        return fail(CHX_E_INVALID, "device=%d outside [0,%d)", device, ndev);
    DeviceGuard g(device);
    if (!g.ok) return fail(CHX_E_CUDA, "cudaSetDevice(%d) failed", device);
    chx_plan *p = new (std::nothrow) chx_plan();
    if (!p) return fail(CHX_E_NOMEM, "host allocation failed");
    p->E = E;
    p->F = F;
    p->T = T;
    p->TA = TA;
    p->ut = ut;
    p->kernel_batch = kernel_batch;
    p->device = device;
    p->NB1 = E / 32;
    p->NB = num_blocks_of(E);
    p->algo = CHX_ALGO_AUTO;
    p->tsplit = 0;
    p->tile = 0;
    p->d_err = nullptr;
    p->d_chans = nullptr;
    cudaError_t e = cudaDeviceGetAttribute(&p->sm_count, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaMalloc(&p->d_err, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(p->d_err, 0, sizeof(int));
    if (e == cudaSuccess) e = build_tc_tables(p);
    if (e != cudaSuccess) {
        free_plan_device(p);
        delete p;
        return cuda_fail(e, "plan device state");
    }
    *plan = p;
    return CHX_OK;
}

int chx_plan_destroy(chx_plan *p) {
    clear_error();
    if (!p) return CHX_OK;
    DeviceGuard g(p->device);
    free_plan_device(p);
    delete p;
    return CHX_OK;
}

int chx_plan_set_option(chx_plan *p, int option, int64_t value) {
    clear_error();
    if (!p) return fail(CHX_E_INVALID, "plan is NULL");
    switch (option) {
    case CHX_OPT_ALGO:
        if (value < CHX_ALGO_AUTO || value > CHX_ALGO_TC)
            return fail(CHX_E_INVALID, "unknown algorithm %lld", (long long)value);
        if (value == CHX_ALGO_TC && !plan_tc_ok(p))
            return fail(CHX_E_UNSUPPORTED, "tensor-core path does not take E=%d T=%d", p->E, p->T);
        p->algo = (int)value;
        return CHX_OK;
    case CHX_OPT_TSPLIT: {
        if (value < 0 || value > 4096) return fail(CHX_E_INVALID, "tsplit %lld", (long long)value);
        p->tsplit = (int)value;
        DeviceGuard g(p->device);
        CHX_CUDA(build_tc_tables(p));
        return CHX_OK;
    }
    case CHX_OPT_TILE: {
        if (value < 0 || value > kTileMax)
            return fail(CHX_E_INVALID,
                        "tile variant %lld (0 auto, 1 one SM, 2 SM pair)",
                        (long long)value);
        p->tile = (int)value;
        DeviceGuard g(p->device);
        CHX_CUDA(build_tc_tables(p));
        return CHX_OK;
    }
    default:
        return fail(CHX_E_INVALID, "unknown option %d", option);
    }
}

int64_t chx_plan_block_words(const chx_plan *p) { return p ? (int64_t)p->F * p->NB * 2048 : -1; }
int64_t chx_plan_input_bytes(const chx_plan *p) {
    return p ? (int64_t)p->T * p->F * p->E : -1;
}
int64_t chx_plan_sum_words(const chx_plan *p) { return p ? (int64_t)p->F * p->E * 2 : -1; }
int64_t chx_plan_triangle_words(const chx_plan *p) {
    return p ? (int64_t)p->F * p->E * (p->E + 1) : -1;
}

// Sample-range splits for a plain-path launch of `units` independent output
// tiles: enough CTAs to fill the SMs several times, never below 1.
static int auto_splits(int64_t units, int T, int sm_count, int min_chunk) {
    int64_t want = (int64_t)sm_count * 4;
    int s = 1;
    while (units * s < want && T / (2 * s) >= min_chunk) s *= 2;
    return s;
}

int chx_correlate(chx_plan *p, const uint8_t *d_packed, int32_t *d_blocks, void *stream,
                  int accumulate) {
    clear_error();
    NvtxRange nvtx_("chx_correlate");
    if (!p || !d_packed || !d_blocks) return fail(CHX_E_INVALID, "NULL argument");
    if (!aligned16(d_packed) || !aligned16(d_blocks))
        return fail(CHX_E_INVALID, "device buffers must be 16-byte aligned");
    DeviceGuard g(p->device);
    cudaStream_t st = (cudaStream_t)stream;
    const bool use_tc =
        (p->algo == CHX_ALGO_TC) || (p->algo == CHX_ALGO_AUTO && plan_tc_ok(p));
    if (use_tc) return run_tc(p, d_packed, d_blocks, MAP_EXACT, accumulate ? 1 : 0, st);
    const int splits =
        p->tsplit ? p->tsplit : auto_splits((int64_t)p->NB * p->F, p->T, p->sm_count, 256);
    int mode;
    if (splits > 1) {
        if (!accumulate)
            CHX_CUDA(cudaMemsetAsync(d_blocks, 0, (size_t)chx_plan_block_words(p) * 4, st));
        mode = 2;
    } else {
        mode = accumulate ? 1 : 0;
    }
    CHX_CUDA(launch_correlate_simt(d_packed, d_blocks, p->E, p->F, p->T, MAP_EXACT, p->ut,
                                   mode, splits, st));
    return CHX_OK;
}

int chx_offset_accumulate(chx_plan *p, const uint8_t *d_packed, uint32_t *d_sums,
                          void *stream, int accumulate) {
    clear_error();
    NvtxRange nvtx_("chx_offset_accumulate");
    if (!p || !d_packed || !d_sums) return fail(CHX_E_INVALID, "NULL argument");
    if (!aligned16(d_packed) || !aligned16(d_sums))
        return fail(CHX_E_INVALID, "device buffers must be 16-byte aligned");
    DeviceGuard g(p->device);
    cudaStream_t st = (cudaStream_t)stream;
    if (!accumulate) CHX_CUDA(launch_zero(d_sums, chx_plan_sum_words(p) * 4, st));
    CHX_CUDA(launch_offset_accumulate(d_packed, d_sums, p->E, p->F, p->T, !accumulate, st));
    return CHX_OK;
}

int chx_preseed(chx_plan *p, const uint32_t *d_sums, int32_t *d_blocks, void *stream) {
    clear_error();
    NvtxRange nvtx_("chx_preseed");
    if (!p || !d_sums || !d_blocks) return fail(CHX_E_INVALID, "NULL argument");
    if (!aligned16(d_sums) || !aligned16(d_blocks))
        return fail(CHX_E_INVALID, "device buffers must be 16-byte aligned");
    DeviceGuard g(p->device);
    CHX_CUDA(launch_preseed(d_sums, d_blocks, p->E, p->F, p->T, p->kernel_batch, p->ut,
                            (cudaStream_t)stream));
    return CHX_OK;
}

int chx_corr_compat(chx_plan *p, const uint8_t *d_packed, int32_t *d_blocks, void *stream) {
    clear_error();
    NvtxRange nvtx_("chx_corr_compat");
    if (!p || !d_packed || !d_blocks) return fail(CHX_E_INVALID, "NULL argument");
    if (!aligned16(d_packed) || !aligned16(d_blocks))
        return fail(CHX_E_INVALID, "device buffers must be 16-byte aligned");
    // The reference kernels' own domain (main_wrapper.c:564-569,
    // pairwise_correlator_UT.cl:82, help text main_wrapper.c:57).
    if (p->T % p->TA != 0)
        return fail(CHX_E_INVALID, "T=%d is not a multiple of time_accum=%d", p->T, p->TA);
    if (p->TA % 8 != 0)
        return fail(CHX_E_INVALID, "time_accum=%d is not a multiple of 8", p->TA);
    if (p->T % 32 != 0) return fail(CHX_E_INVALID, "T=%d is not a multiple of 32", p->T);
    if (p->kernel_batch == CHX_KERNEL_CONFERENCE && p->TA > 291)
        return fail(CHX_E_INVALID, "time_accum=%d > 291 overflows the conference kernel", p->TA);
    if (p->kernel_batch == CHX_KERNEL_PACKED && p->TA > 2272)
        return fail(CHX_E_INVALID, "time_accum=%d > 2272 overflows the packed kernel", p->TA);
    if (p->kernel_batch == CHX_KERNEL_PACKED && p->F != 1)
        return fail(CHX_E_UNSUPPORTED,
                    "the packed reference kernel has no channel index: F must be 1 (F=%d)", p->F);
    DeviceGuard g(p->device);
    cudaStream_t st = (cudaStream_t)stream;
    const int map = p->kernel_batch == CHX_KERNEL_PACKED ? MAP_PACKED : MAP_CONF;
    if (p->algo != CHX_ALGO_SIMT && plan_tc_ok(p))
        return run_tc(p, d_packed, d_blocks, map, 1, st);
    const int splits =
        p->tsplit ? p->tsplit : auto_splits((int64_t)p->NB * p->F, p->T, p->sm_count, 256);
    CHX_CUDA(launch_correlate_simt(d_packed, d_blocks, p->E, p->F, p->T, map, p->ut,
                                   splits > 1 ? 2 : 1, splits, st));
    return CHX_OK;
}

int chx_blocks_to_triangle(chx_plan *p, const int32_t *d_blocks, int32_t *d_tri, void *stream) {
    clear_error();
    NvtxRange nvtx_("chx_blocks_to_triangle");
    if (!p || !d_blocks || !d_tri) return fail(CHX_E_INVALID, "NULL argument");
    if (!aligned16(d_blocks) || !aligned16(d_tri))
        return fail(CHX_E_INVALID, "device buffers must be 16-byte aligned");
    DeviceGuard g(p->device);
    CHX_CUDA(launch_blocks_to_triangle(d_blocks, d_tri, p->E, p->F, (cudaStream_t)stream));
    return CHX_OK;
}

int chx_blocks_to_full(chx_plan *p, const int32_t *d_blocks, int32_t *d_full, void *stream) {
    clear_error();
    NvtxRange nvtx_("chx_blocks_to_full");
    if (!p || !d_blocks || !d_full) return fail(CHX_E_INVALID, "NULL argument");
    if (!aligned16(d_blocks) || !aligned16(d_full))
        return fail(CHX_E_INVALID, "device buffers must be 16-byte aligned");
    DeviceGuard g(p->device);
    CHX_CUDA(launch_blocks_to_full(d_blocks, d_full, p->E, p->F, (cudaStream_t)stream));
    return CHX_OK;
}

int chx_plan_check(chx_plan *p, void *stream) {
    clear_error();
    if (!p) return fail(CHX_E_INVALID, "plan is NULL");
    DeviceGuard g(p->device);
    cudaStream_t st = (cudaStream_t)stream;
    int h = 0;
    CHX_CUDA(cudaMemcpyAsync(&h, p->d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    CHX_CUDA(cudaStreamSynchronize(st));
    if (h != 0) {
        CHX_CUDA(cudaMemsetAsync(p->d_err, 0, sizeof(int), st));
        CHX_CUDA(cudaStreamSynchronize(st));
        return fail(CHX_E_TIMEOUT, "a bounded device wait gave up (code 0x%x)", h);
    }
    return CHX_OK;
}

}  // extern "C"
