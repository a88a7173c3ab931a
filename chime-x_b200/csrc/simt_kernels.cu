// simt_kernels.cu -- CUDA-core kernels of libchimex:
//   * correlate_simt: dp4a correlator over 32x32 blocks (baseline path and the
//     fallback for shapes the tensor-core kernel does not take; also used by
//     chx_corr_compat with the offset-domain value maps),
//   * offset_accumulate: offsetAccumulateElements (offset_accumulator.cl:7-49),
//   * preseed: the four preseed variants (preseed_multifreq*_UT.cl),
//   * block -> triangle / full-matrix reorganisation (gpu_data_reorg.c:36-124).
#include <algorithm>

#include "chimex_internal.h"

namespace chx {

namespace {

// (by, bx) of block b in the row-major upper-triangle enumeration of
// main_wrapper.c:529-540: row y starts at block y nb1 - y (y - 1) / 2.  The root
// of that quadratic, corrected for the float's rounding.
__device__ __forceinline__ void decode_block(int b, int nb1, int &by, int &bx) {
    auto start = [&](int y) { return y * nb1 - y * (y - 1) / 2; };
    const float n = 2.0f * nb1 + 1.0f;
    int y = (int)(0.5f * (n - sqrtf(fmaxf(n * n - 8.0f * (float)b, 0.0f))));
    y = min(max(y, 0), nb1 - 1);
    while (y > 0 && start(y) > b) y--;
    while (y + 1 < nb1 && start(y + 1) <= b) y++;
    by = y;
    bx = y + (b - start(y));
}

// Operand bytes of one packed sample under a value map (see chimex_internal.h).
struct Ops {
    int a0, a1, b0, b1, b2, b3;
};

template <int MAP>
__device__ __forceinline__ Ops map_byte(uint32_t p) {
    const int hi = (p >> 4) & 15, lo = p & 15;
    Ops o;
    if (MAP == MAP_EXACT) {
        o.a0 = hi - 8; o.a1 = lo - 8;
        o.b0 = hi - 8; o.b1 = lo - 8; o.b2 = 8 - lo; o.b3 = hi - 8;
    } else if (MAP == MAP_CONF) {
        o.a0 = hi; o.a1 = lo;
        o.b0 = hi; o.b1 = lo; o.b2 = -lo; o.b3 = hi;
    } else {
        o.a0 = hi; o.a1 = 15 - lo;
        o.b0 = hi; o.b1 = -lo; o.b2 = -lo; o.b3 = -hi;
    }
    return o;
}

__device__ __forceinline__ uint32_t put_byte(uint32_t w, int v, int j) {
    return w | ((uint32_t)(v & 0xFF) << (8 * j));
}

// One CTA = one 32x32 output block of one channel over one sample range.
// Each of the 256 threads owns a 2x2 group of cells.  Samples are staged 32
// at a time: packed bytes -> shared memory -> int8x4 words per element
// ([component][word][element], conflict-free for the compute loop).
template <int MAP>
__global__ void __launch_bounds__(256)
correlate_simt_kernel(const uint8_t *__restrict__ packed, int32_t *__restrict__ blocks,
                      int E, int F, int T, int nb1, int64_t nb, int ut, int mode,
                      int tchunk) {
    __shared__ uint32_t py[32][8];  // [sample][element/4] packed bytes
    __shared__ uint32_t px[32][8];
    __shared__ int32_t A[2][8][32];  // [a0|a1][sample/4][element]
    __shared__ int32_t B[4][8][32];  // [b0..b3][sample/4][element]

    const int b = blockIdx.x, f = blockIdx.y;
    int by, bx;
    decode_block(b, nb1, by, bx);
    const int t_begin = blockIdx.z * tchunk;
    const int t_end = min(T, t_begin + tchunk);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int64_t row = (int64_t)F * E;
    const uint8_t *base = packed + (int64_t)f * E;

    int re[2][2] = {{0, 0}, {0, 0}}, im[2][2] = {{0, 0}, {0, 0}};

    for (int t0 = t_begin; t0 < t_end; t0 += 32) {
        {
            const int r = tid >> 3, c = tid & 7;
            const int t = t0 + r;
            uint32_t vy = 0, vx = 0;
            if (t < t_end) {
                vy = *reinterpret_cast<const uint32_t *>(base + t * row + by * 32 + c * 4);
                vx = *reinterpret_cast<const uint32_t *>(base + t * row + bx * 32 + c * 4);
            }
            py[r][c] = vy;
            px[r][c] = vx;
        }
        __syncthreads();
        {
            const int e = tid & 31, w = tid >> 5;
            uint32_t a0 = 0, a1 = 0, b0 = 0, b1 = 0, b2 = 0, b3 = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int s = 4 * w + j;
                if (t0 + s < t_end) {
                    const uint32_t pyb = (py[s][e >> 2] >> (8 * (e & 3))) & 0xFF;
                    const uint32_t pxb = (px[s][e >> 2] >> (8 * (e & 3))) & 0xFF;
                    const Ops oy = map_byte<MAP>(pyb), ox = map_byte<MAP>(pxb);
                    a0 = put_byte(a0, oy.a0, j);
                    a1 = put_byte(a1, oy.a1, j);
                    b0 = put_byte(b0, ox.b0, j);
                    b1 = put_byte(b1, ox.b1, j);
                    b2 = put_byte(b2, ox.b2, j);
                    b3 = put_byte(b3, ox.b3, j);
                }
            }
            A[0][w][e] = (int32_t)a0;
            A[1][w][e] = (int32_t)a1;
            B[0][w][e] = (int32_t)b0;
            B[1][w][e] = (int32_t)b1;
            B[2][w][e] = (int32_t)b2;
            B[3][w][e] = (int32_t)b3;
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; w++) {
            int ya0[2], ya1[2], xb0[2], xb1[2], xb2[2], xb3[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                ya0[i] = A[0][w][2 * ty + i];
                ya1[i] = A[1][w][2 * ty + i];
                xb0[i] = B[0][w][2 * tx + i];
                xb1[i] = B[1][w][2 * tx + i];
                xb2[i] = B[2][w][2 * tx + i];
                xb3[i] = B[3][w][2 * tx + i];
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    re[i][j] = __dp4a(ya0[i], xb0[j], re[i][j]);
                    re[i][j] = __dp4a(ya1[i], xb1[j], re[i][j]);
                    im[i][j] = __dp4a(ya0[i], xb2[j], im[i][j]);
                    im[i][j] = __dp4a(ya1[i], xb3[j], im[i][j]);
                }
        }
        __syncthreads();
    }

    int32_t *blk = blocks + ((int64_t)f * nb + b) * 2048;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int y = 2 * ty + i, x = 2 * tx + j;
            const int vr = re[i][j];
            const int vi = ut ? im[i][j] : (int)(0u - (uint32_t)im[i][j]);
            int32_t *cell = blk + y * 64 + 2 * x;
            if (mode == 0) {
                *reinterpret_cast<int2 *>(cell) = make_int2(vr, vi);
            } else if (mode == 1) {
                int2 o = *reinterpret_cast<int2 *>(cell);
                o.x = (int)((uint32_t)o.x + (uint32_t)vr);
                o.y = (int)((uint32_t)o.y + (uint32_t)vi);
                *reinterpret_cast<int2 *>(cell) = o;
            } else {
                atomicAdd(cell, vr);
                atomicAdd(cell + 1, vi);
            }
        }
}

// Zeroes words of 16 bytes.  The next kernel may start meanwhile, but not before
// all work ahead of this kernel has ended: it may read its inputs at once and
// waits only before it writes to the zeroed words.
__global__ void zero_kernel(uint4 *out, int64_t n) {
    pdl_wait();
    pdl_launch_dependents();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = make_uint4(0u, 0u, 0u, 0u);
}

// offsetAccumulateElements (offset_accumulator.cl:18-47).  The work is the
// (vector block, 16-sample group) space: a vector block is 32 consecutive
// 16-byte vectors of a sample row (16 (f, e) bytes each), a group 16 samples.
// Each CTA (16 warps per SM, in one CTA unless T is short: offset_split) takes an
// equal, contiguous share of that space, so every SM streams the same number of
// bytes; inside a share, warp w streams the groups w, w + WARPS, ... of one vector
// block at a time (each lane one vector: coalesced 512-byte rows), loading a group's
// 16 vectors at once so that enough bytes are in flight to keep HBM busy (131 KiB
// per SM).  Four samples' words are
// transposed so that a word holds four samples of one element, whose byte sum
// (16 re + im) and low-nibble sum (im) are one dp4a each: three ALU instructions
// per word and 32-bit sums throughout, where masking and adding nibbles in byte
// lanes took six with the flushes.  The warps' sums meet in shared memory, and
// the CTAs' in one atomic add per word for each vector block they touch, after
// the kernel that zeroed the sums (zero_kernel) has ended.  Bound by HBM: with
// the zeroing, E = 2048, F = 8, T = 16384 (268 MB) took 53.1 us with three CTAs of
// 8 warps and byte-lane adds, 48.1 with dp4a and two CTAs, 45.4 with one CTA of
// 16 warps (5.9 TB/s; the read alone 41 us at the copy rate); half as many bytes
// in flight or twice as many CTAs measured slower.  Few samples (us, one CTA per
// eight groups / now; adding): E = 96, F = 55, T = 2 22.2 / 5.9, E = 2048, F = 8, T = 16
// 14.7 / 6.0, E = 2048, F = 200, T = 200 22.3 / 18.2, E = 2048, F = 1024, T = 1 55.6 / 28.0, T = 128 82.5 / 56.5.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, kOaWarps / WARPS)
offset_accumulate_kernel(const uint8_t *packed, uint32_t *sums, int64_t nvec, int T,
                         int64_t ngroups, int64_t nwork, int zeroed) {
    __shared__ uint32_t part[WARPS / 2][32][32];  // [warp pair][word][lane]
    if (!zeroed) pdl_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint4 *p = reinterpret_cast<const uint4 *>(packed);
    const int64_t L1 = nwork * (blockIdx.x + 1) / gridDim.x;
    for (int64_t L = nwork * blockIdx.x / gridDim.x; L < L1;) {  // uniform across the CTA
        const int64_t vb = L / ngroups;
        const int64_t end = min(L1, (vb + 1) * ngroups);  // this vector block's part
        const int64_t g0 = L - vb * ngroups, g1 = end - vb * ngroups;
        const int64_t i = vb * 32 + lane;
        uint32_t tot[16], lo[16];  // per element: sums of the bytes and of their low nibbles
#pragma unroll
        for (int k = 0; k < 16; k++) tot[k] = lo[k] = 0u;
        if (i < nvec) {
            for (int64_t g = g0 + w; g < g1; g += WARPS) {
                const int t = (int)(16 * g);
                const uint4 *row = p + (int64_t)t * nvec + i;
                uint4 v[16];
                if (t + 16 <= T) {  // a full group: 16 independent loads in flight
#pragma unroll
                    for (int k = 0; k < 16; k++) v[k] = __ldcs(row + (int64_t)k * nvec);
                } else {
#pragma unroll
                    for (int k = 0; k < 16; k++)
                        v[k] = t + k < T ? __ldcs(row + (int64_t)k * nvec) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int k = 0; k < 16; k += 4) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        auto word = [&](int s) {
                            const uint4 u = v[k + s];
                            return q == 0 ? u.x : q == 1 ? u.y : q == 2 ? u.z : u.w;
                        };
                        const uint32_t a = word(0), b = word(1), c = word(2), e = word(3);
                        const uint32_t ab0 = __byte_perm(a, b, 0x5140);  // a0 b0 a1 b1
                        const uint32_t ab2 = __byte_perm(a, b, 0x7362);  // a2 b2 a3 b3
                        const uint32_t ce0 = __byte_perm(c, e, 0x5140);
                        const uint32_t ce2 = __byte_perm(c, e, 0x7362);
                        const uint32_t x[4] = {
                            __byte_perm(ab0, ce0, 0x5410), __byte_perm(ab0, ce0, 0x7632),
                            __byte_perm(ab2, ce2, 0x5410), __byte_perm(ab2, ce2, 0x7632)};
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            tot[4 * q + j] = __dp4a(x[j], 0x01010101u, tot[4 * q + j]);
                            lo[4 * q + j] = __dp4a(x[j] & 0x0F0F0F0Fu, 0x01010101u, lo[4 * q + j]);
                        }
                    }
                }
            }
        }
        if (end == L1) pdl_launch_dependents();
        if (w < WARPS / 2)
#pragma unroll
            for (int k = 0; k < 16; k++) {
                part[w][2 * k][lane] = (tot[k] - lo[k]) >> 4;
                part[w][2 * k + 1][lane] = lo[k];
            }
        __syncthreads();
        if (w >= WARPS / 2)
#pragma unroll
            for (int k = 0; k < 16; k++) {
                part[w - WARPS / 2][2 * k][lane] += (tot[k] - lo[k]) >> 4;
                part[w - WARPS / 2][2 * k + 1][lane] += lo[k];
            }
        __syncthreads();
        pdl_wait();  // the sums have been zeroed
        // Thread r handles (word, lane) pairs r, r + 32 WARPS, ...: sum over the warps.
#pragma unroll
        for (int r = threadIdx.x; r < 32 * 32; r += WARPS * 32) {
            const int k = r >> 5, l = r & 31;
            const int64_t iv = vb * 32 + l;
            uint32_t acc = 0u;
#pragma unroll
            for (int ww = 0; ww < WARPS / 2; ww++) acc += part[ww][k][l];
            if (iv < nvec && acc != 0u) atomicAdd(sums + 32 * iv + k, acc);
        }
        __syncthreads();  // part is rewritten for the next vector block
        L = end;
    }
}

// preseed: writes (=) the offset correction of every cell of one block.
// Formulas: preseed_multifreq_UT.cl:54-70 / preseed_multifreq.cl:54-70
// (conference) and preseed_multifreq_highly_packed_correlator_method{_UT,}.cl
// :54-70 (packed); x is the column element, y the row element.  sx / sy hold
// the (re, im) sums of the block's 32 columns / rows; 256 threads write two
// neighbouring cells (xl, xl + 1) per 16-byte store.
__device__ __forceinline__ void preseed_block(const uint32_t *sx, const uint32_t *sy,
                                              int32_t *blk, uint32_t t128,
                                              int packed_variant, int ut, int tid) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int c2 = tid + 256 * k, yl = c2 >> 4, xl0 = (c2 & 15) * 2;
        const uint32_t yr = sy[2 * yl], yi = sy[2 * yl + 1];
        uint32_t v[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int xl = xl0 + h;
            const uint32_t xr = sx[2 * xl], xi = sx[2 * xl + 1];
            uint32_t re, imv;
            if (!packed_variant) {
                re = t128 - 8u * (xr + xi + yr + yi);
                imv = ut ? 8u * ((xi - xr) + (yr - yi)) : 8u * ((xr - xi) + (yi - yr));
            } else {
                re = t128 - 8u * xr + 7u * xi - 8u * (yr + yi);
                imv = ut ? 8u * xi + 7u * xr + 8u * (yr - yi)
                         : 0u - 8u * xi - 7u * xr - 8u * (yr - yi);
            }
            v[2 * h] = re;
            v[2 * h + 1] = imv;
        }
        *reinterpret_cast<int4 *>(blk + (yl * 32 + xl0) * 2) =
            make_int4((int)v[0], (int)v[1], (int)v[2], (int)v[3]);
    }
}

// One CTA per run of kPsBlocks consecutive blocks of one channel: every
// thread issues its 2 x kPsBlocks 16-byte stores back to back (no dependency
// between them), which keeps more bytes in flight per thread than one block
// per CTA.  The blocks' row and column sums are gathered into shared memory
// first.
constexpr int kPsBlocks = 4;

__global__ void __launch_bounds__(256)
preseed_kernel(const uint32_t *sums, int32_t *blocks, int E, int nb1, int64_t nb, uint32_t t128,
               int packed_variant, int ut) {
    __shared__ uint32_t sx[kPsBlocks][64], sy[kPsBlocks][64];
    pdl_launch_dependents();
    pdl_wait();
    const int f = blockIdx.y;
    const int64_t b0 = (int64_t)blockIdx.x * kPsBlocks;
    const int tid = threadIdx.x;
    for (int i = tid; i < kPsBlocks * 64; i += 256) {
        const int k = i >> 6, w = i & 63;
        if (b0 + k < nb) {
            int by, bx;
            decode_block((int)(b0 + k), nb1, by, bx);
            sx[k][w] = sums[((int64_t)f * E + bx * 32) * 2 + w];
            sy[k][w] = sums[((int64_t)f * E + by * 32) * 2 + w];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPsBlocks; k++)
        if (b0 + k < nb)
            preseed_block(sx[k], sy[k], blocks + ((int64_t)f * nb + b0 + k) * 2048, t128,
                          packed_variant, ut, tid);
}

// Block layout -> packed triangle (gpu_data_reorg.c:76-124).  A CTA takes
// kTriBlocks consecutive blocks: all are read into shared memory with 16-byte
// loads first; each block row is a contiguous run of cells in the triangle
// (x >= y only on the diagonal block) starting at any cell index, so every row
// is written as 16-byte stores of cell pairs, with a single 8-byte store for an
// odd first cell and for an odd last cell.  16 threads per row.  Bound by HBM:
// E = 2048, F = 8 (271 MB, three buffer sets in turn) took 48.0 us with one block
// per CTA, 44.0 now (6.2 TB/s; a plain copy of as many bytes 45.1), 45.1 with three
// blocks, 52.4 with four (too few CTAs per SM), 49.3 with streaming loads.
constexpr int kTriBlocks = 2;

__global__ void __launch_bounds__(256)
blocks_to_triangle_kernel(const int32_t *blocks, int32_t *tri, int E, int nb1, int64_t nb) {
    __shared__ __align__(16) int2 cells[kTriBlocks][32 * 32];
    pdl_launch_dependents();
    pdl_wait();
    const int b0 = blockIdx.x * kTriBlocks, f = blockIdx.y;
    const int n = (int)min((int64_t)kTriBlocks, nb - b0);
    const int64_t ntri = (int64_t)E * (E + 1) / 2;
    const int4 *blk = reinterpret_cast<const int4 *>(blocks + ((int64_t)f * nb + b0) * 2048);
    int4 *c4 = reinterpret_cast<int4 *>(cells);
    int4 v[2 * kTriBlocks];
#pragma unroll
    for (int k = 0; k < 2 * kTriBlocks; k++)
        if (k < 2 * n) v[k] = blk[threadIdx.x + 256 * k];
    int by, bx;
    decode_block(b0, nb1, by, bx);
#pragma unroll
    for (int k = 0; k < 2 * kTriBlocks; k++)
        if (k < 2 * n) c4[threadIdx.x + 256 * k] = v[k];
    __syncthreads();
    for (int i = 0; i < n; i++) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int slot = threadIdx.x + 256 * r, yl = slot >> 4, k = slot & 15;
            const int xs = (bx == by) ? yl : 0;  // first cell of the row written
            const int64_t y = by * 32 + yl;
            const int64_t a0 = f * ntri + y * E - (y - 1) * y / 2 + (bx * 32 + xs - y);
            const int head = (int)(a0 & 1);      // odd start: one 8-byte cell first
            const int m = 32 - xs - head;        // cells after the head
            const int2 *row = cells[i] + yl * 32;
            if (k < m / 2) {
                const int x = xs + head + 2 * k;
                const int2 u = row[x], w = row[x + 1];
                *reinterpret_cast<int4 *>(tri + 2 * (a0 + head + 2 * k)) =
                    make_int4(u.x, u.y, w.x, w.y);
            }
            if (k == 15 && head) *reinterpret_cast<int2 *>(tri + 2 * a0) = row[xs];
            if (k == 14 && (m & 1)) *reinterpret_cast<int2 *>(tri + 2 * (a0 + 31 - xs)) = row[31];
        }
        if (++bx == nb1) bx = ++by;  // the next block of the row, or the next row's diagonal
    }
}

// Block layout -> full Hermitian matrix (gpu_data_reorg.c:36-74).  The upper
// triangle is written row by row straight from the block; the mirrored lower
// triangle (conjugates) goes through a shared-memory transpose so that its
// rows are written contiguously too.
__global__ void __launch_bounds__(256)
blocks_to_full_kernel(const int32_t *blocks, int32_t *full, int E, int nb1, int64_t nb) {
    __shared__ int2 tile[32][33];
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.x, f = blockIdx.y;
    int by, bx;
    decode_block(b, nb1, by, bx);
    const int32_t *blk = blocks + ((int64_t)f * nb + b) * 2048;
    int32_t *m = full + (int64_t)f * E * E * 2;
    int2 v[4];  // all loads first: the stores may alias them for the compiler
#pragma unroll
    for (int k = 0; k < 4; k++)
        v[k] = *reinterpret_cast<const int2 *>(blk + 2 * (threadIdx.x + 256 * k));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int c = threadIdx.x + 256 * k, yl = c >> 5, xl = c & 31;
        const int64_t y = by * 32 + yl, x = bx * 32 + xl;
        tile[yl][xl] = v[k];
        if (x >= y) *reinterpret_cast<int2 *>(m + (y * E + x) * 2) = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int c = threadIdx.x + 256 * k, xl = c >> 5, yl = c & 31;
        const int64_t y = by * 32 + yl, x = bx * 32 + xl;
        if (x > y) {
            const int2 v = tile[yl][xl];
            *reinterpret_cast<int2 *>(m + (x * E + y) * 2) = make_int2(v.x, (int)(0u - (uint32_t)v.y));
        }
    }
}

}  // namespace

cudaError_t launch_correlate_simt(const uint8_t *packed, int32_t *blocks, int E, int F,
                                  int T, int map, int ut, int mode, int splits,
                                  cudaStream_t st) {
    const int nb1 = E / 32;
    const int64_t nb = num_blocks_of(E);
    if (splits < 1) splits = 1;
    int tchunk = (T + splits - 1) / splits;
    tchunk = (tchunk + 31) / 32 * 32;
    splits = (T + tchunk - 1) / tchunk;
    dim3 grid((unsigned)nb, (unsigned)F, (unsigned)splits);
    if (map == MAP_EXACT)
        correlate_simt_kernel<MAP_EXACT><<<grid, 256, 0, st>>>(packed, blocks, E, F, T, nb1, nb, ut, mode, tchunk);
    else if (map == MAP_CONF)
        correlate_simt_kernel<MAP_CONF><<<grid, 256, 0, st>>>(packed, blocks, E, F, T, nb1, nb, ut, mode, tchunk);
    else
        correlate_simt_kernel<MAP_PACKED><<<grid, 256, 0, st>>>(packed, blocks, E, F, T, nb1, nb, ut, mode, tchunk);
    return cudaGetLastError();
}

cudaError_t launch_offset_accumulate(const uint8_t *packed, uint32_t *sums, int E, int F,
                                     int T, bool zeroed, cudaStream_t st) {
    const int64_t nvec = (int64_t)F * E / 16;  // E % 32 == 0
    const int64_t vblocks = (nvec + 31) / 32;
    const int64_t ngroups = (T + 15) / 16;
    const int64_t nwork = vblocks * ngroups;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const OffsetSplit split = offset_split(vblocks, ngroups, sms);
    const dim3 grid((unsigned)split.ctas), block(split.warps * 32);
    if (split.warps == kOaWarps)
        return launch_pdl(offset_accumulate_kernel<kOaWarps>, grid, block, 0, st, packed, sums, nvec,
                          T, ngroups, nwork, zeroed ? 1 : 0);
    return launch_pdl(offset_accumulate_kernel<kOaShortWarps>, grid, block, 0, st, packed, sums, nvec,
                      T, ngroups, nwork, zeroed ? 1 : 0);
}

cudaError_t launch_zero(void *out, int64_t bytes, cudaStream_t st) {
    const int64_t n = bytes / 16;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(1184, (n + 1023) / 1024));
    return launch_pdl(zero_kernel, dim3(grid), dim3(256), 0, st, static_cast<uint4 *>(out), n);
}

cudaError_t launch_preseed(const uint32_t *sums, int32_t *blocks, int E, int F, int T,
                           int packed_variant, int ut, cudaStream_t st) {
    const int64_t nb = num_blocks_of(E);
    dim3 grid((unsigned)((nb + kPsBlocks - 1) / kPsBlocks), (unsigned)F);
    return launch_pdl(preseed_kernel, grid, dim3(256), 0, st, sums, blocks, E, E / 32, nb,
                      (uint32_t)T * 128u, packed_variant, ut);
}

cudaError_t launch_blocks_to_triangle(const int32_t *blocks, int32_t *tri, int E, int F,
                                      cudaStream_t st) {
    dim3 grid((unsigned)((num_blocks_of(E) + kTriBlocks - 1) / kTriBlocks), (unsigned)F);
    return launch_pdl(blocks_to_triangle_kernel, grid, dim3(256), 0, st, blocks, tri, E, E / 32,
                      num_blocks_of(E));
}

cudaError_t launch_blocks_to_full(const int32_t *blocks, int32_t *full, int E, int F,
                                  cudaStream_t st) {
    dim3 grid((unsigned)num_blocks_of(E), (unsigned)F);
    return launch_pdl(blocks_to_full_kernel, grid, dim3(256), 0, st, blocks, full, E, E / 32,
                      num_blocks_of(E));
}

}  // namespace chx
