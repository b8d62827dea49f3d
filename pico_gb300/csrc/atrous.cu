// A-trous denoiser (Util::atrous_denoise, Util/Denoisers.cpp:107-126; blend_pixel :18-101).
//
// Five levels with tap spacing 1, 2, 4, 8, 16 over a 5x5 kernel (the reference's
// table, including its 0.09563 entry at index 17).  Per 64x64 tile (the
// reference's Tiler tiles, clamped at the right and bottom edges) and level the
// blend needs the maximum luminance and the min / max |position| over every
// pixel some tap of the tile reads.  That set is rows x columns, each a union of
// five shifted copies of the tile's range, clamped.  The positions are the same
// at every level, so all five levels' |position| ranges are reduced first,
// separably (per image row over each tile column's footprint columns, then per
// tile over its footprint rows), reading the positions once, beside the packing
// of the inputs into records (prepare, tile_range).  Then each level runs:
//
//   white  the maximum luminance of the level's input colour over each tile's
//          footprint: from the luminance cells that the blend before filled, or
//          (first level; images whose last tile is narrower than the spacing)
//          from the colours (stats: four CTAs per tile, each a quarter of the
//          footprint rows).  max / min are exact, so the order is free, and the
//          selects keep std::max / std::min's NaN behaviour.
//   blend  25 taps a pixel, weights
//          w = k[u] * min(exp(-|dn|^2/0.25),1) * min(exp(-|dp|^2/range^2),1)
//                   * min(exp(-|dalbedo|^2/white^2),1),
//          out = sum(w * c) / sum(w), evaluated with one exponential per tap
//          (see the kernel).
//
// 1920 x 1080: 621 us before the records, cells and tiles below, 452 now.
//
// The statistics are exact; the blend agrees with the reference's arithmetic to
// about 1e-6 relative and keeps its NaN pattern.
#include "exact_math.cuh"
#include "kernels_render.h"

#include <algorithm>

namespace pico {

// Base-2 logarithms of the 5x5 table:
//   0.00292, 0.01306, 0.02154, 0.01306, 0.00292
//   0.01306, 0.05855, 0.09653, 0.05855, 0.01306
//   0.02154, 0.09653, 0.15915, 0.09653, 0.02154
//   0.01306, 0.05855, 0.09563, 0.05855, 0.01306
//   0.00292, 0.01306, 0.02154, 0.01306, 0.00292
__constant__ float kAtrousLog2[25] = {
    -8.41981602f, -6.25870132f, -5.53683805f, -6.25870132f, -8.41981602f,
    -6.25870132f, -4.09418678f, -3.37287879f, -4.09418678f, -6.25870132f,
    -5.53683805f, -3.37287879f, -2.65154099f, -3.37287879f, -5.53683805f,
    -6.25870132f, -4.09418678f, -3.38639283f, -4.09418678f, -6.25870132f,
    -8.41981602f, -6.25870132f, -5.53683805f, -6.25870132f, -8.41981602f};

constexpr float kLog2e = 1.44269504f;
constexpr int kTile = 64;
constexpr int kStatsThreads = 256;
constexpr int kStatsSplit = 4;   // CTAs per tile; each reduces every fourth footprint row group
constexpr int kMaxSpan = kTile + 4 * 16;   // tap footprint of a tile along one axis, spacing <= 16

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Coordinates some tap x + k*s (x in [a, b], k in -2..2, clamped to [0, n-1])
// reaches: the union of the five clamped intervals, merged into at most five
// disjoint sorted spans.  Clamping is monotone, so each interval stays whole.
__device__ __forceinline__ int tap_spans(int a, int b, int s, int n, int* lo, int* hi)
{
    int m = 0;
#pragma unroll
    for (int k = -2; k <= 2; ++k) {
        const int l = clampi(a + k * s, 0, n - 1), h = clampi(b + k * s, 0, n - 1);
        if (m > 0 && l <= hi[m - 1] + 1) {
            hi[m - 1] = max(hi[m - 1], h);
        } else {
            lo[m] = l; hi[m] = h; ++m;
        }
    }
    return m;
}

// Lists the members of the spans in out[] with all threads; returns their count.
__device__ __forceinline__ int list_spans(const int* lo, const int* hi, int m, int* out)
{
    int total = 0;
    for (int i = 0; i < m; ++i) total += hi[i] - lo[i] + 1;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int i = 0, base = 0;
        while (t - base > hi[i] - lo[i]) { base += hi[i] - lo[i] + 1; ++i; }
        out[t] = lo[i] + (t - base);
    }
    return total;
}

__device__ __forceinline__ float luminance(float r, float g, float b)
{
    using namespace ex;
    return add(add(mul(r, 0.2126f), mul(g, 0.587f)), mul(b, 0.114f));
}

// Maximum luminance over this CTA's quarter of a tile's footprint rows, into the tile's
// white point (cleared before; non-negative floats order like their bits).
__global__ void __launch_bounds__(kStatsThreads) atrous_stats_kernel(const float* __restrict__ pix, int stride,
                                                                     uint32_t W, uint32_t H, int s,
                                                                     uint32_t* __restrict__ white_bits)
{
    const int tiles_x = (int)((W + kTile - 1) / kTile);
    const int tile = (int)(blockIdx.x / kStatsSplit), part = (int)(blockIdx.x % kStatsSplit);
    const int tx = tile % tiles_x, ty = tile / tiles_x;
    const int x0 = tx * kTile, y0 = ty * kTile;
    const int x1 = min(x0 + kTile, (int)W) - 1, y1 = min(y0 + kTile, (int)H) - 1;
    __shared__ int cols[kMaxSpan], rows[kMaxSpan];
    __shared__ int span[4][5], nspan[2];
    if (threadIdx.x == 0) {
        nspan[0] = tap_spans(x0, x1, s, (int)W, span[0], span[1]);
        nspan[1] = tap_spans(y0, y1, s, (int)H, span[2], span[3]);
    }
    __syncthreads();
    const int ncols = list_spans(span[0], span[1], nspan[0], cols);
    const int nrows = list_spans(span[2], span[3], nspan[1], rows);
    __syncthreads();
    float white = 0.0f;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kStatsThreads / 32;
    for (int r = part * kWarps + warp; r < nrows; r += kStatsSplit * kWarps) {
        const size_t rb = (size_t)rows[r] * W;
        for (int c = lane; c < ncols; c += 32) {
            const size_t f = rb + (size_t)cols[c];
            const float* p = pix + stride * f;
            const float l = luminance(__ldg(p), __ldg(p + 1), __ldg(p + 2));
            white = (white < l) ? l : white;
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        const float w2 = __shfl_down_sync(0xffffffffu, white, off);
        white = (white < w2) ? w2 : white;
    }
    __shared__ float sw[kWarps];
    if (lane == 0) sw[warp] = white;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kWarps; ++w) white = (white < sw[w]) ? sw[w] : white;
        atomicMax(white_bits + tile, __float_as_uint(white));
    }
}

// The min / max |position| over each level's footprint of each tile, in two
// separable steps (the footprint is a set of rows times a set of columns):
//   row_range   one warp per (image row, tile column): |position| of the columns
//               any level's footprint of that tile column can reach ([x0 - 32,
//               x1 + 32], clamped) is read once, then reduced over each level's
//               column spans: rrow[(level * H + y) * tiles_x + tx] = (min, max);
//   tile_range  one warp per (tile, level): the row ranges reduced over the
//               level's row spans: range[level * tiles + tile] = (min, max).
// min / max are exact, so the grouping is free, and the selects keep std::min /
// std::max's NaN behaviour (a NaN |position| never replaces a bound).
constexpr int kRowWarps = 4;
// Whether column (or row) c is read by a tap of the stencil (offsets -2..2 times s, clamped to
// [0, n - 1]) from some pixel of [a, b]: the union tap_spans lists, tested tap by tap so that
// everything stays in registers (span arrays indexed at run time would live in local memory).
__device__ __forceinline__ bool tapped(int c, int a, int b, int s, int n)
{
    bool in = false;
#pragma unroll
    for (int k = -2; k <= 2; ++k) in |= clampi(a + k * s, 0, n - 1) <= c && c <= clampi(b + k * s, 0, n - 1);
    return in;
}

// Rows kRowWarps * block .. of the image's (row, tile column) pairs.
__device__ __forceinline__ void row_range(uint32_t block, const float* __restrict__ pos, uint32_t W, uint32_t H,
                                          float2* __restrict__ rrow)
{
    using namespace ex;
    const int tiles_x = (int)((W + kTile - 1) / kTile);
    const int lane = threadIdx.x & 31;
    const long long task = (long long)block * kRowWarps + (threadIdx.x >> 5);
    if (task >= (long long)H * tiles_x) return;   // the whole warp leaves together
    const int y = (int)(task / tiles_x), tx = (int)(task % tiles_x);
    const int x0 = tx * kTile, x1 = min(x0 + kTile, (int)W) - 1;
    const int rx0 = max(x0 - 32, 0), rx1 = min(x1 + 32, (int)W - 1);
    // the span's positions (at most 128 pixels, 384 floats) staged through shared memory with
    // consecutive lanes reading consecutive floats, all twelve loads in flight before the first
    // store, then |position| of columns rx0 + lane + 32 k
    __shared__ float stage[kRowWarps][3 * 128];
    float* st = stage[threadIdx.x >> 5];
    const int nf = 3 * (rx1 - rx0 + 1);
    const float* row = pos + 3 * ((size_t)y * W + (size_t)rx0);
    float v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = (lane + 32 * k < nf) ? __ldg(row + lane + 32 * k) : 0.0f;
#pragma unroll
    for (int k = 0; k < 12; ++k) st[lane + 32 * k] = v[k];
    __syncwarp();
    float len[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = lane + 32 * k;
        len[k] = (rx0 + j <= rx1) ? length(v3(st[3 * j], st[3 * j + 1], st[3 * j + 2])) : 0.0f;
    }
    const float kInf = __int_as_float(0x7f800000);
    // A tile column at least 16 wide (all but a narrow last one) has overlapping taps at every
    // spacing up to 16: its columns are then the one range [x0 - 2 s, x1 + 2 s], clamped.
    const bool wide = x1 - x0 + 1 >= 16;
#pragma unroll
    for (int level = 0; level < 5; ++level) {
        const int s = 1 << level;
        const int lo = max(x0 - 2 * s, 0), hi = min(x1 + 2 * s, (int)W - 1);
        float mind = kInf, maxd = -kInf;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int c = rx0 + lane + 32 * k;
            if (c >= lo && c <= hi && (wide || tapped(c, x0, x1, s, (int)W))) {
                mind = (len[k] < mind) ? len[k] : mind;
                maxd = (maxd < len[k]) ? len[k] : maxd;
            }
        }
        // neither is a NaN, and lengths order like their bits (the empty maximum, -inf, as a negative integer)
        mind = __int_as_float(__reduce_min_sync(0xffffffffu, __float_as_int(mind)));
        maxd = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(maxd)));
        if (lane == 0) rrow[((size_t)level * H + y) * tiles_x + tx] = make_float2(mind, maxd);
    }
}

__global__ void __launch_bounds__(32 * 5) atrous_tile_range_kernel(const float2* __restrict__ rrow, uint32_t W,
                                                                   uint32_t H, float* __restrict__ pos_scale)
{
    const int tiles_x = (int)((W + kTile - 1) / kTile);
    const int tiles = tiles_x * (int)((H + kTile - 1) / kTile);
    const int tile = (int)blockIdx.x, level = (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int tx = tile % tiles_x, y0 = (tile / tiles_x) * kTile;
    const int y1 = min(y0 + kTile, (int)H) - 1;
    const int s = 1 << level;
    const float kInf = __int_as_float(0x7f800000);
    float mind = kInf, maxd = -kInf;
    // the rows between the first and the last tap, those some tap reads
    for (int r = max(y0 - 2 * s, 0) + lane; r <= min(y1 + 2 * s, (int)H - 1); r += 32)
        if (tapped(r, y0, y1, s, (int)H)) {
            const float2 v = rrow[((size_t)level * H + r) * tiles_x + tx];
            mind = (v.x < mind) ? v.x : mind;
            maxd = (maxd < v.y) ? v.y : maxd;
        }
    for (int off = 16; off > 0; off >>= 1) {
        const float a2 = __shfl_down_sync(0xffffffffu, mind, off);
        const float b2 = __shfl_down_sync(0xffffffffu, maxd, off);
        mind = (a2 < mind) ? a2 : mind;
        maxd = (maxd < b2) ? b2 : maxd;
    }
    if (lane == 0) {
        const float d = __fsub_rn(maxd, mind);
        pos_scale[level * tiles + tile] = -kLog2e * __frcp_rn(__fmul_rn(d, d));   // -inf for a zero range
    }
}

// The blend reads its taps as packed records of 48 bytes a pixel: (normal x, position x, normal y, position y),
// (normal z, position z, albedo x, albedo y) side by side, written once, and (albedo z, colour) in an array of its own,
// written by each level for the next.  A tap is three 128-bit loads instead of twelve of 4 bytes, and the normal and
// the position advance in pairs through packed float operations.
__device__ __forceinline__ void pack(size_t i, const float* __restrict__ pix, const float* __restrict__ nrm,
                                     const float* __restrict__ pos, const float* __restrict__ dif, size_t npx,
                                     float4* __restrict__ ab, float4* __restrict__ c)
{
    if (i >= npx) return;
    const float *n = nrm + 3 * i, *p = pos + 3 * i, *d = dif + 3 * i, *x = pix + 3 * i;
    ab[2 * i] = make_float4(__ldg(n), __ldg(p), __ldg(n + 1), __ldg(p + 1));
    ab[2 * i + 1] = make_float4(__ldg(n + 2), __ldg(p + 2), __ldg(d), __ldg(d + 1));
    c[i] = make_float4(__ldg(d + 2), __ldg(x), __ldg(x + 1), __ldg(x + 2));
}

// Both of these and the clearing of a call's white points and cells in one launch: the row ranges are bound by
// instruction issue (21 us alone) and the packing by memory (31 us), so every third block takes rows and the others
// pack, and they share the SMs.
constexpr int kPrepareThreads = 32 * kRowWarps;
__global__ void __launch_bounds__(kPrepareThreads) atrous_prepare_kernel(
    const float* __restrict__ pix, const float* __restrict__ nrm, const float* __restrict__ pos,
    const float* __restrict__ dif, uint32_t W, uint32_t H, float4* __restrict__ ab, float4* __restrict__ c,
    float2* __restrict__ rrow, uint32_t* __restrict__ white, size_t nwhite, uint32_t* __restrict__ cells, size_t ncells)
{
    if (blockIdx.x % 3 == 0) {
        row_range(blockIdx.x / 3, pos, W, H, rrow);
        return;
    }
    const size_t i = (size_t)(blockIdx.x - blockIdx.x / 3 - 1) * kPrepareThreads + threadIdx.x;
    if (i < nwhite) white[i] = 0;
    if (i < ncells) cells[i] = 0;
    pack(i, pix, nrm, pos, dif, (size_t)W * H, ab, c);
}

// The white points of a level from the cells that the level before it filled: cells of 2 s x 2 s pixels, each with
// its largest luminance (from 0).  A tile's footprint at spacing s is the whole rectangle from its first column and
// row less 2 s to its last plus 2 s, clamped (whole_footprints), and all its sides lie on cell borders or on the
// image's.  One warp per tile.
__global__ void __launch_bounds__(128) atrous_white_kernel(const uint32_t* __restrict__ cells, uint32_t W, uint32_t H,
                                                           int s, float* __restrict__ white)
{
    const uint32_t tiles_x = (W + kTile - 1) / kTile, tiles = tiles_x * ((H + kTile - 1) / kTile);
    const uint32_t tile = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (tile >= tiles) return;   // the whole warp leaves together
    const int x0 = (int)(tile % tiles_x) * kTile, y0 = (int)(tile / tiles_x) * kTile, c = 2 * s;
    const int cx0 = max(x0 - c, 0) / c, cx1 = min(x0 + kTile - 1 + c, (int)W - 1) / c;
    const int cy0 = max(y0 - c, 0) / c, cy1 = min(y0 + kTile - 1 + c, (int)H - 1) / c;
    const int nx = cx1 - cx0 + 1, n = nx * (cy1 - cy0 + 1);
    const size_t pitch = (W + c - 1) / c;
    uint32_t m = 0;   // non-negative floats order like their bits
    for (int k = (int)lane; k < n; k += 32) m = max(m, __ldg(cells + (size_t)(cy0 + k / nx) * pitch + (cx0 + k % nx)));
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) white[tile] = __uint_as_float(m);
}

// Whether every tile's footprint at spacing s is one rectangle: its taps' ranges overlap when the tile is at least s
// wide and high, which only the last column and row of tiles may miss.
static bool whole_footprints(uint32_t W, uint32_t H, int s)
{
    auto whole = [s](uint32_t n) { const uint32_t last = n % kTile; return last == 0 || last >= (uint32_t)s; };
    return whole(W) && whole(H);
}

// The blend: 25 taps per pixel.  The reference's weight
//   k[u] * min(exp(-|dn|^2/0.25),1) * min(exp(-|dp|^2/range^2),1) * min(exp(-|da|^2/white^2),1)
// is evaluated as 2^(log2 k[u] - |dn|^2 4 log2 e - |dp|^2 log2 e / range^2 - |da|^2 log2 e / white^2): the arguments
// of the exponentials are never positive, so the min(., 1) clamps only pass NaN through, and a sum of -inf / NaN
// terms gives the same 0 / NaN as their product.  One hardware exponential per tap; the result stays within 1e-5
// relative of the exact evaluation (the weights enter a normalised sum in which the centre tap, k = 0.159, always
// has exponent 0).
//
// At spacing s every tap of a pixel lands on the pixel's own sub-lattice (x mod s, y mod s), so a CTA takes a
// kLatX x kLatY tile of one sub-lattice at every spacing; the (kLatX + 4) x (kLatY + 4) lattice points its taps read
// (coordinates clamped exactly as the taps clamp them) are copied to shared memory once, asynchronously and past L1.
// Points that only pixels outside the image would read are left out: of a small image at a large spacing they were
// most of a footprint, all clamped to the same few border pixels (65 x 40, spacing 16: 33 us with them, 6 without;
// 1601 x 901 whole: 433 us and 387).
// Each thread blends two neighbouring columns, whose taps overlap, and reads each record once for both; the records of
// a footprint row are split into even and odd columns so that a warp's loads hit consecutive records.
//
// Measured at 1920 x 1080 (start 92-98 us a level with its own tile kernel for spacings 1-4 and a direct one above):
// 68-77 us a level at 65 % of the issue slots, 61-67 % of the LSU wavefronts and half of the FP32 pipe (whose
// 36 us a level are the floor), 24 warps per SM waiting on shared-memory latency between.  Whole call, while footprints
// were copied whole: copies through
// registers 595 us against 534 asynchronous; scalar differences 30 us more than packed ones; two rows per thread
// (fewer reads, 20 warps) 528 against 509, three 605 against 534; 7 or 8 CTAs per SM (72 or 64 registers) 515 and 528;
// tiles of 64 x 8, 32 x 16, 16 x 16 and 16 x 8 points 5, 5, 3 and 1 % slower.
//
// With `cells`, the pixels' luminances go to the next level's white points: the largest of each cell of 4 s x 4 s
// pixels, 4 x 4 points of every sub-lattice.  A level's white points take 4-6 us from cells, 13 from the colours.
__device__ __forceinline__ void copy16(float4* to, const float4* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}

constexpr int kLatX = 32, kLatY = 8, kBlendThreads = kLatX / 2 * kLatY;
constexpr int kFootX = kLatX + 4, kHalfX = kFootX / 2, kFootY = kLatY + 4;

__global__ void __launch_bounds__(kBlendThreads, 6) atrous_blend_kernel(
    const float4* __restrict__ rab, const float4* __restrict__ rc, uint32_t W, uint32_t H, int shift, uint32_t cols,
    const float* __restrict__ white, const float* __restrict__ pos_scale, float4* __restrict__ dst,
    uint32_t* __restrict__ cells, uint32_t cell_pitch)
{
    __shared__ float4 rec[kFootY * kFootX * 3];   // [row][column parity][column / 2] records
    const int s = 1 << shift;
    const int by = (int)(blockIdx.x / cols), bx = (int)(blockIdx.x - (uint32_t)by * cols);
    const int rx = bx & (s - 1), tx = bx >> shift, ry = by & (s - 1), ty = by >> shift;
    const int lx0 = tx * kLatX - 2, ly0 = ty * kLatY - 2;   // lattice coordinate of footprint entry (0, 0)
    int ex = (int)threadIdx.x % kFootX, ey = (int)threadIdx.x / kFootX;
    for (int e = (int)threadIdx.x; e < kFootX * kFootY; e += kBlendThreads) {
        const int x = rx + (lx0 + ex) * s, y = ry + (ly0 + ey) * s;
        if (x < (int)W + 2 * s && y < (int)H + 2 * s) {   // beyond that, only points outside the image read it
            const size_t f = (size_t)clampi(y, 0, (int)H - 1) * W + (size_t)clampi(x, 0, (int)W - 1);
            float4* slot = rec + 3 * ((ey * 2 + (ex & 1)) * kHalfX + (ex >> 1));
            copy16(slot, rab + 2 * f);
            copy16(slot + 1, rab + 2 * f + 1);
            copy16(slot + 2, rc + f);
        }
        ex += kBlendThreads % kFootX;
        ey += kBlendThreads / kFootX;
        if (ex >= kFootX) { ex -= kFootX; ++ey; }
    }
    const int h = (int)(threadIdx.x % (kLatX / 2)), row = (int)(threadIdx.x / (kLatX / 2));
    const uint32_t tiles_x = (W + kTile - 1) / kTile;
    const int x0 = rx + (tx * kLatX + 2 * h) * s, y0 = ry + (ty * kLatY + row) * s;   // the thread's first pixel
    float ctr[2][9], acc[2][4], ip[2], iw[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t x = min((uint32_t)(x0 + k * s), W - 1), y = min((uint32_t)y0, H - 1);
        const size_t tile = (size_t)(y / kTile) * tiles_x + x / kTile;
        const float w = __ldg(white + tile);
        ip[k] = __ldg(pos_scale + tile);                // -log2 e / range^2
        iw[k] = -kLog2e * __frcp_rn(__fmul_rn(w, w));   // -log2 e / white^2
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[k][u] = 0.0f;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float4* c = rec + 3 * (((row + 2) * 2 + k) * kHalfX + h + 1);   // footprint column 2 h + 2 + k
        const float4 a = c[0], b = c[1];
        float* p = ctr[k];
        p[0] = -a.x; p[1] = -a.y; p[2] = -a.z; p[3] = -a.w; p[4] = -b.x; p[5] = -b.y; p[6] = -b.z; p[7] = -b.w;
        p[8] = -c[2].x;
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {   // footprint column 2 h + q: tap column q - k of pixel k
            const float4* t = rec + 3 * (((row + j) * 2 + (q & 1)) * kHalfX + h + (q >> 1));
            const float4 a = t[0], b = t[1], c = t[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = q - k;
                if (i < 0 || i > 4) continue;
                const float* p = ctr[k];
                const float2 x = __fadd2_rn(make_float2(a.x, a.y), make_float2(p[0], p[1]));
                const float2 y = __fadd2_rn(make_float2(a.z, a.w), make_float2(p[2], p[3]));
                const float2 z = __fadd2_rn(make_float2(b.x, b.y), make_float2(p[4], p[5]));
                const float2 v = __fadd2_rn(make_float2(b.z, b.w), make_float2(p[6], p[7]));
                const float az = p[8] + c.x;
                const float2 np = __ffma2_rn(z, z, __ffma2_rn(y, y, __fmul2_rn(x, x)));   // |dn|^2, |dp|^2
                const float2 vv = __fmul2_rn(v, v);
                const float da = fmaf(az, az, vv.x) + vv.y;
                const float e = fmaf(da, iw[k], fmaf(np.y, ip[k], fmaf(np.x, -4.0f * kLog2e, kAtrousLog2[j * 5 + i])));
                float w;
                asm("ex2.approx.f32 %0, %1;" : "=f"(w) : "f"(e));   // keeps subnormal weights
                acc[k][0] = fmaf(c.y, w, acc[k][0]);
                acc[k][1] = fmaf(c.z, w, acc[k][1]);
                acc[k][2] = fmaf(c.w, w, acc[k][2]);
                acc[k][3] += w;
            }
        }
    }
    float bright = 0.0f;   // the thread's largest luminance (a NaN never replaces it)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int x = x0 + k * s;
        if (y0 >= (int)H || x >= (int)W) continue;
        const float* v = acc[k];
        const float red = __fdiv_rn(v[0], v[3]), green = __fdiv_rn(v[1], v[3]), blue = __fdiv_rn(v[2], v[3]);
        dst[(size_t)y0 * W + (size_t)x] = make_float4(-ctr[k][8], red, green, blue);
        const float l = luminance(red, green, blue);
        bright = (bright < l) ? l : bright;
    }
    if (cells) {
        // a cell's four columns are two lanes', its four rows four threads'
        const float o = __shfl_xor_sync(0xffffffffu, bright, 1);
        bright = (bright < o) ? o : bright;
        if (h % 2 == 0 && bright > 0.0f)
            atomicMax(cells + (size_t)(y0 >> (shift + 2)) * cell_pitch + (size_t)(x0 >> (shift + 2)),
                      __float_as_uint(bright));
    }
}

// The last level's colours as the caller's image.  Written by the blend itself, twelve bytes a pixel and those sixteen
// pixels apart, they cost 25 us more than records; this pass over consecutive pixels costs 15-20.
__global__ void __launch_bounds__(256) atrous_unpack_kernel(const float4* __restrict__ c, size_t npx, float* __restrict__ out)
{
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= npx) return;
    const float4 v = __ldg(c + i);
    out[3 * i] = v.y; out[3 * i + 1] = v.z; out[3 * i + 2] = v.w;
}

// Scratch of a call, in floats: the packed records (eight of normal, position and albedo a pixel, then two arrays of
// colours that the levels take in turn), then atrous_stats_floats of statistics.
cudaError_t launch_atrous(const float* pixels, const float* normals, const float* positions, const float* diffuse,
                          uint32_t W, uint32_t H, float* records, float* stats, float* out, cudaStream_t st)
{
    if (W == 0 || H == 0) return cudaSuccess;
    const uint32_t tiles_x = (W + kTile - 1) / kTile, tiles = tiles_x * ((H + kTile - 1) / kTile);
    const size_t npx = (size_t)W * H;
    float4* rab = reinterpret_cast<float4*>(records);
    float4* rc[2] = {rab + 2 * npx, rab + 3 * npx};
    // per level and tile the white point and the scale of the position term; per level, image row and tile column a
    // (min, max) |position|; the cells of levels 1-4
    float* white = stats;
    float* pos_scale = white + (size_t)5 * tiles;
    float2* rrow = reinterpret_cast<float2*>(pos_scale + (size_t)5 * tiles);
    uint32_t* cells = reinterpret_cast<uint32_t*>(rrow + (size_t)5 * H * tiles_x);
    const size_t nwhite = (size_t)5 * tiles, ncells = atrous_cells(W, H);
    const uint64_t row_blocks = ((uint64_t)H * tiles_x + kRowWarps - 1) / kRowWarps;
    const uint64_t pack_blocks = (std::max({npx, nwhite, ncells}) + kPrepareThreads - 1) / kPrepareThreads;
    atrous_prepare_kernel<<<(unsigned)(3 * std::max(row_blocks, (pack_blocks + 1) / 2)), kPrepareThreads, 0, st>>>(
        pixels, normals, positions, diffuse, W, H, rab, rc[0], rrow, reinterpret_cast<uint32_t*>(white), nwhite, cells,
        ncells);
    atrous_tile_range_kernel<<<tiles, 32 * 5, 0, st>>>(rrow, W, H, pos_scale);
    bool filled = false;   // whether the level before filled this one's cells
    for (int level = 0; level < 5; ++level) {
        const int s = 1 << level;
        const float4* src = rc[level % 2];
        float* lwhite = white + (size_t)level * tiles;
        if (filled) {
            atrous_white_kernel<<<(tiles + 3) / 4, 128, 0, st>>>(cells, W, H, s, lwhite);
        } else {
            // the packed colours start at a record's second float
            const float* colour = level == 0 ? pixels : reinterpret_cast<const float*>(src) + 1;
            atrous_stats_kernel<<<tiles * kStatsSplit, kStatsThreads, 0, st>>>(colour, level == 0 ? 3 : 4, W, H, s,
                                                                              reinterpret_cast<uint32_t*>(lwhite));
        }
        if (level > 0) cells += atrous_level_cells(W, H, 2 * s);
        filled = level < 4 && whole_footprints(W, H, 2 * s);
        // one CTA per kLatX x kLatY tile of each of the s x s sub-lattices
        const uint64_t cols = (uint64_t)((W + s - 1) / s + kLatX - 1) / kLatX * s;
        const uint64_t blocks = cols * (((H + s - 1) / s + kLatY - 1) / kLatY * s);
        atrous_blend_kernel<<<(unsigned)blocks, kBlendThreads, 0, st>>>(
            rab, src, W, H, level, (uint32_t)cols, lwhite, pos_scale + (size_t)level * tiles, rc[(level + 1) % 2],
            filled ? cells : nullptr, (W + 4 * (uint32_t)s - 1) / (4 * (uint32_t)s));
    }
    atrous_unpack_kernel<<<(unsigned)((npx + 255) / 256), 256, 0, st>>>(rc[1], npx, out);
    return cudaGetLastError();
}

}  // namespace pico

// ---------------------------------------------------------------------------
// Reinhard tone mapping (Util::reinhard_tone_mapping, Util/ToneMappers.cpp:12-44):
// a global white point = the largest luminance (from 0; NaN luminances are
// skipped, as std::max(white, lum) skips them), then per channel
// p * (1 + p / white^2) / (1 + p), in place.  Non-negative floats order like
// their bit patterns, so the maximum is an atomicMax on the bits.
namespace pico {

__global__ void __launch_bounds__(256) white_point_kernel(const float* __restrict__ pix, size_t npx,
                                                          unsigned* __restrict__ white_bits)
{
    float w = 0.0f;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npx; i += (size_t)gridDim.x * blockDim.x) {
        const float l = luminance(pix[3 * i], pix[3 * i + 1], pix[3 * i + 2]);
        w = (w < l) ? l : w;
    }
    for (int off = 16; off > 0; off >>= 1) {
        const float o = __shfl_down_sync(0xffffffffu, w, off);
        w = (w < o) ? o : w;
    }
    if ((threadIdx.x & 31u) == 0) atomicMax(white_bits, __float_as_uint(w));
}

__global__ void __launch_bounds__(256) reinhard_kernel(float* __restrict__ pix, size_t n,
                                                       const unsigned* __restrict__ white_bits)
{
    using namespace ex;
    const float w = __uint_as_float(*white_bits);
    const float w2 = mul(w, w);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float p = pix[i];
        const float num = mul(p, add(1.0f, div(p, w2)));
        pix[i] = div(num, add(1.0f, p));
    }
}

cudaError_t launch_reinhard(float* pixels, uint32_t W, uint32_t H, unsigned* scratch, cudaStream_t st)
{
    const size_t npx = (size_t)W * H;
    if (npx == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    const unsigned blocks = (unsigned)std::min<size_t>((npx + 255) / 256, (size_t)sm_count() * 8);
    white_point_kernel<<<blocks, 256, 0, st>>>(pixels, npx, scratch);
    reinhard_kernel<<<blocks, 256, 0, st>>>(pixels, 3 * npx, scratch);
    return cudaGetLastError();
}

}  // namespace pico
