// The reference's image output: Scene::render_scene_to_file (Core/Scene.cpp:238-246)
// reverses the flat pixel array and writes it with stb_image_write's
// stbi_write_hdr, a Radiance file of RGBE pixels, run-length coded per
// component on scanlines 8..32767 pixels wide.
//
// On the device: one CTA per scanline encodes its pixels to RGBE (frexp of the
// largest component; mantissa scaled by 256 / max, truncated) as four byte rows in
// shared memory and run-length codes each with a warp, into slots of W + ceil(W / 128)
// bytes (the worst case: all literals); a scan of the codes' lengths gives their places
// in the file, a third kernel moves them there, and the host receives the finished body
// in one copy behind the text header.  NaN or negative components, whose conversion to a
// byte is undefined in the reference, are written as 0.
#include "kernels_render.h"
#include "render_internal.h"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>

namespace pico {
namespace {

__device__ __forceinline__ unsigned char to_byte(float v) { return (v >= 0.0f && v < 256.0f) ? (unsigned char)v : 0; }

__device__ __forceinline__ uchar4 rgbe_of(float r, float g, float b)
{
    const float m12 = (g < b) ? b : g;
    const float maxcomp = (r < m12) ? m12 : r;
    if (maxcomp < 1e-32f) return make_uchar4(0, 0, 0, 0);
    int e;
    const float m = frexpf(maxcomp, &e);
    const float normalize = __fdiv_rn(__fmul_rn(m, 256.0f), maxcomp);
    return make_uchar4(to_byte(__fmul_rn(r, normalize)), to_byte(__fmul_rn(g, normalize)),
                       to_byte(__fmul_rn(b, normalize)), (unsigned char)(e + 128));
}

__global__ void rgbe_kernel(const float* __restrict__ pix, size_t npx, uchar4* __restrict__ out)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npx; i += (size_t)gridDim.x * blockDim.x)
        out[i] = rgbe_of(pix[3 * i], pix[3 * i + 1], pix[3 * i + 2]);
}

size_t rle_slot(uint32_t W) { return (size_t)W + (W + 127) / 128; }

// The stbi_write_hdr run-length scheme, one CTA per scanline and one warp per
// component.  A maximal stretch of three or more equal bytes is a run, coded in pieces
// of up to 127 (two bytes each); what lies between runs is literal, coded in pieces of
// up to 128 behind a length byte.  Both are local: whether a byte belongs to a run shows
// within two bytes of it, a stretch starts where that changes (or a run's value does),
// and its start, the byte's index in it, is the last start at or before the byte.  So a
// warp takes 32 bytes at a time: ballots give each byte the stretch's start and the
// number of bytes coded before it, and the last byte of a piece writes the piece's
// length where the piece began.  One thread per component walking the row byte by byte
// took 781 us for 1920 x 1080, behind 11 us of RGBE conversion; this kernel does both in
// 51 us, the offsets 5 us and the gather 14 us, and the call takes 280 us instead of 2054
// (of which the 25 MB upload takes 150).
__global__ void __launch_bounds__(128) rle_row_kernel(const float* __restrict__ pix, uint32_t W, size_t slot,
                                                      unsigned char* __restrict__ out, uint32_t* __restrict__ lens)
{
    extern __shared__ unsigned char plane[];   // [component][x]
    const uint32_t row = blockIdx.x;
    const float* line = pix + 3 * (size_t)row * W;
    for (uint32_t x = threadIdx.x; x < W; x += blockDim.x) {
        const uchar4 v = rgbe_of(line[3 * x], line[3 * x + 1], line[3 * x + 2]);
        plane[x] = v.x; plane[W + x] = v.y; plane[2 * W + x] = v.z; plane[3 * W + x] = v.w;
    }
    __syncthreads();
    const uint32_t c = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const unsigned char* a = plane + c * W;
    unsigned char* o = out + slot * (4 * (size_t)row + c);
    // bit k of eq(x0): bytes x0 + k and x0 + k + 1 are equal
    auto eq = [&](uint32_t x0) {
        const uint32_t x = x0 + lane;
        return __ballot_sync(0xffffffffu, x + 1 < W && a[x] == a[x + 1]);
    };
    uint32_t start = 0, n = 0;   // the current stretch's start; bytes coded so far
    const unsigned upto = 0xffffffffu >> (31u - lane);   // this lane and those below
    // of the last 32 bytes, these and the next: equal pairs (e), starts of three equal bytes (t), run flags (r)
    unsigned e0 = 0, t0 = 0, r0 = 0, e1 = eq(0);
    for (uint32_t x0 = 0; x0 < W; x0 += 32) {
        const unsigned e2 = eq(x0 + 32);
        const unsigned t1 = e1 & __funnelshift_r(e1, e2, 1);
        const unsigned r1 = t1 | __funnelshift_l(t0, t1, 1) | __funnelshift_l(t0, t1, 2);
        const unsigned r2 = (e2 & (e2 >> 1) & 1u) | (t1 >> 31) | ((t1 >> 30) & 1u);   // the first of the next
        const unsigned valid = W - x0 >= 32 ? 0xffffffffu : (1u << (W - x0)) - 1u;
        const unsigned firsts = valid & ((r1 ^ __funnelshift_l(r0, r1, 1)) | (r1 & ~__funnelshift_l(e0, e1, 1)) |
                                         (x0 == 0 ? 1u : 0u));
        const unsigned lasts = valid & ((r1 ^ __funnelshift_r(r1, r2, 1)) | (r1 & ~e1) |
                                        (W - x0 <= 32 ? 1u << (W - x0 - 1) : 0u));
        const uint32_t x = x0 + lane;
        const bool live = (valid >> lane) & 1u, run = (r1 >> lane) & 1u;
        const unsigned mine = firsts & upto;
        const uint32_t d = x - (mine ? x0 + 31u - (uint32_t)__clz((int)mine) : start);
        const uint32_t i = run ? d % 127u : d % 128u;   // index in the piece
        const unsigned starts = __ballot_sync(0xffffffffu, live && i == 0);
        const unsigned lits = valid & ~r1, heads = starts & ~r1, runs = starts & r1;
        const uint32_t end = n + __popc(lits & upto) + __popc(heads & upto) + 2u * __popc(runs & upto);
        if (live) {
            const bool full = ((lasts >> lane) & 1u) || i == (run ? 126u : 127u);
            if (!run || full) o[end - 1] = a[x];
            if (full) o[run ? end - 2 : end - 2 - i] = (unsigned char)(run ? i + 129 : i + 1);
        }
        n += __popc(lits) + __popc(heads) + 2u * __popc(runs);
        if (firsts) start = x0 + 31u - (uint32_t)__clz((int)firsts);
        e0 = e1; t0 = t1; r0 = r1; e1 = e2;
    }
    if (lane == 0) lens[4 * (size_t)row + c] = n;
}

// Where each code goes in the file's body: off[k] = 4 (k / 4 + 1) + the lengths before k (every row opens with a
// four-byte header), and off[n] the body's length.  One CTA of 1024 threads, eight codes (two rows) a thread.
__global__ void __launch_bounds__(1024) rle_offsets_kernel(const uint32_t* __restrict__ lens, uint32_t n,
                                                           unsigned long long* __restrict__ off)
{
    __shared__ unsigned long long warp_sum[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long base = 0;
    for (uint32_t k0 = 0; k0 < n; k0 += 8192) {
        const uint32_t k = k0 + 8 * threadIdx.x;
        uint32_t len[8], own = 0;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            len[j] = k + j < n ? lens[k + j] : 0u;
            own += len[j] + (j % 4 == 0 && k + j < n ? 4u : 0u);
        }
        unsigned long long sum = own;
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, sum, d);
            if ((int)lane >= d) sum += u;
        }
        if (lane == 31) warp_sum[warp] = sum;
        __syncthreads();
        if (warp == 0) {
            unsigned long long t = warp_sum[lane];
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long u = __shfl_up_sync(0xffffffffu, t, d);
                if ((int)lane >= d) t += u;
            }
            warp_sum[lane] = t;
        }
        __syncthreads();
        unsigned long long at = base + (warp ? warp_sum[warp - 1] : 0ull) + sum - own;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            if (j % 4 == 0) at += 4;
            if (k + j < n) off[k + j] = at;
            at += len[j];
        }
        base += warp_sum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) off[n] = base;
}

// Moves the codes to their places, behind their rows' headers: one CTA per row, one warp per code, in words at the
// destination's alignment (a word's four bytes out of two source words).
__global__ void __launch_bounds__(128) rle_gather_kernel(const unsigned char* __restrict__ codes, uint32_t W,
                                                         size_t slot, const uint32_t* __restrict__ lens,
                                                         const unsigned long long* __restrict__ off,
                                                         unsigned char* __restrict__ body)
{
    const size_t row = blockIdx.x, k = 4 * row + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31u;
    if (threadIdx.x < 4)
        body[off[4 * row] - 4 + threadIdx.x] =
            (unsigned char)(threadIdx.x < 2 ? 2u : threadIdx.x == 2 ? (W & 0xff00u) >> 8 : W & 0xffu);
    const unsigned char* s = codes + slot * k;
    unsigned char* d = body + off[k];
    const uint32_t n = lens[k];
    const uint32_t lead = min((uint32_t)(-(intptr_t)d & 3), n), words = (n - lead) / 4, tail = lead + 4 * words;
    if (lane < lead) d[lane] = s[lane];
    if (tail + lane < n) d[tail + lane] = s[tail + lane];   // at most three
    const uint32_t shift = 8u * (uint32_t)((intptr_t)(s + lead) & 3);
    const uint32_t* sw = reinterpret_cast<const uint32_t*>(s + lead - shift / 8);   // the slots are followed by padding
    uint32_t* dw = reinterpret_cast<uint32_t*>(d + lead);
    for (uint32_t w = lane; w < words; w += 32) dw[w] = __funnelshift_r(sw[w], sw[w + 1], shift);
}

}  // namespace

size_t hdr_bound(uint32_t W, uint32_t H)
{
    return 256 + (size_t)H * (4 + 4 * rle_slot(W)) + (size_t)W * H * 4;
}

// Encodes the device pixels r.hdr_pix into a Radiance file image in `out` (host, `capacity` bytes), its length in
// *length.  The workspaces stay with the context.
static int encode_hdr(pico_gpu_ctx* ctx, RenderBuffers& r, uint32_t W, uint32_t H, unsigned char* out, size_t capacity,
                      size_t* length)
{
    cudaStream_t st = ctx->stream;
    const size_t npx = (size_t)W * H;
    const float* d_pixels = as<float>(r.hdr_pix);
    const bool rle = W >= 8 && W < 32768 && H > 0;
    const size_t slot = rle_slot(W);
    const uint32_t codes = 4 * H;
    unsigned long long body = 4 * (unsigned long long)npx;
    cudaError_t e = cudaSuccess;
    if (rle) {
        e = r.hdr_codes.reserve(slot * 4 * H + 16);   // the gather reads up to a word past the last code
        if (e == cudaSuccess) e = r.hdr_lens.reserve(sizeof(uint32_t) * 4 * (size_t)H);
        if (e == cudaSuccess) e = r.hdr_off.reserve(sizeof(unsigned long long) * (4 * (size_t)H + 1));
        if (e == cudaSuccess) e = r.hdr_body.reserve((size_t)H * (4 + 4 * slot));
        // a scanline's four byte rows in shared memory (W < 32768)
        const size_t smem = 4 * (size_t)W;
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(rle_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) {
            rle_row_kernel<<<H, 128, smem, st>>>(d_pixels, W, slot, as<unsigned char>(r.hdr_codes),
                                                 as<uint32_t>(r.hdr_lens));
            rle_offsets_kernel<<<1, 1024, 0, st>>>(as<uint32_t>(r.hdr_lens), codes, as<unsigned long long>(r.hdr_off));
            rle_gather_kernel<<<H, 128, 0, st>>>(as<unsigned char>(r.hdr_codes), W, slot, as<uint32_t>(r.hdr_lens),
                                                 as<unsigned long long>(r.hdr_off), as<unsigned char>(r.hdr_body));
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&body, as<unsigned long long>(r.hdr_off) + codes, sizeof body, cudaMemcpyDeviceToHost,
                                st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    } else if (npx) {
        e = r.hdr_body.reserve(npx * 4);
        const unsigned blocks = (unsigned)std::min<size_t>((npx + 255) / 256, (size_t)sm_count() * 8);
        if (e == cudaSuccess) {
            rgbe_kernel<<<blocks, 256, 0, st>>>(d_pixels, npx, as<uchar4>(r.hdr_body));
            e = cudaGetLastError();
        }
    }
    if (e != cudaSuccess) return cuda_error(ctx, e, "hdr encode");
    static const char magic[] = "#?RADIANCE\n# Written by stb_image_write.h\nFORMAT=32-bit_rle_rgbe\n";
    char res[128];
    const size_t nm = sizeof(magic) - 1;
    const size_t nr = (size_t)std::snprintf(res, sizeof res, "EXPOSURE=          1.0000000000000\n\n-Y %d +X %d\n",
                                            (int)H, (int)W);
    *length = nm + nr + (size_t)body;
    if (!out || capacity < *length) {
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_error(ctx, e, "hdr encode");
        return set_error(ctx, PICO_ERR_INVALID_ARG, "output buffer too small");
    }
    if (body)
        e = cudaMemcpyAsync(out + nm + nr, r.hdr_body.ptr, (size_t)body, cudaMemcpyDeviceToHost, st);
    std::memcpy(out, magic, nm);
    std::memcpy(out + nm, res, nr);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_error(ctx, e, "hdr encode");
    return PICO_OK;
}

}  // namespace pico

using namespace pico;

extern "C" {

size_t pico_gpu_hdr_bound(uint32_t width, uint32_t height) { return hdr_bound(width, height); }

int pico_gpu_encode_hdr(pico_gpu_ctx* ctx, const float* pixels, uint32_t W, uint32_t H, unsigned char* out,
                        size_t capacity, size_t* length)
{
    if (!ctx || !pixels || !length) return set_error(ctx, PICO_ERR_INVALID_ARG, "null argument");
    const DeviceScope device_scope(ctx->device);
    const size_t n3 = (size_t)W * H * 3;
    RenderBuffers& r = *render_buffers(ctx);
    cudaError_t e = r.hdr_pix.reserve(n3 * sizeof(float));
    if (e == cudaSuccess && n3)
        e = cudaMemcpyAsync(r.hdr_pix.ptr, pixels, n3 * sizeof(float), cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "hdr upload");
    return encode_hdr(ctx, r, W, H, out, capacity, length);
}

int pico_gpu_render_to_file(pico_gpu_ctx* ctx, const pico_gpu_scene* scene, const pico_camera* camera,
                            const pico_render_config* config, float* pixels, uint32_t* sample_count,
                            float* variance, const char* path)
{
    if (!path) return set_error(ctx, PICO_ERR_INVALID_ARG, "null path");
    int32_t quit = 0;
    int st = pico_gpu_render(ctx, scene, camera, config, pixels, sample_count, variance, &quit);
    if (st != PICO_OK) return st;
    // flip the image (std::reverse of the flat array, Scene.cpp:243-244), in the caller's buffer too
    const size_t npx = (size_t)config->width * config->height;
    for (size_t i = 0, j = npx ? npx - 1 : 0; i < j; ++i, --j)
        for (int c = 0; c < 3; ++c) std::swap(pixels[3 * i + c], pixels[3 * j + c]);
    std::vector<unsigned char> file(hdr_bound(config->width, config->height));
    size_t len = 0;
    st = pico_gpu_encode_hdr(ctx, pixels, config->width, config->height, file.data(), file.size(), &len);
    if (st != PICO_OK) return st;
    FILE* f = std::fopen(path, "wb");
    if (!f) return set_error(ctx, PICO_ERR_INVALID_ARG, std::string("cannot open ") + path);
    const size_t w = std::fwrite(file.data(), 1, len, f);
    std::fclose(f);
    if (w != len) return set_error(ctx, PICO_ERR_INVALID_ARG, std::string("short write to ") + path);
    return PICO_OK;
}

}  // extern "C"
