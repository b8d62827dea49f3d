// Host-visible state and launchers of the wavefront renderer and denoiser.
#pragma once

#include "kernels.h"
#include "layout.h"
#include "nrc.h"

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace pico {

// Camera::generate_ray inputs plus host-precomputed glm quantities.
struct CameraView {
    float pos[3], dir[3], up[3];
    float res_x, res_y, aspect, far_plane;
    float right[3];                    // cross(normalize(dir), up), glm operation order
    float view[16];                    // glm::lookAt(pos, pos + dir, up), column-major
};

// The p-th pixel of a W x H image in tile order: bands of 8 rows, in each band tiles of 8 columns from the left
// (narrower and lower at the right and bottom edges), row-major within a tile.  Renders list their pixels in this
// order, so that a warp's 32 paths start from an 8 x 4 block and meet the same nodes for longer than a row of 32
// does: the 1080p lit-field render 66.9 -> 65.9 ms, the physical one of 853 x 479 8.33 -> 8.21 ms, the G-buffer's
// primary rays alike.  Images do not change: a path's random stream depends on its pixel and sample only.
PICO_HD uint32_t tile_pixel(uint32_t p, uint32_t W, uint32_t H)
{
    const uint64_t band = 8ull * W;
    const uint32_t y0 = 8u * (uint32_t)(p / band), h = H - y0 < 8u ? H - y0 : 8u;
    const uint32_t r = (uint32_t)(p % band), x0 = 8u * (r / (8u * h)), w = W - x0 < 8u ? W - x0 : 8u;
    const uint32_t k = r - x0 * h;
    return (y0 + k / w) * W + x0 + k % w;
}

// f(pixel) for every pixel of the image in the same order, on the host.
template <class F>
void for_tile_pixels(uint32_t W, uint32_t H, F&& f)
{
    for (uint64_t y0 = 0; y0 < H; y0 += 8)
        for (uint64_t x0 = 0; x0 < W; x0 += 8)
            for (uint64_t y = y0; y < y0 + 8 && y < H; ++y)
                for (uint64_t x = x0; x < x0 + 8 && x < W; ++x) f((uint32_t)(y * W + x));
}

// The device-side plan of one sample round of a render with the early exit on
// (launch_plan_round, launch_compact_pixels): a batch with a plan reads the round's
// pixel count and samples per pixel from it instead of PathBatch::n / npix and the
// spb argument, so that the host enqueues rounds without knowing how many pixels
// are still sampling.
struct RoundPlan {
    uint32_t npix;        // pixels listed for this round (all still sampling)
    uint32_t spb;         // samples per pixel this round (0: the round does nothing)
    uint32_t n;           // paths of the round: npix * spb
    uint32_t scheduled;   // samples per pixel the rounds so far took
    uint32_t next_npix;   // pixels the compaction kept for the next round
    uint32_t pad[3];
};

// The queue sizes of one depth: its path segments, the shadow rays the shade before it left, and the closest-hit
// launch's claims.  A batch has a ring of kDepthRing of them, cleared in one go before it starts (a depth beyond the
// ring clears its own), so that a depth needs no clearing between its launches.
struct DepthQueues {
    uint32_t paths, shadows;
    unsigned long long work;
};
constexpr uint32_t kDepthRing = 64;

// Structure-of-arrays path state of one batch (capacity >= n) and the
// per-pixel accumulation buffers of the whole image.
struct PathBatch {
    uint32_t n, npix, width;
    uint32_t extend_ctas;              // closest-hit launches: persistent CTAs per SM (0: as many as fit)
    uint32_t extend_threads;           // closest-hit launches: threads per CTA, 64, 128 or 256 (other: 128)
    uint32_t pad;
    const uint32_t* pix_list;          // npix pixel indices
    float4* org; float4* dir; float4* thr; float4* pay;
    float4* hit; uint32_t* hit_tri;
    unsigned long long* rng;
    uint32_t* depth;
    uint32_t* ior_n; float4* ior_lo; float4* ior_hi;   // index-of-refraction stack: size, entries 0-3, 4-7
    float4* sorg; float4* sdir; float4* scontrib; float4* senergy;
    uint32_t* queue[2];
    uint32_t* shadow_queue;
    DepthQueues* depths;               // queue sizes of depth d at d % kDepthRing
    // image state (W*H entries)
    float* pixels; float* variance; uint32_t* count; uint32_t* taken; uint32_t* done;
    unsigned long long* sample_tally;  // samples added to the image (set by launch_render_batch)
    const RoundPlan* plan;             // null, or the round's n / npix / spb (n and npix above are then bounds)
};

// Measurement hooks of a render's closest-hit launches: CUDA events recorded on
// the launching stream before and after each one (timer), or work counters
// (count: the counting kernel variant adds nodes, triangles, instance entries
// and nodes inside instances to `counters`).  Both are off in ordinary renders.
struct LaunchTimer {
    std::vector<cudaEvent_t> events;   // before / after pairs, reused across renders
    size_t used = 0;
    cudaError_t record(cudaStream_t st);
    // Sum of the recorded launches' durations (ms) and their number; the events
    // must have completed.
    cudaError_t total(double& ms, uint64_t& launches) const;
    void reset() { used = 0; }
    ~LaunchTimer();
};
struct RenderProbe {
    LaunchTimer* timer;
    unsigned long long* counters;      // 4 counters, or null
    LaunchTimer* shade_timer;          // events around the shade launches, or null
};

// What the physical shade step does for the radiance cache.
//   kNrcRecord     every shaded vertex of a training path appends a record: the
//                  cache query (4 float4), then the path throughput and payload
//                  on arrival (2 float4 in rec_tp), from which the radiance the
//                  rest of the path reflects there is (final payload - payload)
//                  / throughput;
//   kNrcTerminate  a camera path stops at its vertex after one bounce (after two
//                  when the first vertex has roughness < 0.1) and appends that
//                  vertex's query; the cache's answer times the throughput is
//                  added to the payload after the depth loop.
enum NrcMode { kNrcOff = 0, kNrcRecord = 1, kNrcTerminate = 2 };
constexpr uint32_t kRecordSegment = 4096;   // entries of a CTA of the ordering kernels, 16 a thread
inline size_t record_segments(uint32_t capacity) { return ((size_t)capacity + kRecordSegment - 1) / kRecordSegment; }
PICO_HD size_t record_flags(uint32_t capacity) { return ((size_t)capacity + 15) & ~(size_t)15; }
struct NrcShadeArgs {
    int mode;
    uint32_t passes;          // passes traced together, pass p on paths [p * pass_paths, (p + 1) * pass_paths)
    uint32_t pass_paths;
    uint32_t capacity;        // entries of queries / rec_tp per pass
    uint32_t bounces;         // kNrcTerminate: bounces before the cache answers (one more behind a glossy vertex)
    float4* queries;          // 4 float4 per entry (pico_nrc_query); pass p's from entry p * capacity on
    uint32_t* count;          // entries, per pass
    // kNrcRecord: 2 float4 per entry.  A record's entry is its depth and path (depth * pass_paths + the path's number
    // in its pass), whichever thread shades it first, and order lists the entries written, ascending: a training step's
    // records do not depend on the order in which they arrive.
    float4* rec_tp;
    uint8_t* written;         // per entry 0 or 1; pass p's from p * record_flags(capacity) on
    uint32_t* segments;       // per pass and kRecordSegment entries: how many are written
    uint32_t* order;          // pass p's from p * capacity on
    float* prev_rough;        // kNrcTerminate: per path, roughness of its previous vertex
    // the cache the terminating paths query
    nrc::GridGeometry geo;
    const __half2* table;
    const uint8_t* weights;
    int* err;
    int infer_groups;
    nrc::WaitPolicy wait;
};

cudaError_t launch_render_batch(const SceneView& sc, PathBatch& b, const CameraView& cam, unsigned long long seed,
                                uint32_t spb, uint32_t max_depth, uint32_t max_samples, float max_variance,
                                int estimator, DeviceStatus* status, int order, cudaStream_t st,
                                const RenderProbe* probe = nullptr);
// Exit-aware rounds: plan_init lists npix pixels for the first round; plan_round
// sets the next round from the pixels the compaction kept: samples per pixel
// min(max_samples - scheduled, max_paths / pixels, cap), at most first_cap in the
// first round; compact_pixels keeps the pixels of `in` (plan->npix of them) that
// are not done, in `out`, counting them in plan->next_npix.
cudaError_t launch_plan_init(RoundPlan* plan, uint32_t npix, cudaStream_t st);
cudaError_t launch_plan_round(RoundPlan* plan, uint32_t max_samples, uint32_t first_cap, uint32_t cap,
                              uint32_t max_paths, cudaStream_t st);
cudaError_t launch_compact_pixels(RoundPlan* plan, const uint32_t* in, const uint32_t* done, uint32_t* out,
                                  uint32_t npix_bound, cudaStream_t st);
// The image state of a render into caller device buffers: every pixel listed in
// tile order (tile_pixel), done where count >= max_samples, nothing taken yet.
cudaError_t launch_prepare_image(const uint32_t* count, uint32_t W, uint32_t H, uint32_t max_samples,
                                 uint32_t* pix_list, uint32_t* done, uint32_t* taken, cudaStream_t st);
// The radiance cache's training paths of nrc.passes sample passes: nrc.pass_paths
// full-depth physical paths each, from pseudo-random pixels of the W x H image (path
// slots of b from 0 on; pass p draws with frame + p), recording every shaded vertex
// (kNrcRecord), then the records' order and their targets (4 floats an entry) in `targets`.
cudaError_t launch_training_paths(const SceneView& sc, PathBatch& b, const CameraView& cam, unsigned long long seed,
                                  uint32_t frame, uint32_t W, uint32_t H, uint32_t max_depth, const NrcShadeArgs& nrc,
                                  float4* targets, DeviceStatus* status, int order, cudaStream_t st);
// One sample per pixel of b and pass of nrc (kNrcTerminate), each path up to the vertex
// that it ends at in the cache; launch_cache_answers adds pass p's answers, and
// launch_accumulate then takes the samples of all passes.
cudaError_t launch_cache_paths(const SceneView& sc, PathBatch& b, const CameraView& cam, unsigned long long seed,
                               uint32_t max_depth, const NrcShadeArgs& nrc, DeviceStatus* status, int order,
                               cudaStream_t st);
cudaError_t launch_cache_answers(PathBatch& b, const NrcShadeArgs& nrc, uint32_t pass, cudaStream_t st);
cudaError_t launch_accumulate(PathBatch& b, uint32_t spb, uint32_t max_samples, float max_variance, bool physical,
                              DeviceStatus* status, cudaStream_t st);
// Writes the device's global nanosecond timer to *dst when the stream reaches it.
cudaError_t launch_stamp(unsigned long long* dst, cudaStream_t st);
cudaError_t launch_gbuffer(const SceneView& sc, const CameraView& cam, uint32_t W, uint32_t H, float* normals,
                           float* positions, float* diffuse, DeviceStatus* status, int order, cudaStream_t st);
// Floats of a-trous scratch for a W x H image: the packed records (16 a pixel), and the statistics: per level and
// 64 x 64 tile a white point and the scale of the position term, per level, image row and tile column the (min, max)
// |position|, and the luminance cells, c x c pixels each, of levels 1-4 (c = 4, 8, 16, 32).
inline size_t atrous_record_floats(uint32_t W, uint32_t H) { return (size_t)16 * W * H; }
inline size_t atrous_level_cells(uint32_t W, uint32_t H, int c) { return (((size_t)W + c - 1) / c) * (((size_t)H + c - 1) / c); }
inline size_t atrous_cells(uint32_t W, uint32_t H)
{
    size_t n = 0;
    for (int c = 4; c <= 32; c *= 2) n += atrous_level_cells(W, H, c);
    return n;
}
inline size_t atrous_stats_floats(uint32_t W, uint32_t H)
{
    const size_t tx = ((size_t)W + 63) / 64, ty = ((size_t)H + 63) / 64;
    return tx * ty * (5 + 5) + (size_t)5 * 2 * H * tx + atrous_cells(W, H);
}
cudaError_t launch_atrous(const float* pixels, const float* normals, const float* positions, const float* diffuse,
                          uint32_t W, uint32_t H, float* records, float* stats, float* out, cudaStream_t st);
cudaError_t launch_reinhard(float* pixels, uint32_t W, uint32_t H, unsigned* scratch, cudaStream_t st);

}  // namespace pico
