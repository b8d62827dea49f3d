// Render state shared by the single-render and batched-render entry points.
#pragma once

#include "capi_internal.h"
#include "kernels_render.h"

// Path state and image buffers of one render, grown on demand.
struct RenderBuffers {
    pico::DeviceBuffer org, dir, thr, pay, hit, hit_tri, rng, depth, ior_n, ior_lo, ior_hi, sorg, sdir, scontrib,
        senergy, q0, q1, sq, counters;
    pico::DeviceBuffer pixels, variance, count, taken, done, pix_list;
    pico::DeviceBuffer pix_list2, plan;   // exit-aware rounds: the compacted pixel list, the round plan
    pico::DeviceBuffer gn, gp, gd, ga, stats, out, tonemap;
    pico::DeviceBuffer hdr_pix, hdr_codes, hdr_lens, hdr_off, hdr_body;   // .hdr output: image, codes, their lengths
                                                                          // and places, the file's body
    // radiance cache: training records' queries, throughput and payload, targets, which are written and their order;
    // terminal queries; previous roughness per path; entry counters
    pico::DeviceBuffer nrc_q, nrc_tp, nrc_tgt, nrc_written, nrc_segments, nrc_order, nrc_term, nrc_prev, nrc_count;
    size_t budget = ~size_t(0);   // pico_test_cache_budget
    // the host buffers this render's results will go to, populated once the device has its first work
    struct { void* p; size_t bytes; } results[3] = {};
    void forget_results()
    {
        for (auto& b : results) b = {};
    }
    void populate_results()
    {
        for (const auto& b : results) pico::populate_for_writing(b.p, b.bytes);
        forget_results();
    }
    ~RenderBuffers()
    {
        for (pico::DeviceBuffer* b : {&org, &dir, &thr, &pay, &hit, &hit_tri, &rng, &depth, &ior_n, &ior_lo, &ior_hi,
                                      &sorg, &sdir, &scontrib, &senergy, &q0, &q1, &sq, &counters, &pixels,
                                      &variance, &count, &taken, &done, &pix_list, &pix_list2, &plan, &gn, &gp, &gd,
                                      &ga, &stats,
                                      &out, &tonemap, &hdr_pix, &hdr_codes, &hdr_lens, &hdr_off, &hdr_body, &nrc_q, &nrc_tp, &nrc_tgt, &nrc_written, &nrc_segments, &nrc_order, &nrc_term, &nrc_prev, &nrc_count})
            b->release();
    }
};

namespace pico {

// Paths of one batch of a single render (pixels x samples; 208 B of path state
// each, 14 GB at the limit).  Larger batches amortise each launch and its
// tail: a 1080p render at 64 spp measured 159 / 206 / 267 / 279 / 286 Msamples/s
// with batches of 2^19 / 2^20 / 2^22 / 2^23 / 2^24 paths (physical estimator),
// and 2^25 / 2^26 took the 1080p renders 1.4 / 2.5 % (reference estimator) and
// 1.4 / 2.0 % (physical) below 2^24's time.
constexpr uint32_t kMaxPaths = 1u << 26;
// Device bytes of path state per path that reserve_paths allocates: eleven float4
// arrays, six uint32 arrays and the 64-bit random state.
constexpr size_t kPathStateBytes = 11 * 16 + 6 * 4 + 8;

// What a caller's sample counts say before a render of max_samples per pixel.
struct CountScan {
    size_t unfinished = 0;   // pixels that will take samples
    bool fresh = false;      // no pixel has a sample and all will take one: the mean and variance passed in are not read
};
// Whether no pixel has a sample (false for no pixels): reads up to the first sample.
bool no_samples(const uint32_t* count, size_t npx);
CountScan scan_counts(const uint32_t* count, size_t npx, uint32_t max_samples);

template <class T>
T* as(DeviceBuffer& b) { return static_cast<T*>(b.ptr); }

// Camera::getRight (Core/Camera.hpp:64-65) and Camera::getViewMatrix (glm::lookAtRH).
CameraView make_camera_view(const pico_camera& c);
cudaError_t reserve_paths(RenderBuffers& r, size_t n);
// The path state of a batch of n paths over npix listed pixels, in r's buffers.
PathBatch make_batch(RenderBuffers& r, uint32_t n, uint32_t npix, uint32_t W, const uint32_t* pix_list);

}  // namespace pico
