// Wavefront integrators: the per-sample logic of the reference's stencil,
// depth, ao and pathtracer render_tile methods, split into queue stages.
//
//   camera     one ray per (pixel, position) of every job in the wave
//   extend     closest hit of every queued ray (traverse.cuh)
//   shade      integrator step: contribution of finished paths, next rays of the
//              others appended to the next queue (warp-aggregated atomics); the
//              first pass starts the wave's paths, one per sample, at the hits
//              of their camera rays
//   accumulate per pixel, the samples of the wave folded in sample order into
//              the job's frame exactly as the reference folds them (float
//              colour channels clamped at 0, alpha clamped to [0, 1])
//
// A path's result depends only on (job seed, pixel, sample): the random stream is
// keyed by them, never by a queue slot, and the fold runs in sample order.  So a
// job renders to the same bits alone, split over any number of waves, or merged
// with other jobs.
#pragma once

#include "traverse.cuh"

namespace xtg {

// One job's share of a wave.
struct DevJob {
    int32_t integrator, width, height;
    int32_t spp;                     // samples per pixel: positions x spp1
    int32_t rdepth;
    float ao_maxd;
    uint64_t seed;
    int32_t x0, y0, rw, rh;          // rectangle rendered
    int32_t scene;                   // index in the scene table
    int32_t bounces;                 // extend passes this job needs
    int32_t tile;                    // camera order: square pixel tiles of this edge (0 = rows)
    float4 *frame;                   // rw*rh RGBA accumulation buffer
    int64_t first;                   // first path id of the job in this wave
    int64_t count;                   // paths of the job in this wave
    int64_t offset;                  // wave-local index of the job's first path
    int32_t aa;                      // anti-aliasing level (grid: 1 = pixel centre)
    int32_t spp1;                    // samples per position
    double wt;                       // weight of one sample: 1/positions as a float, times 1/spp1
    float *raygraph;                 // depth integrator: 10 floats per sample (origin, hit
                                     // point, colour after the sample), rectangle pixels
                                     // row-major, each pixel's samples in order; or null
    int32_t dist;                    // XTGPU_SAMPLES_GRID or XTGPU_SAMPLES_RANDOM
    int32_t share;                   // samples in a row that have one camera ray: spp1, or 1 when
                                     // every sample draws its own lens point
    int64_t u0;                      // camera rays of the wave's first (maybe partial) run of them
    int64_t ufirst;                  // wave-local index of the job's first camera ray
    int32_t pix0;                    // wave-local index of the first of its pixels that the
                                     // wave touches
};

// What the wave holds, as the host writes it; the job table follows at CTL_BYTES, so
// that one copy brings both (on lines of its own: beside the counters that shade's
// warps add to, its reads took shade from 121 to 137 us on 256x256x16 spheres).
enum { CTL_QUEUE = 0,                // [0], [1] rays in the queues ([0] starts as the camera rays)
       CTL_FETCH = 2,                // rays taken by the extend kernel
       CTL_JOBS = 4, CTL_PATHS = 5,
       CTL_PIXELS = 6,               // pixels touched, over all jobs
       CTL_RESET = 7 };              // the first wave of a call: counts start at zero
constexpr size_t CTL_BYTES = 256;
// Counters that outlive a wave: rays followed, overflow flag.
constexpr size_t STATE_BYTES = 16;

// Key of the random distribution's offsets of one position of one pixel: a
// stream apart from the paths' (seed ^ this salt).
constexpr uint64_t JITTER_SALT = 0xA0761D6478BD642Full;

// Positions per pixel (aa.cc:7-48): the grid's aa^2, the random
// distribution's aa; level 0 renders as level 1.
inline int sample_positions(int aa, int dist)
{
    const int L = aa > 1 ? aa : 1;
    return dist == XTGPU_SAMPLES_RANDOM ? L : L * L;
}

// Fills the sample fields of a job from params_t's samples, aa and
// sample_distribution (aa.cc:7-77): P positions of weight 1.f/P each taken
// spp times at 1/spp.
inline void set_samples(DevJob &j, int spp, int aa, int dist)
{
    const int L = aa > 1 ? aa : 1, P = sample_positions(aa, dist);
    j.aa = L;
    j.dist = dist;
    j.spp1 = spp;
    j.spp = P * spp;
    j.wt = (P == 1 ? 1.0 : (double)(1.f / (float)P)) * (1.0 / (double)spp);
}

// Camera rays of a wave.  Paths are numbered sample by sample, each sample over
// all pixels, so the `share` samples of one position form a run of
// share * npix paths whose rays repeat every npix: only the first npix of the
// run (or of the part of it that is in the wave) are traced, and k_shade's
// first pass sends every path to its ray.  Fills u0 and ufirst of a job whose
// first and count are set; returns how many camera rays it has in the wave.
inline int64_t set_camera_rays(DevJob &j, bool lens, int64_t ufirst)
{
    const int64_t npix = (int64_t)j.rw * j.rh;
    j.share = lens ? 1 : j.spp1;
    j.ufirst = ufirst;
    const int64_t run = (int64_t)j.share * npix, end = j.first + j.count;
    const int64_t b0 = j.first / run, b1 = (end - 1) / run;
    auto least = [](int64_t a, int64_t b) { return a < b ? a : b; };
    j.u0 = least(npix, least(end, (b0 + 1) * run) - j.first);
    return b1 == b0 ? j.u0 : j.u0 + (b1 - b0 - 1) * npix + least(npix, end - b1 * run);
}

// a / b of non-negative numbers, in 32 bits where both fit: a 64-bit division is
// some hundred instructions, and the first shade pass and k_camera do up to six
// a path with little else to wait for.
__host__ __device__ inline int64_t div64(int64_t a, int64_t b)
{
    return ((uint64_t)(a | b) >> 32) == 0 ? (int64_t)((uint32_t)a / (uint32_t)b) : a / b;
}

// The path whose camera ray is the job's v-th in the wave, and the other way
// round for a path p of sample s and pixel slot pix.
__host__ __device__ inline int64_t camera_ray_path(const DevJob &j, int64_t npix, int64_t v)
{
    if (v < j.u0) return j.first + v;
    const int64_t run = (int64_t)j.share * npix, w = v - j.u0, k = div64(w, npix);
    return (div64(j.first, run) + 1 + k) * run + (w - k * npix);
}
__host__ __device__ inline int64_t camera_ray_of(const DevJob &j, int64_t npix, int64_t p, int64_t s, int64_t pix)
{
    const int64_t b = div64(s, j.share), b0 = div64(j.first, npix * j.share), k = p - j.first;
    return b == b0 ? k - div64(k, npix) * npix : j.u0 + (b - b0 - 1) * npix + pix;
}

// The order in which the first shade pass takes a job's paths of the wave: the
// samples that share a ray next to each other (numbered from 0; the result counts
// from the job's first path).  Their next rays leave one point and stay together
// in the queue: 1.05x on the AO rays of the hairball at 16 spp, 1.02x on terrain
// bounces at 4 spp, 1.06x on the Phong scene's at 8, against sample after sample.
__host__ __device__ inline int64_t first_pass_path(const DevJob &j, int64_t npix, int64_t i)
{
    if (j.share == 1) return i;
    const int64_t run = (int64_t)j.share * npix;
    int64_t start = 0, len = (div64(j.first, run) + 1) * run - j.first;   // the run of path i
    if (i >= len) {
        start = len + div64(i - len, run) * run;
        len = run;
    }
    if (len > j.count - start) len = j.count - start;
    if (len <= npix) return i;
    // the first `more` rays of the run have k paths in the wave, the others k - 1
    const int64_t k = div64(len + npix - 1, npix), more = len - (k - 1) * npix;
    i -= start;
    int64_t ray, rep;
    if (i < more * k) {
        ray = div64(i, k);
        rep = i - ray * k;
    } else {
        const int64_t q = i - more * k, r = div64(q, k - 1);
        ray = more + r;
        rep = q - r * (k - 1);
    }
    return start + rep * npix + ray;
}

struct WaveQueues {
    float4 *org[2], *dir[2];         // (org, tmin), (dir, tmax)
    uint2 *meta[2];                  // (wave-local path index, job slot)
    float4 *P[2];                    // (prefix throughput rgb, rng counter)
    float4 *I[2];                    // (incoming intensity rgb, depth left)
    xtgpu_hit *hit;
    float4 *contrib;                 // per wave-local path: result of the sample
    int32_t *ctl;                    // CTL_*.  The kernels leave the counters as the next one needs
                                     // them: extend clears the queue that shade fills, shade the
                                     // fetch counter (a memset before each cost 2 us and a gap)
    int32_t *over;                   // set when a traversal stack overflows
    unsigned long long *rays;        // rays followed: one per path and pass (paths whose camera
                                     // ray is traced once for all of them count one each)
    unsigned long long *job_rays;    // per job of the wave, or nullptr
    unsigned long long *stats;       // [0] nodes visited, [1] primitives tested, or nullptr
    int64_t capacity;
    int32_t n = -1;                  // rays of queue A, or -1: its count is in ctl
};

}  // namespace xtg
