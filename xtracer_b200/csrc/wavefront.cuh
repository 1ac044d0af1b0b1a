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

// Division by a number known on the host, exact for dividends below 2^31: a high
// product, an addition and a shift where the device's 32-bit division is some 25
// instructions (Granlund and Montgomery, "Division by Invariant Integers using
// Multiplication", PLDI 1994).  k_shade's first pass did ten divisions a path, 250 of
// its 890 instructions: 156 us for 4 Mi paths on terrain200k, 113 so; k_accumulate
// 29 -> 19 us for a 1080p frame of one sample.
struct FastDiv {
    uint32_t d, m, sh;
    __host__ __device__ uint32_t div(uint32_t n) const
    {
#ifdef __CUDA_ARCH__
        return (__umulhi(m, n) + n) >> sh;
#else
        return ((uint32_t)(((uint64_t)m * n) >> 32) + n) >> sh;
#endif
    }
};
inline FastDiv fast_div(int64_t d)   // 1 <= d <= 2^31
{
    FastDiv f;
    f.d = (uint32_t)d;
    f.sh = 0;
    while ((1ll << f.sh) < d) ++f.sh;
    f.m = (uint32_t)((((1ull << f.sh) - (uint64_t)d) << 32) / (uint64_t)d + 1);
    return f;
}

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
    int64_t ufirst;                  // wave-local index of the job's first camera ray
    // Filled by set_camera_rays for the wave: the first path's sample and pixel slot,
    // and the runs of paths that share rays (see there): the first one's part in the
    // wave (0), whole ones (1) and the last one's part (2).
    int64_t run_len;                 // share * pixels
    int32_t first_smp;
    int32_t wide;                    // more pixels than 32-bit divisions hold
    int64_t first_slot;
    int32_t len0, runs;              // paths of part 0; whole runs after it
    int32_t rays0;                   // rays of part 0
    int32_t reps[3], more[3];        // rays with reps[k] paths; the others have one fewer
    FastDiv reps_div[3], less_div[3];
    FastDiv pix_div, run_div;        // by the pixels; by run_len (where there are whole runs)
    // pixel slots in tiles (pixel_of)
    FastDiv band_div, row_div;       // by a band's pixels; by the width (tile <= 1)
    FastDiv tile_div[2], col_div[2]; // by a whole or the last band's tile; by a whole or the last tile's width
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
       CTL_RESET = 7,                // the first wave of a call: counts start at zero
       CTL_FOLLOWED = 8 };           // paths of jobs with passes: what the first pass adds to the ray count
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

// The most pixels of a job for the 32-bit divisions (a wave has at most 2^26 paths, so
// sums of a slot and a path stay below 2^31).  Larger ones divide in 64 bits.
constexpr int64_t MAX_FAST_PIXELS = 1ll << 30;

// Camera rays of a wave.  Paths are numbered sample by sample, each sample over
// all pixels, so the `share` samples of one position form a run of
// share * npix paths whose rays repeat every npix: only the first npix of the
// run (or of the part of it that is in the wave) are traced, and k_shade's
// first pass sends every path to its ray.  Fills the job's fields for the wave
// from its first and count; returns how many camera rays it has in the wave.
inline int64_t set_camera_rays(DevJob &j, bool lens, int64_t ufirst)
{
    const int64_t npix = (int64_t)j.rw * j.rh;
    auto least = [](int64_t a, int64_t b) { return a < b ? a : b; };
    j.share = lens ? 1 : j.spp1;
    j.ufirst = ufirst;
    j.first_smp = (int32_t)(j.first / npix);
    j.first_slot = j.first % npix;
    j.wide = npix > MAX_FAST_PIXELS;
    const int64_t run = j.run_len = (int64_t)j.share * npix;
    j.len0 = (int32_t)least(j.count, (j.first / run + 1) * run - j.first);
    j.runs = (int32_t)((j.count - j.len0) / run);
    const int64_t len[3] = {j.len0, run, j.count - j.len0 - j.runs * run};
    for (int k = 0; k < 3; ++k) {
        const int64_t l = len[k] > 0 && (k != 1 || j.runs > 0) ? len[k] : 1;
        j.reps[k] = (int32_t)((l + npix - 1) / npix);
        j.more[k] = (int32_t)(l - (j.reps[k] - 1) * npix);
        j.reps_div[k] = fast_div(j.reps[k]);
        j.less_div[k] = fast_div(j.reps[k] > 1 ? j.reps[k] - 1 : 1);
    }
    j.rays0 = (int32_t)least(j.len0, npix);
    // (a wide job's wave is shorter than a sample: any number above its paths will do)
    j.pix_div = fast_div(least(npix, MAX_FAST_PIXELS));
    j.run_div = fast_div(j.runs > 0 ? run : 1);
    if (j.tile > 1) {
        const int64_t T = j.tile, bands = (j.rh + T - 1) / T, cols = (j.rw + T - 1) / T;
        const int64_t last_h = j.rh - (bands - 1) * T, last_w = j.rw - (cols - 1) * T;
        j.band_div = fast_div(least(T * j.rw, 1ll << 31));
        j.tile_div[0] = fast_div(T * T);
        j.tile_div[1] = fast_div(T * last_h);
        j.col_div[0] = fast_div(T);
        j.col_div[1] = fast_div(last_w);
    } else {
        j.row_div = fast_div(j.rw);
    }
    const int64_t last = len[2] > 0 ? least(len[2], npix) : 0;
    return j.rays0 + j.runs * npix + last;
}

// Sample and pixel slot of the job's path first + k.
__host__ __device__ inline void sample_of(const DevJob &j, int32_t k, int32_t &smp, int64_t &slot)
{
    if (j.wide) {
        const int64_t npix = (int64_t)j.rw * j.rh, t = j.first_slot + k;
        smp = j.first_smp + (int32_t)(t / npix);
        slot = t % npix;
        return;
    }
    const uint32_t t = (uint32_t)j.first_slot + (uint32_t)k, q = j.pix_div.div(t);
    smp = j.first_smp + (int32_t)q;
    slot = (int64_t)(t - q * j.pix_div.d);
}

// The path, from the job's first, whose camera ray is the job's v-th in the wave.
__host__ __device__ inline int32_t camera_ray_path(const DevJob &j, int32_t v)
{
    if (v < j.rays0) return v;
    const uint32_t w = (uint32_t)(v - j.rays0), k = j.pix_div.div(w);
    return (int32_t)(j.len0 + k * j.run_len + (w - k * j.pix_div.d));
}

// The order in which the first shade pass takes a job's paths of the wave: the
// samples that share a ray next to each other.  The i-th taken: its path, from the
// job's first, and its ray.  Their next rays leave one point and stay together in the
// queue: 1.05x on the AO rays of the hairball at 16 spp, 1.02x on terrain bounces at
// 4 spp, 1.06x on the Phong scene's at 8, against sample after sample.
__host__ __device__ inline int32_t first_pass_path(const DevJob &j, int32_t i, int32_t &ray)
{
    const int32_t npix = (int32_t)j.pix_div.d;
    int part = 0;
    int32_t start = 0, rays = 0;   // of the part's paths and rays
    if (i >= j.len0) {
        const int32_t b = j.runs > 0 ? (int32_t)j.run_div.div((uint32_t)(i - j.len0)) : 0;
        part = b < j.runs ? 1 : 2;
        start = j.len0 + (int32_t)(b * j.run_len);
        rays = j.rays0 + b * npix;
    }
    // the part's first `more` rays have `reps` paths in the wave, the others one fewer
    const int32_t k = j.reps[part], more = j.more[part];
    int32_t n = i - start, r, rep;
    if (n < more * k) {
        r = (int32_t)j.reps_div[part].div((uint32_t)n);
        rep = n - r * k;
    } else {
        n -= more * k;
        const int32_t q = (int32_t)j.less_div[part].div((uint32_t)n);
        r = more + q;
        rep = n - q * (k - 1);
    }
    ray = rays + r;
    return start + rep * npix + r;
}

// Pixel of the k-th pixel slot of a job.  With tiles, slots run through
// square tiles of `tile` pixels (row-major tiles, row-major inside a tile; the
// last band and column may be partial), which keeps the rays of a warp close
// together on screen.  A bijection of [0, rw*rh), so every pixel is visited once.
__host__ __device__ inline void pixel_of(const DevJob &j, int64_t slot, int &x, int &y)
{
    const int T = j.tile;
    if (j.wide) {
        const int64_t band_pixels = T > 1 ? (int64_t)T * j.rw : j.rw, band = slot / band_pixels;
        const int64_t q = slot - band * band_pixels;
        if (T <= 1) {
            x = j.x0 + (int)q;
            y = j.y0 + (int)band;
            return;
        }
        const int64_t rows = j.rh - band * T < T ? j.rh - band * T : T, c = q / (T * rows);
        const int64_t cols = j.rw - c * T < T ? j.rw - c * T : T, r = q - c * T * rows;
        x = j.x0 + (int)(c * T + r % cols);
        y = j.y0 + (int)(band * T + r / cols);
        return;
    }
    const uint32_t k = (uint32_t)slot;
    if (T <= 1) {
        const uint32_t row = j.row_div.div(k);
        x = j.x0 + (int)(k - row * j.row_div.d);
        y = j.y0 + (int)row;
        return;
    }
    const uint32_t band = j.band_div.div(k), q = k - band * j.band_div.d;
    const FastDiv &td = j.tile_div[(int64_t)(band + 1) * T > j.rh];
    const uint32_t c = td.div(q), r = q - c * td.d;
    const FastDiv &cd = j.col_div[(int64_t)(c + 1) * T > j.rw];
    const uint32_t row = cd.div(r);
    x = j.x0 + (int)(c * T + r - row * cd.d);
    y = j.y0 + (int)(band * T + row);
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
