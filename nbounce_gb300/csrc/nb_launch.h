// Kernel parameter blocks and launcher declarations (nb_kernels.cu <-> nb_api.cu, nb_server.cu).
//
// A wave is one wavefront of paths: raygen, then trace + shade per bounce, then accumulate.
// Its paths come from segments; a segment is a run of consecutive samples of one job (one
// render request: scene, camera, environment, image).  The single-image Pathtracer runs
// waves of one segment; the server packs segments of many jobs into one wave.
#pragma once

#include <cstdint>
#include <algorithm>

#include <cuda_runtime.h>

#include "nb_device.cuh"
#include "nb_mlp.cuh"

namespace nb {

constexpr uint32_t kMaxBounceSlots = 64;  // per-bounce queue counters (bounces <= 62)
constexpr uint32_t kMaxWaveJobs = 32;     // jobs per wave
constexpr uint32_t kMaxWaveSegments = 64; // segments per wave
constexpr uint32_t kMaxWaveScenes = 16;   // distinct scenes per wave

struct JobParams {
  float c2w[16];        // clip_to_world, column-major
  nbd::DevEnv env;
  float4* out;          // RGBA32F image, width * height
  uint32_t scene;       // index into WaveTables::scenes
  uint32_t width, height, npix;
  uint32_t bounces;
  float cf;             // contribution_factor
  uint32_t rr_start;    // Russian roulette from this bounce on (0: the reference schedule)
  uint32_t flags;       // kJobEnvNee: environment next-event estimation (k_shade_nee)
};
constexpr uint32_t kJobEnvNee = 1u << 0;

struct Segment {
  uint32_t job;           // index into WaveTables::jobs
  uint32_t first_sample;  // 1-based Sobol row of the segment's first sample
  uint32_t n_samples;
  uint32_t path_begin;    // first path id of the segment in the wave
  uint32_t pix_begin;     // first accumulate thread of the segment
};

// Passed by value to the wave kernels (well under the 32 KB parameter limit).
// flags: kWaveZeroRadiance - raygen zeroes every path's radiance, for waves whose shading adds
// to it (environment NEE, radiance cache); with the reference estimator every path's radiance
// is written once, where the path ends (k_shade), and raygen leaves it alone.
// kWaveDirect - the wave is one launch of k_trace_paths whose paths add to their pixels themselves.
constexpr uint32_t kWaveZeroRadiance = 1u << 0;
constexpr uint32_t kWaveDirect = 1u << 1;
// 64-bit counters per bounce slot of the instrumented traversal (nb_pathtracer_trace_counters):
// 0-4 node / triangle / instance / push counts, 5 rays, 6-10 warp-step statistics
constexpr uint32_t kTraceCounterSlots = 16;
struct WaveTables {
  uint32_t n_segs, n_jobs, n_scenes, n_paths, n_pix;
  uint32_t flags;
  uint32_t group_limit;  // queues of bounces >= 1 up to this long are run to their ends by k_trace_paths
  uint32_t pad;
  Segment segs[kMaxWaveSegments];
  JobParams jobs[kMaxWaveJobs];
  nbd::DevScene scenes[kMaxWaveScenes];
};

// Device work buffers of a wave.  Path p is sample p / npix, pixel p % npix of its segment.
struct PathBatch {
  float4* q_o[2];       // ray origin, .w = path id (bits); double-buffered queues
  float4* q_d[2];       // ray direction, .w = scene index (bits)
  float4* q_t[2];       // throughput
  float4* hits;         // t, u, v, triangle (bits)
  uint32_t* hit_inst;   // TLAS-permuted instance of the hit
  float4* radiance;     // L per path id
  uint32_t* counts;     // rays entering bounce b (kMaxBounceSlots)
  uint32_t* fetch;      // work-fetch cursor per bounce (kMaxBounceSlots)
  uint32_t* status;     // device status word
  const float4* sobol;  // Sobol-Burley table, kLdsStride vec4 per sample row
  uint32_t sobol_entries;
};

// refill: lanes take new rays as theirs finish (for arrays whose neighbouring rays are unrelated)
cudaError_t launch_trace_rays(const nbd::DevScene& s, const float* rays, uint32_t n, bool any, bool refill,
                              float* hits, uint32_t* inst, uint32_t* fetch, uint32_t* status, int sms,
                              cudaStream_t st);

cudaError_t launch_raygen(const PathBatch& pb, const WaveTables& wt, int sms, cudaStream_t st);
struct ShadowQueue;
// single_scene: all paths use wt.scenes[0] (passed by value); otherwise each ray's scene index.
// shadow (optional, bounce >= 1): also traces the shadow rays of the bounce before.
// counters (optional): runs the instrumented traversal, which adds its work counters (TLAS
// node tests, BLAS node tests, triangle tests, instance entries, stack pushes) to
// counters[8 * bounce + 0..4].
cudaError_t launch_trace_wave(const PathBatch& pb, const WaveTables& wt, bool single_scene, uint32_t bounce,
                              const ShadowQueue* shadow, unsigned long long* ray_total, int sms, cudaStream_t st,
                              unsigned long long* counters = nullptr);
cudaError_t launch_shade(const PathBatch& pb, const WaveTables& wt, uint32_t bounce, int sms, cudaStream_t st);
// Shadow rays of environment next-event estimation: one per path and bounce at most.
struct ShadowQueue {
  float4* o;          // origin, .w = path id (bits)
  float4* d;          // direction (unit)
  float4* c;          // radiance the path gains when the direction is unoccluded
  uint32_t* counts;   // rays appended per bounce (kMaxBounceSlots)
  uint32_t* fetch;    // work-fetch cursor per bounce (kMaxBounceSlots)
};

// environment next-event estimation (NB_SAMPLE_ENV_NEE): shade, then the bounce's shadow rays
cudaError_t launch_shade_nee(const PathBatch& pb, const WaveTables& wt, const ShadowQueue& sq, uint32_t bounce,
                             int sms, cudaStream_t st);
cudaError_t launch_trace_shadow(const PathBatch& pb, const WaveTables& wt, const ShadowQueue& sq, uint32_t bounce,
                                int sms, cudaStream_t st);
// directions and densities of env importance samples for uniform pairs u (device arrays)
cudaError_t launch_env_sample(const nbd::DevEnv& env, const float* u, uint32_t n, float4* out, int sms,
                              cudaStream_t st);

struct CacheWave;
// radiance-cache mode shade (nb_mlp.cuh describes the wave state)
cudaError_t launch_shade_cache(const PathBatch& pb, const WaveTables& wt, const CacheWave& cw, uint32_t bounce,
                               int sms, cudaStream_t st);
// nothing to do for a kWaveDirect wave
cudaError_t launch_accumulate(const PathBatch& pb, const WaveTables& wt, int sms, cudaStream_t st);

enum class Estimator { kPlain, kNee, kCache };
// 8 lanes per path, to its end: the camera paths of a whole wave (bounce 0), or a bounce's queue if
// it holds at most wt.group_limit paths (the per-bounce kernels then skip that queue).
cudaError_t launch_trace_paths(const PathBatch& pb, const WaveTables& wt, Estimator est, const CacheWave& cw,
                               uint32_t bounce, unsigned long long* ray_total, int sms, cudaStream_t st);

// Queues and waves up to kGroupPaths paths (fewer where they can have few more rays or have shadow rays:
// launch_bounces), and nb_trace_rays calls up to kGroupRays rays (kGroupScattered with
// NB_TRACE_INCOHERENT), are traced by 8 lanes per ray.  Such a ray costs ~2.5 times the instructions of a
// ray per lane, but a node step takes 0.8 us instead of ~2, and a launch is as long as its longest ray
// until the GPU is full.
// Paths (run to their ends by k_trace_paths), limits of 16K / 24K / 32K / 64K: 160x120 at 1 spp on the
// instanced scene 320 / 260 / 262 / 260 us, 256x256 514 / 516 / 517 / 642, with NEE 1000 / 1000 / 1194 /
// 1544, 400x300 626 / 631 / 594 / 679, 576x320 669 / 657 / 653 / 642, 1013x571 at 3 spp with NEE 3025 / 3090 /
// 3080 / 3348 (queues handed on whatever their length from some bounce on, which is no longer done).  Rays, 8
// lanes against one, closest hits: camera grids of 16,384 rays on soups of 2K, 20K and 1M triangles 24 / 24,
// 50 / 58 and 108 / 145 us, of 32,761 rays 33 / 23, 63 / 59 and 156 / 178; 24,025 scattered rays 37 / 38,
// 76 / 92 and 190 / 250, 32,761 44 / 40, 91 / 94 and 218 / 256.
constexpr uint32_t kGroupPaths = 1u << 15;
constexpr uint32_t kGroupRays = 1u << 14, kGroupScattered = 3u << 13;

// The launch kinds of a wave (nb_kernel_times)
enum class Stage { kStart, kTrace, kShade };

// A wave from its start to its last bounce.  groups: short queues go to k_trace_paths.  counters
// (optional): the instrumented traversal, a ray per lane throughout.  timed(stage, launch) runs one
// launch.  launch_accumulate has to follow (after the lookups of a cache wave).
template <class Timed>
cudaError_t launch_bounces(const PathBatch& pb, WaveTables& wt, Estimator est, bool single_scene, uint32_t max_bounces,
                           const ShadowQueue& sq, const CacheWave& cw, unsigned long long* ray_total, int sms,
                           cudaStream_t st, bool groups, unsigned long long* counters, Timed timed) {
  groups = groups && counters == nullptr;
  wt.group_limit = 0u;
  wt.flags = est != Estimator::kPlain ? kWaveZeroRadiance : 0u;  // their shading adds to radiance
  // Whether a bounce's queue is short (limit) is decided on the device, at each bounce up to the one after
  // that where it is short if half of the paths end per bounce, and at every second one after it: as many
  // of open scenes' queues as ever get short have done so by then, and a check that finds nothing to do, or a
  // bounce whose paths have ended, costs 3 to 4 us a launch.  How many paths a bounce leaves is the
  // scene's: handing every queue to k_trace_paths from that bounce on, whatever its length, saves those
  // launches (576x320 at 1 spp on the instanced scene 662 instead of 731 us), but an enclosed scene keeps
  // most of its paths alive.  The room (scenes.room_scene), with / without that rule: 576x320 at
  // 1 spp 1013 / 583 us, 1920x1080 4186 / 2276, at 12 bounces 5365 / 2575, 256x256 at 16 spp 3474 / 1462, 1920x1080
  // with NEE 8234 / 3318.  Checks at every bounce: 2,000 overlapping spheres at 576x320 11.6 instead of 11.0 ms,
  // the instanced scene 733 us; none after the first kind: 14.1 instead of 12.2 at 12 bounces, 713 us.
  //
  // A path that can have few more rays gains little from a launch of its own to its end, and an enclosed
  // scene's paths have all they can.  181x181 pixels of the room at 0 / 1 / 2 / 3 / 4 / 6 bounces: per bounce 60 / 121 /
  // 174 / 221 / 269 / 360 us, as one launch 90 / 174 / 241 / 298 / 337 / 402; 150x150 at 0 to 4: 62 / 115 / 165 / 212 / 261
  // and 68 / 126 / 174 / 216 / 244.  With NEE, whose shadow rays share the per-bounce launches, 181x181 at 3 / 6
  // bounces 297 / 469 and 651 / 886 us; 1013x571 at 3 spp of the instanced scene takes 2.98 ms, 3.05 with a limit
  // of 32,768.
  const uint32_t cap = est == Estimator::kNee ? 3u * (kGroupPaths / 4u) : kGroupPaths;
  auto limit = [&](uint32_t b) { return std::min(cap, 4096u * (max_bounces + 2u - b)); };
  uint32_t half = 0;
  while (groups && half <= max_bounces && (wt.n_paths >> half) > limit(half)) ++half;
  auto check = [&](uint32_t b) { return groups && b >= 1 && (b <= half + 1 || ((b - half) & 1u)); };
  auto paths = [&](uint32_t b) {
    return timed(Stage::kTrace, [&] { return launch_trace_paths(pb, wt, est, cw, b, ray_total, sms, st); });
  };
  if (groups && half == 0) {
    bool direct = est != Estimator::kCache;
    for (uint32_t k = 0; k < wt.n_segs; ++k) direct = direct && wt.segs[k].n_samples == 1;
    wt.flags = direct ? kWaveDirect : 0u;
    wt.group_limit = 0xFFFFFFFFu;
    return paths(0);
  }
  cudaError_t e = cudaSuccess;
  if (est == Estimator::kNee) e = cudaMemsetAsync(sq.counts, 0, 2 * kMaxBounceSlots * sizeof(uint32_t), st);
  if (e == cudaSuccess) e = timed(Stage::kStart, [&] { return launch_raygen(pb, wt, sms, st); });
  // a bounce's shadow rays run with the next bounce's queue, or in a launch of their own
  const bool nee = est == Estimator::kNee, mixed = nee && counters == nullptr;
  auto shadows = [&](uint32_t b) {
    return timed(Stage::kTrace, [&] { return launch_trace_shadow(pb, wt, sq, b, sms, st); });
  };
  for (uint32_t b = 0; b <= max_bounces && e == cudaSuccess; ++b) {
    wt.group_limit = check(b) ? limit(b) : 0u;
    e = timed(Stage::kTrace, [&] {
      return launch_trace_wave(pb, wt, single_scene, b, mixed ? &sq : nullptr, ray_total, sms, st, counters);
    });
    if (e == cudaSuccess && check(b)) e = paths(b);  // after the shadow rays: it goes on from their sums
    if (e == cudaSuccess)
      e = timed(Stage::kShade, [&] {
        return est == Estimator::kCache ? launch_shade_cache(pb, wt, cw, b, sms, st)
               : nee                    ? launch_shade_nee(pb, wt, sq, b, sms, st)
                                        : launch_shade(pb, wt, b, sms, st);
      });
    if (e == cudaSuccess && nee && (!mixed || b == max_bounces)) e = shadows(b);
  }
  return e;
}

}  // namespace nb
