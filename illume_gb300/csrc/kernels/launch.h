// Host-side launchers of the sm_103a kernels (defined in the .cu files of this folder).
//
// Every wavefront pass runs over a table of jobs. A job is one render (scene, camera,
// Philox key, depth, accumulators, sample range); a plain render is a table of one job.
// The device advances each job's sample range after every pass, so a captured pass can
// be replayed any number of times without the host.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../common/types.h"

namespace illume {

struct Accumulators {
  float* sum32;          // FP32 / Kahan sum (3 per pixel)
  float* comp32;         // Kahan compensation (3 per pixel)
  double* sum64;         // FP64 sum (3 per pixel)
  double* sumsq;         // sum of squares of per-sample radiance (3 per pixel), nullable
};

// One row of the job table (256 bytes).
struct JobDesc {
  SceneView sc;
  CameraView cam;
  Accumulators acc;
  uint32_t seed, job;        // Philox key
  int max_depth;             // closest-hit queries per path
  float ray_bias;
  int flags, accum_mode;      // flags: JOB_EXACT_HG, JOB_NEE, interleave (job_interleave)
  int npix, width;
  // pass state: samples [sample_base, sample_base + nsamples) of every pixel are in the
  // current pass; advanced by k_advance after every pass; nsamples == 0 = idle row
  int sample_base, nsamples, sample_end, per_pass;
  int path_base;             // first path slot of this job in the current pass (k_plan)
  int pixel_base;            // first index of this job's pixels in the accumulation sweep (k_plan)
  unsigned long long rays;   // closest-hit queries traced for this job (running total)
};
static_assert(sizeof(JobDesc) == 256, "JobDesc layout");
enum JobFlags : int { JOB_EXACT_HG = 1, JOB_NEE = 2 };
// Bits 8..15 of the flags: how many job tables take turns on this job's sample ranges
// (0 or 1: this table alone). With n tables, a pass of one table is followed by one pass
// of each other table before its next range, so the row skips the others' samples.
static constexpr int kInterleaveShift = 8;
__host__ __device__ __forceinline__ int job_interleave(int flags) {
  const int n = (flags >> kInterleaveShift) & 0xff;
  return n > 1 ? n : 1;
}
// Pass state after a pass of `nsamples` (the same arithmetic on the host mirror and in
// k_advance).
__host__ __device__ __forceinline__ void advance_pass_state(int& sample_base, int& nsamples, int sample_end,
                                                            int per_pass, int flags) {
  sample_base += nsamples + (job_interleave(flags) - 1) * per_pass;
  const int left = sample_end - sample_base;
  nsamples = left < per_pass ? (left > 0 ? left : 0) : per_pass;
}

// A queued ray's fourth direction word packs its job row and medium:
// (job << kMediumBits) | (medium + 1), medium -1 = air.
static constexpr int kMediumBits = 12;
static constexpr int kMaxMediums = (1 << kMediumBits) - 2;
static constexpr int kMaxJobRows = 1 << 18;

// Wavefront buffers. Queues are double-buffered by bounce parity; a path's slot in the
// current pass indexes its radiance in `contrib`.
struct WaveBuffers {
  float4* q_orig[2];     // origin xyz, path slot (int bits)
  float4* q_dir[2];      // direction xyz, packed job / medium (int bits)
  float4* q_thr[2];      // throughput xyz
  float4* hit;           // t, u, v, prim (int bits), per slot of the current queue
  int* hit_geom;         // instance >= 0, sphere -2 - s, miss -1
  int* evq;              // EV_COUNT queues of `cap` slot indices each
  int* counters;         // see kCounter* below
  float4* contrib;       // per path radiance of the current pass
  float4* s_orig;        // shadow rays of the next-event estimator: origin, job row (int bits)
  float4* s_dir;         //   direction, maximum distance
  float4* s_val;         //   contribution if unoccluded, path slot (int bits)
  unsigned long long* rays;   // closest-hit queries traced (running total)
  unsigned long long* visits; // [node fetches, triangle tests, warp node-fetch slots] of the instrumented trace kernel
  JobDesc* jobs;
  int* job_path_base;    // njobs + 1 prefix sums of the pass's paths (k_plan)
  int* job_pixel_base;   // njobs + 1 prefix sums of the pass's pixels (k_plan)
  // Path regeneration: the bounce of each queued ray, by queue parity. Null: every ray of
  // a queue is at the pass's bounce (the queues hold all the pass's paths at once).
  int* q_bounce[2];
  int njobs;
  int ray_group;         // camera rays in the queue: up to ray_group samples of a pixel together (<= 1: one sample, pixels in tiles)

  int cap;               // path slots of one pass (per-path radiance)
  int qcap;              // queue slots (rays in flight); equal to cap without regeneration
  int part;              // 0: the whole pass; 1, 2: its first and second half of paths (Engine::halves)
};

// counters[]: [0..1] queue sizes by parity, [2 + 16 * parity + class] event counts,
// [kCounterPaths] paths of the pass, [kCounterPixels] pixels of the pass, [42] slot
// overflow flag, [44 + parity] trace ray-fetch counters, [46 + parity] shadow-ray counts,
// [48 + parity] shadow-ray fetch counters, [kCounterStackDrops] set when a traversal
// found its stack full (kept across passes; cleared when the engine is made and read by
// the renderer after each render).
static constexpr int kCounterPaths = 40;
static constexpr int kCounterStackDrops = 50;
// Path regeneration (a pass whose paths outnumber the queue slots): paths started so
// far, the loop's iteration, the next batch of new paths (count, first path, first queue
// position), whether the loop goes on, a flag set when its iteration bound ended a pass
// (kept across passes, like the stack-overflow flag) and the loop's iterations since the
// engine was made.
static constexpr int kCounterGen = 51;
static constexpr int kCounterIter = 52;
static constexpr int kCounterRegenN = 53;
static constexpr int kCounterRegenFirst = 54;
static constexpr int kCounterRegenQ = 55;
static constexpr int kCounterMore = 56;
static constexpr int kCounterLoopLimit = 57;
static constexpr int kCounterIterTotal = 58;
static constexpr int kCounterPixels = 41;
static constexpr int kCounterPathTicket = 59;   // blocks of the path kernel that are done (0 between launches)
// Ray total of the table's first row after the last pass (two words, written by
// k_advance): the words from kCounterStackDrops to here are what a renderer reads back.
static constexpr int kCounterRowRays = 60;
static constexpr int kCounterWords = 64;        // a second half's counters follow the first's

// Iteration of a stage launched with `bounce` (-1 under path regeneration: read from the
// counters), and the bounce of queued ray i.
__device__ __forceinline__ int pass_iteration(const WaveBuffers& w, int bounce) {
  return bounce >= 0 ? bounce : w.counters[kCounterIter];
}
__device__ __forceinline__ int ray_bounce(const WaveBuffers& w, int parity, int i, int it) {
  return w.q_bounce[parity] ? w.q_bounce[parity][i] : it;
}

// Samples of a pixel kept together in a pass's camera-ray queue by default (traversal
// workload, Mrays/s: 1 -> 4168, 4 -> 4249, 8 -> 4311, 16 -> 4349, 32 -> 4266).
static constexpr int kDefaultRayGroup = 16;

// The path kernel (paths.cu): blocks of 128 per SM (at most 128 registers, no spills; 5 and
// 6 blocks spill: a 64x48 render 7-19% slower, a 1280x720 sample 5%), the largest pass that
// runs as one launch of it, and the rays at which a larger pass hands the rest of its paths
// over.
// Pass of 12 bounces, ms, wavefront with hand-over / one path-kernel launch, by paths:
//              2^14        2^16        2^17        2^18        2^19        2^20
//   Cornell    .21 / .12   .22 / .14   .27 / .19   .33 / .32   .48 / .56   .80 / 1.06
//   mixed      .47 / .34   .54 / .45   .63 / .48   .74 / .57   .86 / .70  1.13 / 1.08
//   medium     .38 / .25   .47 / .35   .60 / .52   .93 / .97  1.41 / 1.84 2.14 / 3.58
//   NEE        .48 / .28   .64 / .45   .75 / .61   .96 / 1.01 1.20 / 1.76 1.63 / 3.24
// The wavefront runs lanes of one event class together, which pays once a bounce fills the
// device more than once (155,648 lanes at 64 registers on 152 SMs). One limit for every
// scene: at 2^18 paths a medium and light sampling give away 4 to 5% of a pass, and beyond
// it mixed scenes 4 to 23%; which scene is which is not known before its paths have run.
// Hand-over at 2^16 / 2^17 / 2^18 / 2^19 rays: textured scene 2.54 / 2.19 / 2.21 / 2.37 ms,
// light sampling 7.02 / 7.17 / 7.18 / 7.59, 16 large meshes 5.65 / 5.63 / 5.62 / 5.89.
// Where passes of other tables run beside it the path kernel holds registers they could
// use: there a larger pass hands over at 3 * 2^15 rays, 32 to a warp (light sampling 6.90
// -> 6.68 ms, a textured render of 6M paths 5.00 -> 4.83, instances 3.36 -> 3.23, served
// mixes 0.66 -> 0.61 and 1.50 -> 1.42; at 2^16 16 large meshes lose 5%).
static constexpr int kPathBlocks = 4;
static constexpr int kSplitPass = 1 << 20;   // paths from which a pass may run as two halves (Renderer::init)
static constexpr int kPathPass = 1 << 18;
static constexpr int kPathTail = 1 << 17;
static constexpr int kPathTailOverlap = 3 << 15;

// Settings shared by every job of a table (they select kernel instances).
struct RenderKnobs {
  int isect;           // illume_intersector
  int bvh_kind;        // BvhKind
  int trace_variant;   // see trace_kernel_ptr
  int shade_variant;   // see shade_kernel_ptr
  // 1: passes of other tables may run beside this table's (launch_trace, launch_paths): set for
  // a renderer of several engines and a server of several lanes, whether or not the others
  // have work. A lone request on a server of four lanes (64x48 to 1024x768, six scenes,
  // both tests) takes these settings too: 1.02 to 3.6 times as fast as before they and the
  // path kernel were there.
  int overlap;
};

int kernel_grid_blocks(const void* fn, int block, int device);

// A job row, or its pass state (sample_base, nsamples, sample_end, per_pass), written from
// the launch's arguments.
cudaError_t launch_write_row(JobDesc* dst, const JobDesc& row, cudaStream_t st);
cudaError_t launch_write_pass_state(JobDesc* dst, int4 state, cudaStream_t st);

void launch_plan(const WaveBuffers& w, cudaStream_t st);
void launch_raygen(const WaveBuffers& w, int grid, cudaStream_t st);
// Path regeneration. A pass runs as a loop of iterations (trace, shade, [shadow], plan of
// the next new paths, their camera rays) over queues of qcap rays, new paths entering
// the queue as earlier ones end, until every path of the pass has ended. The stages take
// bounce = -1 and read the iteration from the counters. regen_start: the first
// min(qcap, paths) paths; regen_plan: after an iteration's shading, starts new paths when
// the next queue holds at most threshold x qcap rays (filling it to qcap), and sets the
// loop's condition (through `cond` when launched inside a graph's while node, else only
// counters[kCounterMore]); the loop ends early, raising counters[kCounterLoopLimit], at
// an iteration bound derived from the paths, qcap, threshold and `depth`.
void launch_regen_start(const WaveBuffers& w, cudaStream_t st);
void launch_regen(const WaveBuffers& w, int grid, cudaStream_t st);
void launch_regen_plan(const WaveBuffers& w, cudaGraphConditionalHandle cond, bool use_cond, int depth, float threshold,
                       cudaStream_t st);
void launch_trace(const WaveBuffers& w, const RenderKnobs& k, int bounce, int grid, cudaStream_t st,
                  bool count_visits = false);
void launch_shade(const WaveBuffers& w, const RenderKnobs& k, int bounce, int grid, cudaStream_t st, bool nee = false);
void launch_shadow(const WaveBuffers& w, const RenderKnobs& k, int bounce, int grid, cudaStream_t st);
// Path kernel (paths.cu): bounce < 0 starts every path of the pass and runs it to its end;
// bounce >= 1 takes over the rays queued for that bounce when there are at most `limit`
// (and leaves the queue empty). For the settings paths_kernel_for accepts.
bool paths_kernel_for(const RenderKnobs& k);
void launch_paths(const WaveBuffers& w, const RenderKnobs& k, int bounce, int depth, int limit, int grid,
                  cudaStream_t st, bool nee = false);
void launch_accumulate(const WaveBuffers& w, int grid, cudaStream_t st);
void launch_advance(const WaveBuffers& w, cudaStream_t st);
void launch_tonemap(const Accumulators& acc, int accum_mode, int npix, float samples, int op, uint8_t* rgb8,
                    float* mean, cudaStream_t st);
void launch_clear_accumulators(const Accumulators& acc, int npix, cudaStream_t st);

void launch_face_normals(const int* tris, const float* positions, int n, float4* out, cudaStream_t st);

// test hooks
// d_view: a device copy of sc (read by the persistent 8-wide kernel, bvh_kind 2)
void launch_trace_hook(const SceneView& sc, const SceneView* d_view, const float* rays8, int n, int isect,
                       int bvh_kind, void* hits, cudaStream_t st);
void launch_bsdf_batch(int type, int distribution, const float* in, int n, float* out, cudaStream_t st);

const void* trace_kernel_ptr(int bvh_kind, int variant = 0);
// L2 read-bandwidth probe (measurement only).
void launch_l2_read(const void* buf, size_t bytes, int reps, unsigned* sink, int grid, cudaStream_t st);
const void* l2_read_kernel_ptr();
const void* shade_kernel_ptr(int variant = 0, bool nee = false);
const void* shadow_kernel_ptr(int bvh_kind);
const void* paths_kernel_ptr(int isect, bool nee);

}  // namespace illume
