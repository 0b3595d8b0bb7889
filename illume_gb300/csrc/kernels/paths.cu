// Path kernel: whole paths in one launch, for work too small to fill the device one
// bounce at a time.
//
// The wavefront stages launch once per step and bounce, so a bounce costs at least its
// longest ray and the launches around it however few rays are left. Here a lane carries a
// path from ray to ray (trace, event, shading, shadow ray) without waiting for any other
// warp's path, and a lane whose path has ended takes the next one at its next step. Two
// uses:
//   a pass of few paths runs as one launch, camera rays included (bounce = -1);
//   a larger pass hands over the rest of its paths at a bounce that starts with at most
//   `limit` rays (bounce >= 1: the queue that bounce would trace).
// Every step is the one the wavefront stages run (stages.cuh, closest_hit with the default
// 4-wide kernel's settings), a path's random numbers depend on the path alone, and its
// contributions are added in bounce order, so the image does not depend on the choice.
//
// Bound: latency. A warp's step costs the longest search of its lanes, so when there are
// fewer paths than lanes they are spread over the warps (`width` lanes of each; `spread`),
// unless other tables' passes want the registers of the warps that this saves.
#include <algorithm>

#include "launch.h"
#include "stages.cuh"
#include "trace.cuh"

namespace illume {

template <bool NEE, int ISECT>
__global__ void __launch_bounds__(128, kPathBlocks) k_paths(WaveBuffers w, int bounce, int depth, int limit, int spread) {
  const unsigned FULL = 0xffffffffu;
  const bool start = bounce < 0;
  const int parity = start ? 0 : bounce & 1;
  const int n = start ? w.counters[kCounterPaths] : w.counters[parity];
  if (!start && (n > limit || n == 0)) return;   // the same for every block
  int* fetch = w.counters + 44 + parity;   // zero here: set by the pass plan or the last trace stage
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int width = spread ? min(32, (n + warps - 1) / warps) : 32;
  int stack[kStack];
  float4 qo = make_float4(0, 0, 0, 0), qd = qo, qt = qo;
  int b = 0, job = -1;
  unsigned job_rays = 0;               // rays of `job` not yet added to its total
  unsigned long long all_rays = 0;
  bool alive = false, dropped = false;
  // paths may be left (warp-uniform); warps beyond the paths take none
  bool more = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * width < n;
  for (;;) {
    if (more) {
      const bool want = !alive && lane < width;
      const unsigned idle = __ballot_sync(FULL, want);
      if (idle) {
        const int leader = __ffs(idle) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(fetch, __popc(idle));
        base = __shfl_sync(FULL, base, leader);
        more = base + __popc(idle) < n;
        const int i = base + __popc(idle & ((1u << lane) - 1));
        if (want && i < n) {
          if (start) {
            camera_path(w, i, qo, qd);
            qt = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
            w.contrib[__float_as_int(qo.w)] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            b = 0;
          } else {
            qo = w.q_orig[parity][i];
            qd = w.q_dir[parity][i];
            qt = w.q_thr[parity][i];
            b = bounce;
          }
          alive = true;
          const int j = __float_as_int(qd.w) >> kMediumBits;
          if (j != job) {
            if (job_rays) atomicAdd(&w.jobs[job].rays, (unsigned long long)job_rays);
            job = j;
            job_rays = 0;
          }
        }
      }
    }
    if (__ballot_sync(FULL, alive) == 0) break;   // nothing left to take either
    if (alive) {
      const JobDesc& J = w.jobs[job];
      const SceneView& sc = J.sc;
      const int medium = (__float_as_int(qd.w) & ((1 << kMediumBits) - 1)) - 1;
      float tmax = FLT_MAX;
      if (medium >= 0 && sc.mediums[medium].active)
        tmax = medium_bound(medium_distance(J, sc, __float_as_int(qo.w), medium, b));
      VisitCount vc;
      const HitRecord h = closest_hit<BVH_WIDE4, false, true, false, false, false, true, true, true>(
          sc, v3(qo.x, qo.y, qo.z), v3(qd.x, qd.y, qd.z), ISECT, stack, &vc, tmax);
      dropped |= vc.dropped;
      const int cls = h.geom == -1 && h.t != FLT_MAX ? EV_MEDIUM : surface_class(sc, h);
      ShadeOut out;
      out.cont = out.shadow = false;
      shade_event<NEE>(w, J, cls, qo, qd, qt, make_float4(h.t, h.u, h.v, __int_as_float(h.prim)), h.geom, b, out);
      ++job_rays;
      ++all_rays;
      if (NEE && out.shadow) {
        VisitCount sv;
        const HitRecord s = closest_hit<BVH_WIDE4, false, false, false, true, false, true, false, false>(
            sc, v3(out.so.x, out.so.y, out.so.z), v3(out.sd.x, out.sd.y, out.sd.z), ISECT, stack, &sv, out.sd.w);
        dropped |= sv.dropped;
        if (s.geom == -1) {
          float4* c = w.contrib + __float_as_int(out.sv.w);
          const float4 v = *c;
          *c = make_float4(v.x + out.sv.x, v.y + out.sv.y, v.z + out.sv.z, v.w);
        }
        ++job_rays;
        ++all_rays;
      }
      ++b;
      alive = out.cont && b < depth;
      qo = out.no;
      qd = out.nd;
      qt = out.nt;
    }
    __syncwarp();
  }
  if (dropped) atomicOr(w.counters + kCounterStackDrops, 1);
  const unsigned peers = __match_any_sync(FULL, job);
  const unsigned sum = __reduce_add_sync(peers, job_rays);
  if (job >= 0 && sum && lane == __ffs(peers) - 1) atomicAdd(&w.jobs[job].rays, (unsigned long long)sum);
  for (int off = 16; off > 0; off >>= 1) all_rays += __shfl_down_sync(FULL, all_rays, off);
  if (lane == 0 && all_rays) atomicAdd(w.rays, all_rays);
  if (!start) {
    // the last block empties the queue, so that the pass's later stages find nothing
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(w.counters + kCounterPathTicket, 1) == (int)gridDim.x - 1) {
        w.counters[kCounterPathTicket] = 0;
        w.counters[parity] = 0;
      }
    }
  }
}

const void* paths_kernel_ptr(int isect, bool nee) {
  if (isect == ISECT_MT) return nee ? (const void*)k_paths<true, ISECT_MT> : (const void*)k_paths<false, ISECT_MT>;
  return nee ? (const void*)k_paths<true, ISECT_WATERTIGHT> : (const void*)k_paths<false, ISECT_WATERTIGHT>;
}

void launch_paths(const WaveBuffers& w, const RenderKnobs& k, int bounce, int depth, int limit, int grid,
                  cudaStream_t st, bool nee) {
  int spread = k.overlap ? 0 : 1;
  void* args[] = {const_cast<WaveBuffers*>(&w), &bounce, &depth, &limit, &spread};
  cudaLaunchKernel(paths_kernel_ptr(k.isect, nee), dim3(grid), dim3(128), args, 0, st);
}

bool paths_kernel_for(const RenderKnobs& k) { return k.bvh_kind == BVH_WIDE4 && k.trace_variant == 0; }

}  // namespace illume
