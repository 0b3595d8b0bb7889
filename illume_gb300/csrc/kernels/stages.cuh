// The steps of a path, shared by the wavefront stages (one launch per step and bounce) and
// the path kernel (every step of a path in one launch): camera ray, medium distance and
// search bound, event class, shading of one event. The arithmetic of a step is the same in
// both, so a path does not depend on which of them runs it.
#pragma once

#include "launch.h"
#include "nee.cuh"
#include "shading.cuh"
#include "../common/philox.cuh"

namespace illume {

__device__ __forceinline__ int* ev_counts(const WaveBuffers& w, int parity) { return w.counters + 2 + 16 * parity; }

// Row of the job table that owns index x of a pass-wide numbering (paths or pixels):
// the last row whose first index is <= x. Rows with nothing in the pass share their
// first index with the next row, so the search passes over them.
__device__ __forceinline__ int find_row(const int* base, int n, int x) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(base + mid) <= x) lo = mid + 1;
    else hi = mid;
  }
  return lo - 1;
}

__device__ __forceinline__ float pack_job_medium(int job, int medium) {
  return __int_as_float((job << kMediumBits) | (medium + 1));
}

// init_rays, src/renderer.cu:81-110, for path slot g of job row j: pid = g - path_base
// = sample_in_pass * npix + pixel.
// Pixel of queue position q (0 <= q < w * h) when a sample's camera rays are queued in
// 8x4 tiles: the pixels of whole tiles first, tile after tile in row-major order (so a
// warp's 32 rays cover a compact patch of the image and traverse alike), then the pixels
// of the partial tiles at the right and bottom edges in row-major order.
__device__ __forceinline__ int tiled_pixel(int q, int w, int h) {
  const int tw = w >> 3, th = h >> 2;
  const int full = tw * th * 32;
  if (q < full) {
    const int t = q >> 5, k = q & 31;
    return ((t / tw) * 4 + (k >> 3)) * w + (t % tw) * 8 + (k & 7);
  }
  const int r = q - full, rw = w - tw * 8, right = th * 4 * rw;
  if (r < right) return (r / rw) * w + tw * 8 + r % rw;
  return th * 4 * w + (r - right);
}

// Camera ray of path i of the pass (0 <= i < the pass's paths), as a queue record (origin
// and path slot, direction and packed job / medium; the throughput is 1).
__device__ __forceinline__ void camera_path(const WaveBuffers& w, int i, float4& qo, float4& qd) {
  const int j = find_row(w.job_path_base, w.njobs, i);
  const JobDesc& J = w.jobs[j];
  const int npix = J.npix;
  const CameraView& cam = J.cam;
  // path i (in tile order) is this pixel's; its slot g keys the radiance
  // the pass's samples come in groups of k; a group's paths are queued pixel by pixel
  // (pixels in tile order) with the group's k samples of a pixel next to each other
  const int rel = i - J.path_base;
  const int ns = J.nsamples > 0 ? J.nsamples : 1;
  const int k = w.ray_group > 1 ? (w.ray_group < ns ? w.ray_group : ns) : 1;
  const int grp = rel / (k * npix);
  const int kk = (grp + 1) * k <= ns ? k : ns - grp * k;   // the last group may be smaller
  const int within = rel - grp * k * npix;
  const int s = grp * k + within % kk;
  const int pixel = tiled_pixel(within / kk, cam.width, cam.height);
  const int g = J.path_base + s * npix + pixel;
  const int sample = J.sample_base + s;
  RngStream rng;
  rng.init((uint32_t)pixel, (uint32_t)sample, 0u, J.seed, J.job);
  const int x = pixel % cam.width, y = pixel / cam.width;
  const float left_edge = cam.left + cam.pixel_size * (float)x;
  const float top_edge = cam.top - cam.pixel_size * (float)y;
  const float r_x = left_edge + cam.pixel_size * rng.next();
  const float r_y = top_edge - cam.pixel_size * rng.next();
  V3 pos = v3(0.0f, 0.0f, 0.0f);
  if (cam.aperture > FLT_EPSILON) {
    const float u1 = rng.next(), u2 = rng.next();
    pos = mul(sample_circle(u1, u2), cam.aperture);
  }
  const V3 origin = xform(cam.m, pos, 1.0f);
  const V3 image_pos = xform(cam.m, v3(r_x, r_y, cam.dof), 1.0f);
  const V3 dir = normalize(sub(image_pos, origin));
  qo = make_float4(origin.x, origin.y, origin.z, __int_as_float(g));
  qd = make_float4(dir.x, dir.y, dir.z, pack_job_medium(j, -1));
}

// Distance at which a ray in an active medium scatters: the first number of the path's
// bounce stream, as src/renderer.cu:152-157 draws it.
__device__ __forceinline__ float medium_distance(const JobDesc& J, const SceneView& sc, int g, int medium, int bounce) {
  const int pid = g - J.path_base;
  const uint32_t pixel = (uint32_t)(pid % J.npix), sample = (uint32_t)(J.sample_base + pid / J.npix);
  const Philox4 r = philox4x32_10(pixel, sample, (uint32_t)(bounce + 1), 0u, J.seed, J.job);
  return -logf(philox_unit(r.x)) / sc.mediums[medium].scattering;
}

__device__ __forceinline__ int surface_class(const SceneView& sc, const HitRecord& h) {
  if (h.geom == -1) return EV_MISS;
  const int mat = h.geom >= 0 ? sc.instances[h.geom].material : sc.spheres[-2 - h.geom].material;
  return EV_SURFACE + sc.materials[mat].type;
}

// Search bound of a ray in an active medium. The ray scatters at `dist` unless a surface
// lies at t <= dist, so the search need not look further: hits closer than the next float
// above dist are the ones with t <= dist. A bounded search that finds nothing leaves its
// bound in the hit record (never FLT_MAX), and the ray scatters; one that finds something
// has found the surface before it. Where dist is infinite or NaN the ray cannot scatter
// and the search has no bound (FLT_MAX).
// Subsurface walk (200k triangles, unit mean free path in a body 120 across): 15.1 -> 6.0
// node visits per ray, a 480x360 render at 16 samples 28.3 -> 13.8 ms.
__device__ __forceinline__ float medium_bound(float dist) {
  if (!(fabsf(dist) < FLT_MAX)) return dist < 0.0f ? dist : FLT_MAX;
  const int b = __float_as_int(dist);
  const int next = dist == 0.0f ? 1 : b + (dist > 0.0f ? 1 : -1);
  return fminf(__int_as_float(next), 3.4028233e38f);   // the float below FLT_MAX
}

// A path's radiance: the reference estimator ends a path at its one contribution, so
// the slot is written once; with next-event estimation contributions add up.
template <bool NEE>
__device__ __forceinline__ void add_radiance(float4* c, V3 L) {
  if (NEE) {
    const float4 v = *c;
    *c = make_float4(v.x + L.x, v.y + L.y, v.z + L.z, 0.0f);
  } else {
    *c = make_float4(L.x, L.y, L.z, 0.0f);
  }
}

struct BounceRng {
  RngStream s;
  __device__ __forceinline__ float operator()() { return s.next(); }
};

// Geometric normal of a triangle, as shading uses it (src/primitives/mesh.cu computes it at
// every hit).
__device__ __forceinline__ V3 face_normal(const float* positions, int i0, int i1, int i2) {
  const V3 v0 = v3(__ldg(positions + 3 * i0), __ldg(positions + 3 * i0 + 1), __ldg(positions + 3 * i0 + 2));
  const V3 v1 = v3(__ldg(positions + 3 * i1), __ldg(positions + 3 * i1 + 1), __ldg(positions + 3 * i1 + 2));
  const V3 v2 = v3(__ldg(positions + 3 * i2), __ldg(positions + 3 * i2 + 1), __ldg(positions + 3 * i2 + 2));
  return normalize(cross(sub(v1, v0), sub(v2, v0)));
}

// What one event leaves behind: the path's next ray, and a shadow ray of the next-event
// estimator (queue records).
struct ShadeOut {
  bool cont, shadow;
  float4 no, nd, nt;
  float4 so, sd, sv;
};

// One event of one path: its radiance goes to its slot, its next ray and shadow ray to
// `out`. qo, qd, qt: the ray's queue record; hv, geom: its hit record (not read for
// scatter events in a medium).
template <bool NEE>
__device__ __forceinline__ void shade_event(const WaveBuffers& w, const JobDesc& J, int cls, float4 qo, float4 qd,
                                            float4 qt, float4 hv, int geom, int bounce, ShadeOut& out) {
  const int g = __float_as_int(qo.w);
  const int packed = __float_as_int(qd.w);
  const int job = packed >> kMediumBits;
  int medium = (packed & ((1 << kMediumBits) - 1)) - 1;
  const SceneView sc = J.sc;
  const int pid = g - J.path_base;
  const int npix = J.npix;
  const V3 o = v3(qo.x, qo.y, qo.z), d = v3(qd.x, qd.y, qd.z);
  V3 thr = v3(qt.x, qt.y, qt.z);
  const float t = hv.x;
  BounceRng rng;
  rng.s.init((uint32_t)(pid % npix), (uint32_t)(J.sample_base + pid / npix), (uint32_t)(bounce + 1), J.seed,
             J.job);
  float4* contrib = w.contrib + g;
  const bool last = bounce + 1 >= J.max_depth;
  const bool nee = NEE && (J.flags & JOB_NEE) != 0;
  const float pdf_prev = qt.w;   // density of the BSDF sample that led here (next-event paths)
  if (medium >= 0 && sc.mediums[medium].active) {
    const DevMedium md = sc.mediums[medium];
    const float u = rng();
    const float dist = -logf(u) / md.scattering;
    if (cls == EV_MEDIUM) {
      const float u1 = rng(), u2 = rng();
      const V3 dir = to_basis(sample_hg(md.g, u1, u2, (J.flags & JOB_EXACT_HG) != 0), d);
      const V3 no3 = add(o, mul(d, dist));
      const V3 nd3 = normalize(dir);
      thr = mulv(thr, v3(expf(-1.0f * dist * md.absorption[0]), expf(-1.0f * dist * md.absorption[1]),
                         expf(-1.0f * dist * md.absorption[2])));
      if (!((double)length2(thr) < 1e-4) && !last) {
        out.cont = true;
        out.no = make_float4(no3.x, no3.y, no3.z, qo.w);
        out.nd = make_float4(nd3.x, nd3.y, nd3.z, qd.w);
        out.nt = make_float4(thr.x, thr.y, thr.z, 0.0f);
      }
      return;
    }
    thr = mulv(thr, v3(expf(-1.0f * t * md.absorption[0]), expf(-1.0f * t * md.absorption[1]),
                       expf(-1.0f * t * md.absorption[2])));
  }
  if (cls == EV_MISS) {
    V3 L = mulv(thr, env_eval(sc, d));
    if (nee && pdf_prev > 0.0f) L = mul(L, power_heuristic(pdf_prev, env_light_pdf(*sc.lights, d)));
    add_radiance<NEE>(contrib, L);
    return;
  }
  {
    // shading frame of the hit
    V3 N;
    float uv0, uv1;
    int matid;
    if (geom >= 0) {
      const DevInstance& in = sc.instances[geom];
      const DevMesh& m = sc.meshes[in.mesh];
      const int prim = __float_as_int(hv.w);
      const float bu = hv.y, bv = hv.z;
      // A face normal is one 16-byte gather; vertex indices are read only where something
      // needs them (12 scattered words and a normalisation otherwise: shading of the
      // traversal scene 1.526 -> 1.464 ms per 16-sample pass, 16 meshes 0.359 -> 0.343).
      const bool indexed = m.normals || m.texcoords || !m.face_normals;
      int i0 = 0, i1 = 0, i2 = 0;
      if (indexed) {
        i0 = __ldg(m.tris + 3 * prim);
        i1 = __ldg(m.tris + 3 * prim + 1);
        i2 = __ldg(m.tris + 3 * prim + 2);
      }
      V3 n;
      if (!m.normals) {
        if (m.face_normals) {
          const float4 f = __ldg(m.face_normals + prim);
          n = v3(f.x, f.y, f.z);
        } else {
          n = face_normal(m.positions, i0, i1, i2);
        }
      } else {
        const V3 n0 = v3(__ldg(m.normals + 3 * i0), __ldg(m.normals + 3 * i0 + 1), __ldg(m.normals + 3 * i0 + 2));
        const V3 n1 = v3(__ldg(m.normals + 3 * i1), __ldg(m.normals + 3 * i1 + 1), __ldg(m.normals + 3 * i1 + 2));
        const V3 n2 = v3(__ldg(m.normals + 3 * i2), __ldg(m.normals + 3 * i2 + 1), __ldg(m.normals + 3 * i2 + 2));
        n = normalize(add(mul(n0, 1.0f - bu - bv), add(mul(n1, bu), mul(n2, bv))));
      }
      N = normalize(xform(in.trans_inv, n, 0.0f));
      if (m.texcoords) {
        const float w0 = 1.0f - bu - bv;
        uv0 = (__ldg(m.texcoords + 2 * i0) * w0 + __ldg(m.texcoords + 2 * i1) * bu) + __ldg(m.texcoords + 2 * i2) * bv;
        uv1 = (__ldg(m.texcoords + 2 * i0 + 1) * w0 + __ldg(m.texcoords + 2 * i1 + 1) * bu) +
              __ldg(m.texcoords + 2 * i2 + 1) * bv;
      } else {
        uv0 = bu;
        uv1 = bv;
      }
      matid = in.material;
    } else {
      const DevSphere sp = sc.spheres[-2 - geom];
      const V3 pos = add(o, mul(d, t));
      N = normalize(sub(pos, v3(sp.cx, sp.cy, sp.cz)));
      uv0 = (float)((double)(atan2f(N.z, N.x) * 0.5f) * ILLUME_INV_PI_D + 0.5);
      uv1 = (float)(0.5 - (double)asinf(N.y) * ILLUME_INV_PI_D);
      matid = sp.material;
    }
    const DevMaterial mat = sc.materials[matid];
    const V3 albedo = tex_eval(sc, mat.albedo_tex, uv0, uv1);
    const float roughness = tex_eval(sc, mat.roughness_tex, uv0, uv1).x;
    if (mat.type == MAT_EMISSIVE) {
      V3 L = mulv(thr, albedo);
      if (nee && pdf_prev > 0.0f && geom >= 0) {
        const LightView& LV = *sc.lights;
        const int base = LV.num_tri > 0 ? __ldg(LV.inst_light_base + geom) : -1;
        if (base >= 0) {
          const int l = base + __float_as_int(hv.w);
          const float4 e1 = __ldg(&LV.tri[3 * l + 1]), e2 = __ldg(&LV.tri[3 * l + 2]);
          const V3 ln = cross(v3(e1.x, e1.y, e1.z), v3(e2.x, e2.y, e2.z));
          const float lnl = sqrtf(dot(ln, ln));
          const float cos_l = lnl > 0.0f ? dot(ln, d) / lnl : 0.0f;
          L = mul(L, power_heuristic(pdf_prev, tri_light_pdf(LV, l, t, cos_l)));
        }
      }
      add_radiance<NEE>(contrib, L);
      return;
    }
    if (last) return;   // the path has used all its closest-hit queries
    // next-event estimation: one light sample at a non-delta reflection vertex in air
    if (nee && (medium < 0 || !sc.mediums[medium].active) &&
        (mat.type == MAT_LAMBERT || mat.type == MAT_ROUGHCONDUCTOR || mat.type == MAT_ROUGHREFLECTIVE)) {
      RngStream nr;
      nr.init((uint32_t)(pid % npix), (uint32_t)(J.sample_base + pid / npix), 0x40000000u | (uint32_t)(bounce + 1),
              J.seed, J.job);
      const float u0 = nr.next(), u1 = nr.next(), u2 = nr.next();
      const V3 ph = add(o, mul(d, t));
      const LightSample ls = sample_light(sc, *sc.lights, ph, u0, u1, u2);
      V3 fcos;
      float pdf_b = 0.0f;
      if (ls.ok && bsdf_eval_cos(mat, d, N, albedo, roughness, ls.dir, fcos, pdf_b)) {
        const V3 Cn = mul(mulv(mulv(thr, fcos), ls.Le), power_heuristic(ls.pdf, pdf_b) / ls.pdf);
        if (isfinite(Cn.x + Cn.y + Cn.z) && (Cn.x > 0.0f || Cn.y > 0.0f || Cn.z > 0.0f)) {
          const V3 norm_o = mul(N, dot(N, d) > 0.0f ? -1.0f : 1.0f);
          const V3 org = add(ph, mul(norm_o, J.ray_bias));
          const float tmax = ls.dist == FLT_MAX ? FLT_MAX : ls.dist * (1.0f - 1e-4f) - J.ray_bias;
          if (tmax > 0.0f) {
            out.shadow = true;
            out.so = make_float4(org.x, org.y, org.z, __int_as_float(job));
            out.sd = make_float4(ls.dir.x, ls.dir.y, ls.dir.z, tmax);
            out.sv = make_float4(Cn.x, Cn.y, Cn.z, __int_as_float(g));
          }
        }
      }
    }
    const ScatterResult s = scatter(mat, d, N, albedo, roughness, rng);
    if (s.status == SCATTER_KILLED) return;
    if (s.medium != kMediumUnchanged) medium = s.medium;
    thr = mulv(thr, s.weight);
    const V3 p = add(add(o, mul(d, t)), mul(s.offset_dir, s.offset_sign * J.ray_bias));
    const V3 dir = normalize(s.dir);
    out.cont = true;
    out.no = make_float4(p.x, p.y, p.z, qo.w);
    out.nd = make_float4(dir.x, dir.y, dir.z, pack_job_medium(job, medium));
    out.nt = make_float4(thr.x, thr.y, thr.z, nee ? bsdf_sampled_pdf(mat, s, d, N) : 0.0f);
  }
}

}  // namespace illume
