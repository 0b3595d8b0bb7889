// A host-only stand-in for the CUDA runtime and the kernels, linked with the library's host
// sources (test_host_runtime.py). Every asynchronous operation (copy, clear, kernel, graph
// launch) waits in one queue and runs when the host waits for the device: a copy may read
// or write host memory at any time until then, which is all the runtime promises for
// memory that is not page-locked. Device memory is host memory with an optional limit.
//
// Usage: host_device_fake SCENARIO; prints what failed and returns 1, or returns 0.
#include <cuda_runtime.h>

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <functional>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "handles.h"
#include "../kernels/bvh_device.h"
#include "../kernels/launch.h"

using namespace illume;

// ---------------------------------------------------------------- the device
using Op = std::function<void()>;
static std::vector<Op> g_queue;                    // not yet run
static std::vector<Op>* g_capture = nullptr;       // operations of the graph being captured
static std::map<void*, size_t> g_memory;
static size_t g_used = 0, g_limit = 0;             // g_limit 0: none
static int g_fail_graph_launch = -1;               // countdown to a failing graph launch
static cudaError_t g_error = cudaSuccess;          // what cudaGetLastError reports
static int g_pass_kernels = 0;                     // kernels of passes that have run
static std::vector<std::pair<int, int>> g_samples; // sample ranges accumulated

static void push(Op f) { (g_capture ? *g_capture : g_queue).push_back(std::move(f)); }
static void drain() {
  std::vector<Op> q;
  q.swap(g_queue);
  for (Op& f : q) f();
}

struct FakeGraph { std::vector<Op> ops; };

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 4; return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_error;
  g_error = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake device error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_limit && g_used + n > g_limit) return g_error = cudaErrorMemoryAllocation;
  *p = aligned_alloc(256, (n + 255) & ~(size_t)255);
  g_memory[*p] = n;
  g_used += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  drain();
  if (p) { g_used -= g_memory.at(p); g_memory.erase(p); }
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *t = g_limit ? g_limit : (size_t)1 << 40;
  *f = *t - g_used;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  push([=] { memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { drain(); memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { push([=] { memset(d, v, n); }); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { drain(); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }   // one queue: in order
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { drain(); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { g_capture = new std::vector<Op>; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t) new FakeGraph{std::move(*g_capture)};
  delete g_capture;
  g_capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t) new FakeGraph(*(FakeGraph*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (FakeGraph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete (FakeGraph*)e; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  if (g_fail_graph_launch >= 0 && g_fail_graph_launch-- == 0) return g_error = cudaErrorUnknown;
  for (const Op& f : ((FakeGraph*)e)->ops) g_queue.push_back(f);
  return cudaSuccess;
}
// path regeneration's loop nodes: not used here
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                             cudaGraphNodeParams*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                          cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus*, unsigned long long*, cudaGraph_t*,
                                     const cudaGraphNode_t**, const cudaGraphEdgeData**, size_t*) { return cudaErrorNotSupported; }
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, unsigned) {
  return cudaErrorNotSupported;
}
}

// ---------------------------------------------------------------- the kernels
// A pass traces kRaysPerSample rays for every sample of its rows.
static constexpr int kRaysPerSample = 1000;
namespace illume {
int kernel_grid_blocks(const void*, int, int) { return 4; }
static int anchor;
const void* trace_kernel_ptr(int, int) { return &anchor; }
const void* l2_read_kernel_ptr() { return &anchor; }
const void* shade_kernel_ptr(int, bool) { return &anchor; }
const void* shadow_kernel_ptr(int) { return &anchor; }
const void* paths_kernel_ptr(int, bool) { return &anchor; }
bool paths_kernel_for(const RenderKnobs& k) { return k.bvh_kind == BVH_WIDE4 && k.trace_variant == 0; }
static void pass_kernel() { push([] { ++g_pass_kernels; }); }
void launch_plan(const WaveBuffers&, cudaStream_t) { pass_kernel(); }
void launch_raygen(const WaveBuffers&, int, cudaStream_t) { pass_kernel(); }
void launch_regen_start(const WaveBuffers&, cudaStream_t) {}
void launch_regen(const WaveBuffers&, int, cudaStream_t) {}
void launch_regen_plan(const WaveBuffers&, cudaGraphConditionalHandle, bool, int, float, cudaStream_t) {}
void launch_trace(const WaveBuffers&, const RenderKnobs&, int, int, cudaStream_t, bool) { pass_kernel(); }
void launch_shade(const WaveBuffers&, const RenderKnobs&, int, int, cudaStream_t, bool) { pass_kernel(); }
void launch_shadow(const WaveBuffers&, const RenderKnobs&, int, int, cudaStream_t) { pass_kernel(); }
void launch_paths(const WaveBuffers&, const RenderKnobs&, int, int, int, int, cudaStream_t, bool) { pass_kernel(); }
void launch_accumulate(const WaveBuffers& w, int, cudaStream_t) {
  pass_kernel();
  push([w] {
    for (int j = 0; j < w.njobs; ++j)
      if (w.jobs[j].nsamples > 0) {
        w.jobs[j].rays += (unsigned long long)kRaysPerSample * w.jobs[j].nsamples;
        g_samples.emplace_back(w.jobs[j].sample_base, w.jobs[j].sample_base + w.jobs[j].nsamples);
      }
  });
}
void launch_advance(const WaveBuffers& w, cudaStream_t) {
  pass_kernel();
  push([w] {
    for (int j = 0; j < w.njobs; ++j) {
      JobDesc& J = w.jobs[j];
      if (j == 0) memcpy(w.counters + kCounterRowRays, &J.rays, 8);
      if (J.nsamples > 0) advance_pass_state(J.sample_base, J.nsamples, J.sample_end, J.per_pass, J.flags);
    }
  });
}
void launch_tonemap(const Accumulators&, int, int npix, float, int, uint8_t* rgb8, float* mean, cudaStream_t) {
  push([=] {
    for (int i = 0; i < 3 * npix; ++i) { mean[i] = 0.5f; rgb8[i] = 7; }
  });
}
void launch_clear_accumulators(const Accumulators&, int, cudaStream_t) {}
cudaError_t launch_write_row(JobDesc* dst, const JobDesc& row, cudaStream_t) {
  push([=] { *dst = row; });
  return cudaSuccess;
}
cudaError_t launch_write_pass_state(JobDesc* dst, int4 s, cudaStream_t) {
  push([=] { dst->sample_base = s.x; dst->nsamples = s.y; dst->sample_end = s.z; dst->per_pass = s.w; });
  return cudaSuccess;
}
void launch_face_normals(const int*, const float*, int n, float4* out, cudaStream_t) {
  push([=] { memset(out, 0, sizeof(float4) * n); });
}
void launch_trace_hook(const SceneView&, const SceneView*, const float* rays, int n, int, int, void* hits, cudaStream_t) {
  push([=] {   // a hit's distance: the ray's first number
    for (int i = 0; i < n; ++i) ((illume_hit*)hits)[i].t = rays[8 * (size_t)i];
  });
}
void launch_bsdf_batch(int, int, const float*, int, float*, cudaStream_t) {}
void launch_l2_read(const void*, size_t, int, unsigned*, int, cudaStream_t) {}
int build_cluster_tree_device(Context*, const float*, int, ClusterTree*, std::string*) { return ILLUME_ERR_UNSUPPORTED; }
}  // namespace illume

// ---------------------------------------------------------------- scenarios
static int g_failed = 0;
#define EXPECT(cond) \
  do { if (!(cond)) { printf("%s:%d: %s (last error: %s)\n", __FILE__, __LINE__, #cond, illume_last_error()); ++g_failed; } } while (0)

struct World {
  illume_context* ctx = nullptr;
  illume_scene* scene = nullptr;
  int status;
  World(int tris = 2, int bitmap = 0) {
    illume_context_create(0, 0, &ctx);
    status = load(tris, bitmap);
  }
  // one instance of a strip of triangles without normals; its albedo is constant, or a bitmap
  int load(int ntris, int bitmap) {
    std::vector<float> P;
    std::vector<int32_t> T;
    for (int i = 0; i < ntris + 2; ++i) { P.push_back((float)(i / 2)); P.push_back((float)(i % 2)); P.push_back(0.0f); }
    for (int i = 0; i < ntris; ++i) { T.push_back(i); T.push_back(i + 1); T.push_back(i + 2); }
    const int32_t zero = 0, nv = ntris + 2, nt = ntris, leaf = 4, lambert = ILLUME_MAT_LAMBERT, air = -1;
    const float eye[12] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0}, one = 1.0f, grey[3] = {0.5f, 0.5f, 0.5f}, scale[2] = {1, 1};
    const int64_t off = 0;
    illume_scene_desc d;
    memset(&d, 0, sizeof(d));
    d.num_meshes = 1;
    d.mesh_vertex_offset = d.mesh_tri_offset = d.mesh_has_normals = d.mesh_has_texcoords = &zero;
    d.mesh_num_vertices = &nv;
    d.mesh_num_tris = &nt;
    d.mesh_bvh_leaf_size = &leaf;
    d.positions = P.data();
    d.tris = T.data();
    d.num_instances = 1;
    d.inst_mesh = d.inst_material = &zero;
    d.inst_mat = d.inst_inv = d.inst_trans_inv = eye;
    d.num_materials = 1;
    d.mat_type = &lambert;
    d.mat_albedo_tex = d.mat_roughness_tex = d.mat_distribution = &zero;
    d.mat_medium = &air;
    d.mat_ior = d.mat_diffuse_fresnel = &one;
    d.mat_eta = d.mat_k = grey;
    const int32_t type = bitmap ? ILLUME_TEX_BITMAP : ILLUME_TEX_CONSTANT, size = bitmap;
    const std::vector<float> texels(4 * (size_t)bitmap * bitmap, 0.5f);
    d.num_textures = 1;
    d.tex_type = &type;
    d.tex_width = d.tex_height = &size;
    d.tex_hdr = &zero;
    d.texels = texels.data();
    d.tex_color = d.tex_off = grey;
    d.tex_scale = scale;
    d.tex_texel_offset = &off;
    d.env_tex = -1;
    memcpy(d.camera_transform, eye, sizeof(eye));
    d.camera_fov = 40.0f;
    d.camera_dof = 1.0f;
    d.width = d.height = 16;
    return illume_scene_create(ctx, &d, &scene);
  }
  illume_renderer* renderer(int w, int h, int spp, int per_pass = 0, int engines = 0, int estimator = 0, int depth = 5) {
    illume_render_params p;
    illume_render_params_default(scene, spp, depth, &p);
    p.width = w; p.height = h;
    p.samples_per_pass = per_pass; p.engines = engines; p.estimator = estimator;
    illume_renderer* r = nullptr;
    illume_renderer_create(ctx, scene, &p, &r);
    return r;
  }
  ~World() {
    if (scene) illume_scene_destroy(scene);
    illume_context_destroy(ctx);
  }
};

// The passes of a call get the sample ranges the call set, however late the device takes
// them: on one engine and several, in renders that follow one another, and in a server
// whose jobs share a table and whose shares change between steps.
static void pass_state() {
  World x;
  for (int engines = 1; engines <= 3; ++engines) {
    illume_renderer* r = x.renderer(16, 16, 7, 2, engines);
    EXPECT(r);
    if (!r) return;
    for (int call = 0; call < 2; ++call) {
      g_samples.clear();
      illume_render_stats st;
      EXPECT(illume_render_device(r, 0, &st) == ILLUME_OK);
      std::vector<int> seen(7, 0);
      for (auto& s : g_samples)
        for (int k = s.first; k < s.second; ++k)
          if (k >= 0 && k < 7) ++seen[k];
          else EXPECT(!"sample outside the call");
      for (int k : seen) EXPECT(k == 1);
      EXPECT(st.rays == 7 * kRaysPerSample);
    }
    illume_renderer_destroy(r);
  }
  illume_server* s = nullptr;
  EXPECT(illume_server_create(x.ctx, 0, 4, &s) == ILLUME_OK);
  EXPECT(illume_server_set_option(s, ILLUME_SERVER_PATH_CAPACITY, 3 * 256) == ILLUME_OK);
  EXPECT(illume_server_set_option(s, ILLUME_SERVER_LANES, 1) == ILLUME_OK);
  const int spp[3] = {5, 2, 9};
  illume_job_id id[3];
  for (int j = 0; j < 3; ++j) {
    illume_render_params p;
    illume_render_params_default(x.scene, spp[j], 5, &p);
    p.width = p.height = 16;
    EXPECT(illume_job_submit(s, x.scene, &p, &id[j]) == ILLUME_OK);
  }
  for (int left = 1, k = 0; left && k < 100; ++k) EXPECT(illume_server_step(s, &left) == ILLUME_OK);
  for (int j = 0; j < 3; ++j) {
    illume_render_stats st;
    EXPECT(illume_job_poll(s, id[j], nullptr, nullptr, &st) == ILLUME_OK);
    EXPECT(st.rays == spp[j] * kRaysPerSample);
  }
  illume_server_destroy(s);
}

// The table of face normals is an extra: a scene loads wherever there is memory for the
// rest of it, and the table leaves most of what is left to the renders that follow.
static void face_normal_memory() {
  const int tris = 5000;
  const size_t table = sizeof(float4) * tris;
  size_t need;
  {
    World x(tris, 128);
    EXPECT(x.status == ILLUME_OK && x.scene->s.t_meshes[0].face_normals);
    need = g_used - table;
  }
  for (size_t spare : {(size_t)0, table, 15 * table, 16 * table}) {
    g_limit = need + spare;
    World x(tris, 128);
    EXPECT(x.status == ILLUME_OK);
    if (x.status != ILLUME_OK) continue;
    DevMesh m;   // as the device has it
    memcpy(&m, x.scene->s.view.meshes, sizeof(m));
    EXPECT((m.face_normals != nullptr) == (spare == 16 * table));
    EXPECT(m.face_normals == x.scene->s.t_meshes[0].face_normals);
    EXPECT(g_used == need + (m.face_normals ? table : 0));
    size_t bytes = 0;
    EXPECT(illume_scene_upload(x.scene, &bytes) == ILLUME_OK);
    drain();
    EXPECT(memcmp(&m, x.scene->s.view.meshes, sizeof(m)) == 0);
  }
  g_limit = need - 1;
  World x(tris, 128);
  EXPECT(x.status == ILLUME_ERR_OOM && g_queue.empty());
  g_limit = 0;
}

// A render whose outputs cannot be allocated, or whose passes cannot all be launched, returns
// with nothing of it left to run: the next call's staging memory and ray counts are its own.
static void failed_render() {
  World x;
  for (int midway = 0; midway < 2; ++midway) {
    illume_renderer* r = midway ? x.renderer(16, 16, 4, 1, 2) : x.renderer(16, 16, 4);
    EXPECT(r);
    if (!r) return;
    std::vector<float> mean(3 * 256);
    illume_render_stats st;
    if (midway) g_fail_graph_launch = 2;              // the second pass's first graph
    else x.ctx->c.budget = x.ctx->c.used.load() + 64; // no room for the output images
    EXPECT(illume_render(r, mean.data(), nullptr, nullptr, nullptr, &st) == (midway ? ILLUME_ERR_CUDA : ILLUME_ERR_BUDGET));
    x.ctx->c.budget = 0;
    g_fail_graph_launch = -1;
    EXPECT(g_queue.empty());
    float rays[8] = {11, 0, 0, 0, 0, 0, 1, 0};
    illume_hit hit;
    memset(&hit, 0, sizeof(hit));
    EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE4, &hit) == ILLUME_OK);
    EXPECT(hit.t == 11.0f);
    EXPECT(illume_render(r, mean.data(), nullptr, nullptr, nullptr, &st) == ILLUME_OK);
    EXPECT(st.rays == 4 * kRaysPerSample);
    EXPECT(mean[0] == 0.5f && mean[767] == 0.5f);
    illume_renderer_destroy(r);
  }
}

// The device memory that small queries keep between calls is given back when an allocation
// of the context needs it, and not while a query is using it.
static void query_memory() {
  World x;
  float rays[8] = {3, 0, 0, 0, 0, 0, 1, 0};
  illume_hit hit;
  EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE4, &hit) == ILLUME_OK);
  EXPECT(x.ctx->c.query_ws && hit.t == 3.0f);
  g_limit = g_used + 4096;
  {
    DevBuffer b;
    EXPECT(b.alloc(&x.ctx->c, 500000) == ILLUME_OK);
    EXPECT(!x.ctx->c.query_ws && cudaGetLastError() == cudaSuccess);
    // with none to give back the allocation is refused, and its error does not linger
    DevBuffer more;
    EXPECT(more.alloc(&x.ctx->c, 800000) == ILLUME_ERR_OOM && cudaGetLastError() == cudaSuccess);
    // a query without memory to keep takes what it needs
    hit.t = 0;
    EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE4, &hit) == ILLUME_OK);
    EXPECT(hit.t == 3.0f && !x.ctx->c.query_ws);
  }
  EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE4, &hit) == ILLUME_OK);
  EXPECT(x.ctx->c.query_ws);
  // the first 8-wide query allocates its layout while it holds the kept memory
  g_limit = g_used;
  EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE8, &hit) == ILLUME_ERR_OOM);
  EXPECT(x.ctx->c.query_ws && g_memory.count(x.ctx->c.query_ws) && g_queue.empty());
  g_limit = 0;
}

// An 8-wide query that finds no memory for the layout uploads it when it is asked again.
static void wide_layout_memory() {
  World x(200);
  float rays[8] = {3, 0, 0, 0, 0, 0, 1, 0};
  illume_hit hit;
  const size_t before = g_used, listed = x.scene->s.device_bytes;
  for (size_t room : {(size_t)0, (size_t)64, (size_t)4096}) {
    g_limit = before + 64 + room;   // (the rays and the hit take 64 bytes)
    EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE8, &hit) == ILLUME_ERR_OOM);
    EXPECT(g_used == before && x.scene->s.device_bytes == listed);
  }
  g_limit = 0;
  EXPECT(illume_trace_closest(x.ctx, x.scene, rays, 1, ILLUME_ISECT_MT, ILLUME_BVH_WIDE8, &hit) == ILLUME_OK);
  DevMesh m;
  memcpy(&m, x.scene->s.view.meshes, sizeof(m));
  const MeshBvh& b = x.scene->s.bvhs[0];
  EXPECT(b.wide.size() > 0 && g_memory[(void*)m.wide] == b.wide.size() * sizeof(WideNode));
  EXPECT(g_memory[(void*)m.wide_tris] == b.wide_tris.size() * sizeof(float4));
  if (!g_failed) EXPECT(memcmp(m.wide, b.wide.data(), b.wide.size() * sizeof(WideNode)) == 0);
}

// The launches a call reports are the ones its passes made.
static void launch_counts() {
  World x;
  x.scene->s.room = true;   // (a strip of triangles otherwise, whose passes run whole)
  illume_render_stats st;
  for (int depth : {0, 1, 3, 9})
    for (int estimator = 0; estimator < 2; ++estimator)
      // passes of the path kernel alone, of bounces with hand-over, of two halves, of engines
      for (int k = 0; k < 4; ++k) {
        illume_renderer* r = k == 0 ? x.renderer(64, 48, 5, 2, 0, estimator, depth)
                             : k == 1 ? x.renderer(600, 500, 3, 1, 1, estimator, depth)
                             : k == 2 ? x.renderer(1024, 1024, 2, 1, 0, estimator, depth)
                                      : x.renderer(600, 500, 5, 2, 2, estimator, depth);
        EXPECT(r);
        if (!r) return;
        const long long before = x.ctx->c.launches.load();
        g_pass_kernels = 0;
        EXPECT(illume_render_device(r, 0, &st) == ILLUME_OK);
        EXPECT(st.kernel_launches == g_pass_kernels && x.ctx->c.launches.load() - before == g_pass_kernels);
        illume_profile prof;
        const long long at = x.ctx->c.launches.load();
        g_pass_kernels = 0;
        EXPECT(illume_renderer_profile(r, 0, &prof) == ILLUME_OK);
        EXPECT(x.ctx->c.launches.load() - at == g_pass_kernels);
        illume_renderer_destroy(r);
      }
}

// The largest sample count renders all its samples.
static void largest_sample_count() {
  World x;
  const int spp = 0x7fffffff;
  illume_renderer* r = x.renderer(16, 16, spp, 4000000, 1);
  EXPECT(r);
  if (!r) return;
  g_samples.clear();
  EXPECT(illume_render_device(r, 0, nullptr) == ILLUME_OK);
  long long n = 0;
  for (auto& s : g_samples) {
    EXPECT(s.first == n);
    n = s.second;
  }
  EXPECT(n == spp);
  illume_renderer_destroy(r);
}

int main(int argc, char** argv) {
  const std::string s = argc > 1 ? argv[1] : "";
  if (s == "pass_state") pass_state();
  else if (s == "face_normal_memory") face_normal_memory();
  else if (s == "query_memory") query_memory();
  else if (s == "wide_layout_memory") wide_layout_memory();
  else if (s == "launch_counts") launch_counts();
  else if (s == "largest_sample_count") largest_sample_count();
  else if (s == "failed_render") failed_render();
  else { printf("unknown scenario\n"); return 2; }
  if (g_failed) printf("%d expectations failed\n", g_failed);
  return g_failed ? 1 : 0;
}
