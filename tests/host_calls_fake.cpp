// Host calls of libtpt_cuda.so against a CUDA runtime made of this file: the
// library's C++ objects are linked with the functions below instead of the
// runtime and the kernels.  Memory is host memory, copies happen at once, and each
// stream counts its operations, so that a program can tell which of them a call
// has waited for when it returns, and what memory a launch or copy touches.
//
//   host_calls_fake share <outer> <inner>   one call begun while another is in
//       flight on the same context, as by a second thread
//   host_calls_fake fail <call> <k>         the k-th launch of a call fails
//   host_calls_fake wait <call> 1           a call alone
//   host_calls_fake trim <call> <mib>       what a call keeps is at most <mib> MiB and
//       goes back with tpt_context_trim
//   host_calls_fake records <t> <bytes>     <bytes> a triangle are what a scene of <t>
//       triangles with a material holds over one without
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "../include/tpt.h"
#include "../toy-path-tracing_b200/csrc/api/internal.h"

namespace {
using Clock = std::map<void*, long>;  // operations of each stream that something comes after
std::map<void*, Clock> streams;       // [s][s]: operations issued on s
std::map<void*, Clock> events;
Clock done;
std::map<char*, size_t> blocks;  // live memory
std::set<char*> in_use;          // blocks that a call in flight works on
bool pinned = false;
std::string failure;
std::function<void()> at_launch;  // what runs inside the call's first launch of `at_kind`
std::string at_kind;
int launches = 0, fail_launch = 0;

void join(Clock& a, const Clock& b) {
  for (auto& [s, n] : b) a[s] = std::max(a[s], n);
}
void issue(void* s) { ++streams[s][s]; }
bool idle() {
  for (auto& [s, c] : streams)
    if (c[s] > done[s]) return false;
  return true;
}
char* block_of(const void* p) {
  auto it = blocks.upper_bound((char*)p);
  if (it == blocks.begin()) return nullptr;
  --it;
  return (char*)p < it->first + it->second ? it->first : nullptr;
}
size_t live_bytes() {
  size_t n = 0;
  for (auto& [p, bytes] : blocks) n += bytes;
  return n;
}
void touch(const void* p) {
  if (char* b = block_of(p); b && in_use.count(b)) failure = "memory of a call in flight is written by another";
}
cudaError_t get(void** p, size_t n) {
  *p = calloc(n + 1, 1);
  blocks[(char*)*p] = n + 1;
  return cudaSuccess;
}
cudaError_t drop(void* p) {
  if (!p) return cudaSuccess;
  if (in_use.count((char*)p)) failure = "memory of a call in flight is freed";
  blocks.erase((char*)p);
  free(p);
  return cudaSuccess;
}
cudaError_t launch(const char* kind, cudaStream_t s, std::initializer_list<const void*> writes) {
  issue(s);
  for (const void* p : writes) touch(p);
  if (++launches == fail_launch) return cudaErrorLaunchFailure;
  if (at_launch && in_use.empty() && at_kind == kind) {
    for (const void* p : writes)
      if (char* b = block_of(p)) in_use.insert(b);
    auto f = at_launch;
    f();
    in_use.clear();
    at_launch = nullptr;
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
const char* cudaGetErrorName(cudaError_t) { return "error"; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return get(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return get(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return get(p, n); }
cudaError_t cudaFree(void* p) { return drop(p); }
cudaError_t cudaFreeHost(void* p) { return drop(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return drop(p); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { join(done, streams[s]); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { touch(p); std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { issue(s); return cudaMemset(p, v, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  issue(st);
  touch(d);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
// a copy from pageable memory returns when it has read the memory: its last bytes
// may reach the device later, in the order of the legacy stream
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  cudaMemcpyAsync(d, s, n, k, cudaStreamLegacy);
  return k == cudaMemcpyHostToDevice ? cudaSuccess : cudaStreamSynchronize(cudaStreamLegacy);
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k,
                              cudaStream_t st) {
  for (size_t r = 0; r < h; ++r) cudaMemcpyAsync((char*)d + r * dp, (const char*)s + r * sp, w, k, st);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  a->type = pinned ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  for (auto& [s, c] : streams) join(done, c);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { events[e] = streams[s]; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { join(done, events[e]); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { join(streams[s], events[e]); return cudaSuccess; }
}

namespace tpt {
cudaError_t launch_traverse_strided(const DevGeometry&, const float* rays, uint64_t, uint64_t, int, int32_t* prim,
                                    float* t, int32_t*, float*, uint64_t, unsigned long long*, uint32_t*, int,
                                    cudaStream_t s, uint32_t*, uint32_t*, const uint32_t*, const DevJob*,
                                    const uint32_t*, unsigned long long*, uint32_t*, const uint32_t*) {
  return launch("traverse", s, {rays, prim, t});
}
cudaError_t launch_wf_generate(const DevGeometry&, const DevRenderData&, const RenderLaunch&, const WfBuffers&,
                               uint64_t, uint32_t, cudaStream_t s, const float*) {
  issue(s);
  return cudaSuccess;
}
cudaError_t launch_wf_generate_batch(const DevJob*, uint32_t, const WfBuffers&, uint64_t, uint32_t, cudaStream_t s) {
  issue(s);
  return cudaSuccess;
}
cudaError_t launch_wf_shade(const DevGeometry&, const DevRenderData&, const RenderLaunch&, const WfBuffers&, int,
                            cudaStream_t s, const DevAdjoint*, int) {
  issue(s);
  return cudaSuccess;
}
cudaError_t launch_wf_shade_batch(const DevJob*, const WfBuffers&, int, cudaStream_t s, int, bool) {
  issue(s);
  return cudaSuccess;
}
cudaError_t launch_wf_resolve(const WfBuffers&, cudaStream_t s, const DevAdjoint*) {
  issue(s);
  return cudaSuccess;
}
cudaError_t launch_wf_accumulate(const WfBuffers&, uint32_t, uint32_t, uint32_t, uint32_t, float, float* image,
                                 cudaStream_t s) {
  return launch("image", s, {image});
}
cudaError_t launch_bake_shade_tris(const MeshSpan* m, uint32_t, const float* pos, const float*, const float*,
                                   const uint32_t* idx, uint64_t, DevShadeTri* out, cudaStream_t s) {
  return launch("upload", s, {m, pos, idx, out});
}
}  // namespace tpt

namespace {
tpt_context* ctx;
tpt_scene* scene;

tpt_status upload(uint32_t triangles, tpt_scene** out, uint32_t materials = 1) {
  std::vector<float> p(9 * (size_t)triangles);
  std::vector<uint32_t> idx(3 * (size_t)triangles);
  for (uint32_t t = 0; t < triangles; ++t) {
    const float x = (float)t, tri[9] = {x, 0, 0, x + 1, 0, 0, x, 1, 0};
    std::memcpy(&p[9 * t], tri, sizeof tri);
    for (uint32_t k = 0; k < 3; ++k) idx[3 * t + k] = 3 * t + k;
  }
  tpt_mesh_desc m{};
  m.positions = p.data();
  m.num_vertices = 3 * (uint64_t)triangles;
  m.indices = idx.data();
  m.num_indices = idx.size();
  tpt_instance_desc inst{};
  for (int k = 0; k < 4; ++k) inst.local_to_world[5 * k] = inst.world_to_local[5 * k] = 1.0f;
  for (int k = 0; k < 3; ++k) inst.normal_to_world[4 * k] = 1.0f;
  tpt_material_desc mat{};
  mat.kind = TPT_MATERIAL_NORMALIZED_LAMBERT;
  tpt_scene_desc d{};
  d.meshes = &m;
  d.num_meshes = 1;
  d.instances = &inst;
  d.num_instances = 1;
  d.materials = &mat;
  d.num_materials = materials;
  return tpt_scene_upload(ctx, &d, out);
}

tpt_status call(const std::string& what) {
  if (what.rfind("traverse", 0) == 0) {
    const uint64_t n = 300001;
    std::vector<float> rays(7 * n), t(n);
    std::vector<int32_t> prim(n);
    pinned = what == "traverse_pinned";
    return tpt_traverse(ctx, scene, rays.data(), n, TPT_CLOSEST_HIT, prim.data(), t.data(), nullptr, nullptr);
  }
  if (what.rfind("upload", 0) == 0) {
    tpt_scene* s = nullptr;
    const tpt_status st = upload(what == "upload_large" ? 1u << 18 : 100, &s);
    tpt_scene_release(s);
    return st;
  }
  const int side = what == "render_large" ? 2000 : what == "render_own_memory" ? 3400 : 64, jobs = what == "render_batch" ? 3 : 1;
  tpt_render_job j{};
  j.scene = scene;
  j.camera.look_at[2] = -1.0f;
  j.camera.up[1] = j.camera.fov_y = j.camera.exposure = 1.0f;
  j.width = j.height = side;
  j.spp = j.max_depth = 1;
  std::vector<float> image(3 * (size_t)side * side);
  std::vector<tpt_render_job> js(jobs, j);
  std::vector<float*> out(jobs, image.data());
  return tpt_render(ctx, js.data(), jobs, out.data());
}

int bad(const char* what) {
  std::printf("%s\n", what);
  return 1;
}
}  // namespace

int main(int argc, char** argv) {
  if (argc != 4 || tpt_context_create(0, &ctx) || tpt_context_set_graphs(ctx, 0) ||
      tpt_context_set_wavefront_capacity(ctx, 1 << 16) || upload(100, &scene))
    return bad("set-up failed");
  cudaDeviceSynchronize();
  const std::string mode = argv[1], what = argv[2], arg = argv[3];
  launches = 0;
  if (mode == "share") {
    tpt_status inner = TPT_ERR_INVALID_ARG;
    at_kind = what.rfind("render", 0) == 0 ? "image" : "traverse";
    at_launch = [&] { inner = call(arg); };
    if (call(what) || inner) return bad("a call failed");
    if (call(what) || call(arg)) return bad("a later call failed");
    if (!failure.empty()) return bad(failure.c_str());
  } else if (mode == "wait") {
    if (call(what)) return bad("a call failed");
  } else if (mode == "trim") {
    const size_t most = (size_t)std::atoi(argv[3]) << 20;
    if (call(what) || tpt_context_trim(ctx)) return bad("a call failed");
    const size_t before = live_bytes();  // arenas of renders stay
    if (call(what)) return bad("a call failed");
    if (live_bytes() == before || live_bytes() > before + most) return bad("memory kept by the call");
    if (tpt_context_trim(ctx)) return bad("a call failed");
    if (live_bytes() != before) return bad("memory not given back");
    if (call(what)) return bad("a call after it failed");
  } else if (mode == "records") {
    tpt_scene *a = nullptr, *b = nullptr;
    uint64_t with = 0, without = 0;
    const uint64_t t = std::atoi(argv[2]), bytes = std::atoi(argv[3]);
    if (upload(t, &a) || upload(t, &b, 0) || tpt_scene_device_bytes(a, &with) || tpt_scene_device_bytes(b, &without))
      return bad("a call failed");
    if (with < without + bytes * t) return bad("a scene for queries alone holds shading records");
  } else {
    fail_launch = std::atoi(argv[3]);
    const bool failed = call(what) != TPT_OK;
    if (failed != (launches >= fail_launch)) return bad("the failed launch is not reported");
    if (!failed) return bad("no such launch");
  }
  if (!idle()) return bad("the call returned with work in flight");
  std::printf("ok\n");
  return 0;
}
