// Scene upload: per-triangle shading records from the meshes' vertex arrays.
#include "../api/internal.h"

namespace tpt {

// One thread per triangle: three indices and vertices gathered into one 96-byte
// record (bound by its writes: 1M triangles, 96 MB, take some 30 us).
__global__ void __launch_bounds__(256) bake_shade_tris(const MeshSpan* __restrict__ meshes, uint32_t n_meshes,
                                                       const float* __restrict__ pos, const float* __restrict__ nrm,
                                                       const float* __restrict__ uv, const uint32_t* __restrict__ idx,
                                                       uint64_t n, DevShadeTri* __restrict__ out) {
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  // the last mesh whose first triangle is at most g
  uint32_t lo = 0, hi = n_meshes;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (meshes[mid].tri_base <= g) lo = mid;
    else hi = mid;
  }
  DevShadeTri t;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const size_t v = (size_t)meshes[lo].vtx_base + idx[3 * g + k];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      t.p[3 * k + c] = pos[3 * v + c];
      t.n[3 * k + c] = nrm[3 * v + c];
    }
    t.uv[2 * k] = uv[2 * v];
    t.uv[2 * k + 1] = uv[2 * v + 1];
  }
  out[g] = t;
}

cudaError_t launch_bake_shade_tris(const MeshSpan* meshes, uint32_t n_meshes, const float* pos, const float* nrm,
                                   const float* uv, const uint32_t* idx, uint64_t n, DevShadeTri* out,
                                   cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  bake_shade_tris<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(meshes, n_meshes, pos, nrm, uv, idx, n, out);
  return cudaGetLastError();
}

}  // namespace tpt
