// Wavefront path tracing: the MIS integrator of integrator/mis.rs split into
// stage kernels over compacted queues of path slots,
//
//   generate -> [ traverse(closest) -> shade -> traverse(shadow) -> resolve ]
//               x (max_depth + 1) -> accumulate (finalize where samples are asked for)
//
// Traversal runs in the persistent-warp kernel of traverse_kernels.cu; shade
// handles one path vertex (emission with MIS against the previous vertex, NEE
// preparation, BSDF sampling, Russian roulette) and appends the next ray and
// the shadow ray with warp-aggregated atomics; resolve adds the NEE
// contribution of visible shadow rays.  Each path's radiance is updated in the
// reference's order (emission of vertex d, then NEE of vertex d, then emission
// of vertex d + 1), so the result equals the megakernel's bit for bit.
// Stage launch shapes do not depend on queue lengths (those live on the
// device), so one bounce is a fixed launch sequence that a CUDA graph replays.
//
// The batched instantiation (BATCH = true) runs many jobs (scenes, cameras,
// resolutions, spp, depths) through one launch sequence: slot i of a chunk is
// global path first_path + i of the batch, whose job is found by binary search
// over the jobs' path bases; every slot, queued ray and shadow ray carries its
// job index, and each stage reads the job's scene and launch record from the
// DevJob array instead of its kernel parameters.
//
// The adjoint instantiation (ADJ = true) replays the same paths with the
// radiance planes holding R, the part of the path's radiance still to come:
// generate starts R at the path's radiance from the forward pass, shade and
// resolve subtract what each vertex collects, and shade adds, at every rough
// OpenPBR vertex, dLoss/dL * R * (df/dtheta) / f to the per-material gradients.
// A light sample C at an OpenPBR vertex (directional lights) is only known to
// count once its shadow ray is resolved, while shade has already used R with C
// still in it; shade therefore queues, with the shadow ray, the change
// dLoss/dL * C * [(df/dtheta) / f at the light direction - the same at the
// sampled direction], which resolve adds when the ray is unoccluded.
#include "wf_shade.cuh"

namespace tpt {

// Job of global path g: the last job whose path_base <= g (jobs sorted by path_base).
__device__ __forceinline__ uint32_t job_of_path(const DevJob* __restrict__ jobs, uint32_t n_jobs, uint64_t g) {
  uint32_t lo = 0, hi = n_jobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].path_base <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <bool ADJ, bool BATCH>
__global__ void __launch_bounds__(kWfBlock) wf_generate(const __grid_constant__ DevRender S0,
                                                                 const __grid_constant__ RenderLaunch P0, WfBuffers B,
                                                        uint64_t first_path, uint32_t n_paths,
                                                        const float* __restrict__ primal,
                                                        const DevJob* __restrict__ jobs, uint32_t n_jobs) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    B.counts[0] = n_paths;
    B.counts[1] = 0;
    B.counts[2] = 0;
    // the chunk's first path, for the later stages (which a graph replays
    // unchanged from chunk to chunk)
    B.counts[4] = (uint32_t)first_path;
    B.counts[5] = (uint32_t)(first_path >> 32);
  }
  if (i >= n_paths) return;
  const uint32_t C = B.capacity;
  const uint32_t jb = BATCH ? job_of_path(jobs, n_jobs, first_path + i) : 0u;
  const RenderLaunch& P = BATCH ? jobs[jb].P : P0;
  const uint64_t path = first_path + i - (BATCH ? jobs[jb].path_base : 0ull);
  const uint32_t pixel = (uint32_t)(path / P.spp), sample = (uint32_t)(path % P.spp);
  const uint32_t px = pixel % P.width, py = pixel / P.width;
  PathSamplerDev ps;
  ps.init(px, py, sample, P.log2_spp, P.n_base4_digits, P.seed);
  float c0, c1;
  ps.sample_2d(kDimCamera, c0, c1);
  const float fx = ((float)px + 0.5f) + 0.5f * tent(c0);
  const float fy = ((float)py + 0.5f) + 0.5f * tent(c1);
  const V3 d = camera_dir(P.cam, P.width, P.height, fx, fy);
  float* q = B.q_ray[0];
  q[i] = P.cam.eye[0];
  q[C + i] = P.cam.eye[1];
  q[2 * C + i] = P.cam.eye[2];
  q[3 * C + i] = d.x;
  q[4 * C + i] = d.y;
  q[5 * C + i] = d.z;
  q[6 * C + i] = __int_as_float(0x7f800000);
  B.q_slot[0][i] = i;
  if (BATCH) {
    B.job[i] = jb;
    B.q_job[0][i] = jb;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    B.beta[k * C + i] = 1.0f;
    B.L[k * C + i] = ADJ ? primal[3 * (uint64_t)i + k] : 0.0f;
  }
  B.depth[i] = 0;
  B.lock[i] = -1.0f;
  // alpha tests: the camera ray's AuxRng (mis.rs: the initial seed; nee.rs /
  // pt.rs: depth 0's seed)
  if (B.q_aux && (BATCH ? jobs[jb].render.geo.inst_alpha : S0.geo.inst_alpha) != nullptr)
    B.q_aux[i] = aux_from_seed(ps, P.integrator == kIntegMis ? -1 : 0);
}

// unoccluded_ray (integrator/mod.rs:239-265): visible when nothing is hit, the
// first hit is the sampled emitter triangle, or (point and spot lights) the
// first hit lies beyond the light.
template <bool ADJ>
__global__ void __launch_bounds__(kWfBlock) wf_resolve(WfBuffers B, const __grid_constant__ DevAdjoint A) {
  __shared__ float grad_sh[ADJ ? kWfBlock * kGradParams : 1];
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= B.counts[2]) return;
  const uint32_t C = B.capacity;
  // MIS with alpha tests: the bounce ray continues the shadow ray's AuxRng
  if (B.s_aux_cont && B.s_aux_cont[j]) B.q_aux[B.s_slot[j]] = B.s_aux[j];
  const uint32_t tgt_inst = B.s_target[j];
  // the distance plane is written for delta-light shadow rays only
  const bool visible = shadow_visible(B.s_tri[j], B.s_inst[j], B.s_t[j], tgt_inst, B.s_target[C + j],
                                      tgt_inst == 0xFFFFFFFFu ? B.s_dist[j] : 0.0f);
  if (visible) {
    const uint32_t slot = B.s_slot[j];
    const float sgn = ADJ ? -1.0f : 1.0f;
    B.L[slot] = B.L[slot] + sgn * B.s_contrib[j];
    B.L[C + slot] = B.L[C + slot] + sgn * B.s_contrib[C + j];
    B.L[2 * C + slot] = B.L[2 * C + slot] + sgn * B.s_contrib[2 * C + j];
  }
  if (ADJ && A.s_gkey) {
    const uint32_t key = visible ? A.s_gkey[j] : 0xFFFFFFFFu;
    float vals[kGradParams];
#pragma unroll
    for (int k = 0; k < (int)kGradParams; ++k) vals[k] = key != 0xFFFFFFFFu ? A.s_grad[(size_t)k * C + j] : 0.0f;
    warp_accumulate_grads(A.grad, key, vals, grad_sh + (threadIdx.x & ~31u) * kGradParams);
  }
}

__global__ void __launch_bounds__(kWfBlock) wf_finalize(WfBuffers B, uint32_t n_paths, float* samples) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_paths) return;
  const uint32_t C = B.capacity;
  samples[3 * (uint64_t)i] = B.L[i];
  samples[3 * (uint64_t)i + 1] = B.L[C + i];
  samples[3 * (uint64_t)i + 2] = B.L[2 * C + i];
}

// finalize and accumulate in one, without the per-sample buffer between them: the
// running mean of each pixel's radiance planes, color += (sample - color) / (i + 1)
// in sample order, then * exposure (main.rs:107-123), of the n_pixels pixels whose
// samples start at slot `first_slot`.  Bound by the chain of divisions of a pixel:
// a thread per pixel and channel, its samples loaded eight at a time ahead of the
// chain.  It spares the buffer (12 bytes a path, 50 MB for 256 x 256 x 64) and a pass;
// the time saved is within the noise (that render 7.40 -> 7.37 ms).
__global__ void __launch_bounds__(kWfBlock) wf_accumulate(const float* __restrict__ L, uint32_t C, uint32_t first_slot,
                                                          uint32_t spp, uint32_t first_pixel, uint32_t n_pixels,
                                                          float exposure, float* __restrict__ image) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3ull * n_pixels) return;
  const uint32_t i = (uint32_t)(t / 3u), c = (uint32_t)(t - 3ull * i);
  const float* s = L + (size_t)c * C + first_slot + (size_t)spp * i;
  float mean = 0.0f;
  uint32_t k = 0;
  for (; k + 8 <= spp; k += 8) {
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = s[k + u];
#pragma unroll
    for (int u = 0; u < 8; ++u) mean = mean + (x[u] - mean) / (float)(k + u + 1);
  }
  for (; k < spp; ++k) mean = mean + (s[k] - mean) / (float)(k + 1);
  image[3ull * first_pixel + t] = mean * exposure;
}

cudaError_t launch_wf_generate(const DevGeometry& geo, const DevRenderData& rd, const RenderLaunch& P,
                               const WfBuffers& B, uint64_t first_path, uint32_t n_paths, cudaStream_t s,
                               const float* primal) {
  DevRender S{geo, rd};
  if (primal)
    wf_generate<true, false><<<grid_for(std::max(n_paths, 1u)), kWfBlock, 0, s>>>(S, P, B, first_path, n_paths,
                                                                                  primal, nullptr, 0);
  else
    wf_generate<false, false><<<grid_for(std::max(n_paths, 1u)), kWfBlock, 0, s>>>(S, P, B, first_path, n_paths,
                                                                                   nullptr, nullptr, 0);
  return cudaGetLastError();
}

cudaError_t launch_wf_generate_batch(const DevJob* jobs, uint32_t n_jobs, const WfBuffers& B, uint64_t first_path,
                                     uint32_t n_paths, cudaStream_t s) {
  wf_generate<false, true><<<grid_for(std::max(n_paths, 1u)), kWfBlock, 0, s>>>(
      DevRender{}, RenderLaunch{}, B, first_path, n_paths, nullptr, jobs, n_jobs);
  return cudaGetLastError();
}

cudaError_t launch_wf_resolve(const WfBuffers& B, cudaStream_t s, const DevAdjoint* A) {
  if (A) wf_resolve<true><<<grid_for(B.capacity), kWfBlock, 0, s>>>(B, *A);
  else wf_resolve<false><<<grid_for(B.capacity), kWfBlock, 0, s>>>(B, DevAdjoint{});
  return cudaGetLastError();
}

cudaError_t launch_wf_finalize(const WfBuffers& B, uint32_t n_paths, float* samples, cudaStream_t s) {
  wf_finalize<<<grid_for(std::max(n_paths, 1u)), kWfBlock, 0, s>>>(B, n_paths, samples);
  return cudaGetLastError();
}

cudaError_t launch_wf_accumulate(const WfBuffers& B, uint32_t first_slot, uint32_t spp, uint32_t first_pixel,
                                 uint32_t n_pixels, float exposure, float* image, cudaStream_t s) {
  if (n_pixels == 0) return cudaSuccess;
  wf_accumulate<<<(unsigned)((3ull * n_pixels + kWfBlock - 1) / kWfBlock), kWfBlock, 0, s>>>(
      B.L, B.capacity, first_slot, spp, first_pixel, n_pixels, exposure, image);
  return cudaGetLastError();
}

}  // namespace tpt
