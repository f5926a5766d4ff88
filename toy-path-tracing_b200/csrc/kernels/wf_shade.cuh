// The shade stage of the wavefront (wavefront_kernels.cu describes the
// pipeline): one path vertex per queue entry.  A template in a header because
// its instantiations (render, batch, adjoint) are compiled in parallel, each in
// its own wf_shade_*.cu.
#pragma once
#include "../api/internal.h"
#include "../device/adjoint.cuh"
#include "../device/render.cuh"

namespace tpt {

constexpr int kWfBlock = 256;  // threads per block of the small stages
// Threads and blocks per SM of the shade stage.  A vertex runs some 4,000
// instructions nearly without loops, so the stage is bound by instruction
// fetches: the warps of a block run it in step (StageSync, a block barrier
// between its parts), which lets them share each fetch, and large blocks share
// more.  Two blocks per SM cover each other's barriers and ends.  Measured
// (Cornell OpenPBR 256x256x64 / dispersive glass 320x200x32 / 2.1M triangles
// 1080p x 8, ms per image): blocks of 256 without barriers 8.50 / 14.3 / 46.1;
// with one call site of the BSDF evaluation and barriers 1 x 640 8.26 / 6.84 / 37.7,
// 2 x 512 8.29 / 7.33 / 38.0, 2 x 384 7.79 / 7.65 / 38.7, 3 x 256 7.79 / 8.74 / 40.3;
// 1 x 640 without barriers 7.86 / 9.87 / 38.1, 2 x 256 with warp-level ones
// 7.94 / 12.6 / 42.4.
constexpr int kShadeBlock = 384, kShadeMinBlocks = 2;
// The adjoint variant spends its time in the sensitivities' loop over parameter
// groups, which fits the instruction cache: inverse-rendering step of the 64-patch
// box at 16 / 64 spp 7.94 / 16.1 ms; 1 x 256 8.33 / 17.8, 2 x 384 8.29 / 16.4,
// 1 x 640 8.40 / 16.2.
constexpr int kAdjointBlock = 256, kAdjointMinBlocks = 2;
struct StageSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// The launch's block for tpt_context_set_shade_block's setting: 128, or 256 for
// the stage's full blocks.
static inline int shade_launch_block(int setting) { return setting == 128 ? 128 : kShadeBlock; }

static inline unsigned grid_for(uint32_t n, int block = kWfBlock) { return (n + block - 1) / block; }

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool pred) {
  const unsigned act = __activemask();
  const unsigned m = __ballot_sync(act, pred);
  const unsigned lane = threadIdx.x & 31u;
  const int leader = __ffs(act) - 1;
  uint32_t base = 0;
  if ((int)lane == leader && m) base = atomicAdd(counter, (uint32_t)__popc(m));
  base = __shfl_sync(act, base, leader);
  return base + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// One vertex per queue entry of queue `cur`; appends to queue `cur ^ 1` and the shadow queue.
// LIGHTS: the scene (any scene of a batch) has point, spot or directional
// lights (prepare_direct's specialisation).
template <bool ADJ, bool BATCH, bool LIGHTS>
__global__ void __launch_bounds__(ADJ ? kAdjointBlock : kShadeBlock, ADJ ? kAdjointMinBlocks : kShadeMinBlocks)
    wf_shade(const __grid_constant__ DevRender S0, const __grid_constant__ RenderLaunch P0, WfBuffers B, int cur,
             const __grid_constant__ DevAdjoint A, const DevJob* __restrict__ jobs) {
  __shared__ float grad_sh[ADJ ? kAdjointBlock * kGradParams : 1];
  const StageSync sync;
  const uint32_t n_queue = B.counts[cur];
  if (blockIdx.x * blockDim.x >= n_queue) return;
  // threads past the queue's end stay for the barriers, on its last entry,
  // without a hit
  const bool valid = blockIdx.x * blockDim.x + threadIdx.x < n_queue;
  const uint32_t j = valid ? blockIdx.x * blockDim.x + threadIdx.x : n_queue - 1;
  const uint64_t first_path = (uint64_t)B.counts[4] | ((uint64_t)B.counts[5] << 32);
  const float sgn = ADJ ? -1.0f : 1.0f;  // the adjoint takes collected radiance off R
  uint32_t grad_key = 0xFFFFFFFFu, s_key = 0xFFFFFFFFu;
  float grad_v[ADJ ? kGradParams : 1], s_grad[ADJ ? kGradParams : 1];
  const uint32_t C = B.capacity;
  const uint32_t slot = B.q_slot[cur][j];
  const uint32_t jb = BATCH ? B.job[slot] : 0u;
  const DevRender& S = BATCH ? jobs[jb].render : S0;
  const RenderLaunch& P = BATCH ? jobs[jb].P : P0;
  const uint32_t d = B.depth[slot];
  bool push_next = false, push_shadow = false;
  V3 next_o, next_d;
  DirectPrep dp;
  V3 beta = V3{B.beta[slot], B.beta[C + slot], B.beta[2 * C + slot]};
  // The path's radiance: read and written back where the vertex collects some (the
  // adjoint reads R at every vertex).  Most vertices collect nothing, and a path that
  // ends needs no throughput: leaving those planes alone took the Cornell box
  // 256 x 256 x 64 from 7.18 to 7.02 ms, the batch of eight from 188.4 to 185.2.
  const auto load_L = [&] { return V3{B.L[slot], B.L[C + slot], B.L[2 * C + slot]}; };
  V3 L;
  if (ADJ) L = load_L();
  bool collected = false;
  // alpha tests (integrator order, see render_kernels.cu): the shadow ray's
  // AuxRng start, the bounce ray's, and whether the bounce continues from the
  // shadow ray's final state (MIS; the resolve stage copies it over)
  const bool alpha = B.q_aux != nullptr && S.geo.inst_alpha != nullptr;
  uint32_t sh_aux = 0, nx_aux = 0, aux_cont = 0;
  const int32_t tri = valid ? B.h_tri[j] : -1;
  Vertex v;
  DevMaterialRec m;
  uint32_t mi = 0;
  if (tri >= 0) {
    TraceResult h;
    h.tri = tri;
    h.inst = B.h_inst[j];
    h.b0 = B.h_bary[j];
    h.b1 = B.h_bary[C + j];
    h.b2 = B.h_bary[2 * C + j];
    const float* qr = B.q_ray[cur];
    const V3 rd = V3{qr[3 * C + j], qr[4 * C + j], qr[5 * C + j]};
    v = shade_hit<int>(S, h, rd);
    v.thr = beta;  // the path state of the vertex (mis.rs:54-55)
    v.lock = B.lock[slot];
    mi = __ldg(&S.d.inst[v.inst].material);
    m = S.d.mats[mi];
    // emission of this vertex (mis.rs:45-47 for the camera vertex, 101-117
    // after a bounce; PT counts every hit in full, NEE only from the camera
    // and after delta samples)
    V3 le;
    if (may_emit(m) && material_le(S, m, v, le)) {
      collected = true;
      if (!ADJ) L = load_L();
      if (d == 0) {
        L = L + sgn * le;
      } else {
        const uint32_t pm = B.prev_mat[slot];
        if ((pm >> 31) || P.integrator == kIntegPt) {
          L = L + sgn * (beta * le);
        } else if (P.integrator == kIntegMis) {
          Vertex pv;
          pv.p = V3{B.prev[slot], B.prev[C + slot], B.prev[2 * C + slot]};
          pv.ns = V3{B.prev[3 * C + slot], B.prev[4 * C + slot], B.prev[5 * C + slot]};
          const float lp = light_pdf_for_hit(S, S.d.mats[pm & 0x7FFFFFFFu], pv, v);
          L = L + sgn * (beta * le * balance_heuristic(B.prev[6 * C + slot], lp));
        }
      }
    }
  }
  sync();
  const bool scatters = tri >= 0 && d < P.max_depth && m.kind != kDevEmissive;
  PathSamplerDev ps;
  V3 dl = V3{0.0f, 0.0f, 0.0f};
  if (scatters) {
    const uint64_t path = first_path + slot - (BATCH ? jobs[jb].path_base : 0ull);
    if (ADJ) {
      const uint64_t di = 3ull * ((uint32_t)(path / P.spp) - A.pixel_base);
      dl = V3{A.d_image[di], A.d_image[di + 1], A.d_image[di + 2]} * A.scale;
    }
    const uint32_t pixel = (uint32_t)(path / P.spp), sample = (uint32_t)(path % P.spp);
    ps.init(pixel % P.width, pixel / P.width, sample, P.log2_spp, P.n_base4_digits, P.seed);
    if (alpha) {
      if (P.integrator == kIntegMis) {
        sh_aux = nx_aux = aux_from_seed(ps, (int)d);
        aux_cont = 1u;
      } else {
        sh_aux = B.q_aux[slot];  // NEE: after the arriving ray's draws
        nx_aux = aux_from_seed(ps, (int)d + 1);
      }
    }
    // (PT: BSDF sampling only)
    if (P.integrator != kIntegPt &&
        prepare_direct<LIGHTS>(S, m, v, ps, d, dp, P.integrator == kIntegNee)) {
      dp.contrib = beta * dp.contrib;
      push_shadow = true;
    }
  }
  sync();
  BsdfSampleOut s;
  const bool sampled = material_sample(S, m, v, ps, d, s, scatters, sync);
  if (scatters) {
    bool sampled_grads = false;
    float sens_s[ADJ ? 3 * kGradGroups : 1];
    if (sampled) {
      beta = beta * s.weight;
      if (s.lock >= 0.0f) B.lock[slot] = s.lock;
      bool alive = true;
      if (d + 1 >= 4) {
        const float q = clampf(max_element(beta), 0.05f, 1.0f);
        if (ps.sample_1d(vertex_dim(d, kOffRr)) > q) alive = false;
        else beta = beta / q;
      }
      if (alive) {
        push_next = true;
        if (ADJ && m.kind == kDevOpenPbr && !s.delta) {
          // R (= L here) still holds this vertex's light sample, if any:
          // resolve corrects for it once the shadow ray is known unoccluded
          openpbr_vertex_sens(S, A, m.openpbr, v, s.wi, sens_s);
          grads_from_sens(sens_s, dl * L, grad_v);
          grad_key = mi;
          sampled_grads = true;
        }
        next_o = offset_origin(v.p, v.ng, s.wi);
        next_d = s.wi;
        B.prev[slot] = v.p.x;
        B.prev[C + slot] = v.p.y;
        B.prev[2 * C + slot] = v.p.z;
        B.prev[3 * C + slot] = v.ns.x;
        B.prev[4 * C + slot] = v.ns.y;
        B.prev[5 * C + slot] = v.ns.z;
        B.prev[6 * C + slot] = s.pdf;
        B.prev_mat[slot] = mi | (s.delta ? 0x80000000u : 0u);
        B.depth[slot] = d + 1;
      }
    }
    if (ADJ && push_shadow && A.s_gkey) {
      s_key = 0xFFFFFFFFu;
      if (m.kind == kDevOpenPbr) {
        float sens_l[3 * kGradGroups], t[kGradParams];
        openpbr_vertex_sens(S, A, m.openpbr, v, dp.wi, sens_l);
        const V3 w = dl * dp.contrib;
        grads_from_sens(sens_l, w, s_grad);
        if (sampled_grads) {
          grads_from_sens(sens_s, w, t);
#pragma unroll
          for (int k = 0; k < (int)kGradParams; ++k) s_grad[k] -= t[k];
        }
        s_key = mi;
      }
    }
  }
  if (LIGHTS && valid && tri < 0 && S.d.has_env) {
    // the ray left the scene: the environment's radiance (mis.rs:33-35,
    // 127-135; PT in full, pt.rs:36-39; NEE from the camera and after delta
    // samples only, nee.rs:37-42)
    const uint32_t pm = d == 0 ? 0u : B.prev_mat[slot];
    const bool full = d == 0 || (pm >> 31) != 0 || P.integrator == kIntegPt;
    if (full || P.integrator == kIntegMis) {
      const float* qr = B.q_ray[cur];
      const V3 rd = V3{qr[3 * C + j], qr[4 * C + j], qr[5 * C + j]};
      const V3 le = env_escape(S.d, rd, full, false, full ? 0.0f : B.prev[6 * C + slot]);
      collected = true;
      if (!ADJ) L = load_L();
      L = L + sgn * (d == 0 ? le : beta * le);
    }
  }
  sync();
  if (!valid) return;
  if (collected) {
    B.L[slot] = L.x;
    B.L[C + slot] = L.y;
    B.L[2 * C + slot] = L.z;
  }
  if (push_next) {
    B.beta[slot] = beta.x;
    B.beta[C + slot] = beta.y;
    B.beta[2 * C + slot] = beta.z;
  }
  const int nxt = cur ^ 1;
  const uint32_t qn = warp_append(&B.counts[nxt], push_next);
  const uint32_t qs = warp_append(&B.counts[2], push_shadow);
  if (push_next) {
    float* q = B.q_ray[nxt];
    q[qn] = next_o.x;
    q[C + qn] = next_o.y;
    q[2 * C + qn] = next_o.z;
    q[3 * C + qn] = next_d.x;
    q[4 * C + qn] = next_d.y;
    q[5 * C + qn] = next_d.z;
    q[6 * C + qn] = __int_as_float(0x7f800000);
    B.q_slot[nxt][qn] = slot;
    if (BATCH) B.q_job[nxt][qn] = jb;
    if (alpha) B.q_aux[slot] = nx_aux;
  }
  if (push_shadow) {
    float* q = B.s_ray;
    q[qs] = dp.so.x;
    q[C + qs] = dp.so.y;
    q[2 * C + qs] = dp.so.z;
    q[3 * C + qs] = dp.wi.x;
    q[4 * C + qs] = dp.wi.y;
    q[5 * C + qs] = dp.wi.z;
    q[6 * C + qs] = __int_as_float(0x7f800000);
    B.s_slot[qs] = slot;
    if (BATCH) B.s_job[qs] = jb;
    if (alpha) {
      B.s_aux[qs] = sh_aux;
      B.s_aux_cont[qs] = aux_cont;
    } else if (B.s_aux_cont) {
      B.s_aux_cont[qs] = 0u;  // a batch mixes scenes with and without alpha tests
    }
    B.s_target[qs] = dp.inst;
    B.s_target[C + qs] = dp.tri;
    if (LIGHTS) B.s_dist[qs] = dp.dist;
    B.s_contrib[qs] = dp.contrib.x;
    B.s_contrib[C + qs] = dp.contrib.y;
    B.s_contrib[2 * C + qs] = dp.contrib.z;
    if (ADJ && A.s_gkey) {
      A.s_gkey[qs] = s_key;
      if (s_key != 0xFFFFFFFFu) {
#pragma unroll
        for (int k = 0; k < (int)kGradParams; ++k) A.s_grad[(size_t)k * C + qs] = s_grad[k];
      }
    }
  }
  if (ADJ) warp_accumulate_grads(A.grad, grad_key, grad_v, grad_sh + (threadIdx.x & ~31u) * kGradParams);
}

}  // namespace tpt
