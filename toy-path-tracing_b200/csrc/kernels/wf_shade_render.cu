// Shade stage of single-job renders and of the adjoint replay: launches.
#include "wf_shade.cuh"

namespace tpt {

cudaError_t launch_wf_shade_adjoint(const DevGeometry& geo, const DevRenderData& rd, const RenderLaunch& P,
                                    const WfBuffers& B, int cur, cudaStream_t s, const DevAdjoint& A);

cudaError_t launch_wf_shade(const DevGeometry& geo, const DevRenderData& rd, const RenderLaunch& P,
                            const WfBuffers& B, int cur, cudaStream_t s, const DevAdjoint* A, int block) {
  if (A) return launch_wf_shade_adjoint(geo, rd, P, B, cur, s, *A);
  DevRender S{geo, rd};
  const DevAdjoint none{};
  const int bs = shade_launch_block(block);
  if (rd.num_extra_lights > 0)
    wf_shade<false, false, true><<<grid_for(B.capacity, bs), bs, 0, s>>>(S, P, B, cur, none, nullptr);
  else
    wf_shade<false, false, false><<<grid_for(B.capacity, bs), bs, 0, s>>>(S, P, B, cur, none, nullptr);
  return cudaGetLastError();
}

}  // namespace tpt
