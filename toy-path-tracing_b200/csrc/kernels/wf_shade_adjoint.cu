// Shade stage of the adjoint replay: one instantiation, with the delta-light paths.
#include "wf_shade.cuh"

namespace tpt {

cudaError_t launch_wf_shade_adjoint(const DevGeometry& geo, const DevRenderData& rd, const RenderLaunch& P,
                                    const WfBuffers& B, int cur, cudaStream_t s, const DevAdjoint& A) {
  wf_shade<true, false, true><<<grid_for(B.capacity, kAdjointBlock), kAdjointBlock, 0, s>>>(DevRender{geo, rd}, P, B, cur, A,
                                                                                            nullptr);
  return cudaGetLastError();
}

}  // namespace tpt
