// Shade stage of batched renders: launches.
#include "wf_shade.cuh"

namespace tpt {

cudaError_t launch_wf_shade_batch(const DevJob* jobs, const WfBuffers& B, int cur, cudaStream_t s, int block,
                                  bool lights) {
  const DevRender S{};
  const RenderLaunch P{};
  const DevAdjoint none{};
  const int bs = shade_launch_block(block);
  if (lights)
    wf_shade<false, true, true><<<grid_for(B.capacity, bs), bs, 0, s>>>(S, P, B, cur, none, jobs);
  else
    wf_shade<false, true, false><<<grid_for(B.capacity, bs), bs, 0, s>>>(S, P, B, cur, none, jobs);
  return cudaGetLastError();
}

}  // namespace tpt
