// Kernels of the splitting sort for 4-byte keys.
#include "b2s_split.cuh"
namespace b2s {
template <>
cudaError_t launch_split<4>(int xf, const SplitPlan& plan, const SplitJob& job, Ctrl* ctrl, cudaStream_t stream)
{
  return split_any<4>(xf, plan, job, ctrl, stream);
}
}
