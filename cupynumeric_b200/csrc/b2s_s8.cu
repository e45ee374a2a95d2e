// Kernels of the splitting sort for 8-byte keys.
#include "b2s_split.cuh"
namespace b2s {
template <>
cudaError_t launch_split<8>(int xf, const SplitPlan& plan, const SplitJob& job, Ctrl* ctrl, cudaStream_t stream)
{
  return split_any<8>(xf, plan, job, ctrl, stream);
}
}
