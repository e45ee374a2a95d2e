// Kernels of the local sort for 4-byte keys.
#include "b2s_launch.cuh"
namespace b2s {
B2S_INSTANTIATE_KEY_WIDTH(4, true, false)

cudaError_t selftest_sweeps(int which, Ctrl* ctrl, unsigned int* lookback, unsigned int tiles, SegGeom geo, cudaStream_t stream)
{
  if (which == SELFTEST_SHORT) return launch_sweeps<4, XF_UNSIGNED, false, SWEEP_SMALL, true>(ctrl, lookback, tiles, geo, 0, stream);
  if (which == SELFTEST_ROWS) return launch_sweeps<4, XF_UNSIGNED, false>(ctrl, lookback, tiles, geo, 0, stream);
  return launch_sweeps<4, XF_UNSIGNED, false, SWEEP_LARGE, false>(ctrl, lookback, tiles, geo, 0, stream);
}
}
