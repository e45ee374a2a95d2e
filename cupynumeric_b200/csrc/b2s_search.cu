// SEARCHSORTED: for every value, its insertion position in a sorted 1-D array that may be tiled
// over ranks.  Same per-tile contract as the reference's kernels
// (src/cupynumeric/sort/searchsorted.cu:25-74): a tile contributes its lower bound (left) only
// when it lies inside the tile, its upper bound (right) only when it is positive, shifted by
// the tile's global offset, and contributions combine by MIN (left) / MAX (right) into an
// output the caller pre-filled with the global size (left) or 0 (right).  Keys compare in the
// same total order the sort produces (NaN last).
#include "../../include/b200sort.h"
#include "b2s_common.cuh"
#include "b2s_prof.h"

#include <type_traits>

namespace b2s {

constexpr int SS_SAMPLES  = 4096;
constexpr size_t SS_MANY  = (size_t)1 << 20;  // values from which on a long tile is searched without samples
constexpr size_t SS_BYTES = (size_t)1 << 28;  // longest tile that the L2 holds well enough

// SAMPLES > 0: every CTA first puts SS_SAMPLES evenly spaced keys of the tile (their images) into shared memory and
// searches there; only the levels below go to memory.  A warp's 32 probes at different places of
// memory cost the L1 a lookup each, 32 cycles per level, while shared memory answers 32 random
// probes in about 3.5: that, and not the bytes, is what bounds a search without the samples, even though
// its upper levels sit in the L1 (10^6 values in 2^24 doubles: 114 us, 94 with the samples).  More samples
// would cost each CTA more to fetch than they save.
// SAMPLES == 0: every value is searched for in memory from the start.
// STORE: the tile is the whole array, positions are stored; else they are combined with what is there.
template <int KB, bool STORE, int SAMPLES, int THREADS>
__global__ void __launch_bounds__(THREADS)
searchsorted_kernel(const typename KeyOf<KB>::type* __restrict__ sorted, long long n, long long global_offset,
                    const typename KeyOf<KB>::type* __restrict__ values, long long num_values, int left, int xf,
                    long long* __restrict__ positions)
{
  using K = typename KeyOf<KB>::type;
  __shared__ K sample[SAMPLES > 0 ? SAMPLES : 1];
  const long long step = SAMPLES > 0 ? (n + SAMPLES - 1) / (SAMPLES > 0 ? SAMPLES : 1) : 0;
  const int m          = SAMPLES > 0 && n > 0 ? (int)((n + step - 1) / step) : 0;
  if (SAMPLES > 0) {
    for (int k = threadIdx.x; k < m; k += THREADS) sample[k] = to_ordered_rt<KB>(sorted[k * step], xf);
    __syncthreads();
  }
  for (long long i = (long long)blockIdx.x * THREADS + threadIdx.x; i < num_values; i += (long long)gridDim.x * THREADS) {
    const K v = to_ordered_rt<KB>(values[i], xf);
    long long lo = 0, hi = n;
    if (SAMPLES > 0) {
      int below = 0, top = m;  // samples in front of the position
      while (below < top) {
        const int mid       = (below + top) >> 1;
        const K k           = sample[mid];
        const bool go_right = left ? (k < v) : (k <= v);
        if (go_right) below = mid + 1; else top = mid;
      }
      // the position lies behind sample below - 1 and not behind sample `below`
      lo = below == 0 ? 0 : (below - 1) * step + 1;
      hi = below == 0 ? 0 : (below * step < n ? below * step : n);
    }
    using Len     = typename std::conditional<SAMPLES != 0, unsigned int, long long>::type;  // (a step of up to 2^44 keys)
    const K* base = sorted + lo;
    Len len       = (Len)(hi - lo);
    Len first     = 0;
    while (first < len) {
      const Len mid          = first + ((len - first) >> 1);
      const K k              = to_ordered_rt<KB>(base[mid], xf);
      const bool go_right    = left ? (k < v) : (k <= v);
      if (go_right) first = mid + 1; else len = mid;
    }
    lo += first;
    if (STORE) {
      positions[i] = lo + global_offset;
    } else if (left) {
      if (lo < n) atomicMin(positions + i, lo + global_offset);
    } else {
      if (lo > 0) atomicMax(positions + i, lo + global_offset);
    }
  }
}

template <int KB>
static cudaError_t searchsorted_launch(const void* sorted, size_t n, int64_t global_offset, const void* values, size_t num_values,
                                       int left, int xf, int64_t* positions, bool whole, cudaStream_t stream)
{
  using K = typename KeyOf<KB>::type;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  prof::Scope ps(prof::K_DIST, stream);
  auto launch = [&](auto kern, int threads, size_t grid) {
    kern<<<(unsigned int)grid, threads, 0, stream>>>(static_cast<const K*>(sorted), (long long)n, global_offset,
                                                     static_cast<const K*>(values), (long long)num_values, left, xf,
                                                     reinterpret_cast<long long*>(positions));
    return cudaGetLastError();
  };
  // The samples pay where a CTA has more than one round of values for the ones it fetched (10^5 values in 2^24 doubles
  // take 19 us with them and 13 without, 2 * 10^5 26 and 20, 4 * 10^5 47 and 50, 2^20 95 and 110), and, for many
  // values, where the probes below them find the tile in the L2: in 2^26 doubles (512 MiB) 4 * 10^5 values take 111
  // us with them and 138 without, but 2^22 values 1071 and 994.
  const size_t grid_all = (size_t)sms * 4;  // all resident: the samples are fetched once per CTA
  if (num_values > grid_all * 512 && (num_values < SS_MANY || n <= SS_BYTES / KB)) {
    const size_t grid = grid_all;
    return whole ? launch(searchsorted_kernel<KB, true, SS_SAMPLES, 512>, 512, grid)
                 : launch(searchsorted_kernel<KB, false, SS_SAMPLES, 512>, 512, grid);
  }
  size_t grid = (num_values + 255) / 256;
  if (grid > (1ull << 30)) grid = 1ull << 30;
  return whole ? launch(searchsorted_kernel<KB, true, 0, 256>, 256, grid) : launch(searchsorted_kernel<KB, false, 0, 256>, 256, grid);
}

}  // namespace b2s

using namespace b2s;

static int searchsorted_any(int dtype, const void* sorted_tile, size_t n_tile, int64_t global_offset, const void* values,
                            size_t num_values, int left, int64_t* positions, bool whole, void* cuda_stream)
{
  int kb = 0, xf = 0;
  switch (dtype) {
    case B2S_BOOL: case B2S_UINT8: kb = 1; xf = XF_UNSIGNED; break;
    case B2S_INT8: kb = 1; xf = XF_SIGNED; break;
    case B2S_UINT16: kb = 2; xf = XF_UNSIGNED; break;
    case B2S_INT16: kb = 2; xf = XF_SIGNED; break;
    case B2S_FLOAT16: kb = 2; xf = XF_FLOAT; break;
    case B2S_UINT32: kb = 4; xf = XF_UNSIGNED; break;
    case B2S_INT32: kb = 4; xf = XF_SIGNED; break;
    case B2S_FLOAT32: kb = 4; xf = XF_FLOAT; break;
    case B2S_UINT64: kb = 8; xf = XF_UNSIGNED; break;
    case B2S_INT64: kb = 8; xf = XF_SIGNED; break;
    case B2S_FLOAT64: kb = 8; xf = XF_FLOAT; break;
    case B2S_COMPLEX64: kb = 8; xf = XF_CFLOAT; break;
    default: return B2S_ERR_UNSUPPORTED;
  }
  if (num_values == 0) return B2S_OK;
  if (values == nullptr || positions == nullptr || (n_tile > 0 && sorted_tile == nullptr)) return B2S_ERR_INVALID_ARG;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  cudaError_t e;
  switch (kb) {
    case 1: e = searchsorted_launch<1>(sorted_tile, n_tile, global_offset, values, num_values, left, xf, positions, whole, stream); break;
    case 2: e = searchsorted_launch<2>(sorted_tile, n_tile, global_offset, values, num_values, left, xf, positions, whole, stream); break;
    case 4: e = searchsorted_launch<4>(sorted_tile, n_tile, global_offset, values, num_values, left, xf, positions, whole, stream); break;
    default: e = searchsorted_launch<8>(sorted_tile, n_tile, global_offset, values, num_values, left, xf, positions, whole, stream); break;
  }
  return e == cudaSuccess ? B2S_OK : B2S_ERR_CUDA;
}

extern "C" {

int b2s_searchsorted(int dtype, const void* sorted_tile, size_t n_tile, int64_t global_offset, const void* values,
                     size_t num_values, int left, int64_t* positions, void* cuda_stream)
{
  return searchsorted_any(dtype, sorted_tile, n_tile, global_offset, values, num_values, left, positions, false, cuda_stream);
}

int b2s_searchsorted_whole(int dtype, const void* sorted, size_t n, const void* values, size_t num_values, int left,
                           int64_t* positions, void* cuda_stream)
{
  return searchsorted_any(dtype, sorted, n, 0, values, num_values, left, positions, true, cuda_stream);
}
}
