// UNIQUE on sorted data: keeps the first element of every run of equal keys.  With the sort in
// front of it this replaces the local part of the reference's UNIQUE task, which is a
// thrust::sort followed by thrust::unique (src/cupynumeric/set/unique.cu:150-208).  Keys are
// equal when their ordered images are equal: all NaNs are one value, -0.0 equals +0.0.
#include "../../include/b200sort.h"
#include "b2s_common.cuh"
#include "b2s_prof.h"

namespace b2s {

constexpr int UQ_THREADS = 256;
constexpr int UQ_WARPS   = UQ_THREADS / 32;
constexpr int UQ_ITEMS   = 16;  // keys per thread of short arrays
constexpr int UQ_TILE    = UQ_THREADS * UQ_ITEMS;
// From here on a thread takes twice as many.  The chain over the tiles advances by about 50 of them per microsecond
// whatever they hold, which bounds long arrays: 2^27 uint8 keys 660 -> 560 us, int64 with few distinct ones 712 ->
// 588.  (A look-back of 128 tiles per round trip instead of 32 made it worse: 907 us.)  10^5 keys take 28 us with
// the small tiles and 35 with the large ones.
constexpr long long UQ_LONG = 1ll << 22;

// Head of the workspace; one state word per tile follows (0: nothing yet).
struct UniqueCtrl {
  unsigned long long total;  // heads in the whole array, written by the last tile
  unsigned int ticket;       // next tile
  unsigned int status;       // 0 or DEV_ERR_TIMEOUT
  unsigned int spin_limit;   // 0: SPIN_LIMIT; else the poll limit of the look-back wait (self-test)
  unsigned int pad_;
};
constexpr unsigned long long UQ_AGG = 1ull << 62, UQ_INCL = 2ull << 62, UQ_VALUE = UQ_AGG - 1;

__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p)
{
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One pass over the sorted keys: a CTA takes the next tile (ticket), counts its heads, chains the count
// to its predecessors (decoupled look-back, 32 tiles per round trip, one lane each) and writes its heads
// in order.  Bound by memory: every key is read once from HBM (its left neighbour comes from the L1),
// every head written once; counting, scanning and writing in three launches read the keys twice (2^25 float32
// keys, most of them heads: 214 -> 170 us, few heads 197 -> 147; uint8 163 -> 145; int64 225 -> 209 and 190 -> 170).
template <int KB, int ITEMS>
__global__ void __launch_bounds__(UQ_THREADS)
unique_kernel(const typename KeyOf<KB>::type* __restrict__ a, long long n, int xf, UniqueCtrl* ctrl,
              unsigned long long* __restrict__ state, typename KeyOf<KB>::type* __restrict__ out)
{
  using K = typename KeyOf<KB>::type;
  constexpr int TILE = UQ_THREADS * ITEMS;
  __shared__ unsigned int heads[ITEMS * UQ_WARPS];  // per group of 32 keys, in key order; then their prefix
  __shared__ unsigned int tile_sh;
  __shared__ unsigned long long before_sh;
  if (threadIdx.x == 0) tile_sh = atomicAdd(&ctrl->ticket, 1u);
  __syncthreads();
  const unsigned int tile = tile_sh;
  const long long base    = (long long)tile * TILE;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  K key[ITEMS];
  unsigned int bal[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const long long i = base + j * UQ_THREADS + threadIdx.x;
    key[j]            = i < n ? a[i] : (K)0;
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const long long i = base + j * UQ_THREADS + threadIdx.x;
    const bool head   = i < n && (i == 0 || to_ordered_rt<KB>(key[j], xf) != to_ordered_rt<KB>(a[i - 1], xf));
    bal[j]            = __ballot_sync(0xFFFFFFFFu, head);
    if (lane == 0) heads[j * UQ_WARPS + w] = __popc(bal[j]);
  }
  __syncthreads();
  if (w == 0) {
    // one count per group, PER consecutive ones per lane
    constexpr int PER = ITEMS * UQ_WARPS / 32;
    unsigned int c[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      c[j] = heads[lane * PER + j];
      sum += c[j];
    }
    unsigned int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += t;
    }
    unsigned int run = incl - sum;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      heads[lane * PER + j] = run;
      run += c[j];
    }
    const unsigned long long mine = __shfl_sync(0xFFFFFFFFu, incl, 31);
    unsigned long long before     = 0;
    if (tile != 0) {
      if (lane == 0) st_relaxed64(state + tile, UQ_AGG | mine);
      long long t        = (long long)tile - 1 - lane;
      unsigned int spins = 0, spin_cap = SPIN_LIMIT;
      while (true) {
        const unsigned long long v  = t >= 0 ? ld_relaxed64(state + t) : UQ_INCL;
        const unsigned int missing  = __ballot_sync(0xFFFFFFFFu, v == 0);
        const unsigned int inclusive = __ballot_sync(0xFFFFFFFFu, (v >> 62) == 2);
        // the nearest entries up to the first gap; up to and with the first inclusive one
        const int gap   = missing ? __ffs(missing) - 1 : 32;
        const int stop  = inclusive ? __ffs(inclusive) - 1 : 32;
        const int used  = stop < gap ? stop + 1 : gap;
        unsigned long long add = lane < used ? v & UQ_VALUE : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xFFFFFFFFu, add, o);
        before += add;
        t -= used;
        if (stop < gap) break;
        if (used == 0) {
          // one lane decides for the warp: the status may change between two lanes' loads of it, and lanes
          // that left would be missing from the votes of those that stayed
          ++spins;
          int give_up = 0;
          if (lane == 0) {
            if (spins == 1 && ctrl->spin_limit != 0) spin_cap = ctrl->spin_limit;
            give_up = spins > spin_cap || ((spins & 1023u) == 0 && ld_relaxed(&ctrl->status) != 0);
            if (give_up) atomicMax(&ctrl->status, DEV_ERR_TIMEOUT);
          }
          if (__shfl_sync(0xFFFFFFFFu, give_up, 0)) break;
          if (spins > 4) __nanosleep(64);
        }
      }
    }
    if (lane == 0) {
      st_relaxed64(state + tile, UQ_INCL | (before + mine));
      before_sh = before;
      if (base + TILE >= n) ctrl->total = before + mine;
    }
  }
  __syncthreads();
  K* dst = out + before_sh;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if ((bal[j] >> lane) & 1u) dst[heads[j * UQ_WARPS + w] + __popc(bal[j] & ((1u << lane) - 1))] = key[j];
}

// skip > 0 (self-test): the first `skip` tiles are left to nobody, and waits give up after spin_limit polls.
template <int KB, int ITEMS>
static cudaError_t unique_launch_items(const void* a, long long n, int xf, void* out, unsigned char* ws, cudaStream_t stream,
                                       unsigned int skip, unsigned int spin_limit)
{
  using K = typename KeyOf<KB>::type;
  const long long ntiles    = (n + UQ_THREADS * ITEMS - 1) / (UQ_THREADS * ITEMS);
  UniqueCtrl* ctrl          = reinterpret_cast<UniqueCtrl*>(ws);
  unsigned long long* state = reinterpret_cast<unsigned long long*>(ws + 256);
  cudaError_t e             = cudaMemsetAsync(ws, 0, 256 + (size_t)ntiles * 8, stream);
  if (e != cudaSuccess) return e;
  if (skip != 0) {
    UniqueCtrl start{};
    start.ticket     = skip;
    start.spin_limit = spin_limit;
    e                = cudaMemcpyAsync(ctrl, &start, sizeof(start), cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
  }
  prof::Scope ps(prof::K_DIST, stream);
  unique_kernel<KB, ITEMS><<<(unsigned int)(ntiles - skip), UQ_THREADS, 0, stream>>>(static_cast<const K*>(a), n, xf, ctrl, state,
                                                                                     static_cast<K*>(out));
  return cudaGetLastError();
}

template <int KB>
static cudaError_t unique_launch(const void* a, long long n, int xf, void* out, unsigned char* ws, cudaStream_t stream)
{
  return n < UQ_LONG ? unique_launch_items<KB, UQ_ITEMS>(a, n, xf, out, ws, stream, 0, 0)
                     : unique_launch_items<KB, 2 * UQ_ITEMS>(a, n, xf, out, ws, stream, 0, 0);
}

// Waits for the launch above and reads its result: a b2s_status_t, and the number of heads.
static int unique_result(const unsigned char* ws, size_t* out_len, cudaStream_t stream)
{
  UniqueCtrl done{};
  if (cudaMemcpyAsync(&done, ws, sizeof(done), cudaMemcpyDeviceToHost, stream) != cudaSuccess) return B2S_ERR_CUDA;
  if (cudaStreamSynchronize(stream) != cudaSuccess) return B2S_ERR_CUDA;
  if (done.status != 0) return (int)done.status;
  *out_len = (size_t)done.total;
  return B2S_OK;
}

}  // namespace b2s

using namespace b2s;

extern "C" {

int b2s_unique_workspace_bytes(size_t n, size_t* bytes)
{
  if (bytes == nullptr) return B2S_ERR_INVALID_ARG;
  const size_t ntiles = (n + UQ_TILE - 1) / UQ_TILE;
  *bytes              = 256 + align_up(ntiles * 8, 256);
  return B2S_OK;
}

int b2s_unique_sorted(int dtype, const void* sorted, size_t n, void* out, size_t* out_len, void* ws,
                      size_t ws_bytes, void* cuda_stream)
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
  if (out_len == nullptr) return B2S_ERR_INVALID_ARG;
  *out_len = 0;
  if (n == 0) return B2S_OK;
  size_t need = 0;
  b2s_unique_workspace_bytes(n, &need);
  if (sorted == nullptr || out == nullptr || out == sorted) return B2S_ERR_INVALID_ARG;
  if (ws == nullptr || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 255u)) return B2S_ERR_WORKSPACE;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  unsigned char* w    = static_cast<unsigned char*>(ws);
  cudaError_t e;
  switch (kb) {
    case 1: e = unique_launch<1>(sorted, (long long)n, xf, out, w, stream); break;
    case 2: e = unique_launch<2>(sorted, (long long)n, xf, out, w, stream); break;
    case 4: e = unique_launch<4>(sorted, (long long)n, xf, out, w, stream); break;
    default: e = unique_launch<8>(sorted, (long long)n, xf, out, w, stream); break;
  }
  if (e != cudaSuccess) return B2S_ERR_CUDA;
  return unique_result(w, out_len, stream);
}

int b2s_selftest_unique_timeout(void* ws, size_t ws_bytes, void* cuda_stream)
{
  // 80 tiles of equal keys, then 40 larger ones: more than one look-back window
  constexpr size_t N = (size_t)UQ_TILE * 80;
  size_t need        = 0;
  b2s_unique_workspace_bytes(N, &need);
  if (ws == nullptr || ws_bytes < need + 2 * N || (reinterpret_cast<uintptr_t>(ws) & 255u)) return B2S_ERR_WORKSPACE;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  unsigned char* w    = static_cast<unsigned char*>(ws);
  unsigned char* keys = w + need;
  size_t heads        = 0;
  if (cudaMemsetAsync(keys, 0, N, stream) != cudaSuccess) return B2S_ERR_CUDA;
  if (unique_launch_items<1, UQ_ITEMS>(keys, (long long)N, XF_UNSIGNED, keys + N, w, stream, 1, 4096) != cudaSuccess) return B2S_ERR_CUDA;
  const int rc = unique_result(w, &heads, stream);
  if (rc != B2S_ERR_TIMEOUT) return rc;
  if (unique_launch_items<1, 2 * UQ_ITEMS>(keys, (long long)N, XF_UNSIGNED, keys + N, w, stream, 1, 4096) != cudaSuccess) return B2S_ERR_CUDA;
  return unique_result(w, &heads, stream);
}
}
