// Lexicographic argsort over several keys along the last axis (the last key is the most
// significant): one stable radix argsort per key, least significant key first, each applied to
// that key gathered through the order found so far.  On 1-D tiles the 32-bit positions travel
// through the radix passes of every key as the payload, so a key costs one gather and one sort;
// nothing leaves the library between the keys (the reference chains argsort tasks and index
// gathers from Python, cupynumeric/_module/ssc_sorting.py:423-444).
//
// Neighbouring keys of at most eight bytes together are one key to the radix passes: the gather puts their
// order-preserving images side by side.  The passes are those of the bytes that differ, as before; a gather, a histogram and
// the passes that find nothing to do are saved for every key that joins another (4000037 rows of float64, int32, int16:
// the two integers 220 -> 150 us), but every pass moves 8-byte keys: see lex_worth.
#include <cuda_runtime.h>

#include "../../include/b200sort.h"
#include "b2s_common.cuh"
#include "b2s_prof.h"

namespace b2s {
bool local_sort_pos32_supported(size_t n);
int local_sort_payload32(int dtype, const void* keys_in, const uint32_t* pay_in, int64_t* idx_out, size_t n,
                         int64_t index_offset, void* ws, size_t ws_bytes, cudaStream_t stream, int out32 = 0);
unsigned int argsort_pass_waves(int kb, size_t n);

static size_t lex_elem_bytes(int dtype)
{
  switch (dtype) {
    case B2S_BOOL: case B2S_INT8: case B2S_UINT8: return 1;
    case B2S_INT16: case B2S_UINT16: case B2S_FLOAT16: return 2;
    case B2S_INT32: case B2S_UINT32: case B2S_FLOAT32: return 4;
    case B2S_INT64: case B2S_UINT64: case B2S_FLOAT64: case B2S_COMPLEX64: return 8;
    case B2S_COMPLEX128: return 16;
    default: return 0;
  }
}

// out[i] = in[row(i) * segment + order[i]]   (order holds positions inside the row)
template <typename T, typename I>
__global__ void lex_gather_kernel(const T* __restrict__ in, const I* __restrict__ order, size_t volume, size_t segment,
                                  T* __restrict__ out)
{
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < volume; i += stride)
    out[i] = in[(i / segment) * segment + (size_t)order[i]];
}

// order_out[i] = order_in[row(i) * segment + pick[i]]
__global__ void lex_compose_kernel(const int64_t* __restrict__ order_in, const int64_t* __restrict__ pick, size_t volume,
                                   size_t segment, int64_t* __restrict__ order_out)
{
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < volume; i += stride)
    order_out[i] = order_in[(i / segment) * segment + (size_t)pick[i]];
}

// Several keys as one 8-byte key: images side by side, the major key uppermost.
struct LexPart {
  const void* keys;
  int bytes, xf, shift;
};
struct LexParts {
  LexPart part[8];
  int n;
};

__device__ __forceinline__ unsigned long long lex_image(const LexPart& p, size_t i)
{
  if (p.bytes == 4) return to_ordered_rt<4>(__ldg(static_cast<const unsigned int*>(p.keys) + i), p.xf);
  if (p.bytes == 2) return to_ordered_rt<2>(__ldg(static_cast<const unsigned short*>(p.keys) + i), p.xf);
  return to_ordered_rt<1>(__ldg(static_cast<const unsigned char*>(p.keys) + i), p.xf);
}

// out[i] = the parts' images of row order[i] (null: i)
__global__ void lex_join_kernel(LexParts parts, const uint32_t* __restrict__ order, size_t volume, unsigned long long* __restrict__ out)
{
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < volume; i += stride) {
    const size_t row     = order != nullptr ? order[i] : i;
    unsigned long long k = 0;
    for (int p = 0; p < parts.n; ++p) k |= lex_image(parts.part[p], row) << parts.part[p].shift;
    out[i] = k;
  }
}

// Whether joining `m` keys of `bytes` together pays.  A joined pass moves 8-byte keys: a round of its resident blocks takes
// 15 us where one of a 4-byte pass takes 18.7 for 1.7 times the keys, so it pays where the rounds are about as many, and what
// joining saves besides, a gather and a histogram per key, tells where both last one round.  Key by key against joined,
// us, every byte differing:
//   int32, int32      3 * 10^5 rows 103 -> 93, 8 * 10^5 210 -> 143, 2 * 10^6 (a round each) 215 -> 205, 3 (one, two) 262 -> 297,
//                     4 (two each) 403 -> 333, 5 (two, three) 439 -> 459, 7 (two, four) 525 -> 602, 16 (five, eight) 1069 -> 1126;
//                     2^20 rows, whose 4-byte tiles are all full, 151 -> 160
//   float32, uint16   2 * 10^6 182 -> 161, 3 219 -> 234, 4 317 -> 262, 16 * 10^6 707 -> 866
//   uint8, uint8      3 * 10^5 45 -> 47, 2 * 10^6 72 -> 81, 16 * 10^6 287 -> 394: short keys have cheap passes of their own
//   eight of uint8    3 * 10^5 198 -> 99, 3 * 10^6 405 -> 327, 7 711 -> 671, 16 * 10^6 1401 -> 1289: many keys save many gathers
static bool lex_worth(int m, size_t bytes, size_t volume)
{
  if (m >= 5) return true;
  if (m == 2 && bytes <= 4) return false;
  return argsort_pass_waves(8, volume) * 4 <= argsort_pass_waves(4, volume) * 5;
}

// Keys k .. k + lex_group() - 1 are sorted as one.
static int lex_group(int nkeys, const int* dtypes, int k, size_t volume)
{
  size_t bytes = 0;
  int m        = 0;
  while (k + m < nkeys && m < 8 && bytes + lex_elem_bytes(dtypes[k + m]) <= 8) bytes += lex_elem_bytes(dtypes[k + m++]);
  return m > 1 && lex_worth(m, bytes, volume) ? m : 1;
}

static int lex_xf(int dtype)
{
  switch (dtype) {
    case B2S_INT8: case B2S_INT16: case B2S_INT32: return XF_SIGNED;
    case B2S_FLOAT16: case B2S_FLOAT32: return XF_FLOAT;
    default: return XF_UNSIGNED;
  }
}

template <typename I>
static cudaError_t lex_gather(size_t eb, const void* in, const I* order, size_t volume, size_t segment, void* out,
                              cudaStream_t stream)
{
  prof::Scope ps(prof::K_FIXUP, stream);
  unsigned int grid = (unsigned int)((volume + 1023) / 1024);
  if (grid > 148 * 16) grid = 148 * 16;
  if (grid == 0) grid = 1;
  switch (eb) {
    case 1: lex_gather_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint8_t*>(in), order, volume, segment, static_cast<uint8_t*>(out)); break;
    case 2: lex_gather_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(in), order, volume, segment, static_cast<uint16_t*>(out)); break;
    case 4: lex_gather_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint32_t*>(in), order, volume, segment, static_cast<uint32_t*>(out)); break;
    case 8: lex_gather_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint64_t*>(in), order, volume, segment, static_cast<uint64_t*>(out)); break;
    default: lex_gather_kernel<<<grid, 256, 0, stream>>>(static_cast<const ulonglong2*>(in), order, volume, segment, static_cast<ulonglong2*>(out)); break;
  }
  return cudaGetLastError();
}

struct LexLayout {
  size_t off_gather, off_ord[2], off_pick, off_sort, sort_bytes, total;
};

// `joined`: with room for joined keys.
static int lex_layout(int nkeys, const int* dtypes, size_t volume, size_t segment, LexLayout* l, bool joined)
{
  size_t max_eb = 0, max_ws = 0;
  if (joined) {
    for (int k = 0; k < nkeys; k += lex_group(nkeys, dtypes, k, volume)) {
      if (lex_group(nkeys, dtypes, k, volume) < 2) continue;
      const int rc = b2s_workspace_bytes(B2S_UINT64, volume, segment, 1, &max_ws);
      if (rc != B2S_OK) return rc;
      max_eb = 8;
    }
  }
  for (int k = 0; k < nkeys; ++k) {
    const size_t eb = lex_elem_bytes(dtypes[k]);
    if (eb == 0) return B2S_ERR_UNSUPPORTED;
    size_t ws = 0;
    const int rc = b2s_workspace_bytes(dtypes[k], volume, segment, 1, &ws);
    if (rc != B2S_OK) return rc;
    max_eb = eb > max_eb ? eb : max_eb;
    max_ws = ws > max_ws ? ws : max_ws;
  }
  size_t off = 0;
  l->off_gather = off; off += align_up(volume * max_eb, 256);
  l->off_ord[0] = off; off += align_up(volume * 8, 256);
  l->off_ord[1] = off; off += align_up(volume * 8, 256);
  l->off_pick   = off; off += align_up(volume * 8, 256);
  l->off_sort   = off; off += align_up(max_ws, 256);
  l->sort_bytes = max_ws;
  l->total      = off;
  return B2S_OK;
}

// Whether neighbouring keys may be sorted as one: 1-D tiles whose order is carried through the passes.
static bool lex_joins(const int* dtypes, int nkeys, size_t volume, size_t segment)
{
  bool some = false;
  for (int k = 0; k < nkeys; ++k) {
    if (dtypes[k] == B2S_COMPLEX128) return false;
    some = some || lex_group(nkeys, dtypes, k, volume) > 1;
  }
  return some && volume == segment && local_sort_pos32_supported(volume);
}

}  // namespace b2s

using namespace b2s;

extern "C" {

int b2s_lexsort_workspace_bytes(int nkeys, const int* dtypes, size_t volume, size_t segment, size_t* bytes)
{
  if (nkeys < 1 || dtypes == nullptr || bytes == nullptr) return B2S_ERR_INVALID_ARG;
  if (volume > 0 && (segment == 0 || volume % segment != 0)) return B2S_ERR_INVALID_ARG;
  LexLayout l{};
  const int rc = lex_layout(nkeys, dtypes, volume, segment ? segment : 1, &l, lex_joins(dtypes, nkeys, volume, segment));
  if (rc == B2S_OK) *bytes = l.total;
  return rc;
}

int b2s_lexsort(int nkeys, const int* dtypes, const void* const* keys, int64_t* idx_out, size_t volume, size_t segment,
                void* ws, size_t ws_bytes, void* cuda_stream)
{
  if (nkeys < 1 || dtypes == nullptr || keys == nullptr) return B2S_ERR_INVALID_ARG;
  if (volume == 0) return B2S_OK;
  if (idx_out == nullptr || segment == 0 || volume % segment != 0) return B2S_ERR_INVALID_ARG;
  for (int k = 0; k < nkeys; ++k)
    if (keys[k] == nullptr) return B2S_ERR_INVALID_ARG;
  LexLayout l{};
  bool joined = lex_joins(dtypes, nkeys, volume, segment);
  int rc      = lex_layout(nkeys, dtypes, volume, segment, &l, joined);
  if (rc != B2S_OK) return rc;
  if (joined && ws_bytes < l.total) {
    // a workspace without that room: key by key
    joined = false;
    rc     = lex_layout(nkeys, dtypes, volume, segment, &l, joined);
    if (rc != B2S_OK) return rc;
  }
  if (ws == nullptr || ws_bytes < l.total || (reinterpret_cast<uintptr_t>(ws) & 255u) != 0) return B2S_ERR_WORKSPACE;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  unsigned char* base = static_cast<unsigned char*>(ws);
  void* gathered      = base + l.off_gather;
  int64_t* ord[2]     = {reinterpret_cast<int64_t*>(base + l.off_ord[0]), reinterpret_cast<int64_t*>(base + l.off_ord[1])};
  int64_t* pick       = reinterpret_cast<int64_t*>(base + l.off_pick);
  void* sort_ws       = base + l.off_sort;
  const int one_d     = volume == segment;

  // 1-D tiles of a size the single radix sort takes (and no 16-byte keys): the order so far rides
  // through the passes as a 32-bit payload
  bool carry = one_d && local_sort_pos32_supported(volume);
  for (int k = 0; k < nkeys; ++k) carry = carry && dtypes[k] != B2S_COMPLEX128;
  if (carry) {
    uint32_t* pos[2] = {reinterpret_cast<uint32_t*>(ord[0]), reinterpret_cast<uint32_t*>(ord[1])};
    int cur = 0;
    for (int k = 0, step = 1; k < nkeys; k += step) {
      step = joined ? lex_group(nkeys, dtypes, k, volume) : 1;
      const bool last = k + step == nkeys;
      const int dtype = step > 1 ? (int)B2S_UINT64 : dtypes[k];
      // joined keys lie in clusters and later keys have few values: the splits give up on them, late (two int32 keys of 100000 and 200
      // values by 1.6 * 10^7 rows 631 us by the passes, 851 after the splits)
      const int how = step > 1 || k > 0 ? IDX_PASSES_ONLY : 0;
      const void* src = keys[k];
      if (step > 1) {
        LexParts parts{};
        int shift = 0;
        for (int i = 0; i < step; ++i) {
          parts.part[i] = LexPart{keys[k + i], (int)lex_elem_bytes(dtypes[k + i]), lex_xf(dtypes[k + i]), shift};
          shift += 8 * parts.part[i].bytes;
        }
        parts.n           = step;
        unsigned int grid = (unsigned int)((volume + 1023) / 1024);
        if (grid > 148 * 16) grid = 148 * 16;
        prof::Scope ps(prof::K_FIXUP, stream);
        lex_join_kernel<<<grid, 256, 0, stream>>>(parts, k > 0 ? pos[cur] : nullptr, volume, static_cast<unsigned long long*>(gathered));
        if (cudaGetLastError() != cudaSuccess) return B2S_ERR_CUDA;
        src = gathered;
      } else if (k > 0) {
        if (lex_gather<uint32_t>(lex_elem_bytes(dtypes[k]), keys[k], pos[cur], volume, segment, gathered, stream) != cudaSuccess)
          return B2S_ERR_CUDA;
        src = gathered;
      }
      if (last) {
        rc = local_sort_payload32(dtype, src, k == 0 ? nullptr : pos[cur], idx_out, volume, 0, sort_ws, l.sort_bytes, stream, how);
      } else {
        rc = local_sort_payload32(dtype, src, k == 0 ? nullptr : pos[cur], reinterpret_cast<int64_t*>(pos[cur ^ 1]), volume, 0,
                                  sort_ws, l.sort_bytes, stream, how | IDX_32);
        cur ^= 1;
      }
      if (rc != B2S_OK) return rc;
    }
    return B2S_OK;
  }

  // every other shape: argsort of the gathered key, then the order so far taken through it
  int cur = 0;
  for (int k = 0; k < nkeys; ++k) {
    const bool last = k == nkeys - 1;
    if (k == 0) {
      rc = b2s_local_sort(dtypes[0], keys[0], nullptr, last ? idx_out : ord[cur], volume, segment, 0, one_d, 1, sort_ws, l.sort_bytes, stream);
      if (rc != B2S_OK) return rc;
      continue;
    }
    if (lex_gather<int64_t>(lex_elem_bytes(dtypes[k]), keys[k], ord[cur], volume, segment, gathered, stream) != cudaSuccess) return B2S_ERR_CUDA;
    rc = b2s_local_sort(dtypes[k], gathered, nullptr, pick, volume, segment, 0, one_d, 1, sort_ws, l.sort_bytes, stream);
    if (rc != B2S_OK) return rc;
    {
      prof::Scope ps(prof::K_FIXUP, stream);
      unsigned int grid = (unsigned int)((volume + 1023) / 1024);
      if (grid > 148 * 16) grid = 148 * 16;
      lex_compose_kernel<<<grid, 256, 0, stream>>>(ord[cur], pick, volume, segment, last ? idx_out : ord[cur ^ 1]);
      if (cudaGetLastError() != cudaSuccess) return B2S_ERR_CUDA;
    }
    cur ^= 1;
  }
  return B2S_OK;
}
}
