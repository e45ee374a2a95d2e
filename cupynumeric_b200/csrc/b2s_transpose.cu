// Transposes the last two dimensions of a dense array: the copy in front of a sort along another axis than
// the last (the reference swaps the axes and copies, cupynumeric/_thunk/_sort.py:50-76).
#include "../../include/b200sort.h"
#include "b2s_common.cuh"
#include "b2s_prof.h"

namespace b2s {

constexpr int TR_TILE = 64;   // a tile is TR_TILE x TR_TILE elements
constexpr int TR_ROWS = 8;    // rows that the CTA's 256 threads take at a time, half a tile row each

// Bound by HBM: every element is read and written once, with 32 consecutive elements per warp on both
// sides; the tile goes through shared memory with one spare element per row, so that its columns hit
// all banks.  Copying through strides instead reads a memory sector per element: the whole sort of 257
// float32 columns of 100003 went from 669 to 607 us with this kernel and the faster row histograms.
template <typename T>
__global__ void __launch_bounds__(256)
transpose_kernel(const T* __restrict__ in, T* __restrict__ out, unsigned long long rows, unsigned long long cols,
                 unsigned int tiles_x, unsigned int tiles_y)
{
  __shared__ T tile[TR_TILE][TR_TILE + 1];
  unsigned long long b     = blockIdx.x;
  const unsigned int tx    = (unsigned int)(b % tiles_x);
  b /= tiles_x;
  const unsigned int ty    = (unsigned int)(b % tiles_y);
  const unsigned long long batch = b / tiles_y;
  in += batch * rows * cols;
  out += batch * rows * cols;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned long long r0 = (unsigned long long)ty * TR_TILE, c0 = (unsigned long long)tx * TR_TILE;
#pragma unroll
  for (int i = 0; i < TR_TILE; i += TR_ROWS)
#pragma unroll
    for (int h = 0; h < TR_TILE; h += 32) {
      const unsigned long long r = r0 + i + w, c = c0 + h + lane;
      if (r < rows && c < cols) tile[i + w][h + lane] = in[r * cols + c];
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TR_TILE; i += TR_ROWS)
#pragma unroll
    for (int h = 0; h < TR_TILE; h += 32) {
      const unsigned long long c = c0 + i + w, r = r0 + h + lane;
      if (r < rows && c < cols) out[c * rows + r] = tile[h + lane][i + w];
    }
}

template <typename T>
static cudaError_t transpose_launch(const void* in, void* out, size_t batch, size_t rows, size_t cols, cudaStream_t stream)
{
  const size_t tx = (cols + TR_TILE - 1) / TR_TILE, ty = (rows + TR_TILE - 1) / TR_TILE;
  prof::Scope ps(prof::K_FIXUP, stream);
  transpose_kernel<T><<<(unsigned int)(batch * tx * ty), 256, 0, stream>>>(static_cast<const T*>(in), static_cast<T*>(out), rows, cols,
                                                                          (unsigned int)tx, (unsigned int)ty);
  return cudaGetLastError();
}

}  // namespace b2s

using namespace b2s;

extern "C" int b2s_transpose(size_t elem_bytes, const void* in, void* out, size_t batch, size_t rows, size_t cols, void* cuda_stream)
{
  if (batch == 0 || rows == 0 || cols == 0) return B2S_OK;
  if (in == nullptr || out == nullptr || in == out) return B2S_ERR_INVALID_ARG;
  const size_t tx = (cols + TR_TILE - 1) / TR_TILE, ty = (rows + TR_TILE - 1) / TR_TILE;
  if (tx > 0x7FFFFFFFull / ty || batch > 0x7FFFFFFFull / (tx * ty)) return B2S_ERR_UNSUPPORTED;  // tiles are a 31-bit grid
  if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % (elem_bytes ? elem_bytes : 1)) return B2S_ERR_INVALID_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  cudaError_t e;
  switch (elem_bytes) {
    case 1: e = transpose_launch<uint8_t>(in, out, batch, rows, cols, s); break;
    case 2: e = transpose_launch<uint16_t>(in, out, batch, rows, cols, s); break;
    case 4: e = transpose_launch<uint32_t>(in, out, batch, rows, cols, s); break;
    case 8: e = transpose_launch<uint64_t>(in, out, batch, rows, cols, s); break;
    default: return B2S_ERR_UNSUPPORTED;
  }
  return e == cudaSuccess ? B2S_OK : B2S_ERR_CUDA;
}
