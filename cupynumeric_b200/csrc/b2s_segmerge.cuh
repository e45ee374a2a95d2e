// Segmented sort of rows that fit in shared memory (513 to 8192 elements of 4 or 8 bytes), one CTA per row,
// one read and one write of HBM per element.  Two methods share the kernel:
//
// * Buckets.  A linear function of the key that never inverts the order maps the row's keys to twice as
//   many buckets as there are keys; counting and a scan give every bucket its place, and what is left is
//   the order inside the buckets.  If none holds more than nine keys, two sorting networks over 16
//   neighbours (the second one halfway between the first one's blocks) finish the row.  About 160 thread
//   instructions per 8-byte key.
// * Merging, for rows whose keys crowd: every thread sorts 16 consecutive elements in registers, then
//   log2(threads) rounds of pairwise merge-path merges run in one shared-memory buffer; about 480
//   instructions per 8-byte key.  A row finds out after its counting step, a sixth of the work of merging.
//
// Both are bound by instruction issue and the shared-memory pipe, not by HBM.  2^24 elements with NaNs and
// duplicates, merging only -> buckets: float64 rows of 4096 0.390 -> 0.171 ms, of 1000 0.321 -> 0.146;
// float32 with positions, rows of 2000 0.345 -> 0.135 ms.  The registers the compiler may use (64 for 512
// threads, 80 for 256, 100 below) are the measured best per block size for the sort of keys and for 4-byte keys;
// 8-byte keys with positions need 124 KB of shared memory for 512 threads, so that one block is all an SM
// takes, and get the registers of two (2^22 int64 in rows of 8192, three values, argsort 6 to 18 % faster).
//
// A row is merged where its keys crowd: heavy duplicates in an argsort, an outlier that takes most buckets for
// itself, doubles whose spread is below 1e-33 or above float32's range (the scale is computed in float32).
//
// Stands, like the on-chip radix kernel beside it, for cub::DeviceSegmentedRadixSort and the
// short-segment thrust sort (src/cupynumeric/sort/cub_sort.cuh:73-107,145-184,
// src/cupynumeric/sort/thrust_sort.cuh:61-123).
//
// Keys are merged as their order-preserving unsigned images (to_ordered).  For floats that image
// folds -0.0 onto +0.0 and every NaN onto one value, so that the stable merge leaves them in input
// order; the way back yields +0.0 and the canonical quiet NaN, and a row that held a -0.0 or
// another NaN pattern gets those elements rewritten from the input, in input order, afterwards.
#pragma once

#include "b2s_common.cuh"

#include <type_traits>

namespace b2s {

constexpr int SM_VT     = 16;  // elements per thread
constexpr int SM_BUCKET = 9;   // most keys of a bucket: half a block of SM_VT, and one

// shared-memory index of logical position i: one spare slot per 16 keeps a warp's blocked accesses
// (stride 16) off a single bank
__device__ __host__ __forceinline__ constexpr int smpad(int i) { return i + (i >> 4); }
static_assert(SM_VT == 16, "the padding rule and the counters assume 16 elements per thread");

template <int KB> struct SmWord { using type = unsigned long long; };
template <> struct SmWord<4> { using type = unsigned int; };

// inverse of to_ordered: integers exactly; floats up to the folding described above
template <int KB>
__device__ __forceinline__ typename KeyOf<KB>::type sm_from_ordered(typename KeyOf<KB>::type o, int xf)
{
  using K        = typename KeyOf<KB>::type;
  constexpr K SB = (K)((K)1 << (8 * KB - 1));
  if (xf == XF_UNSIGNED) return o;
  if (xf == XF_SIGNED) return (K)(o ^ SB);
  constexpr K QNAN = KB == 4 ? (K)0x7FC00000u : (K)0x7FF8000000000000ull;
  if (o == (K)~(K)0) return QNAN;
  return (o & SB) ? (K)(o ^ SB) : (K)~o;
}

// rows whose float keys need the rewrite: a -0.0, or a NaN that is not the canonical quiet NaN
template <int KB>
__device__ __forceinline__ bool sm_is_special(typename KeyOf<KB>::type raw, int xf)
{
  using K = typename KeyOf<KB>::type;
  if (xf != XF_FLOAT) return false;
  constexpr K SB   = (K)((K)1 << (8 * KB - 1));
  constexpr K EXP  = KB == 4 ? (K)0x7F800000u : (K)0x7FF0000000000000ull;
  constexpr K QNAN = KB == 4 ? (K)0x7FC00000u : (K)0x7FF8000000000000ull;
  const K mag      = (K)(raw & (K)~SB);
  return raw == SB || (mag > EXP && raw != QNAN);
}
template <int KB>
__device__ __forceinline__ bool sm_is_zero(typename KeyOf<KB>::type raw)
{
  using K = typename KeyOf<KB>::type;
  return (K)(raw << 1) == 0;
}
template <int KB>
__device__ __forceinline__ bool sm_is_nan(typename KeyOf<KB>::type raw)
{
  using K         = typename KeyOf<KB>::type;
  constexpr K SB  = (K)((K)1 << (8 * KB - 1));
  constexpr K EXP = KB == 4 ? (K)0x7F800000u : (K)0x7FF0000000000000ull;
  return (K)(raw & (K)~SB) > EXP;
}

// Batcher's odd-even merge sort of N (a power of two) elements from blocks of FROM elements that are
// sorted already (1: from scratch; N / 2: one merge of two halves; K. E. Batcher, "Sorting networks and
// their applications", 1968).  cmp_swap(i, j) puts elements i < j in order.
template <int N, int FROM, typename CmpSwap>
__device__ __forceinline__ void odd_even_merge_sort(CmpSwap cmp_swap)
{
#pragma unroll
  for (int p = FROM; p < N; p <<= 1) {
#pragma unroll
    for (int k = p; k >= 1; k >>= 1) {
#pragma unroll
      for (int j = 0; j + k < N; ++j) {
        // j is the lower end of a comparator where it lies in the lower half of a block of 2k that
        // starts k % p after a multiple of 2k, and both ends lie in the same block of 2p
        const int off = j - k % p;
        if (off >= 0 && off % (2 * k) < k && j / (2 * p) == (j + k) / (2 * p)) cmp_swap(j, j + k);
      }
    }
  }
}

template <int KB, bool PAIRS, int THREADS> struct SegMergeSmem {
  static constexpr int TILE   = THREADS * SM_VT;
  static constexpr int PADDED = TILE + TILE / 16 + 1;
  // 4-byte keys with payload travel as one 64-bit word (image << 32 | position); 8-byte keys with
  // payload keep the positions in a 16-bit array beside the images
  static constexpr bool PACK   = PAIRS && KB == 4;
  static constexpr bool SIDE   = PAIRS && KB == 8;
  static constexpr size_t WB   = (KB == 8 || PACK) ? 8 : 4;
  // two buckets per element, a 16-bit count or place each; four spare words after every 32
  static constexpr int NB          = 2 * TILE;
  static constexpr size_t OFF_PAY  = ((size_t)PADDED * WB + 15) / 16 * 16;
  static constexpr size_t OFF_CNT  = (OFF_PAY + (SIDE ? (size_t)PADDED * 2 : 0) + 15) / 16 * 16;
  static constexpr size_t CNT_BYTES = (size_t)NB * 2 + (size_t)NB / 64 * 16;
  static constexpr size_t OFF_MISC = OFF_CNT + CNT_BYTES;
  static constexpr size_t BYTES    = OFF_MISC + 64 + (THREADS / 32) * 16;
};

// A row's bucket function: maps keys to 0 .. NB - 1 without ever inverting the sort order, equal keys to
// equal buckets.  Integers (and complex images): linear in the image.  Floats: linear in the value, since
// the image is logarithmic; infinities and NaNs go to the end buckets.
template <int KB, int NB> struct RowBuckets {
  using K = typename KeyOf<KB>::type;
  using F = typename std::conditional<KB == 8, double, float>::type;
  // images of finite floats, compared by their upper 32 bits
  static constexpr unsigned int FIN_LO = KB == 8 ? 0x00100000u : 0x00800000u;  // lowest finite
  static constexpr unsigned int FIN_N  = 0u - 2u * FIN_LO;                     // as many upper words
  F fmin, fscale;
  K imin;
  unsigned int mult;
  unsigned int range;  // exact: the last bucket in use
  int shift;
  bool ok, exact;  // exact: a bucket holds equal keys only

  static __device__ __forceinline__ F value(K bits)
  {
    if constexpr (KB == 8) return __longlong_as_double((long long)bits); else return __uint_as_float((unsigned int)bits);
  }
  static __device__ __forceinline__ unsigned int upper(K o) { return KB == 8 ? (unsigned int)((unsigned long long)o >> 32) : (unsigned int)o; }

  // from the smallest and largest upper words of the finite images
  __device__ __forceinline__ void from_floats(unsigned int lo, unsigned int hi)
  {
    const K a = KB == 8 ? (K)((unsigned long long)lo << 32) : (K)lo;
    const K b = KB == 8 ? (K)(((unsigned long long)hi << 32) | 0xFFFFFFFFull) : (K)hi;
    fmin      = value(sm_from_ordered<KB>(a, XF_FLOAT));
    // a rough quotient will do: any positive scale keeps the order, and buckets are clamped
    fscale    = (F)__fdividef((float)NB, (float)(value(sm_from_ordered<KB>(b, XF_FLOAT)) - fmin));
    ok        = lo <= hi && fscale > (F)0 && fscale < (F)1e37f;
    exact     = false;
  }
  __device__ __forceinline__ unsigned int bucket_float(K o) const
  {
    const unsigned int u = upper(o);
    const K flip         = (K)((K)1 << (8 * KB - 1)) | (K)~(K)((typename std::make_signed<K>::type)o >> (8 * KB - 1));
    const K raw          = (K)(o ^ flip);  // the key's bits, but for signed zeros and NaNs
    unsigned int b;
    // the addition of 2^23 (2^52) leaves the rounded product in the low bits
    if constexpr (KB == 8) b = (unsigned int)__double_as_longlong(fma(value(raw) - fmin, fscale, 4503599627370496.0));
    else b = __float_as_uint(fmaf(value(raw) - fmin, fscale, 8388608.0f)) & 0x7FFFFFu;
    b = min(b, (unsigned int)NB - 1);
    return u - FIN_LO < FIN_N ? b : (u >> 31) * (NB - 1);
  }
  // from the smallest and largest images
  __device__ __forceinline__ void from_images(K lo, K hi)
  {
    const unsigned long long span = (unsigned long long)hi - (unsigned long long)lo;
    imin  = lo;
    range = (unsigned int)span;
    exact = span < NB;
    shift = KB == 8 && (span >> 32) != 0 ? 32 - __clz((int)(span >> 32)) : 0;
    mult  = exact ? 0u : __float2uint_rz(__fdividef((float)NB * 4294967296.0f, (float)(unsigned int)(span >> shift)));
    ok    = true;
  }
  __device__ __forceinline__ unsigned int bucket_image(K o) const
  {
    const unsigned int x = (unsigned int)((unsigned long long)(K)(o - imin) >> shift);
    return exact ? x : min(__umulhi(x, mult), (unsigned int)NB - 1);
  }
};

// How a kernel turns keys into images: integers share one form (flip is the sign bit or nothing).
enum : int { SM_INT = 0, SM_FLOAT = 1, SM_COMPLEX = 2 };

// One CTA sorts one row at a time (grid-stride over rows); seg_len <= THREADS * 16.
template <int KB, bool PAIRS, int THREADS, int FORM>
__global__ void __launch_bounds__(THREADS, THREADS == 512 ? (PAIRS && KB == 8 ? 1 : 2) : THREADS == 256 ? 3 : THREADS == 128 ? 5 : 10)
segmerge_kernel(const typename KeyOf<KB>::type* in, typename KeyOf<KB>::type* out /* may be `in`: no __restrict__ */, int64_t* idx_out, unsigned int seg_len, unsigned long long nseg, int xf, int64_t index_offset,
                unsigned int* __restrict__ status)
{
  using K = typename KeyOf<KB>::type;
  using S = SegMergeSmem<KB, PAIRS, THREADS>;
  using W = typename SmWord<S::WB>::type;
  constexpr int TILE  = S::TILE;
  constexpr int WARPS = THREADS / 32;
  constexpr bool PACK = S::PACK, SIDE = S::SIDE;
  extern __shared__ __align__(16) unsigned char smem[];
  W* sw                  = reinterpret_cast<W*>(smem);
  unsigned short* sp     = reinterpret_cast<unsigned short*>(smem + S::OFF_PAY);
  unsigned int* misc     = reinterpret_cast<unsigned int*>(smem + S::OFF_MISC);   // [0..3] block bounds
  unsigned int* wsum     = misc + 16;                                             // per-warp counts and bounds
  unsigned char* cnt     = smem + S::OFF_CNT;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = tid * SM_VT;
  constexpr W WMAX = (W)~(W)0;
  const K flip = xf == XF_SIGNED ? (K)((K)1 << (8 * KB - 1)) : (K)0;
  auto image = [&](K raw) {
    if constexpr (FORM == SM_FLOAT) return to_ordered<KB, XF_FLOAT>(raw);
    else if constexpr (FORM == SM_COMPLEX) return to_ordered<8, XF_CFLOAT>(raw);
    else return (K)(raw ^ flip);
  };
  auto from_image = [&](K o) {
    if constexpr (FORM == SM_FLOAT) return sm_from_ordered<KB>(o, XF_FLOAT);
    else return (K)(o ^ flip);
  };

  if (blockIdx.x == 0 && tid == 0) *status = 0;  // nothing here waits, so nothing can time out
  for (unsigned long long seg = blockIdx.x; seg < nseg; seg += gridDim.x) {
    const K* src = in + seg * seg_len;
    // ---- load: consecutive threads read consecutive elements ----
    int special = 0;
    K img[SM_VT];
#pragma unroll
    for (int j = 0; j < SM_VT; ++j) {
      const int e = j * THREADS + tid;
      img[j]      = (unsigned int)e < seg_len ? src[e] : (K)0;
    }
#pragma unroll
    for (int j = 0; j < SM_VT; ++j) {
      const K raw = img[j];
      img[j]      = image(raw);
      if constexpr (FORM == SM_FLOAT && !PAIRS) {
        // only zeros and NaNs can be special
        const unsigned int u = RowBuckets<KB, S::NB>::upper(img[j]);
        if (u == 0xFFFFFFFFu || u == 0x80000000u) special |= sm_is_special<KB>(raw, XF_FLOAT) ? 1 : 0;
      }
    }
    auto word_of = [&](K o, int e) { return PACK ? (W)(((unsigned long long)o << 32) | (unsigned int)e) : (W)o; };
    W key[SM_VT];
    unsigned int pay[SIDE ? SM_VT : 1];
    auto cmp_swap = [&](int a, int b) {
      const W x = key[a], y = key[b];
      if (SIDE) {
        const unsigned int p = pay[SIDE ? a : 0], q = pay[SIDE ? b : 0];
        const bool sw_ = y < x || (y == x && q < p);
        key[a] = sw_ ? y : x;
        key[b] = sw_ ? x : y;
        pay[SIDE ? a : 0] = sw_ ? q : p;
        pay[SIDE ? b : 0] = sw_ ? p : q;
      } else {
        const bool sw_ = y < x;
        key[a] = sw_ ? y : x;
        key[b] = sw_ ? x : y;
      }
    };
    auto read_words = [&](int at) {
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        key[j] = sw[smpad(at + j)];
        if (SIDE) pay[SIDE ? j : 0] = sp[smpad(at + j)];
      }
    };
    auto write_words = [&](int at) {
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        sw[smpad(at + j)] = key[j];
        if (SIDE) sp[smpad(at + j)] = (unsigned short)pay[SIDE ? j : 0];
      }
    };

    // ---- the row's bounds, then a bucket per key ----
    bool sorted = false;
    {
      constexpr int NB = S::NB;
      RowBuckets<KB, NB> rb;
      for (int i = tid; i < (int)(S::CNT_BYTES / 16); i += THREADS) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (FORM == SM_FLOAT) {
        unsigned int lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
        for (int j = 0; j < SM_VT; ++j) {
          if ((unsigned int)(j * THREADS + tid) < seg_len) {
            const unsigned int u = RowBuckets<KB, NB>::upper(img[j]);
            if (u - RowBuckets<KB, NB>::FIN_LO < RowBuckets<KB, NB>::FIN_N) {
              lo = min(lo, u);
              hi = max(hi, u);
            }
          }
        }
        lo = __reduce_min_sync(0xFFFFFFFFu, lo);
        hi = __reduce_max_sync(0xFFFFFFFFu, hi);
        if (lane == 0) {
          wsum[2 * warp]     = lo;
          wsum[2 * warp + 1] = hi;
        }
        special = __syncthreads_or(special);
        for (int w = 0; w < WARPS; ++w) {
          lo = min(lo, wsum[2 * w]);
          hi = max(hi, wsum[2 * w + 1]);
        }
        rb.from_floats(lo, hi);
      } else {
        K lo = (K)~(K)0, hi = 0;
#pragma unroll
        for (int j = 0; j < SM_VT; ++j) {
          if ((unsigned int)(j * THREADS + tid) < seg_len) {
            lo = img[j] < lo ? img[j] : lo;
            hi = img[j] > hi ? img[j] : hi;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const K l = __shfl_xor_sync(0xFFFFFFFFu, lo, o), h = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
          lo        = l < lo ? l : lo;
          hi        = h > hi ? h : hi;
        }
        K* bounds = reinterpret_cast<K*>(wsum);
        if (lane == 0) {
          bounds[2 * warp]     = lo;
          bounds[2 * warp + 1] = hi;
        }
        __syncthreads();
        for (int w = 0; w < WARPS; ++w) {
          const K l = bounds[2 * w], h = bounds[2 * w + 1];
          lo        = l < lo ? l : lo;
          hi        = h > hi ? h : hi;
        }
        rb.from_images(lo, hi);
      }
      // equal keys of a sort need no order among themselves: a row with fewer values than buckets is
      // done once it is counted
      const bool counted = !PAIRS && rb.exact;
      unsigned int br[SM_VT];  // where the bucket's counter is | rank in the bucket << 16
      // fewer values than a ninth of the row: some bucket is too full, whatever the row holds
      const bool full = PAIRS && rb.exact && (rb.range + 1) * SM_BUCKET < seg_len;
      int over = rb.ok && !full ? 0 : 1;
      if (!over) {
#pragma unroll
        for (int j = 0; j < SM_VT; ++j) {
          if ((unsigned int)(j * THREADS + tid) < seg_len) {
            const unsigned int b  = FORM == SM_FLOAT ? rb.bucket_float(img[j]) : rb.bucket_image(img[j]);
            const unsigned int at = b * 2 + (b >> 6) * 16;  // of the bucket's 16 bits
            const unsigned int h  = (b & 1u) * 16u;
            const unsigned int r  = (atomicAdd(reinterpret_cast<unsigned int*>(cnt + (at & ~3u)), 1u << h) >> h) & 0xFFFFu;
            over |= r >= (unsigned int)SM_BUCKET ? 1 : 0;
            br[j] = at | (r << 16);
          }
        }
      }
      if (counted) over = 0;
      sorted = !__syncthreads_or(over);
      if (sorted) {
        // counts -> places: my 32 buckets, then the threads before me
        uint4* mine = reinterpret_cast<uint4*>(cnt) + 4 * tid + (tid >> 1);
        unsigned int sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 c = mine[j];
          sum += c.x + c.y + c.z + c.w;  // two counts per word, added side by side
        }
        sum = (sum & 0xFFFFu) + (sum >> 16);
        unsigned int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        unsigned int run = incl - sum;
        for (int w = 0; w < warp; ++w) run += wsum[w];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 c = mine[j];
          auto place = [&](unsigned int& two) {
            const unsigned int first_n = two & 0xFFFFu, both = first_n + (two >> 16);
            two = run | ((run + first_n) << 16);
            run += both;
          };
          place(c.x);
          place(c.y);
          place(c.z);
          place(c.w);
          mine[j] = c;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SM_VT; ++j) {
          const int e = j * THREADS + tid;
          if ((unsigned int)e < seg_len) {
            const unsigned int p = *reinterpret_cast<const unsigned short*>(cnt + (br[j] & 0xFFFFu)) + (br[j] >> 16);
            sw[smpad(p)] = word_of(img[j], e);
            if (SIDE) sp[smpad(p)] = (unsigned short)e;
          } else {
            sw[smpad(e)] = WMAX;
            if (SIDE) sp[smpad(e)] = (unsigned short)e;
          }
        }
        __syncthreads();
        if (!counted) {
          // Elements are at most SM_BUCKET - 1 places from where they belong.  Sorting every block of
          // 16 settles the buckets inside a block; the windows halfway between the blocks settle the
          // buckets that lie across a block's end, whose parts reach at most 8 into either block.
          read_words(first);
          odd_even_merge_sort<SM_VT, 1>(cmp_swap);
          write_words(first);
          __syncthreads();
          if (tid < THREADS - 1) {
            read_words(first + SM_VT / 2);
            odd_even_merge_sort<SM_VT, SM_VT / 2>(cmp_swap);
            write_words(first + SM_VT / 2);
          }
          __syncthreads();
        }
      }
    }

    // ---- rows whose keys crowd in few buckets: merge sort, from runs of 16 per thread ----
    if (!sorted) {
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        const int e  = j * THREADS + tid;
        sw[smpad(e)] = (unsigned int)e < seg_len ? word_of(img[j], e) : WMAX;
        if (SIDE) sp[smpad(e)] = (unsigned short)e;
      }
      __syncthreads();
      read_words(first);
      // rows of one value (which the buckets of floats and complex keys do not tell from crowded ones) and rows
      // that come in order have nothing to sort
      int back = tid < THREADS - 1 && sw[smpad(first + SM_VT)] < key[SM_VT - 1] ? 1 : 0;
#pragma unroll
      for (int j = 0; j + 1 < SM_VT; ++j) back |= key[j + 1] < key[j] ? 1 : 0;
      sorted = !__syncthreads_or(back);  // (and everybody holds its elements: the buffer may be rewritten)
      if (!sorted) {
        odd_even_merge_sort<SM_VT, 1>(cmp_swap);
        write_words(first);
        __syncthreads();
      }
    }
    // ---- merge rounds: runs of `run` elements, pairwise; my 16 outputs start at `first` ----
    for (int run = sorted ? TILE : SM_VT; run < TILE; run <<= 1) {
      const int pbase = first & ~(2 * run - 1);
      const int diag  = first - pbase;
      const int a0 = pbase, b0 = pbase + run;
      int lo = max(0, diag - run), hi = min(diag, run);
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sw[smpad(a0 + mid)] <= sw[smpad(b0 + diag - 1 - mid)]) lo = mid + 1; else hi = mid;
      }
      int ia = lo, ib = diag - lo;
      W ka = ia < run ? sw[smpad(a0 + ia)] : WMAX, kb = ib < run ? sw[smpad(b0 + ib)] : WMAX;
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        // on equal words the lower run goes first; an exhausted run shows the largest word, which only its like
        // ties with (beside positions of their own that would matter, so it must not win there)
        const bool take_a = SIDE ? ib >= run || (ia < run && ka <= kb) : ka <= kb;
        key[j]            = take_a ? ka : kb;
        if (SIDE) pay[j] = sp[smpad(take_a ? a0 + ia : b0 + ib)];
        ia += take_a ? 1 : 0;
        ib += take_a ? 0 : 1;
        const int nxt = take_a ? a0 + ia : b0 + ib;
        const bool ok = take_a ? ia < run : ib < run;
        const W v     = ok ? sw[smpad(nxt)] : WMAX;
        ka = take_a ? v : ka;
        kb = take_a ? kb : v;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        sw[smpad(first + j)] = key[j];
        if (SIDE) sp[smpad(first + j)] = (unsigned short)pay[j];
      }
      __syncthreads();
    }

    // ---- rows with -0.0 or unusual NaNs (sorts of keys): the elements the image folded are
    // fetched from the input in input order, to be written over their blocks after the store ----
    K fix_raw[FORM == SM_FLOAT && !PAIRS ? SM_VT : 1];
    int fix_at[FORM == SM_FLOAT && !PAIRS ? SM_VT : 1];
    int nfix = 0;
    if constexpr (FORM == SM_FLOAT && !PAIRS) if (special) {
      if (tid == 0) {
        // block of zeros [z0, z1) and start of the NaN block in the sorted images
        const W zimg = (W)image((K)0);
        int a = 0, b = (int)seg_len;
        while (a < b) { const int m = (a + b) >> 1; if (sw[smpad(m)] < zimg) a = m + 1; else b = m; }
        misc[0] = a;
        a = 0; b = (int)seg_len;
        while (a < b) { const int m = (a + b) >> 1; if (sw[smpad(m)] < WMAX) a = m + 1; else b = m; }
        misc[1] = a;
      }
      // my 16 consecutive input elements: how many zeros / NaNs come before them
      unsigned int cz = 0, cn = 0;
      K raw[SM_VT];
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        raw[j] = (unsigned int)(first + j) < seg_len ? src[first + j] : (K)1;
        cz += sm_is_zero<KB>(raw[j]) ? 1u : 0u;
        cn += sm_is_nan<KB>(raw[j]) ? 1u : 0u;
      }
      unsigned int packed = cz | (cn << 16), incl = packed;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
      }
      if (lane == 31) wsum[warp] = incl;
      __syncthreads();
      unsigned int before = incl - packed;
      for (int w = 0; w < warp; ++w) before += wsum[w];
      int rz = (int)(before & 0xFFFFu) + (int)misc[0], rn = (int)(before >> 16) + (int)misc[1];
#pragma unroll
      for (int j = 0; j < SM_VT; ++j) {
        const bool z = sm_is_zero<KB>(raw[j]), nn = sm_is_nan<KB>(raw[j]);
        if (z || nn) {
          fix_raw[nfix] = raw[j];
          fix_at[nfix]  = z ? rz : rn;
          ++nfix;
        }
        rz += z ? 1 : 0;
        rn += nn ? 1 : 0;
      }
    }

    // ---- store (coalesced) ----
    K* dst = out ? out + seg * seg_len : nullptr;
    if (!PAIRS) {
      for (int e = tid; e < (int)seg_len; e += THREADS) dst[e] = from_image((K)sw[smpad(e)]);
      if (special) {
        __syncthreads();  // the plain store of the row is complete
        for (int f = 0; f < nfix; ++f) dst[fix_at[f]] = fix_raw[f];
      }
    } else {
      int64_t* idst = idx_out ? idx_out + seg * seg_len : nullptr;
      if (dst != nullptr) {
        // keys as well: fetched through the positions before anything of the row is written
        // (the output may be the input)
        K kraw[SM_VT];
#pragma unroll
        for (int j = 0; j < SM_VT; ++j) {
          const int e = j * THREADS + tid;
          if (e < (int)seg_len) kraw[j] = src[PACK ? (unsigned int)sw[smpad(e)] : (unsigned int)sp[smpad(e)]];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SM_VT; ++j) {
          const int e = j * THREADS + tid;
          if (e < (int)seg_len) dst[e] = kraw[j];
        }
      }
      for (int e = tid; idx_out != nullptr && e < (int)seg_len; e += THREADS) {
        const unsigned int p = PACK ? (unsigned int)sw[smpad(e)] : (unsigned int)sp[smpad(e)];
        idst[e]              = (int64_t)p + index_offset;
      }
    }
    __syncthreads();  // all reads of shared memory are done before the next row's load
  }
}

}  // namespace b2s
