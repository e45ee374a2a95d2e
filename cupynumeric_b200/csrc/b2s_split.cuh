// Splitting sort of long arrays and long rows (4- and 8-byte keys): the keys are moved once or twice into
// buckets of ascending key ranges until a bucket fits a block's shared memory, and sorted there.
//
// Why: a stable 8-bit radix pass costs 105 to 115 thread instructions per key, most of them for ranking
// equal digits in input order, and 4-byte keys need four of them.  A split needs no order inside a bucket: one
// shared-memory atomic takes the place of the ranking (53 instructions per int32 key), two splits of a few hundred
// buckets each leave rows of a few thousand keys, and the last step orders those by (key, position), so that
// an argsort is stable although the splits are not.  Equal keys of a sort have nothing to be told apart by.
// 2^24 int32 keys: four passes of 84 us and a histogram of 26 against two splits of 51 and 57, counts of 21 and 18 and leaves
// of 68; 2^28 int64 Zipf keys 7174 -> 3120 us.  Pairs of 4-byte keys, with four passes to save, gain least (float32 argsort of
// 2 * 10^7 keys 583 -> 517 us).
//
// Steps, all on the stream, with no word back to the host:
//   sample    per segment (the array, a row, or a bucket of the first split): bounds of 4096 keys, from
//             which a monotone function of the key to C cells is chosen (SplitMap)
//   cells     counts the keys per cell
//   pack      cuts the cells into buckets of at most `cap` keys each, so that the split has exact places
//   split     moves keys (and positions) to their buckets
//   leaves    sorts every bucket of the last split and writes the result
//
// A cell that holds a single value of which a sort has many copies is not moved at all: its place in the
// result is filled in at the end.  What cannot be cut finely enough (a heavily repeated key of an argsort,
// values that crowd at a scale of their own) or needs input order among keys of equal image (zeros of both signs, NaNs of
// several patterns) is left to the radix passes: `route` in the control block says so before anything of the output is
// written, and the radix kernels, launched behind, return at once where it says otherwise.
#pragma once

#include "b2s_common.cuh"
#include "b2s_prof.h"
#include "b2s_segmerge.cuh"
#include "b2s_split_plan.cuh"

namespace b2s {

// How the keys of a level are held: as they come (integers, floats), or, after the first split of floats, as their images.
enum : int { FORM_INT = 0, FORM_FLOAT = 1, FORM_IMAGE = 2 };
constexpr unsigned short LUT_DROP = 0xFFFF;
constexpr int SPLIT_THREADS       = 512;
constexpr int SPLIT_SAMPLES       = 4096;  // of a segment of the input
constexpr int SPLIT_SAMPLES_NEXT  = 2048;  // of a bucket of the first split
// Places for the samples' fingerprints by how often the samples are drawn: of argsorts, whose copies decide (below), twice from
// 1.6 * 10^7 keys on, where a dozen copies of each value are too few pairs among 4096.  (Four rounds cost 2^27 uint64 keys 15 us.)
inline unsigned int split_rounds(unsigned int len, unsigned int nseg, bool pairs) { return pairs && nseg == 1 && len > 16000000u ? 2 : 1; }
__host__ __device__ constexpr unsigned int split_prints(unsigned int rounds) { return rounds == 1 ? 8192 : 32768; }

template <int KB, bool PAIRS> struct SplitCfg {
  // (two blocks per SM, each with its tile, the counters and the table of up to 8192 cells)
  // Keys per thread, by sweeps: more spill more, fewer make shorter runs (int64 14 -> 12: a split of 2^25 keys 176 -> 160 us; float32
  // with positions 14 -> 12: the second split of 2^25 179 -> 160).  These spill 48 to 104 bytes of a thread's each way in the moves.
  static constexpr int ITEMS = KB == 8 && PAIRS ? 9 : KB == 8 || PAIRS ? 12 : 16;
  static constexpr int TILE  = SPLIT_THREADS * ITEMS;
};

// One split: its segments, cells and buckets.
struct SplitLevel {
  SplitSeg* segs;
  unsigned int* hist;         // [segment][cells]
  unsigned short* lut;        // [segment][cells]: bucket
  unsigned int* cursor;       // [segment][SPLIT_BINS]: next free place of the bucket
  const unsigned short* tile_seg;  // tile -> segment; null: tiles_per_seg each
  unsigned int nseg, tiles_per_seg, seg_len;  // (of equal segments)
  unsigned int cells, cap;
  unsigned int last;          // buckets are leaves (else segments of the next level)
  unsigned int pos_n;         // positions lie below this
  unsigned int radix_if;      // bit k: keys that differ in k bytes are left to the radix passes
  unsigned int rounds;        // of samples
  unsigned int most_copies;   // of a key, above which the radix passes are faster
  unsigned int leaf_cap;      // `cap` of the last split
  SplitMarks* marks;
  const void* src_keys;
  const uint32_t* src_pos;    // null: the place inside the segment
  void* dst_keys;
  uint32_t* dst_pos;
};

// NaNs of an argsort need many cells: they are ordered by position.
__host__ __device__ constexpr unsigned int split_nan_cells(int form, bool pairs, unsigned int cells)
{
  return form != FORM_INT ? (pairs ? cells / 8 : 1) : 0;
}

template <int KB, int FORM>
__device__ __forceinline__ typename KeyOf<KB>::type split_image(typename KeyOf<KB>::type raw, typename KeyOf<KB>::type flip)
{
  if constexpr (FORM == FORM_FLOAT) return to_ordered<KB, XF_FLOAT>(raw);
  else if constexpr (FORM == FORM_IMAGE) return raw;
  else return (typename KeyOf<KB>::type)(raw ^ flip);
}

// Zeros of both signs have one image, and so have all NaNs.  Where a sort holds one pattern of each, that is what its result gets;
// of several it would have to keep the input order, which the radix passes do.  Key j of a thread: the usual patterns
// into `flags`, others into `odd`, to be looked at by mark().
template <int KB>
__device__ __forceinline__ void mark_usual(typename KeyOf<KB>::type raw, typename KeyOf<KB>::type image, unsigned int& flags, unsigned int& odd, int j)
{
  using K = typename KeyOf<KB>::type;
  if (image == (K)~(K)0 || image == (K)((K)1 << (8 * KB - 1))) {
    if (sm_is_special<KB>(raw, XF_FLOAT)) odd |= 1u << j;
    else flags |= image == (K)~(K)0 ? MARK_NAN : MARK_ZERO;
  }
}
// `block` lies in shared memory.
template <int KB>
__device__ __forceinline__ void mark(typename KeyOf<KB>::type raw, typename KeyOf<KB>::type image, unsigned int& flags, SplitMarks* block)
{
  if (image != (typename KeyOf<KB>::type)~(typename KeyOf<KB>::type)0) {
    flags |= MARK_NEG_ZERO;
    return;
  }
  flags |= MARK_OTHER;
  if (*reinterpret_cast<volatile unsigned long long*>(&block->nan) != (unsigned long long)raw) {
    const unsigned long long old = atomicCAS(&block->nan, 0ull, (unsigned long long)raw);
    if (old != 0 && old != (unsigned long long)raw) flags |= MARK_MIXED;
  }
}
__device__ __forceinline__ bool marks_mixed(unsigned long long nan, unsigned int flags)
{
  return (flags & MARK_MIXED) != 0 || (flags & (MARK_ZERO | MARK_NEG_ZERO)) == (MARK_ZERO | MARK_NEG_ZERO) || ((flags & MARK_NAN) != 0 && nan != 0);
}
// A key from its image.
template <int KB>
__device__ __forceinline__ typename KeyOf<KB>::type marked_raw(typename KeyOf<KB>::type o, const SplitMarks* m)
{
  using K        = typename KeyOf<KB>::type;
  constexpr K SB = (K)((K)1 << (8 * KB - 1));
  if (o == (K)~(K)0 && m->nan != 0) return (K)m->nan;
  if (o == SB && (m->flags & MARK_NEG_ZERO) != 0) return SB;
  return sm_from_ordered<KB>(o, XF_FLOAT);
}

template <int KB> struct FloatOf { using type = float; };
template <> struct FloatOf<8> { using type = double; };
template <int KB>  // (not of NaNs)
__device__ __forceinline__ typename FloatOf<KB>::type value_of(typename KeyOf<KB>::type image)
{
  using K        = typename KeyOf<KB>::type;
  constexpr K SB = (K)((K)1 << (8 * KB - 1));
  const K raw    = (K)(image ^ (SB | (K)~(K)((typename std::make_signed<K>::type)image >> (8 * KB - 1))));
  if constexpr (KB == 8) return __longlong_as_double((long long)raw); else return __uint_as_float((unsigned int)raw);
}

template <int KB, int FORM, bool PAIRS, unsigned int MODE>
__device__ __forceinline__ unsigned int cell_of(typename KeyOf<KB>::type x, unsigned int pos, const SplitMap& m, unsigned int ci)
{
  using K   = typename KeyOf<KB>::type;
  const K y = (K)(x - (K)m.lo);
  if (y > (K)m.range) {
    // outside (rare, hence a branch of its own); a segment of nothing but NaNs takes them for its one image
    if (FORM != FORM_INT && x == (K)~(K)0) return ci + 2 + (PAIRS ? __umulhi(pos, m.nscale) : 0u);
    return x < (K)m.lo ? 0u : ci + 1;
  }
  unsigned int t;
  if constexpr (MODE == MAP_LIN || MODE == MAP_TOP) {
    if constexpr (KB == 8) {
      const unsigned int a = (unsigned int)y, b = (unsigned int)(y >> 32);
      t = __funnelshift_r(m.shift < 32 ? a : b, m.shift < 32 ? b : 0u, m.shift & 31u);
    } else {
      t = y >> m.shift;
    }
    if constexpr (MODE == MAP_TOP) t += (y >= (K)m.top ? 1u : 0u) + (y > (K)m.top ? 1u : 0u);
  } else if constexpr (MODE == MAP_POS) {
    t = (unsigned int)y * m.mult + __umulhi(pos, m.pscale);
  } else if constexpr (MODE == MAP_VAL) {
    // (adding 2^23 or 2^52 leaves the rounded product in the low bits; the product of the range is at most ci - 1)
    using F   = typename FloatOf<KB>::type;
    const F v = value_of<KB>(x);
    if constexpr (KB == 8) {
      t = (unsigned int)__double_as_longlong(fma(v - __longlong_as_double((long long)m.vmin), __longlong_as_double((long long)m.top), 4503599627370496.0));
    } else {
      t = __float_as_uint(fmaf(v - __uint_as_float((unsigned int)m.vmin), (float)__longlong_as_double((long long)m.top), 8388608.0f)) & 0x7FFFFFu;
    }
    t = min(t, ci - 1);
  } else {
    const float f = KB == 8 ? __ull2float_rz((unsigned long long)y) : __uint2float_rz((unsigned int)y);
    t             = (unsigned int)max((int)(__float_as_uint(f) >> m.shift) - (int)m.mult, 0);
  }
  return t + 1;
}
template <int FORM, bool PAIRS, typename F>
__device__ __forceinline__ void with_mode(unsigned int mode, F f)
{
  if (mode == MAP_LIN) f(std::integral_constant<unsigned int, MAP_LIN>{});
  else if (mode == (FORM != FORM_INT ? MAP_VAL : MAP_LOG)) f(std::integral_constant<unsigned int, FORM != FORM_INT ? MAP_VAL : MAP_LOG>{});
  else f(std::integral_constant<unsigned int, PAIRS ? MAP_POS : MAP_TOP>{});
}

// MAP_LOG: where, from m.lo on, cell q + 1 starts (2^64 - 1 also for what lies beyond).
__device__ __forceinline__ unsigned long long log_from(const SplitMap& m, unsigned int q)
{
  return q == 0 ? 0ull : __float2ull_ru(__uint_as_float((q + m.mult) << m.shift));
}

// The last image of that cell.
__device__ __forceinline__ unsigned long long log_last(const SplitMap& m, unsigned int q)
{
  const unsigned long long next = log_from(m, q + 1);
  return next == ~0ull ? next : next - 1;
}

// The only image of a cell, where it has one.
template <int KB, int FORM, bool PAIRS>
__device__ __forceinline__ bool cell_value(const SplitMap& m, unsigned int c, unsigned int ci, unsigned long long* image)
{
  if (FORM != FORM_INT && !PAIRS && c == ci + 2) {
    *image = KB == 8 ? ~0ull : 0xFFFFFFFFull;
    return true;
  }
  if (c < 1 || c > ci) return false;
  if (m.mode == MAP_LIN && m.shift == 0) {
    *image = m.lo + (c - 1);
    return true;
  }
  if (m.mode == MAP_TOP && c == (unsigned int)(m.top >> m.shift) + 2) {
    *image = m.lo + m.top;
    return true;
  }
  if (m.mode == MAP_LOG) {
    const unsigned long long z = log_from(m, c - 1);
    if (log_last(m, c - 1) != z) return false;
    *image = m.lo + z;
    return true;
  }
  return false;
}

// The images that cells c0 .. c1 - 1 can hold, where the mapping tells.
__device__ __forceinline__ bool cell_bounds(const SplitMap& m, unsigned int c0, unsigned int c1, unsigned int ci, unsigned long long* lo, unsigned long long* span)
{
  if (c0 < 1 || c1 - 1 > ci) return false;
  unsigned long long a, b;  // first and last image, from m.lo on
  // (cells of a mapping may reach beyond the range, and beyond 64 bits)
  auto step = [&](unsigned int c) { return c > (m.range >> m.shift) ? m.range : ((unsigned long long)c << m.shift) - 1; };   // the last of c linear cells
  if (m.mode == MAP_LIN) {
    a = (unsigned long long)(c0 - 1) << m.shift;
    b = step(c1 - 1);
  } else if (m.mode == MAP_TOP) {
    // (cells from the one of lo + top on are two further up, with it and after it)
    const unsigned int t = (unsigned int)(m.top >> m.shift) + 1;
    a = c0 <= t ? (unsigned long long)(c0 - 1) << m.shift : c0 == t + 1 ? m.top : c0 == t + 2 ? m.top + 1 : (unsigned long long)(c0 - 3) << m.shift;
    b = c1 <= t ? step(c1 - 1) : c1 == t + 1 ? m.top - 1 : c1 == t + 2 ? m.top : step(c1 - 3);
    if (c1 == t + 1 && m.top == 0) return false;
  } else if (m.mode == MAP_LOG) {
    a = log_from(m, c0 - 1);
    b = log_last(m, c1 - 2);
  } else {
    return false;
  }
  b     = min(b, m.range);
  if (a > b) return false;
  *lo   = m.lo + a;
  *span = b - a;
  return true;
}

// Places of a tile: which segment, where in it.
struct TileRange {
  unsigned int first, end;
};
__device__ __forceinline__ TileRange my_tiles(unsigned int ntiles)
{
  TileRange r;
  r.first = (unsigned int)((unsigned long long)blockIdx.x * ntiles / gridDim.x);
  r.end   = (unsigned int)((unsigned long long)(blockIdx.x + 1) * ntiles / gridDim.x);
  return r;
}

// ---- sample: one block per segment ----
// Latency of scattered loads: 7 to 13 us for an array, 33 us for the 187 segments of 2^28 keys.  More samples would narrow
// what lies outside their range: with 1024 per segment of the second split one sort of 2^27 keys in a few had a cell
// of outsiders that no bucket holds.  Two blocks per SM at 64 registers (1000 rows of 12000 float64 88 -> 70 us); argsorts of float64
// would spill (2 * 10^6 keys 138.9 -> 140.7).
template <int KB, int FORM, bool PAIRS, int SAMPLES>
__global__ void __launch_bounds__(SPLIT_THREADS, KB == 8 && FORM == FORM_FLOAT && PAIRS ? 1 : 2) split_sample_kernel(Ctrl* ctrl, SplitLevel L, unsigned int decide, typename KeyOf<KB>::type flip)
{
  using K = typename KeyOf<KB>::type;
  extern __shared__ unsigned int sh_cells[];
  __shared__ K sh_b[2 * SPLIT_THREADS / 32];
  __shared__ unsigned int sh_n[2], sh_most[2], sh_eq[2];
  __shared__ unsigned long long sh_lo, sh_hi;
  __shared__ SplitMarks sh_marks;
  const unsigned int seg = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  chain_wait();
  if (!decide && ctrl->route != ROUTE_SPLIT) return;
  if (L.tile_seg != nullptr && seg >= ctrl->split_nseg) return;
  unsigned int begin, len;
  if (L.tile_seg == nullptr) {
    begin = seg * L.seg_len;
    len   = L.seg_len;
  } else {
    begin = L.segs[seg].begin;
    len   = L.segs[seg].len;
  }
  if (len == 0) return;
  const K* src          = static_cast<const K*>(L.src_keys) + begin;
  const unsigned int ns = min(len, (unsigned int)SAMPLES);
  constexpr int PER     = SAMPLES / SPLIT_THREADS;
  constexpr unsigned int FIN_LO = KB == 8 ? 0x00100000u : 0x00800000u;  // upper words of finite images start here
  K img[PER];
  unsigned int at[PER];
  // one key of every stretch of len / SAMPLES, at a scattered place inside it
  auto place = [&](unsigned int i) {
    unsigned int h = i * 2654435761u;
    h ^= h >> 15;
    h *= 2246822519u;
    return len <= SAMPLES ? i : (unsigned int)(((unsigned long long)i * len) / SAMPLES) + __umulhi(h, len / SAMPLES);
  };
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const unsigned int i = j * SPLIT_THREADS + tid;
    at[j]  = place(i);
    img[j] = i < ns ? src[at[j]] : (K)0;
    if (PAIRS && L.src_pos != nullptr) at[j] = i < ns ? L.src_pos[begin + at[j]] : 0u;
  }
  // one more key of every stretch per round (of argsorts), from parts of it that do not meet; on their way into the L2 early, since a round
  // waits for its own
  const unsigned int part = PAIRS && L.rounds > 1 ? len / SAMPLES / (L.rounds - 1) : 0;
  auto further = [&](unsigned int i, unsigned int r) {
    return (unsigned int)(((unsigned long long)i * len) / SAMPLES) + (r - 1) * part + __umulhi((i + r) * 2654435761u, part);
  };
  if (PAIRS && decide) {
    for (unsigned int r = 1; r < L.rounds; ++r) {
#pragma unroll
      for (int j = 0; j < PER; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + further(j * SPLIT_THREADS + tid, r)));
    }
  }
  auto mine = [&](int j) { return j * SPLIT_THREADS + tid < ns; };
  K lo = (K)~(K)0, hi = 0;
  unsigned int flags = 0, odd = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const K raw = img[j];
    img[j] = split_image<KB, FORM>(img[j], flip);
    if (FORM == FORM_FLOAT && !PAIRS && mine(j)) mark_usual<KB>(raw, img[j], flags, odd, j);
    // (of floats the finite ones count)
    if (mine(j) && !(FORM != FORM_INT && (unsigned int)(img[j] >> (8 * KB - 32)) - FIN_LO >= 0u - 2u * FIN_LO)) {
      lo = img[j] < lo ? img[j] : lo;
      hi = img[j] > hi ? img[j] : hi;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const K l = __shfl_xor_sync(0xFFFFFFFFu, lo, o), h = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
    lo = l < lo ? l : lo;
    hi = h > hi ? h : hi;
  }
  if (lane == 0) {
    sh_b[2 * warp]     = lo;
    sh_b[2 * warp + 1] = hi;
  }
  if (tid < 2) sh_n[tid] = sh_most[tid] = sh_eq[tid] = 0;
  if (tid == 0) {
    sh_lo = ~0ull;
    sh_hi = 0;
  }
  for (unsigned int i = tid; i < L.cells; i += SPLIT_THREADS) sh_cells[i] = 0;
  __syncthreads();
  for (int w = 0; w < SPLIT_THREADS / 32; ++w) {
    const K l = sh_b[2 * w], h = sh_b[2 * w + 1];
    lo = l < lo ? l : lo;
    hi = h > hi ? h : hi;
  }
  if (lo > hi) lo = hi = (K)~(K)0;  // no finite ones: taken for NaNs
  const unsigned int nan = split_nan_cells(FORM, PAIRS, L.cells), ci = L.cells - 2 - nan;
  const K lo_seen = lo, hi_seen = hi;
  const bool narrow = (unsigned long long)(hi - lo) < ci;
  if (!narrow || (FORM == FORM_INT && !PAIRS)) {
    // some room for the keys outside the sampled range, which would all lie in one cell; a narrow range of integers has cells to
    // spare (10^7 keys around one place, a hundredth elsewhere: rare values of the crowd that 2048 samples missed filled that cell)
    const K room = narrow ? (K)((ci - 1 - (unsigned int)(hi - lo)) / 2) : (K)((hi - lo) >> 6);
    const K least = FORM != FORM_INT ? (K)((K)FIN_LO << (8 * KB - 32)) : (K)0, most_ = FORM != FORM_INT ? (K)~least : (K)~(K)0;
    lo = lo - least > room ? (K)(lo - room) : least;
    hi = most_ - hi > room ? (K)(hi + room) : most_;
  }
  SplitMap m{};
  m.lo    = (unsigned long long)lo;
  m.range = (unsigned long long)hi - (unsigned long long)lo;
  m.mode  = MAP_LIN;
  auto scale_of = [&](unsigned int parts) {
    return (unsigned int)min(((unsigned long long)parts << 32) / L.pos_n, 0xFFFFFFFFull);
  };
  m.nscale = PAIRS && FORM != FORM_INT ? scale_of(nan) : 0u;
  SplitMap alt = m;
  bool two     = false;
  if (m.range < ci) {
    if (PAIRS && 2 * (m.range + 1) <= ci) {
      m.mode   = MAP_POS;
      m.mult   = ci / ((unsigned int)m.range + 1);
      m.pscale = scale_of(m.mult);
    }
  } else {
    while ((m.range >> m.shift) >= ci - 2) ++m.shift;
    if constexpr (FORM != FORM_INT) {
      using F = typename FloatOf<KB>::type;
      const F room = (value_of<KB>(hi_seen) - value_of<KB>(lo_seen)) * (F)0.015625;
      const F a = value_of<KB>(lo_seen) - room, b = value_of<KB>(hi_seen) + room, w = b - a;
      const double scale = (double)(ci - 2) / (double)w;
      alt.mode = MAP_VAL;
      if constexpr (KB == 8) {
        alt.vmin  = (unsigned long long)__double_as_longlong(a);
        alt.lo    = (unsigned long long)to_ordered<8, XF_FLOAT>((uint64_t)__double_as_longlong(a));
        alt.range = (unsigned long long)to_ordered<8, XF_FLOAT>((uint64_t)__double_as_longlong(b)) - alt.lo;
      } else {
        alt.vmin  = __float_as_uint(a);
        alt.lo    = to_ordered<4, XF_FLOAT>(__float_as_uint(a));
        alt.range = to_ordered<4, XF_FLOAT>(__float_as_uint(b)) - (unsigned int)alt.lo;
      }
      alt.top = (unsigned long long)__double_as_longlong(scale);
      two     = scale > 1e-30 && scale < 1e30 && (double)a > -1e300 && (double)b < 1e300;   // (nothing overflows)
    } else {
      alt.lo    = (unsigned long long)lo_seen;
      alt.range = (unsigned long long)hi - (unsigned long long)lo_seen;
      const unsigned int oct = 64 - __clzll((long long)alt.range);
      unsigned int bits      = 0;
      while (bits < 22 && ((unsigned long long)oct << (bits + 1)) < ci) ++bits;
      alt.mode  = MAP_LOG;
      alt.shift = 23 - bits;
      alt.mult  = (127u << bits) - 1;
      two       = true;
    }
  }
  // samples that lie in cells which alone fill a bucket (the mapping with fewer of them is taken), and the
  // fullest cell
  const unsigned int heavy = max(6u, (unsigned int)((unsigned long long)ns * L.cap / len / 2));
  auto score = [&](const SplitMap& f, int slot) {
    unsigned int c[PER];
    with_mode<FORM, PAIRS>(f.mode, [&](auto md) {
#pragma unroll
      for (int j = 0; j < PER; ++j) c[j] = cell_of<KB, FORM, PAIRS, decltype(md)::value>(img[j], at[j], f, ci);
    });
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (mine(j)) atomicAdd(&sh_cells[c[j]], 1u);
    __syncthreads();
    unsigned int n = 0, mx = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (mine(j)) {
        const unsigned int k = sh_cells[c[j]];
        n += k > heavy ? 1u : 0u;
        mx = max(mx, (k << 16) | c[j]);
      }
    }
    n  = __reduce_add_sync(0xFFFFFFFFu, n);
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    if (lane == 0) {
      if (n) atomicAdd(&sh_n[slot], n);
      atomicMax(&sh_most[slot], mx);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (mine(j)) sh_cells[c[j]] = 0;
    __syncthreads();
  };
  score(m, 0);
  unsigned int most = sh_most[0];
  if (m.mode == MAP_LIN && m.shift > 0 && sh_n[0] > 0) {
    // one value with many copies among others: is it the smallest or the largest one of the fullest cell?
    bool top           = false;
    unsigned int crowd = sh_n[0];
    if (!PAIRS) {
      const unsigned int cell = most & 0xFFFFu;
      bool in[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        in[j] = mine(j) && cell_of<KB, FORM, PAIRS, MAP_LIN>(img[j], at[j], m, ci) == cell && cell >= 1 && cell <= ci;
        if (in[j]) {
          atomicMin(&sh_lo, (unsigned long long)img[j]);
          atomicMax(&sh_hi, (unsigned long long)img[j]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        if (in[j] && (unsigned long long)img[j] == sh_lo) atomicAdd(&sh_eq[0], 1u);
        if (in[j] && (unsigned long long)img[j] == sh_hi) atomicAdd(&sh_eq[1], 1u);
      }
      __syncthreads();
      const int w = sh_eq[1] >= sh_eq[0] ? 1 : 0;
      top         = 2 * sh_eq[w] > (most >> 16);
      if (top) {
        m.top = (w ? sh_hi : sh_lo) - m.lo;
        crowd -= min(crowd, most >> 16);
      }
    }
    if (two) score(alt, 1);
    if (two && sh_n[1] < crowd) {
      m    = alt;
      most = sh_most[1];
    } else if (top) {
      m.mode = MAP_TOP;
    }
  }
  if (tid == 0) {
    SplitSeg& s = L.segs[seg];
    s.map       = m;
    if (L.tile_seg == nullptr) {
      s.begin = begin;
      s.len   = len;
      s.tile0 = seg * L.tiles_per_seg;
      s.drops = 0;
    }
  }
  if (decide) {
    // Who sorts.  Copies of a key among the samples, by a table of fingerprints (NaNs apart), as if every value
    // had as many
    __syncthreads();
    unsigned int* table       = sh_cells;
    const unsigned int prints = split_prints(L.rounds);
    for (unsigned int i = tid; i < prints; i += SPLIT_THREADS) table[i] = 0;
    if (tid == 0) {
      sh_n[0] = sh_n[1] = 0;
      sh_marks = SplitMarks{};
    }
    __syncthreads();
    if (FORM == FORM_FLOAT && !PAIRS) {
      while (odd) {
        const K raw = src[place((__ffs(odd) - 1) * SPLIT_THREADS + tid)];
        odd &= odd - 1;
        mark<KB>(raw, split_image<KB, FORM>(raw, flip), flags, &sh_marks);
      }
      flags = __reduce_or_sync(0xFFFFFFFFu, flags);
      if (lane == 0 && flags) atomicOr(&sh_marks.flags, flags);
    }
    // What a leaf, or a later split, cannot take apart would be found out late: the fullest cell, if its samples say so by three
    // standard deviations.  (A cell of one value is filled in, one of a few is counted.)
    const unsigned int cell = most & 0xFFFFu;
    const float k_ = (float)(most >> 16), sure = k_ - 3.0f * sqrtf(k_), leaf = (float)L.leaf_cap * __fdividef((float)ns, (float)len);
    constexpr float NEXT = SPLIT_BINS * 15 / 16;   // leaves of a segment
    // of the integers of a sort those in that cell
    unsigned int in_fullest = 0;
    if (!PAIRS && FORM == FORM_INT && !L.last && sure > NEXT * leaf) {
      with_mode<FORM, PAIRS>(m.mode, [&](auto md) {
#pragma unroll
        for (int j = 0; j < PER; ++j) in_fullest |= cell_of<KB, FORM, PAIRS, decltype(md)::value>(img[j], at[j], m, ci) == cell ? 1u << j : 0u;
      });
    }
    unsigned int same = 0, bytes = 0;
    auto print = [&](K image) {
      if (FORM != FORM_INT && image == (K)~(K)0) return;
      unsigned int h = (unsigned int)image * 2654435761u ^ (unsigned int)((unsigned long long)image >> 32) * 2246822519u;
      h ^= h >> 15;
      h = h * 3266489917u | 1u;
      const unsigned int old = atomicCAS(&table[__umulhi(h, prints)], 0u, h);
      same += old == h ? 1u : 0u;
    };
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (mine(j)) {
        const unsigned long long d = (unsigned long long)(img[j] ^ lo_seen);
#pragma unroll
        for (int k = 0; k < KB; ++k) bytes |= (d >> (8 * k) & 0xFFu) ? 1u << k : 0u;
        if (PAIRS || FORM != FORM_INT || (in_fullest >> j & 1u)) print(img[j]);
      }
    }
    if (PAIRS) {
      for (unsigned int r = 1; r < L.rounds; ++r) {
        K more[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) more[j] = src[further(j * SPLIT_THREADS + tid, r)];
#pragma unroll
        for (int j = 0; j < PER; ++j)
          if (further(j * SPLIT_THREADS + tid, r) != place(j * SPLIT_THREADS + tid)) print(split_image<KB, FORM>(more[j], flip));
      }
    }
    same  = __reduce_add_sync(0xFFFFFFFFu, same);
    bytes = __reduce_or_sync(0xFFFFFFFFu, bytes);
    if (lane == 0) {
      if (same) atomicAdd(&sh_n[0], same);
      atomicOr(&sh_n[1], bytes);
    }
    __syncthreads();
    if (tid == 0) {
      unsigned int route = FORM == FORM_FLOAT && !PAIRS && marks_mixed(sh_marks.nan, sh_marks.flags) ? ROUTE_RADIX : ROUTE_SPLIT;
      // A sample finds its copies among those before it: half of the square, as long as few have any; then what counts is how many
      // others there are.
      const unsigned int eq = sh_n[0];
      const float drawn     = (float)(ns * L.rounds);
      float copies          = 2.0f * (float)eq * __fdividef((float)len, drawn * drawn);
      if (2.0f * (float)eq > drawn) copies = fmaxf(copies, __fdividef((float)len, fmaxf(drawn - (float)eq, 1.0f)));
      // (of an argsort equal keys have to be taken apart; in a sort of floats, whose cells cannot be seen to hold one value, they
      // fill cells that nothing splits)
      const bool each = decide == 1 && !PAIRS && m.mode == MAP_LIN && m.shift == 0;   // (a row of few values has a cell for each)
      if ((PAIRS || FORM != FORM_INT) && m.mode != MAP_POS && !each && eq >= 6 && copies > (float)L.most_copies) route = ROUTE_RADIX;
      if (m.mode == MAP_TOP) {
        // (the fullest cell is the value's own)
      } else if (PAIRS) {
        if (sure > (L.last ? 4.0f : NEXT) * leaf) route = ROUTE_RADIX;
      } else if (!L.last) {
        if (sure - (FORM == FORM_INT ? 2.0f * (float)eq : 0.0f) > NEXT * leaf && !(FORM != FORM_INT && cell == ci + 2)) route = ROUTE_RADIX;
      } else if (sure > leaf) {
        unsigned long long first, span;
        const bool known = cell_bounds(m, cell, cell + 1, ci, &first, &span);
        if (!(FORM != FORM_INT && cell == ci + 2) && (!known || span > (sure > COUNT_MOST * leaf ? 0u : COUNT_SPAN))) route = ROUTE_RADIX;
      }
      // (a short row of few leaves has its tail in one of them, whose cells are linear)
      if (KB == 4 && decide == 1 && m.mode == MAP_LOG && len < 6 * L.cap) route = ROUTE_RADIX;
      if (decide == 2 && (L.radix_if >> __popc(sh_n[1]) & 1u)) route = ROUTE_RADIX;
      atomicMax(&ctrl->route, route);
    }
  }
}

// ---- cells: counts per cell; a block takes a run of consecutive tiles ----
// One shared-memory reduction per key.  8-byte keys are bound by memory (2^28 uint64 keys 332 us, 6.5 TB/s), 4-byte keys by
// issue (2^26 int32 keys 62 us, 4.3 TB/s).
template <int KB, int FORM, bool PAIRS>
__global__ void __launch_bounds__(SPLIT_THREADS, 3) split_cells_kernel(Ctrl* ctrl, SplitLevel L, typename KeyOf<KB>::type flip)
{
  using K             = typename KeyOf<KB>::type;
  constexpr int ITEMS = SplitCfg<KB, PAIRS>::ITEMS, TILE = SplitCfg<KB, PAIRS>::TILE;
  extern __shared__ unsigned int h[];
  __shared__ SplitMarks sh_marks;
  chain_wait();
  if (__syncthreads_or(ld_relaxed(&ctrl->route) != ROUTE_SPLIT)) return;  // (other blocks may be changing it)
  const unsigned int tid = threadIdx.x;
  const TileRange r = my_tiles(L.tile_seg ? ctrl->split_ntiles : L.nseg * L.tiles_per_seg);
  if (r.first >= r.end) return;
  for (unsigned int i = tid; i < L.cells; i += SPLIT_THREADS) h[i] = 0;
  if (tid == 0) sh_marks = SplitMarks{};
  __syncthreads();
  const unsigned int ci = L.cells - 2 - split_nan_cells(FORM, PAIRS, L.cells);
  unsigned int cur = 0xFFFFFFFFu;
  SplitSeg s{};
  unsigned int flags = 0;
  auto flush = [&] {
    __syncthreads();
    unsigned int* out = L.hist + (size_t)cur * L.cells;
    for (unsigned int i = tid; i < L.cells; i += SPLIT_THREADS) {
      const unsigned int c = h[i];
      if (c) {
        atomicAdd(out + i, c);
        h[i] = 0;
      }
    }
    __syncthreads();
  };
  for (unsigned int t = r.first; t < r.end; ++t) {
    const unsigned int seg = L.tile_seg ? L.tile_seg[t] : t / L.tiles_per_seg;
    if (seg != cur) {
      if (cur != 0xFFFFFFFFu) flush();
      cur = seg;
      s   = L.segs[seg];
    }
    const unsigned int at    = (t - s.tile0) * TILE;
    const unsigned int valid = min((unsigned int)TILE, s.len - at);
    const K* src             = static_cast<const K*>(L.src_keys) + s.begin + at;
    const uint32_t* psrc     = PAIRS && L.src_pos ? L.src_pos + s.begin + at : nullptr;
    K key[ITEMS];
    auto count = [&](auto md, auto part) {
      constexpr unsigned int MODE = decltype(md)::value;
      constexpr bool PART         = decltype(part)::value;
      unsigned int nans = 0, odd = 0;
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned int e = j * SPLIT_THREADS + tid;
        key[j]               = !PART || e < valid ? src[e] : (K)0;
      }
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned int e = j * SPLIT_THREADS + tid;
        if (PART && e >= valid) continue;
        const K x = split_image<KB, FORM>(key[j], flip);
        if (FORM == FORM_FLOAT && !PAIRS) mark_usual<KB>(key[j], x, flags, odd, j);
        if (PAIRS && MODE != MAP_POS && FORM != FORM_INT && x == (K)~(K)0) {
          nans |= 1u << j;   // ordered by position, which is fetched for them alone
          continue;
        }
        const unsigned int pos = !PAIRS || MODE != MAP_POS ? 0u : psrc == nullptr ? at + e : psrc[e];
        atomicAdd(&h[cell_of<KB, FORM, PAIRS, MODE>(x, pos, s.map, ci)], 1u);
      }
      if (FORM == FORM_FLOAT && !PAIRS) {
        while (odd) {   // negative zeros and other NaNs, fetched once more: kept until here they would spill
          const int j = __ffs(odd) - 1;
          odd &= odd - 1;
          const K raw = src[j * SPLIT_THREADS + tid];
          mark<KB>(raw, split_image<KB, FORM>(raw, flip), flags, &sh_marks);
        }
      }
      if (PAIRS && FORM != FORM_INT) {
        while (nans) {
          const int j = __ffs(nans) - 1;
          nans &= nans - 1;
          const unsigned int e = j * SPLIT_THREADS + tid;
          atomicAdd(&h[cell_of<KB, FORM, PAIRS, MODE>((K)~(K)0, psrc == nullptr ? at + e : psrc[e], s.map, ci)], 1u);
        }
      }
    };
    with_mode<FORM, PAIRS>(s.map.mode, [&](auto md) {
      if (valid == TILE) count(md, std::false_type{});
      else count(md, std::true_type{});
    });
  }
  flush();
  if (FORM == FORM_FLOAT && !PAIRS) {
    if (__syncthreads_or(flags)) {
      flags = __reduce_or_sync(0xFFFFFFFFu, flags);
      if ((tid & 31) == 0 && flags) atomicOr(&sh_marks.flags, flags);
      __syncthreads();
      if (tid == 0) {
        flags = sh_marks.flags;
        if (sh_marks.nan != 0) {
          const unsigned long long old = atomicCAS(&L.marks->nan, 0ull, sh_marks.nan);
          if (old != 0 && old != sh_marks.nan) flags |= MARK_MIXED;
        }
        atomicOr(&L.marks->flags, flags);
      }
    }
  }
}

// ---- pack: one block per segment cuts its cells into buckets ----
// Latency of a handful of dependent steps on chip: 8 to 9 us, up to 50 where many values are filled in.  Walking from bucket to
// bucket costs 35 cycles each with one lookup per step (220 with the four it takes to tell what a bucket is, hence
// the list that the block looks at afterwards: float32 sort of 7 * 10^5 keys, this kernel 30 -> 8 us); cells that are small
// need no walk at all.
constexpr int PACK_THREADS = 1024;
inline size_t pack_smem(unsigned int cells) { return (size_t)(cells + 1) * 4 + (size_t)cells * 6; }

template <int KB, int FORM, bool PAIRS>
__global__ void __launch_bounds__(PACK_THREADS)
split_pack_kernel(Ctrl* ctrl, SplitLevel L, SplitLeaf* leaves, SplitSeg* next_segs, unsigned short* next_tile_seg, unsigned int next_nseg, unsigned int next_tile, typename KeyOf<KB>::type flip)
{
  using K = typename KeyOf<KB>::type;
  extern __shared__ unsigned int pre[];
  unsigned short* nxt  = reinterpret_cast<unsigned short*>(pre + L.cells + 1);
  unsigned short* stop = nxt + L.cells;   // the first cell from here on that is filled in
  unsigned short* list = stop + L.cells;  // the first cells of the buckets, and the cells between them
  __shared__ unsigned int wsum[PACK_THREADS / 32], wstop[PACK_THREADS / 32], wmost[PACK_THREADS / 32];
  __shared__ unsigned int sh_nb, sh_leaf0;
  __shared__ unsigned int bin_cell[SPLIT_BINS], bin_end[SPLIT_BINS], bin_tile[SPLIT_BINS], bin_tiles[SPLIT_BINS];
  const unsigned int seg = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  chain_wait();
  const bool mixed = FORM == FORM_FLOAT && !PAIRS && marks_mixed(L.marks->nan, L.marks->flags);
  if (__syncthreads_or(ld_relaxed(&ctrl->route) != ROUTE_SPLIT)) return;  // (other blocks may be changing it)
  if (mixed) {
    if (tid == 0) atomicMax(&ctrl->route, (unsigned int)ROUTE_LATE);
    return;
  }
  if (L.tile_seg != nullptr && seg >= ctrl->split_nseg) return;
  const SplitSeg s = L.segs[seg];
  if (s.len == 0) return;
  const unsigned int C = L.cells, ci = C - 2 - split_nan_cells(FORM, PAIRS, C);
  const unsigned int* cnt = L.hist + (size_t)seg * C;
  // exclusive prefix of the counts: a warp takes a run of cells, 32 at a time
  const unsigned int per = C / (PACK_THREADS / 32);
  {
    constexpr int MOST = SPLIT_MAX_CELLS / PACK_THREADS;
    unsigned int run = 0, got[MOST];
#pragma unroll
    for (int k = 0; k < MOST; ++k) got[k] = k * 32 + lane < per ? cnt[warp * per + k * 32 + lane] : 0u;
#pragma unroll
    for (int k = 0; k < MOST; ++k) {
      const unsigned int i = k * 32 + lane;
      const unsigned int v = got[k];
      unsigned int incl    = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (unsigned int)o) incl += u;
      }
      if (i < per) pre[warp * per + i] = run + incl - v;
      run += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    if (lane == 0) wsum[warp] = run;
    __syncthreads();
    const unsigned int before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? wsum[lane] : 0u);
    for (unsigned int i = lane; i < per; i += 32) pre[warp * per + i] += before;
    if (tid == 0) pre[C] = s.len;
  }
  __syncthreads();
  auto scan = [&](unsigned int v, unsigned int* total) {  // exclusive, over the block
    unsigned int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= (unsigned int)o) incl += u;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    const unsigned int w = wsum[lane];
    *total = __reduce_add_sync(0xFFFFFFFFu, w);
    return incl - v + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u);
  };
  // values with many copies are filled in at the end: nothing of them is moved
  auto filled = [&](unsigned int c, unsigned long long* image) {
    return !PAIRS && pre[c + 1] - pre[c] > L.cap / 4 && cell_value<KB, FORM, PAIRS>(s.map, c, ci, image);
  };
  bool drops = false, crowded = false;
  unsigned int most = 0;
  for (unsigned int c = tid; c < C; c += PACK_THREADS) {
    const unsigned int n = pre[c + 1] - pre[c];
    unsigned long long image;
    crowded |= filled(c, &image);
    most = max(most, n);
  }
  most = __reduce_max_sync(0xFFFFFFFFu, most);
  if (lane == 0) wmost[warp] = most;
  crowded = __syncthreads_or(crowded);
  most    = __reduce_max_sync(0xFFFFFFFFu, wmost[lane]);
  // Small cells: buckets of `step` keys and up to one cell more, every cell for itself
  const unsigned int step = L.cap - min(most, L.cap / 2) - 8;
  if (!crowded && (most <= L.cap / 8 || (most <= L.cap / 3 && s.len / step < SPLIT_BINS * 15 / 16))) {
    const float inv         = __fdividef(1.0f, (float)step);
    auto bin_of = [&](unsigned int c) {
      // the exact quotient: the rounded one is off by one at most
      unsigned int q = (unsigned int)((float)pre[c] * inv);
      if (q * step > pre[c]) --q;
      if (pre[c] - q * step >= step) ++q;
      return q;
    };
    const unsigned int n = bin_of(C - 1) + 1;
    for (unsigned int c = tid; c < C; c += PACK_THREADS) {
      const unsigned int q    = bin_of(c);
      const unsigned int last = c == 0 ? 0xFFFFFFFFu : bin_of(c - 1);
      if (q != last && q < SPLIT_BINS) {   // (no bucket is left out: a cell is shorter than a step)
        bin_cell[q] = c;
        if (q > 0) bin_end[q - 1] = c;
      }
      if (c == C - 1 && q < SPLIT_BINS) bin_end[q] = C;
    }
    if (tid == 0) sh_nb = n;
  } else {
    {
      unsigned int next = C;   // in the cells of this warp that lie above
      for (unsigned int i = per - per % 32 + lane; i - lane < C; i -= 32) {
        unsigned long long image;
        const unsigned int c   = warp * per + i;
        const unsigned int set = __ballot_sync(0xFFFFFFFFu, i < per && filled(c, &image)) & (0xFFFFFFFFu << lane);
        if (i < per) stop[c] = (unsigned short)(set ? c - lane + (__ffs(set) - 1) : next);
        const unsigned int low = __shfl_sync(0xFFFFFFFFu, set, 0);
        if (low) next = c - lane + (__ffs(low) - 1);
        if (i < 32) break;
      }
      if (lane == 0) wstop[warp] = next;
      __syncthreads();
      const unsigned int above = __reduce_min_sync(0xFFFFFFFFu, lane > warp ? wstop[lane] : C);
      for (unsigned int i = lane; i < per; i += 32)
        if (stop[warp * per + i] == C) stop[warp * per + i] = (unsigned short)above;
    }
    __syncthreads();
    // the end of the longest bucket that starts at each cell
    for (unsigned int c = tid; c < C; c += PACK_THREADS) {
      const unsigned int lim = pre[c] + L.cap;
      unsigned int a = c + 1, b = stop[c];   // largest q in [c + 1, stop] with pre[q] <= lim, or c + 1
      unsigned long long image;
      if (b == c && filled(c, &image)) {
        const unsigned int len = pre[c + 1] - pre[c], begin = s.begin + pre[c];
        unsigned long long raw;
        if constexpr (FORM != FORM_INT)
          raw = (unsigned long long)marked_raw<KB>((K)image, L.marks);
        else raw = (unsigned long long)(K)((K)image ^ flip);
        const unsigned int parts = (len + FILL_CHUNK - 1) / FILL_CHUNK, e = atomicAdd(&ctrl->split_nleaf, parts);
        for (unsigned int i = 0; i < parts; ++i)
          leaves[e + i] = SplitLeaf{begin + i * FILL_CHUNK, min(FILL_CHUNK, len - i * FILL_CHUNK) | LEAF_FILL, raw, 0};
        L.lut[(size_t)seg * C + c] = LUT_DROP;
        drops = true;
      } else {
        while (a < b) {
          const unsigned int q = (a + b + 1) >> 1;
          if (pre[q] <= lim) a = q; else b = q - 1;
        }
      }
      nxt[c] = (unsigned short)a;
    }
    drops = __syncthreads_or(drops);
    if (tid == 0) {
      unsigned int p = 0, n = 0;
      while (p < C) {
        list[n++] = (unsigned short)p;
        p         = nxt[p];
      }
      sh_leaf0 = n;
    }
    __syncthreads();
    const unsigned int chain = sh_leaf0;
    unsigned int nb0         = 0;
    for (unsigned int i0 = 0; i0 < chain; i0 += PACK_THREADS) {
      const unsigned int i = i0 + tid, p = i < chain ? list[i] : 0, q = i < chain ? nxt[p] : 0;
      // (cells without keys between two values that are filled in make no bucket)
      const bool bin = i < chain && stop[p] != p && pre[q] != pre[p];
      unsigned int all;
      const unsigned int at = nb0 + scan(bin ? 1u : 0u, &all);
      if (bin && at < SPLIT_BINS) {
        bin_cell[at] = p;
        bin_end[at]  = q;
      }
      nb0 += all;
    }
    if (tid == 0) sh_nb = nb0;
  }
  if (tid == 0) L.segs[seg].drops = drops;
  __syncthreads();
  const unsigned int nb = sh_nb;
  bool fail = nb > SPLIT_BINS || (!L.last && nb > next_nseg);
  unsigned int entries = 0, tiles = 0, len = 0, begin = 0;
  SplitLeaf leaf{};
  if (!fail && tid < nb) {
    const unsigned int c0 = bin_cell[tid], c1 = bin_end[tid];
    len     = pre[c1] - pre[c0];
    begin   = s.begin + pre[c0];
    if (L.last && len > 0) {
      if (cell_bounds(s.map, c0, c1, ci, &leaf.lo, &leaf.span)) leaf.len |= LEAF_BOUNDED;
      if (len > L.cap) {
        // more than fits the chip: keys of a few values are counted, others are left to the radix passes
        fail = PAIRS || !(leaf.len & LEAF_BOUNDED) || leaf.span > COUNT_SPAN || len > COUNT_MOST * L.cap;
        leaf.len |= LEAF_COUNT;
      }
    }
    entries = L.last && len > 0 ? 1 : 0;
    tiles   = L.last ? 0 : (len + next_tile - 1) / next_tile;
  }
  if (__syncthreads_or(fail)) {
    if (tid == 0) atomicMax(&ctrl->route, (unsigned int)ROUTE_LATE);
    return;
  }
  unsigned int all_entries, all_tiles;
  const unsigned int e0 = scan(entries, &all_entries), t0 = scan(tiles, &all_tiles);
  if (tid == 0) {
    sh_leaf0 = all_entries ? atomicAdd(&ctrl->split_nleaf, all_entries) : 0;
    if (!L.last) {
      ctrl->split_nseg   = nb;
      ctrl->split_ntiles = all_tiles;
    }
  }
  __syncthreads();
  if (tid < nb) {
    bin_tile[tid]  = t0;
    bin_tiles[tid] = tiles;
    L.cursor[(size_t)seg * SPLIT_BINS + tid] = begin;
    if (entries) {
      leaf.begin = begin;
      leaf.len |= len;
      leaves[sh_leaf0 + e0] = leaf;
    }
    if (!L.last) {
      next_segs[tid].begin = begin;
      next_segs[tid].len   = len;
      next_segs[tid].tile0 = t0;
      next_segs[tid].drops = 0;
    }
  }
  __syncthreads();
  // the table cell -> bucket, and tile -> segment of the next level: a warp per bucket
  unsigned short* lut = L.lut + (size_t)seg * C;
  for (unsigned int b = warp; b < nb; b += PACK_THREADS / 32) {
    for (unsigned int c = bin_cell[b] + lane; c < bin_end[b]; c += 32) lut[c] = (unsigned short)b;
    if (!L.last)
      for (unsigned int i = lane; i < bin_tiles[b]; i += 32) next_tile_seg[bin_tile[b] + i] = (unsigned short)b;
  }
}

// ---- split: moves the keys of a tile to their buckets ----
// What bounds it is the shared-memory pipe (81 % busy for int32 keys, 17.5 wavefronts per 32 keys) and, with two blocks of 64
// registers per thread on an SM, latency; DRAM is 30 to 40 % busy.  2^28 int32 keys: shared counters and staged
// bucket numbers 1.12 ms, the counters below 0.99, the next tile's keys on their way while a tile goes out 0.79; 2^28 uint64 keys
// with positions in order 2.5 -> 1.9 -> 1.6.  Three blocks with smaller tiles lose (int32 2^25 96 -> 122 us: shorter runs, and
// the counters' scan is shared by fewer keys); a product instead of the table where keys lie evenly takes three
// wavefronts away and 2 % of the time.
//
// 32 random words lie three or four deep in the banks.  So every lane
// has counters of its own, in its own bank: counting a key and looking its place up take one wavefront each, whatever
// the keys (keys that come in order would meet in one counter, at two cycles per lane).  The order inside
// a bucket is the lanes'; bucket and destination of a staged key are found once more from the key, by neighbours that
// look at neighbouring words, instead of travelling with it through random places.
template <int KB, bool PAIRS> struct SplitSmem {
  static constexpr int TILE = SplitCfg<KB, PAIRS>::TILE;
  static constexpr size_t OFF_POS  = (size_t)TILE * KB;
  static constexpr size_t OFF_CNT  = OFF_POS + (PAIRS ? (size_t)TILE * 4 : 0);
  static constexpr size_t OFF_GOFS = OFF_CNT + (size_t)SPLIT_BINS * 128;
  static constexpr size_t OFF_LUT  = OFF_GOFS + SPLIT_BINS * 4;
  static __host__ __device__ size_t bytes(unsigned int cells) { return OFF_LUT + (size_t)cells * 2; }
};

template <int KB, int FORM, bool PAIRS>
__global__ void __launch_bounds__(SPLIT_THREADS, 2) split_move_kernel(Ctrl* ctrl, SplitLevel L, typename KeyOf<KB>::type flip)
{
  using K             = typename KeyOf<KB>::type;
  using S             = SplitSmem<KB, PAIRS>;
  constexpr int ITEMS = SplitCfg<KB, PAIRS>::ITEMS, TILE = SplitCfg<KB, PAIRS>::TILE;
  static_assert(SPLIT_THREADS == 2 * SPLIT_BINS, "two threads per bucket");
  extern __shared__ __align__(16) unsigned char smem[];
  K* skey             = reinterpret_cast<K*>(smem);
  uint2* sboth        = reinterpret_cast<uint2*>(smem);   // 4-byte keys with positions: side by side
  uint32_t* spos      = reinterpret_cast<uint32_t*>(smem + S::OFF_POS);
  unsigned char* cnt  = smem + S::OFF_CNT;   // [bucket][lane]
  unsigned int* gofs  = reinterpret_cast<unsigned int*>(smem + S::OFF_GOFS);
  unsigned short* lut = reinterpret_cast<unsigned short*>(smem + S::OFF_LUT);
  __shared__ unsigned int wsum[SPLIT_THREADS / 32];
  __shared__ SplitSeg ss;
  chain_wait();
  if (ctrl->route != ROUTE_SPLIT) return;
  const unsigned int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const TileRange r = my_tiles(L.tile_seg ? ctrl->split_ntiles : L.nseg * L.tiles_per_seg);
  if (r.first >= r.end) return;
  const unsigned int ci = L.cells - 2 - split_nan_cells(FORM, PAIRS, L.cells);
  K* dst                = static_cast<K*>(L.dst_keys);
  // my half of bucket tid / 2's counters, 16 bytes at a time from a place that keeps the banks apart
  unsigned char* half = cnt + tid * 64;
  auto quad = [&](unsigned int k) -> uint4& { return *reinterpret_cast<uint4*>(half + ((k * 16 + tid * 8) & 48u)); };
#pragma unroll
  for (unsigned int k = 0; k < 4; ++k) quad(k) = make_uint4(0u, 0u, 0u, 0u);
  K key[ITEMS];
  unsigned int pos[PAIRS ? ITEMS : 1];
  unsigned int seg = 0, at = 0, valid = 0;   // of the tile in the registers
  auto fetch = [&](unsigned int t) {
    seg = L.tile_seg ? L.tile_seg[t] : t / L.tiles_per_seg;
    const SplitSeg* g = L.segs + seg;
    at                = (t - g->tile0) * TILE;
    valid             = min((unsigned int)TILE, g->len - at);
    const K* src      = static_cast<const K*>(L.src_keys) + g->begin + at + tid;
    if (valid == TILE) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) key[j] = src[j * SPLIT_THREADS];
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) key[j] = j * SPLIT_THREADS + tid < valid ? src[j * SPLIT_THREADS] : (K)0;
    }
    if constexpr (PAIRS) {
      if (L.src_pos != nullptr) {
        const uint32_t* psrc = L.src_pos + g->begin + at + tid;
        if (valid == TILE) {
#pragma unroll
          for (int j = 0; j < ITEMS; ++j) pos[j] = psrc[j * SPLIT_THREADS];
        } else {
#pragma unroll
          for (int j = 0; j < ITEMS; ++j) pos[j] = j * SPLIT_THREADS + tid < valid ? psrc[j * SPLIT_THREADS] : 0u;
        }
      }
    }
  };
  fetch(r.first);
  unsigned int cur = 0xFFFFFFFFu;
  for (unsigned int t = r.first; t < r.end; ++t) {
    if (seg != cur) {
      cur = seg;
      __syncthreads();  // (nobody looks at the last segment's table any more)
      const unsigned int* g = reinterpret_cast<const unsigned int*>(L.lut + (size_t)seg * L.cells);
      for (unsigned int i = tid; i < L.cells / 2; i += SPLIT_THREADS) reinterpret_cast<unsigned int*>(lut)[i] = g[i];
      if (tid < sizeof(SplitSeg) / 4) reinterpret_cast<unsigned int*>(&ss)[tid] = reinterpret_cast<const unsigned int*>(L.segs + seg)[tid];
    }
    __syncthreads();  // the counters are clear, the table is loaded, the last tile is out
    auto tile = [&](auto md, auto part_c) {
      constexpr unsigned int MODE = decltype(md)::value;
      constexpr bool PART         = decltype(part_c)::value;  // not full, or not all of its keys are moved
      const SplitMap m = ss.map;
      auto bucket_of = [&](K x, unsigned int p) -> unsigned int { return lut[cell_of<KB, FORM, PAIRS, MODE>(x, p, m, ci)]; };
      if (PAIRS && L.src_pos == nullptr) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) pos[PAIRS ? j : 0] = at + j * SPLIT_THREADS + tid;
      }
      // bucket << 8 | rank among the lane's keys of the bucket, two to a word
      unsigned int br[(ITEMS + 1) / 2], moved = 0;
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        unsigned int v = 0;
        key[j]         = split_image<KB, FORM>(key[j], flip);   // (what is staged)
        if (!PART || j * SPLIT_THREADS + tid < valid) {
          const unsigned int b = bucket_of(key[j], pos[PAIRS ? j : 0]);
          if (!PART || b != LUT_DROP) {
            v = (b << 8) | atomicAdd(reinterpret_cast<unsigned int*>(cnt + b * 128 + lane * 4), 1u);
            if (PART) moved |= 1u << j;
          }
        }
        if (j & 1) br[j / 2] |= v << 16; else br[j / 2] = v;
      }
      __syncthreads();
      // room in the buckets, and the places inside the tile
      unsigned int mine = 0;
#pragma unroll
      for (unsigned int k = 0; k < 4; ++k) {
        const uint4 c = quad(k);
        mine += c.x + c.y + c.z + c.w;
      }
      const unsigned int other = __shfl_xor_sync(0xFFFFFFFFu, mine, 1), both = mine + other;
      unsigned int g = 0;
      if ((tid & 1) == 0 && both) g = atomicAdd(&L.cursor[(size_t)seg * SPLIT_BINS + (tid >> 1)], both);
      unsigned int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (unsigned int)o) incl += u;
      }
      if (lane == 31) wsum[warp] = incl;
      __syncthreads();
      const unsigned int w     = lane < SPLIT_THREADS / 32 ? wsum[lane] : 0u;
      const unsigned int total = PART ? __reduce_add_sync(0xFFFFFFFFu, w) : (unsigned int)TILE;
      unsigned int run         = incl - mine + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u);
      const unsigned int start = run;
#pragma unroll
      for (unsigned int k = 0; k < 4; ++k) {
        const uint4 c = quad(k);
        uint4 p;
        p.x = run;
        p.y = p.x + c.x;
        p.z = p.y + c.y;
        p.w = p.z + c.z;
        run = p.w + c.w;
        quad(k) = p;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (!PART || (moved >> j & 1u)) {
          const unsigned int v = j & 1 ? br[j / 2] >> 16 : br[j / 2] & 0xFFFFu;
          const unsigned int p = *reinterpret_cast<const unsigned int*>(cnt + (v >> 8) * 128 + lane * 4) + (v & 0xFFu);
          if constexpr (PAIRS && KB == 4) {
            sboth[p] = make_uint2(key[j], pos[j]);
          } else {
            skey[p] = key[j];
            if (PAIRS) spos[p] = pos[PAIRS ? j : 0];
          }
        }
      }
      if ((tid & 1) == 0) gofs[tid >> 1] = g - start;
      __syncthreads();
      if (t + 1 < r.end) fetch(t + 1);  // (on its way while this tile goes out)
#pragma unroll
      for (unsigned int k = 0; k < 4; ++k) quad(k) = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned int p = j * SPLIT_THREADS + tid;
        if (!PART || p < total) {
          K k;
          unsigned int q = 0;
          if constexpr (PAIRS && KB == 4) {
            const uint2 both = sboth[p];
            k = both.x;
            q = both.y;
          } else {
            k = skey[p];
            if (PAIRS) q = spos[p];
          }
          const unsigned int d = gofs[bucket_of(k, q)] + p;
          dst[d]               = FORM == FORM_INT ? (K)(k ^ flip) : k;
          if (PAIRS) L.dst_pos[d] = q;
        }
      }
    };
    const bool part = valid < TILE || ss.drops;
    with_mode<FORM, PAIRS>(ss.map.mode, [&](auto md) {
      if (part) tile(md, std::true_type{});
      else tile(md, std::false_type{});
    });
  }
}

// ---- leaves: sorts a bucket on chip ----
// Like rows of one block (segmerge_kernel): a bucket per key, then networks of 16; bound by issue (81 thread instructions per
// int32 key, 140 per int64 key, 147 per float32 key with its position) and the shared-memory pipe.  2^26 int32 keys 281 us, 2^25
// int64 keys 228, 2^25 float32 keys with positions 257.  Bounds that the cells imply save the search for them (int64
// 2^27 1097 -> 893 us), and buckets of one word each the networks (uint64 argsort of 2^28 keys almost in order 2.7 -> 1.9 ms).  8-byte
// words get the registers of 24 warps per SM (80): with 64 they spill (int64 2^27 1271 -> 1058 us).  Fetching the next bucket's
// keys early gained nothing and made 8-byte pairs spill.
constexpr int LEAF_VT = 16;
template <int KB, bool PAIRS, int THREADS> struct LeafSmem {
  static constexpr int TILE   = THREADS * LEAF_VT;
  static constexpr int PADDED = TILE + TILE / 16 + 1;
  static constexpr bool WIDE  = PAIRS && KB == 8;              // images that need all 64 bits: positions beside them
  static constexpr size_t WB  = PAIRS || KB == 8 ? 8 : 4;
  static constexpr size_t OFF_PAY  = ((size_t)PADDED * WB + 15) / 16 * 16;
  static constexpr size_t OFF_CNT  = (OFF_PAY + (WIDE ? (size_t)PADDED * 4 : 0) + 15) / 16 * 16;
  static constexpr size_t CNT_BYTES = (size_t)TILE * 4 + (size_t)TILE / 16 * 16;
  static constexpr size_t BYTES     = OFF_CNT + CNT_BYTES;
};

struct LeafArgs {
  const SplitLeaf* leaves;
  const SplitMarks* marks;
  const void* keys;
  const uint32_t* pos;
  void* out;
  int64_t* idx64;
  uint32_t* idx32;
  const uint32_t* payload;  // null: the position itself
  int64_t index_offset;
  unsigned int pos_n;
};

// Sorts the block's words: w[j] (and its payload) has bucket bk[j] < TILE, or LEAF_NONE: beyond the bucket's end, or the
// largest word.  Buckets rise with the words.  The result stands in sw (and sp), padded, the largest words behind the
// others.  `done_when_placed`: a bucket's words are all equal.
constexpr unsigned int LEAF_NONE = 0xFFFFFFFFu;
template <typename W, bool SIDE, int THREADS>
__device__ __forceinline__ void leaf_order(W (&w)[LEAF_VT], unsigned int (&pay)[SIDE ? LEAF_VT : 1], unsigned int (&bk)[LEAF_VT], bool done_when_placed, W* sw,
                                           unsigned int* sp, unsigned char* cnt, unsigned int* wsum)
{
  constexpr int TILE = THREADS * LEAF_VT, WARPS = THREADS / 32;
  constexpr W WMAX   = (W)~(W)0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, first = tid * LEAF_VT;
  unsigned int rank = 0;
#pragma unroll
  for (int j = 0; j < LEAF_VT; ++j) {
    if (bk[j] != LEAF_NONE) {
      const unsigned int at = (bk[j] << 2) + (bk[j] & ~15u);
      const unsigned int r  = atomicAdd(reinterpret_cast<unsigned int*>(cnt + at), 1u);
      rank  = max(rank, r);
      bk[j] = at | (r << 16);
    }
  }
  // (a word to a bucket: nothing is left to do once they are placed)
  if (!__syncthreads_or(rank)) done_when_placed = true;
  int over;
  unsigned int total;
  {
    uint4* mine = reinterpret_cast<uint4*>(cnt + (size_t)tid * 80);
    uint4 c[4];
    unsigned int sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      c[j] = mine[j];
      sum += c[j].x + c[j].y + c[j].z + c[j].w;
    }
    unsigned int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    over = __syncthreads_or(rank >= (unsigned int)SM_BUCKET);
    const unsigned int u = lane < WARPS ? wsum[lane] : 0u;
    unsigned int run     = incl - sum + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? u : 0u);
    total                = __reduce_add_sync(0xFFFFFFFFu, u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 p;
      p.x = run;
      p.y = p.x + c[j].x;
      p.z = p.y + c[j].y;
      p.w = p.z + c[j].z;
      run = p.w + c[j].w;
      mine[j] = p;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < LEAF_VT; ++j) {
    if (bk[j] != LEAF_NONE) {
      const unsigned int p = *reinterpret_cast<const unsigned int*>(cnt + (bk[j] & 0xFFFFu)) + (bk[j] >> 16);
      sw[smpad(p)]         = w[j];
      if (SIDE) sp[smpad(p)] = pay[SIDE ? j : 0];
    }
  }
  for (unsigned int e = total + tid; e < (unsigned int)TILE; e += THREADS) {
    sw[smpad(e)] = WMAX;
    if (SIDE) sp[smpad(e)] = 0xFFFFFFFFu;
  }
  __syncthreads();
  if (done_when_placed) return;
  auto cmp_swap = [&](int a, int b) {
    const W x = w[a], y = w[b];
    bool s;
    if (SIDE) {
      const unsigned int p = pay[SIDE ? a : 0], q = pay[SIDE ? b : 0];
      s = y < x || (y == x && q < p);
      pay[SIDE ? a : 0] = s ? q : p;
      pay[SIDE ? b : 0] = s ? p : q;
    } else {
      s = y < x;
    }
    w[a] = s ? y : x;
    w[b] = s ? x : y;
  };
  auto read_words = [&](int at) {
#pragma unroll
    for (int j = 0; j < LEAF_VT; ++j) {
      w[j] = sw[smpad(at + j)];
      if (SIDE) pay[SIDE ? j : 0] = sp[smpad(at + j)];
    }
  };
  auto write_words = [&](int at) {
#pragma unroll
    for (int j = 0; j < LEAF_VT; ++j) {
      sw[smpad(at + j)] = w[j];
      if (SIDE) sp[smpad(at + j)] = pay[SIDE ? j : 0];
    }
  };
  // Blocks of 16, then the windows halfway between them: settles buckets of up to nine words (segmerge_kernel);
  // fuller ones take more rounds, and what three do not settle is merged.
  bool sorted = false;
  for (int round = 0; round < 3 && !sorted; ++round) {
    read_words(first);
    odd_even_merge_sort<LEAF_VT, 1>(cmp_swap);
    write_words(first);
    __syncthreads();
    if (tid < THREADS - 1) {
      read_words(first + LEAF_VT / 2);
      odd_even_merge_sort<LEAF_VT, LEAF_VT / 2>(cmp_swap);
      write_words(first + LEAF_VT / 2);
    }
    __syncthreads();
    sorted = !over;
    if (!sorted) {
      // every window is in order, and so are the eight words before the first and after the last one: what
      // remains are the steps between them
      const int i = first + LEAF_VT / 2 - 1;
      const W a = sw[smpad(i)], b = sw[smpad(i + 1)];
      sorted = !__syncthreads_or(b < a || (SIDE && a == b && sp[smpad(i + 1)] < sp[smpad(i)]));
    }
  }
  if (sorted) return;
  read_words(first);
  odd_even_merge_sort<LEAF_VT, 1>(cmp_swap);
  __syncthreads();
  write_words(first);
  __syncthreads();
  for (int run = LEAF_VT; run < TILE; run <<= 1) {
    const int pbase = first & ~(2 * run - 1);
    const int diag  = first - pbase;
    const int a0 = pbase, b0 = pbase + run;
    const int la = min(run, TILE - a0), lb = max(0, min(run, TILE - b0));   // (the block need not be a power of two)
    int lo = max(0, diag - lb), hi = min(diag, la);
    auto not_after = [&](int a, int b) {  // word a <= word b
      const W x = sw[smpad(a)], y = sw[smpad(b)];
      return x < y || (x == y && (!SIDE || sp[smpad(a)] <= sp[smpad(b)]));
    };
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (not_after(a0 + mid, b0 + diag - 1 - mid)) lo = mid + 1; else hi = mid;
    }
    int ia = lo, ib = diag - lo;
#pragma unroll
    for (int j = 0; j < LEAF_VT; ++j) {
      const bool take_a = ib >= lb || (ia < la && not_after(a0 + ia, b0 + ib));
      const int from    = smpad(take_a ? a0 + ia : b0 + ib);
      w[j]              = sw[from];
      if (SIDE) pay[SIDE ? j : 0] = sp[from];
      ia += take_a ? 1 : 0;
      ib += take_a ? 0 : 1;
    }
    __syncthreads();
    write_words(first);
    __syncthreads();
  }
}

template <int KB, bool PAIRS, int THREADS>
constexpr int LEAF_PER_SM = (KB == 8 || PAIRS ? 768 : 1280) / THREADS;

template <int KB, int FORM, bool PAIRS, int THREADS>
__global__ void __launch_bounds__(THREADS, LEAF_PER_SM<KB, PAIRS, THREADS>)
split_leaf_kernel(const Ctrl* ctrl, LeafArgs A, typename KeyOf<KB>::type flip)
{
  using K = typename KeyOf<KB>::type;
  using S = LeafSmem<KB, PAIRS, THREADS>;
  using W = typename KeyOf<(int)S::WB>::type;
  constexpr unsigned int NB = S::TILE;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ K bounds[2 * THREADS / 32];
  __shared__ unsigned int wsum[THREADS / 32];
  W* sw              = reinterpret_cast<W*>(smem);
  unsigned int* sp   = reinterpret_cast<unsigned int*>(smem + S::OFF_PAY);
  unsigned char* cnt = smem + S::OFF_CNT;
  chain_wait();
  if (ctrl->route != ROUTE_SPLIT) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned int nleaf = ctrl->split_nleaf;
  // (other patterns than the usual ones of NaNs and zeros: a loop of its own, so that the usual one costs no more for it)
  const bool marked = FORM != FORM_INT && !PAIRS && (A.marks->nan != 0 || (A.marks->flags & MARK_NEG_ZERO) != 0);
  for (unsigned int l = blockIdx.x; l < nleaf; l += gridDim.x) {
    const SplitLeaf leaf = A.leaves[l];
    if (leaf.len & LEAF_FILL) {
      if (!PAIRS) {
        K* dst = static_cast<K*>(A.out) + leaf.begin;
        const unsigned int n = leaf.len & ~LEAF_FILL;
        for (unsigned int i = tid; i < n; i += THREADS) dst[i] = (K)leaf.lo;
      }
      continue;
    }
    const unsigned int n = leaf.len & LEAF_LEN;
    if (!PAIRS && (leaf.len & LEAF_COUNT)) {
      // few values, many keys: counted, and written by their places
      unsigned int* count = reinterpret_cast<unsigned int*>(cnt);
      const K* from       = static_cast<const K*>(A.keys) + leaf.begin;
      K* to               = static_cast<K*>(A.out) + leaf.begin;
      const unsigned int values = (unsigned int)leaf.span + 1;
      for (unsigned int i = tid; i < (values + 31) / 32 * 32; i += THREADS) count[i] = 0;
      __syncthreads();
      constexpr unsigned int AHEAD = 8;
      for (unsigned int i = tid; i < n; i += AHEAD * THREADS) {
        K k[AHEAD];
#pragma unroll
        for (unsigned int j = 0; j < AHEAD; ++j) k[j] = i + j * THREADS < n ? from[i + j * THREADS] : (K)0;
#pragma unroll
        for (unsigned int j = 0; j < AHEAD; ++j)
          if (i + j * THREADS < n) atomicAdd(&count[(unsigned int)(split_image<KB, FORM>(k[j], flip) - (K)leaf.lo)], 1u);
      }
      __syncthreads();
      if (warp == 0) {   // counts -> ends
        unsigned int run = 0;
        for (unsigned int i = lane; i < (values + 31) / 32 * 32; i += 32) {
          unsigned int incl = count[i];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const unsigned int u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += u;
          }
          count[i] = run + incl;
          run += __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
      }
      __syncthreads();
      auto raw_of = [&](unsigned int v) -> K {
        const K o = (K)((K)leaf.lo + v);
        if constexpr (FORM != FORM_INT) return marked_raw<KB>(o, A.marks);
        else return (K)(o ^ flip);
      };
      if (n > 32 * values) {
        for (unsigned int v = warp; v < values; v += THREADS / 32) {   // a warp writes the copies of a value
          const unsigned int first = v ? count[v - 1] : 0u, end = count[v];
          const K raw = raw_of(v);
          for (unsigned int i = first + lane; i < end; i += 32) to[i] = raw;
        }
      } else {
        for (unsigned int i = tid; i < n; i += THREADS) {
          unsigned int a = 0, b = values - 1;   // the first value that ends behind i
          while (a < b) {
            const unsigned int mid = (a + b) >> 1;
            if (count[mid] > i) b = mid; else a = mid + 1;
          }
          to[i] = raw_of(a);
        }
      }
      __syncthreads();
      continue;
    }
    const K* src         = static_cast<const K*>(A.keys) + leaf.begin;
    const uint32_t* psrc = PAIRS ? A.pos + leaf.begin : nullptr;
    K img[LEAF_VT];
    unsigned int pos[PAIRS ? LEAF_VT : 1];
#pragma unroll
    for (int j = 0; j < LEAF_VT; ++j) {
      const unsigned int e = j * THREADS + tid;
      img[j]               = e < n ? src[e] : (K)0;
      if (PAIRS) pos[PAIRS ? j : 0] = e < n ? psrc[e] : 0xFFFFFFFFu;
    }
    for (int i = tid; i < (int)(S::CNT_BYTES / 16); i += THREADS) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
    using RB = RowBuckets<KB, (int)NB>;
    K lo = (K)leaf.lo, hi = (K)(leaf.lo + leaf.span);
#pragma unroll
    for (int j = 0; j < LEAF_VT; ++j) img[j] = split_image<KB, FORM>(img[j], flip);
    if (leaf.len & LEAF_BOUNDED) {
      __syncthreads();
    } else {
      lo = (K)~(K)0, hi = 0;
#pragma unroll
      for (int j = 0; j < LEAF_VT; ++j) {
        if ((unsigned int)(j * THREADS + tid) < n && (FORM == FORM_INT || RB::upper(img[j]) - RB::FIN_LO < RB::FIN_N)) {
          lo = img[j] < lo ? img[j] : lo;
          hi = img[j] > hi ? img[j] : hi;
        }
      }
      if constexpr (KB == 4) {
        lo = __reduce_min_sync(0xFFFFFFFFu, lo);
        hi = __reduce_max_sync(0xFFFFFFFFu, hi);
      } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const K a = __shfl_xor_sync(0xFFFFFFFFu, lo, o), b = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
          lo = a < lo ? a : lo;
          hi = b > hi ? b : hi;
        }
      }
      if (lane == 0) {
        bounds[2 * warp]     = lo;
        bounds[2 * warp + 1] = hi;
      }
      __syncthreads();
#pragma unroll
      for (int v = 0; v < THREADS / 32; ++v) {
        const K a = bounds[2 * v], b = bounds[2 * v + 1];
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
      }
    }
    if (FORM != FORM_INT && lo > hi) lo = hi = (K)~(K)0;  // nothing finite: NaNs are taken for one image
    // Bucket: a narrow range of images has buckets for each of them, of argsorts cut by position; else linear in
    // the value of floats (infinities and NaNs at the ends), in the image of integers.
    const unsigned long long span = (unsigned long long)hi - (unsigned long long)lo;
    const bool exact = span < NB;
    unsigned int bk[LEAF_VT];
    if (exact) {
      const unsigned int mult   = PAIRS ? NB / ((unsigned int)span + 1) : 1u;
      const unsigned int pscale = PAIRS && mult > 1 ? (unsigned int)min(((unsigned long long)mult << 32) / A.pos_n, 0xFFFFFFFFull) : 0u;
#pragma unroll
      for (int j = 0; j < LEAF_VT; ++j) {
        bk[j] = (unsigned int)(img[j] - lo) * mult + (PAIRS ? __umulhi(pos[PAIRS ? j : 0], pscale) : 0u);
        if (FORM != FORM_INT) bk[j] = img[j] < lo ? 0u : img[j] > hi ? NB - 1 : bk[j];
      }
    } else {
      // NaNs have the last buckets to themselves, by position (argsorts), or need none at all
      constexpr unsigned int NANS = FORM != FORM_INT && PAIRS ? NB / 8 : 0;
      using RN = RowBuckets<KB, (int)(NB - NANS)>;
      RN rb;
      const unsigned int nscale = NANS ? (unsigned int)(((unsigned long long)NANS << 32) / A.pos_n) : 0u;
      if constexpr (FORM != FORM_INT) rb.from_floats(RN::upper(lo), RN::upper(hi));
      // (within a binade or two the image is as good)
      constexpr unsigned long long BINADES = 2ull << (KB == 8 ? 52 : 23);
      if (FORM == FORM_INT || !rb.ok || span < BINADES) {
        rb.from_images(lo, hi);
#pragma unroll
        for (int j = 0; j < LEAF_VT; ++j) {
          bk[j] = rb.bucket_image(img[j]);
          if (FORM != FORM_INT) bk[j] = img[j] < lo ? 0u : img[j] > hi ? NB - NANS - 1 : bk[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < LEAF_VT; ++j) bk[j] = rb.bucket_float(img[j]);
      }
      if constexpr (FORM != FORM_INT) {
#pragma unroll
        for (int j = 0; j < LEAF_VT; ++j)
          if (img[j] == (K)~(K)0) bk[j] = PAIRS ? NB - NANS + __umulhi(pos[PAIRS ? j : 0], nscale) : LEAF_NONE;
      }
    }
#pragma unroll
    for (int j = 0; j < LEAF_VT; ++j)
      if ((unsigned int)(j * THREADS + tid) >= n) bk[j] = LEAF_NONE;
    if constexpr (PAIRS) {
      bool wide = false;
      if constexpr (KB == 8) wide = (span >> 32) != 0 || FORM != FORM_INT;
      if (wide) {
        if constexpr (KB == 8) leaf_order<W, true, THREADS>(img, pos, bk, false, sw, sp, cnt, wsum);
      } else {
        W w[LEAF_VT];
        unsigned int none[1];
#pragma unroll
        for (int j = 0; j < LEAF_VT; ++j) w[j] = ((unsigned long long)(unsigned int)(KB == 4 ? img[j] : img[j] - lo) << 32) | pos[PAIRS ? j : 0];
        leaf_order<W, false, THREADS>(w, none, bk, false, sw, sp, cnt, wsum);
      }
      for (unsigned int e = tid; e < n; e += THREADS) {
        const unsigned int p = wide ? sp[smpad(e)] : (unsigned int)sw[smpad(e)];
        const unsigned int v = A.payload ? A.payload[p] : p;
        if (A.idx64) A.idx64[leaf.begin + e] = A.index_offset + (int64_t)v;
        else A.idx32[leaf.begin + e] = v;
      }
    } else {
      unsigned int none[1];
      K* dst = static_cast<K*>(A.out) + leaf.begin;
      bool narrow = false;
      if constexpr (KB == 8 && FORM == FORM_INT) {
        // images within 2^32: half the words
        narrow = (span >> 32) == 0;
        if (narrow) {
          uint32_t w[LEAF_VT];
          uint32_t* sw32 = reinterpret_cast<uint32_t*>(smem);
#pragma unroll
          for (int j = 0; j < LEAF_VT; ++j) w[j] = (uint32_t)(img[j] - lo);
          leaf_order<uint32_t, false, THREADS>(w, none, bk, exact, sw32, sp, cnt, wsum);
          for (unsigned int e = tid; e < n; e += THREADS) dst[e] = (K)((lo + sw32[smpad(e)]) ^ flip);
        }
      }
      if (!narrow) {
        leaf_order<W, false, THREADS>(img, none, bk, exact && FORM == FORM_INT, sw, sp, cnt, wsum);
        if (FORM != FORM_INT && marked) {
          for (unsigned int e = tid; e < n; e += THREADS) dst[e] = marked_raw<KB>((K)sw[smpad(e)], A.marks);
        } else {
          for (unsigned int e = tid; e < n; e += THREADS) {
            const K o = (K)sw[smpad(e)];
            if constexpr (FORM != FORM_INT) dst[e] = sm_from_ordered<KB>(o, XF_FLOAT);
            else dst[e] = (K)(o ^ flip);
          }
        }
      }
    }
    __syncthreads();
  }
}

// ---- host side ----
inline int split_sms()
{
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
template <typename Kern>
inline cudaError_t split_smem(Kern kern, size_t smem)
{
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Copies of each key above which the passes are faster: the positions of equal keys are put in order by the networks and the merging of
// leaf_order.  Time of the splits in parts of the passes' for argsorts of n / c evenly used values:
//   float32, 6 * 10^6 (two splits)   c = 8 0.90, 20 1.25, 100 1.50, 400 1.68;  2 * 10^7  0.89, 1.30, 1.75, 1.97
//   float32, 7 * 10^5 (one split)    c = 20 0.90, 100 0.93, 150 1.02, 400 1.06
//   float64, 2.5 * 10^5              c = 8 0.79, 20 1.04, 100 1.21;  8 * 10^6  c = 8 0.63, 20 0.92, 40 1.07, 250 1.43
//   int64, 2.4 * 10^7                c = 8 0.66, 20 0.93, 40 1.19, 400 1.46
//   float32, 300 rows of 16400       c = 8 0.85, 20 1.16, 40 1.34 (int32 0.81, 1.10, 1.30);  sent back 1.15
//   float64, rows                    30000 of 300 copies 1.09, 100003 of 1000 0.95; sent back 1.06 to 1.12
// Sorts have no positions to be put in order, but of floats values that fill cells.
inline unsigned int split_most_copies(int kb, bool pairs, unsigned int nseg, const SplitPlan& plan)
{
  if (!pairs) return plan.lev[plan.levels - 1].cap / 2;
  if (kb == 8) return nseg != 1 ? 2048 : 24;
  return nseg != 1 ? 24 : plan.levels == 1 ? 128 : 12;
}

template <int KB, int FORM0, bool PAIRS>
inline cudaError_t split_form(typename KeyOf<KB>::type flip, const SplitPlan& plan, const SplitJob& job, Ctrl* ctrl, cudaStream_t stream)
{
  constexpr unsigned int TILE = SplitCfg<KB, PAIRS>::TILE;
  const size_t volume         = (size_t)job.seg_len * job.nseg;
  SplitLeaf* leaves           = reinterpret_cast<SplitLeaf*>(job.tables + plan.off_leaves);
  unsigned short* tile_seg    = reinterpret_cast<unsigned short*>(job.tables + plan.off_tile_seg);
  auto segs_of = [&](int l) { return reinterpret_cast<SplitSeg*>(job.tables + plan.off_segs[l]); };
  constexpr int FORM1 = FORM0 == FORM_FLOAT ? FORM_IMAGE : FORM0;   // after the first split
  cudaError_t e;
  const unsigned int sms = (unsigned int)split_sms();
  for (int l = 0; l < plan.levels; ++l) {
    const SplitShape& sh = plan.lev[l];
    SplitLevel L{};
    L.segs          = segs_of(l);
    L.hist          = reinterpret_cast<unsigned int*>(job.tables + plan.off_hist[l]);
    L.lut           = reinterpret_cast<unsigned short*>(job.tables + plan.off_lut[l]);
    L.cursor        = reinterpret_cast<unsigned int*>(job.tables + plan.off_cursor[l]);
    L.tile_seg      = l == 0 ? nullptr : tile_seg;
    L.nseg          = sh.nseg;
    L.tiles_per_seg = (job.seg_len + TILE - 1) / TILE;
    L.seg_len       = job.seg_len;
    L.cells         = sh.cells;
    L.cap           = sh.cap;
    L.last          = l == plan.levels - 1;
    L.pos_n         = job.seg_len;
    L.radix_if      = plan.radix_if;
    L.rounds        = l == 0 ? split_rounds(job.seg_len, job.nseg, PAIRS) : 1;
    L.leaf_cap      = plan.lev[plan.levels - 1].cap;
    L.most_copies   = split_most_copies(KB, PAIRS, job.nseg, plan);
    L.marks         = reinterpret_cast<SplitMarks*>(job.tables + plan.off_marks);
    L.src_keys      = l == 0 ? job.in : job.tmp_keys[0];
    L.src_pos       = PAIRS && l > 0 ? job.tmp_pos[0] : nullptr;
    L.dst_keys      = job.tmp_keys[l];
    L.dst_pos       = PAIRS ? job.tmp_pos[l] : nullptr;
    const unsigned int most_tiles = (unsigned int)(l == 0 ? (size_t)L.tiles_per_seg * job.nseg : volume / TILE + sh.nseg);
    {
      prof::Scope ps(prof::K_HIST, stream);
      auto sample = l == 0 ? split_sample_kernel<KB, FORM0, PAIRS, SPLIT_SAMPLES> : split_sample_kernel<KB, FORM1, PAIRS, SPLIT_SAMPLES_NEXT>;
      const unsigned int prints = split_prints(L.rounds);
      const size_t smem         = (size_t)(sh.cells > prints ? sh.cells : prints) * 4;
      e = split_smem(sample, smem);
      if (e != cudaSuccess) return e;
      e = launch_chained(sample, sh.nseg, SPLIT_THREADS, smem, stream, ctrl, L, l > 0 ? 0u : job.nseg == 1 ? 2u : 1u, flip);
      if (e != cudaSuccess) return e;
    }
    {
      prof::Scope ps(prof::K_HIST, stream);
      auto cells = l == 0 ? split_cells_kernel<KB, FORM0, PAIRS> : split_cells_kernel<KB, FORM1, PAIRS>;
      e = split_smem(cells, (size_t)sh.cells * 4);
      if (e != cudaSuccess) return e;
      const unsigned int grid = sms * 3;
      e = launch_chained(cells, grid < most_tiles ? grid : most_tiles, SPLIT_THREADS, (size_t)sh.cells * 4, stream, ctrl, L, flip);
      if (e != cudaSuccess) return e;
    }
    {
      prof::Scope ps(prof::K_SCAN, stream);
      auto pack         = l == 0 ? split_pack_kernel<KB, FORM0, PAIRS> : split_pack_kernel<KB, FORM1, PAIRS>;
      const size_t smem = pack_smem(sh.cells);
      e = split_smem(pack, smem);
      if (e != cudaSuccess) return e;
      e = launch_chained(pack, sh.nseg, PACK_THREADS, smem, stream, ctrl, L, leaves, L.last ? nullptr : segs_of(l + 1), tile_seg, L.last ? 0u : plan.lev[l + 1].nseg, TILE, flip);
      if (e != cudaSuccess) return e;
    }
    {
      prof::Scope ps(prof::K_SWEEP, stream);
      auto move         = l == 0 ? split_move_kernel<KB, FORM0, PAIRS> : split_move_kernel<KB, FORM1, PAIRS>;
      const size_t smem = SplitSmem<KB, PAIRS>::bytes(sh.cells);
      e = split_smem(move, smem);
      if (e != cudaSuccess) return e;
      const unsigned int grid = sms * 2;
      e = launch_chained(move, grid < most_tiles ? grid : most_tiles, SPLIT_THREADS, smem, stream, ctrl, L, flip);
      if (e != cudaSuccess) return e;
    }
  }
  LeafArgs A{};
  A.leaves       = leaves;
  A.marks        = reinterpret_cast<const SplitMarks*>(job.tables + plan.off_marks);
  A.keys         = job.tmp_keys[plan.levels - 1];
  A.pos          = PAIRS ? job.tmp_pos[plan.levels - 1] : nullptr;
  A.out          = job.out;
  A.idx64        = job.idx64;
  A.idx32        = job.idx32;
  A.payload      = job.payload;
  A.index_offset = job.index_offset;
  A.pos_n        = job.seg_len;
  auto leaf_of   = [&](auto threads) {
    constexpr int THREADS = decltype(threads)::value;
    prof::Scope ps(prof::K_SEGSORT, stream);
    auto leaf         = split_leaf_kernel<KB, FORM1, PAIRS, THREADS>;
    const size_t smem = LeafSmem<KB, PAIRS, THREADS>::BYTES;
    cudaError_t err = split_smem(leaf, smem);
    if (err != cudaSuccess) return err;
    return launch_chained(leaf, sms * LEAF_PER_SM<KB, PAIRS, THREADS>, THREADS, smem, stream, ctrl, A, flip);
  };
  const unsigned int cap = plan.lev[plan.levels - 1].cap;
  if (cap <= 128 * LEAF_VT) return leaf_of(std::integral_constant<int, 128>{});
  if (cap <= 256 * LEAF_VT) return leaf_of(std::integral_constant<int, 256>{});
  return leaf_of(std::integral_constant<int, (PAIRS ? LEAF_MOST_PAIRS : LEAF_MOST) / LEAF_VT>{});
}

template <int KB>
inline cudaError_t split_any(int xf, const SplitPlan& plan, const SplitJob& job, Ctrl* ctrl, cudaStream_t stream)
{
  using K      = typename KeyOf<KB>::type;
  const K flip = xf == XF_SIGNED ? (K)((K)1 << (8 * KB - 1)) : (K)0;
  const bool pairs = job.idx64 != nullptr || job.idx32 != nullptr;
  if (xf == XF_FLOAT)
    return pairs ? split_form<KB, FORM_FLOAT, true>(flip, plan, job, ctrl, stream) : split_form<KB, FORM_FLOAT, false>(flip, plan, job, ctrl, stream);
  return pairs ? split_form<KB, FORM_INT, true>(flip, plan, job, ctrl, stream) : split_form<KB, FORM_INT, false>(flip, plan, job, ctrl, stream);
}

}  // namespace b2s
