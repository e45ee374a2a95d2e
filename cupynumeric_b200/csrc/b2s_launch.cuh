// Host-side launchers of the local sort kernels, templated on the key width so that each width
// compiles in a translation unit of its own.
#pragma once

#include "b2s_prof.h"
#include "b2s_radix.cuh"
#include "b2s_segsort.cuh"
#include "b2s_segmerge.cuh"
#include "b2s_segwarp.cuh"
#include "b2s_split_plan.cuh"

#include <cstdlib>
#include <type_traits>

namespace b2s {

// Largest segment the on-chip segmented kernel takes.
constexpr unsigned int SEG_CAP = 8192;

// Tile shapes of the onesweep pass: threads, keys per thread, CTAs per SM and look-back window by key
// width, payload and size class, found by sweeps on B200.
//
// Short arrays (1-D sorts of up to SMALL_MAX keys) take small tiles: with the others 10^5 keys are 13 to 20
// tiles on 148 SMs, and a pass lasts as long as one tile's chain of loading, ranking and looking back.
// Their walks read 16 entries per round trip, since most tiles run at once and few prefixes are ready.
// Measured, medium -> small tiles: float32 argsort of 20000 116 -> 63 us, of 100003 106 -> 65, of 400000 122 ->
// 73; int64 argsort of 20000 169 -> 110 us; int32 sort of 400000 73 -> 67; at 2^20 keys the medium tiles win
// (float32 argsort 95 against 124 us).  4 keys per thread lose to 8 from 4-byte keys on, 12 at the short end.
//
// Long arrays (1-D sorts of more than MEDIUM_MAX keys), medium -> large tiles: int32 sort of 2^28 4.94 -> 4.71
// ms (24 keys per thread amortise the work per tile better), float16 sort of 2^27 1.66 -> 1.54 (384
// threads), int64 sort of 2^28 Zipf keys 7.45 -> 7.33 and float64 sort of 2^27 6.52 -> 6.24 (20 keys leave
// the registers of a fourth CTA per SM), int64 argsort of 2^27 7.67 -> 7.44 (longer digit runs).  The border
// is where the scratch of b2s_local_sort_noalloc ends: the smaller tiles need a larger look-back table,
// and what fits that scratch has to go on fitting.  Segments keep the medium tiles, whose last tile wastes least.
enum : int { SWEEP_SMALL = 0, SWEEP_MEDIUM = 1, SWEEP_LARGE = 2 };
constexpr size_t SMALL_TILE = 256 * 8;
constexpr size_t SMALL_MAX  = 240 * SMALL_TILE;
constexpr size_t MEDIUM_MAX = (size_t)1 << 21;
template <int KB, bool PAIRS, int SIZE = SWEEP_MEDIUM> struct SweepCfg {
  static constexpr bool LARGE  = SIZE == SWEEP_LARGE && !(PAIRS && KB < 8);
  static constexpr int THREADS = SIZE == SWEEP_SMALL || !LARGE ? 256 : PAIRS ? 512 : KB == 2 ? 384 : 256;
  static constexpr int ITEMS   = SIZE == SWEEP_SMALL ? (int)(SMALL_TILE / 256)
                               : LARGE               ? (PAIRS ? 14 : KB == 8 || KB == 2 ? 20 : 24)
                                                     : (PAIRS ? (KB == 8 ? 20 : 32) : (KB == 8 ? 28 : 20));
  static constexpr int MINCTAS = SIZE == SWEEP_SMALL ? 4
                               : LARGE               ? (PAIRS ? 2 : KB == 2 ? 3 : 4)
                                                     : (PAIRS ? 3 : (KB == 8 ? 3 : 4));
  static constexpr int CHAINS  = 1;
  static constexpr int TILE    = THREADS * ITEMS;
  static constexpr int WINDOW  = SIZE == SWEEP_SMALL ? 16 : LB_WINDOW;
};

// Where the look-back table of every workspace starts: behind the control block and nothing else, since the short
// window of a first tile's successors reads that far in front of the table (look_back), without using what it finds.
constexpr size_t LOOKBACK_OFFSET = (sizeof(Ctrl) + 255) / 256 * 256;
static_assert(LOOKBACK_OFFSET >= (LB_WINDOW - 1) * RADIX * sizeof(unsigned int), "a short window may read the control block");

struct Radix1dLayout {
  size_t off_lookback, lookback_used, off_keys[2], off_idx[2], total;
  unsigned int tiles;
};

template <int KB>
inline Radix1dLayout radix_1d_layout(size_t n, bool pairs)
{
  Radix1dLayout l{};
  const size_t small = SMALL_TILE, medium = pairs ? SweepCfg<KB, true>::TILE : SweepCfg<KB, false>::TILE,
               large = pairs ? SweepCfg<KB, true, SWEEP_LARGE>::TILE : SweepCfg<KB, false, SWEEP_LARGE>::TILE;
  auto tiles_of = [&](size_t m) {
    const size_t tile = m <= SMALL_MAX ? small : m <= MEDIUM_MAX ? medium : large;
    return (m + tile - 1) / tile;
  };
  l.tiles = (unsigned int)tiles_of(n);
  // room for the table of every shorter sort too, so that a workspace serves any length below its own
  size_t rows = tiles_of(n);
  if (n > SMALL_MAX && tiles_of(SMALL_MAX) > rows) rows = tiles_of(SMALL_MAX);
  if (n > MEDIUM_MAX && tiles_of(MEDIUM_MAX) > rows) rows = tiles_of(MEDIUM_MAX);
  size_t off           = LOOKBACK_OFFSET;
  l.off_lookback       = off;
  l.lookback_used      = align_up((size_t)KB * l.tiles * RADIX * sizeof(unsigned int), 256);
  off += align_up((size_t)KB * rows * RADIX * sizeof(unsigned int), 256);
  for (int i = 0; i < 2; ++i) {
    l.off_keys[i] = off;
    off += align_up(n * KB, 256);
  }
  for (int i = 0; i < 2; ++i) {
    l.off_idx[i] = off;
    if (pairs) off += align_up(n * 4, 256);
  }
  l.total = off;
  return l;
}

// Launches a kernel that calls chain_wait() before it reads anything its predecessor in the stream wrote:
// its launch and first instructions overlap the predecessor's end.  A sort of 10^5 keys is a chain of six
// launches: float32 argsort 67 -> 53 us, float64 sort of 2^20 163 -> 142.  Letting the CTAs in earlier, as soon as
// the predecessor's have all started, crowds them on the SMs that have room then: float64 sort of 2^20 194 us.
// Beyond CHAIN_MAX keys the launches no longer matter, and a pass that takes its ticket only after the
// wait loses more than it hides (Zipf int64 sort of 2^28 7.17 -> 7.29 ms; at 2^22 keys int64 argsort still
// gains, 343 -> 320 us): those sorts, and segments, launch their passes the plain way.
constexpr size_t CHAIN_MAX = (size_t)1 << 23;
template <int KB, int XF, bool PAIRS, int SIZE = SWEEP_MEDIUM, bool CHAINED = false>
inline cudaError_t launch_sweeps(Ctrl* ctrl, unsigned int* lookback, unsigned int tiles, SegGeom geo,
                                 int64_t index_offset, cudaStream_t stream)
{
  using C   = SweepCfg<KB, PAIRS, SIZE>;
  using S   = SweepSmem<KB, PAIRS, C::THREADS, C::ITEMS, C::CHAINS>;
  auto kern = onesweep_kernel<KB, XF, PAIRS, C::THREADS, C::ITEMS, C::CHAINS, C::MINCTAS, C::WINDOW, CHAINED>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::BYTES);
  if (e != cudaSuccess) return e;
  for (int pass = 0; pass < KB; ++pass) {
    prof::Scope ps(prof::K_SWEEP, stream);
    unsigned int* table = lookback + (size_t)pass * tiles * RADIX;
    if (CHAINED) e = launch_chained(kern, tiles, C::THREADS, S::BYTES, stream, ctrl, table, pass, geo, index_offset);
    else kern<<<tiles, C::THREADS, S::BYTES, stream>>>(ctrl, table, pass, geo, index_offset);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

// Testing aid and comparisons: B2S_SPLIT=0 leaves every sort to the radix passes, another number is the length from which
// 1-D sorts are tried by the splitting kernels, whatever bytes of the keys differ; rows are tried then at every length.
inline long long split_override()
{
  const char* e = std::getenv("B2S_SPLIT");
  return e == nullptr ? -1 : std::atoll(e);
}

// Whether a 1-D sort is tried by the splitting kernels first, and which keys the sample then sends back to the radix
// passes.  Measured on one GPU, radix passes -> splits, us per call:
//   int32 sort, full range         10^7 253 -> 195, 2^24 371 -> 272, 8 * 10^7 1450 -> 1016
//   float32 sort, normal           1.1 * 10^6 (one split) 69 -> 61, 3.5 (two) 117 -> 119, 6 191 -> 177, 20 450 -> 371, 80 1517 -> 1163
//   float32 argsort                7 * 10^5 97 -> 61, 2 * 10^6 99 -> 100, 6 230 -> 209, 20 583 -> 517, 80 1853 -> 1747
//   int64 sort, full range         2.5 * 10^7 1298 -> 586, 8 3780 -> 1875
//   int64 argsort, full range      2.5 * 10^7 1541 -> 807, 8 4495 -> 2435
//   float64 sort, normal           2 * 10^5 84 -> 69, 7 131 -> 70, 80 * 10^6 3702 -> 2006
//   float64 argsort                2 * 10^5 87 -> 70, 4 103 -> 75, 80 * 10^6 4587 -> 2536
//   uint64 argsort, almost in order  3 * 10^7 940 -> 769, 2^28 8094 -> 6225
//   int64 sort, Zipf               3 * 10^7 921 -> 468, 2^28 7174 -> 3120
// Whether bytes are constant is not known before the sample; keys that are sent back have paid for it and for the launches: 13
// to 17 us for one split, 22 to 30 for two.  On both sides of the borders, passes -> splits, and what goes back:
//   int32 sort 16       full range 10^7 264 -> 197 and 14 * 10^6 335 -> 241, but of 65536 values 154 -> 176 and 185 -> 208; 16 * 10^6
//                       365 -> 264, 205 -> 227: a tenth.  A hundred values stay, one byte differing: 16 134 -> 134, 40 259 -> 237, 160 * 10^6
//                       856 -> 683; two and three go back (65536 values, 16 * 10^6 by splits 234 and more)
//   int32 argsort none  full range 16 * 10^6 494 -> 370, 40 1012 -> 819, but Zipf 453 -> 492, 942 -> 980, 2^24 values 774 -> 829
//   int64 24            sort, full range 8 * 10^6 513 -> 250, 12 702 -> 335, 20 1071 -> 490, but Zipf 8 377 -> 502 (12 514 -> 270), 65536
//                       values, which go back, 8 166 -> 191, 20 338 -> 363, 24 397 -> 417
//   float32 sort 0.9    one split 0.7 * 10^6 60 -> 59, 0.85 66 -> 61, 1.3 74 -> 65; two (5) 1.7 85 -> 93, 2.5 98 -> 115, 3.5 124 -> 140, 4.5 169 -> 152
//                       (scores 164 -> 163), 5 179 -> 168
//   float32 argsort 0.6 one split 0.3 * 10^6 55 -> 55, 0.45 63 -> 55, 0.6 98 -> 59; to 10^8: 0.9 * 10^8 2062 -> 1832, 1.6 3540 -> 3229 (with
//                       NaNs and copies 3377), 2.7 5769 -> 5497 (5736)
//   float64 0.2         sort 10^5 76 -> 64, 2 * 10^5 83 -> 64; what goes back 54 -> 68
// Float64 keys that hold whole numbers differ in five bytes; many copies crowd their cells (unique of ids, 5 * 10^6: 334 us, by
// splits 450, sent back by the sample 361).  Of int64 sorts two differing bytes go back (65536 values, 8 * 10^7 1110 -> 1655),
// one and three do not (a hundred values 670 -> 644, 2^24 values 2.4 * 10^7 544 -> 503, 8 1559 -> 1629).
// Argsorts of keys that are alike as far as the sample sees need few passes, and the splits, which cut them by position, give up
// late: they go back (one value, 2.4 * 10^7 int64 148 us by the passes, by the splits 519; 8 * 10^6 float64 73, 935).  Sorts of such
// integers stay: one value costs more (2.4 * 10^7 int64 176 -> 245, int32 of 1.6 * 10^7 70 -> 130), but one value and a few others less.
template <int KB, int XF>
inline SplitPlan split_plan_1d(size_t n, bool pairs, bool keys_too, size_t room)
{
  const long long over = split_override();
  if (!(KB == 4 || KB == 8) || XF == XF_CFLOAT || (pairs && keys_too) || over == 0) return SplitPlan{};
  SplitPlan p          = split_plan(n, 1, pairs, room);
  constexpr bool FLOAT = XF == XF_FLOAT;
  size_t least;
  if (KB == 4) least = !FLOAT ? (pairs ? SIZE_MAX : 16000000) : p.levels != 1 ? 5000000 : pairs ? 600000 : 900000;
  else least = FLOAT ? 200000 : 24000000;
  if (n < (over > 0 ? (size_t)over : least)) p.ok = false;
  // (above, the gain shrinks to that of the noise for keys with NaNs and copies)
  if (KB == 4 && pairs && n > 100000000 && over < 0) p.ok = false;
  // each byte in which the keys differ is a radix pass
  if (over <= 0) p.radix_if = KB == 4 ? (pairs ? 0xFu : p.levels == 1 ? 0xEu : 0xCu) : FLOAT ? (pairs ? 0x3Fu : 0x3Eu) : pairs ? 0xFu : 0x4u;
  return p;
}

#ifndef B2S_HIST_LANES
#define B2S_HIST_LANES 1
#endif

template <int KB, int XF>
inline cudaError_t radix_1d_xf(const void* in, void* out, int64_t* idx_out, unsigned int n,
                               int64_t index_offset, unsigned char* ws, cudaStream_t stream, int idx32,
                               const uint32_t* idx_in, const unsigned int* hist_parts, int hist_nparts)
{
  using K            = typename KeyOf<KB>::type;
  const bool pairs   = idx_out != nullptr;
  const auto lay     = radix_1d_layout<KB>(n, pairs);
  Ctrl* ctrl         = reinterpret_cast<Ctrl*>(ws);
  unsigned int* lb   = reinterpret_cast<unsigned int*>(ws + lay.off_lookback);
  // control block; the look-back tables too unless the histogram kernel clears them
  const bool own_hist = hist_parts == nullptr;
  const SplitPlan plan = own_hist && !(idx32 & IDX_PASSES_ONLY) ? split_plan_1d<KB, XF>(n, pairs, out != nullptr, lay.off_keys[0] - lay.off_lookback) : SplitPlan{};
  cudaError_t e        = cudaMemsetAsync(ws, 0, lay.off_lookback + (plan.ok ? plan.zero_bytes : own_hist ? 0 : lay.lookback_used), stream);
  if (e != cudaSuccess) return e;
  if constexpr ((KB == 4 || KB == 8) && XF != XF_CFLOAT) {
    // the splitting kernels first; the radix passes behind them find out whether anything is left to do
    if (plan.ok) {
      SplitJob job{};
      job.in           = in;
      job.out          = out;
      job.idx64        = (idx32 & IDX_32) ? nullptr : idx_out;
      job.idx32        = (idx32 & IDX_32) ? reinterpret_cast<uint32_t*>(idx_out) : nullptr;
      job.payload      = idx_in;
      job.seg_len      = n;
      job.nseg         = 1;
      job.index_offset = index_offset;
      for (int i = 0; i < 2; ++i) {
        job.tmp_keys[i] = ws + lay.off_keys[i];
        job.tmp_pos[i]  = reinterpret_cast<uint32_t*>(ws + lay.off_idx[i]);
      }
      job.tables = ws + lay.off_lookback;
      e = launch_split<KB>(XF, plan, job, ctrl, stream);
      if (e != cudaSuccess) return e;
    }
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const unsigned int per_cta = HIST_THREADS * 16;
  unsigned int hgrid         = (n + per_cta - 1) / per_cta;
  if (hgrid > (unsigned int)sms * 4) hgrid = sms * 4;
  RouteArgs ra{};
  ra.keys_in     = in;
  ra.keys_out    = out;
  ra.idx_out     = (idx32 & IDX_32) ? nullptr : idx_out;
  ra.idx_out32   = (idx32 & IDX_32) ? reinterpret_cast<uint32_t*>(idx_out) : nullptr;
  ra.idx_in      = idx_in;
  ra.tmp_keys[0] = ws + lay.off_keys[0];
  ra.tmp_keys[1] = ws + lay.off_keys[1];
  ra.tmp_idx[0]  = reinterpret_cast<uint32_t*>(ws + lay.off_idx[0]);
  ra.tmp_idx[1]  = reinterpret_cast<uint32_t*>(ws + lay.off_idx[1]);
  ra.n           = n;
  ra.npass       = KB;
  ra.key_bytes   = KB;
  ra.zero_ptr    = own_hist ? reinterpret_cast<uint4*>(ws + lay.off_lookback) : nullptr;
  ra.zero_vecs   = own_hist ? lay.lookback_used / 16 : 0;
  if (hist_parts != nullptr) {
    // the histograms were counted elsewhere (by the ranks that sent this GPU its keys)
    prof::Scope ps(prof::K_SCAN, stream);
    hist_from_parts_kernel<<<1, RADIX, 0, stream>>>(ctrl, hist_parts, hist_nparts, ra);
  } else {
    // digit histograms of all passes; the CTA that finishes last scans them and routes the passes
    prof::Scope ps(prof::K_HIST, stream);
#if B2S_HIST_LANES
    // one CTA per SM with a copy of the tables per lane; inputs too small to give every SM a few
    // thousand keys take the single-table kernel
    if (n >= (unsigned int)sms * HISTL_THREADS * 16) {
      auto kern = hist_lanes_kernel<KB, XF>;
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HistLanes<KB>::BYTES);
      if (e != cudaSuccess) return e;
      kern<<<sms, HISTL_THREADS, HistLanes<KB>::BYTES, stream>>>(static_cast<const K*>(in), n, ctrl, ra);
    } else
#endif
    hist_kernel<KB, XF><<<hgrid, HIST_THREADS, 0, stream>>>(static_cast<const K*>(in), n, ctrl, ra);
  }
  const SegGeom geo{n, lay.tiles, 1u, KB, nullptr};
  auto sweeps = [&](auto size, auto chained) {
    constexpr int SIZE     = decltype(size)::value;
    constexpr bool CHAINED = decltype(chained)::value;
    return pairs ? launch_sweeps<KB, XF, true, SIZE, CHAINED>(ctrl, lb, lay.tiles, geo, index_offset, stream)
                 : launch_sweeps<KB, XF, false, SIZE, CHAINED>(ctrl, lb, lay.tiles, geo, index_offset, stream);
  };
  e = n <= SMALL_MAX    ? sweeps(std::integral_constant<int, SWEEP_SMALL>{}, std::true_type{})
      : n <= MEDIUM_MAX ? sweeps(std::integral_constant<int, SWEEP_MEDIUM>{}, std::true_type{})
      : n <= CHAIN_MAX  ? sweeps(std::integral_constant<int, SWEEP_LARGE>{}, std::true_type{})
                        : sweeps(std::integral_constant<int, SWEEP_LARGE>{}, std::false_type{});
  if (e != cudaSuccess) return e;
  unsigned int fgrid = (n + 256 * 16 - 1) / (256 * 16);
  if (fgrid > (unsigned int)sms * 8) fgrid = sms * 8;
  {
    prof::Scope ps(prof::K_FIXUP, stream);
    e = launch_chained(fixup_kernel, fgrid, 256, 0, stream, ctrl, n, index_offset);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

// ---- segments too long for the on-chip kernel: onesweep passes whose tiles stay inside segments ----
struct RadixSegLayout {
  size_t off_lookback, off_seghist, off_keys[2], off_idx[2], total;
  unsigned int tiles_per_seg, tiles;
};

template <int KB>
inline RadixSegLayout radix_seg_layout(size_t seg_len, size_t nseg, bool pairs)
{
  RadixSegLayout l{};
  const unsigned int tile = pairs ? SweepCfg<KB, true>::TILE : SweepCfg<KB, false>::TILE;
  l.tiles_per_seg         = (unsigned int)((seg_len + tile - 1) / tile);
  l.tiles                 = (unsigned int)(l.tiles_per_seg * nseg);
  const size_t volume     = seg_len * nseg;
  size_t off              = LOOKBACK_OFFSET;
  l.off_lookback          = off;
  off += align_up((size_t)KB * l.tiles * RADIX * sizeof(unsigned int), 256);
  l.off_seghist = off;
  off += align_up(nseg * KB * RADIX * sizeof(unsigned int), 256);
  for (int i = 0; i < 2; ++i) {
    l.off_keys[i] = off;
    off += align_up(volume * KB, 256);
  }
  for (int i = 0; i < 2; ++i) {
    l.off_idx[i] = off;
    if (pairs) off += align_up(volume * 4, 256);
  }
  l.total = off;
  return l;
}

template <int KB, int XF>
inline cudaError_t radix_seg_xf(const void* in, void* out, int64_t* idx_out, unsigned int seg_len, unsigned int nseg,
                                int64_t index_offset, unsigned char* ws, cudaStream_t stream)
{
  using K          = typename KeyOf<KB>::type;
  const bool pairs = idx_out != nullptr;
  const auto lay   = radix_seg_layout<KB>(seg_len, nseg, pairs);
  Ctrl* ctrl       = reinterpret_cast<Ctrl*>(ws);
  unsigned int* lb = reinterpret_cast<unsigned int*>(ws + lay.off_lookback);
  unsigned int* sh = reinterpret_cast<unsigned int*>(ws + lay.off_seghist);
  // control block and histograms; the look-back table is cleared by the histogram kernel, since the tables of the
  // splitting kernels take its place until then
  cudaError_t e = cudaMemsetAsync(ws, 0, lay.off_lookback, stream);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(ws + lay.off_seghist, 0, lay.off_keys[0] - lay.off_seghist, stream);
  if (e != cudaSuccess) return e;
  if constexpr ((KB == 4 || KB == 8) && XF != XF_CFLOAT) {
    // 8-byte keys and argsorts gain at every length (time in parts of the passes': int64 and float64 sorts 0.65 for 3 rows of 8200,
    // 0.37 to 0.5 for 1000 rows; argsorts of float32 0.7 for 3 rows of 20011, 0.6 for 1000 of 16400).  4-byte sorts need 10^6 keys
    // (float32, 7 rows of 90000 66 -> 73 us, 10 rows of 10^6 271 -> 177), and rows of two leaves do not gain enough for what
    // crowded ones lose (1000 rows of 8200, full range 0.91, 40 copies of each key 1.28, Zipf 1.61; of 12000 0.71, Zipf 1.19).
    const bool enough = KB == 8 || pairs || ((size_t)seg_len * nseg >= 1000000 && seg_len >= 10000) || split_override() > 0;
    if (!(pairs && out != nullptr) && split_override() != 0 && enough) {
      const SplitPlan plan = split_plan(seg_len, nseg, pairs, lay.off_seghist - lay.off_lookback);
      if (plan.ok) {
        e = cudaMemsetAsync(ws + lay.off_lookback, 0, plan.zero_bytes, stream);
        if (e != cudaSuccess) return e;
        SplitJob job{};
        job.in           = in;
        job.out          = out;
        job.idx64        = idx_out;
        job.seg_len      = seg_len;
        job.nseg         = nseg;
        job.index_offset = index_offset;
        for (int i = 0; i < 2; ++i) {
          job.tmp_keys[i] = ws + lay.off_keys[i];
          job.tmp_pos[i]  = reinterpret_cast<uint32_t*>(ws + lay.off_idx[i]);
        }
        job.tables = ws + lay.off_lookback;
        e = launch_split<KB>(XF, plan, job, ctrl, stream);
        if (e != cudaSuccess) return e;
      }
    }
  }
  const unsigned int chunks = (seg_len + SEG_HIST_CHUNK - 1) / SEG_HIST_CHUNK;
  {
    prof::Scope ps(prof::K_HIST, stream);
    seg_hist_kernel<KB, XF><<<nseg * chunks, 256, 0, stream>>>(static_cast<const K*>(in), seg_len, chunks, sh, ctrl,
                                                                  reinterpret_cast<uint4*>(ws + lay.off_lookback),
                                                                  (lay.off_seghist - lay.off_lookback) / 16);
  }
  {
    prof::Scope ps(prof::K_SCAN, stream);
    seg_scan_kernel<<<nseg * KB, RADIX, 0, stream>>>(sh);
  }
  RouteArgs ra{};
  ra.keys_in     = in;
  ra.keys_out    = out;
  ra.idx_out     = idx_out;
  ra.tmp_keys[0] = ws + lay.off_keys[0];
  ra.tmp_keys[1] = ws + lay.off_keys[1];
  ra.tmp_idx[0]  = reinterpret_cast<uint32_t*>(ws + lay.off_idx[0]);
  ra.tmp_idx[1]  = reinterpret_cast<uint32_t*>(ws + lay.off_idx[1]);
  ra.n           = seg_len * nseg;
  ra.npass       = KB;
  ra.key_bytes   = KB;
  {
    // the global histogram stays empty here, so every pass is routed as active
    prof::Scope ps(prof::K_SCAN, stream);
    scan_route_kernel<<<1, RADIX, 0, stream>>>(ctrl, ra);
  }
  // every pass is active here (empty global histogram), so the only leftover is the copy of an
  // in-place single-pass sort out of its temporary
  const SegGeom geo{seg_len, lay.tiles_per_seg, nseg, KB, sh};
  e = pairs ? launch_sweeps<KB, XF, true>(ctrl, lb, lay.tiles, geo, index_offset, stream)
            : launch_sweeps<KB, XF, false>(ctrl, lb, lay.tiles, geo, index_offset, stream);
  if (e != cudaSuccess) return e;
  if (out != nullptr && out == in) {
    prof::Scope ps(prof::K_FIXUP, stream);
    fixup_kernel<<<148 * 4, 256, 0, stream>>>(ctrl, seg_len * nseg, index_offset);
  }
  return cudaGetLastError();
}

// The self-test's way to the passes of uint32 keys as the sorts launch them: of short 1-D arrays (dependent launches),
// of rows longer than SEG_CAP, of long 1-D arrays.
enum : int { SELFTEST_SHORT = 0, SELFTEST_ROWS = 1, SELFTEST_LONG = 2 };
cudaError_t selftest_sweeps(int which, Ctrl* ctrl, unsigned int* lookback, unsigned int tiles, SegGeom geo, cudaStream_t stream);

// Segments of more than SEG_CAP elements (each below 2^30, fewer than 2^32 elements in all).
template <int KB>
cudaError_t launch_radix_seg(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                             unsigned int nseg, int64_t index_offset, unsigned char* ws, cudaStream_t stream);

// 1-D stable sort of n < 2^30 keys. `ws` must hold radix_1d_layout<KB>(n, idx_out != null).total bytes.
// idx32: IDX_32: idx_out points to n uint32 values and receives positions 0..n-1 without the offset; IDX_PASSES_ONLY: by the
// radix passes alone.
// idx_in != null: the payload of element i is idx_in[i] instead of i (stable argsort of data that
// already carries 32-bit payloads); the output index is index_offset + payload.
// hist_parts != null: hist_nparts ready-made digit histograms ([part][KB][256]) to add up instead
// of reading the keys for them.
template <int KB>
cudaError_t launch_radix_1d(int xf, const void* in, void* out, int64_t* idx_out, unsigned int n,
                            int64_t index_offset, unsigned char* ws, cudaStream_t stream, int idx32 = 0,
                            const uint32_t* idx_in = nullptr, const unsigned int* hist_parts = nullptr,
                            int hist_nparts = 0);

// Segments of seg_len <= SEG_CAP elements, sorted on chip. `status` (the workspace's
// status word) is set to 0 by the kernels, which have nothing to report.
template <int KB>
cudaError_t launch_segsort(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                           unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream);

template <int KB, bool PAIRS, int THREADS, int ITEMS>
inline cudaError_t segsort_cfg(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                               unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  using K   = typename KeyOf<KB>::type;
  using S   = SegSmem<KB, PAIRS, THREADS, ITEMS>;
  auto kern = segsort_kernel<KB, PAIRS, THREADS, ITEMS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::BYTES);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, S::BYTES);
  if (per_sm < 1) per_sm = 1;
  unsigned long long grid = (unsigned long long)sms * per_sm;
  if (grid > nseg) grid = nseg;
  {
    prof::Scope ps(prof::K_SEGSORT, stream);
    kern<<<(unsigned int)grid, THREADS, S::BYTES, stream>>>(static_cast<const K*>(in), static_cast<K*>(out),
                                                             idx_out, seg_len, nseg, xf, index_offset, status);
  }
  return cudaGetLastError();
}

// Rows of one block: buckets, merging where the keys crowd (4- and 8-byte keys, rows of more than 512 elements).
template <int KB, bool PAIRS, int THREADS, int FORM>
inline cudaError_t segmerge_cfg(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                                unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  using K   = typename KeyOf<KB>::type;
  using S   = SegMergeSmem<KB, PAIRS, THREADS>;
  auto kern = segmerge_kernel<KB, PAIRS, THREADS, FORM>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::BYTES);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, S::BYTES);
  if (per_sm < 1) per_sm = 1;
  unsigned long long grid = (unsigned long long)sms * per_sm;
  if (grid > nseg) grid = nseg;
  {
    prof::Scope ps(prof::K_SEGSORT, stream);
    kern<<<(unsigned int)grid, THREADS, S::BYTES, stream>>>(static_cast<const K*>(in), static_cast<K*>(out), idx_out, seg_len,
                                                             nseg, xf, index_offset, status);
  }
  return cudaGetLastError();
}

// Rows of up to SW_MAX elements: one warp per 32 / group rows.
template <int KB, bool PAIRS, int VT, int GL>
inline cudaError_t segwarp_cfg(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                               unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  using K = typename KeyOf<KB>::type;
  constexpr unsigned long long ROWS = (unsigned long long)SW_WARPS * (32 >> GL);
  unsigned long long grid = (nseg + ROWS - 1) / ROWS;
  if (grid > (1ull << 30)) grid = 1ull << 30;
  {
    prof::Scope ps(prof::K_SEGSORT, stream);
    segwarp_kernel<KB, PAIRS, VT, GL><<<(unsigned int)grid, SW_WARPS * 32, 0, stream>>>(
      static_cast<const K*>(in), static_cast<K*>(out), idx_out, seg_len, nseg, xf, index_offset, status);
  }
  return cudaGetLastError();
}

template <int KB, bool PAIRS>
inline cudaError_t segwarp_any(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                               unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  if (seg_len <= 2) return segwarp_cfg<KB, PAIRS, 2, 0>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 4) return segwarp_cfg<KB, PAIRS, 4, 0>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 8) return segwarp_cfg<KB, PAIRS, 8, 0>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 16) return segwarp_cfg<KB, PAIRS, 16, 0>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 32) return segwarp_cfg<KB, PAIRS, 16, 1>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 64) return segwarp_cfg<KB, PAIRS, 16, 2>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 128) return segwarp_cfg<KB, PAIRS, 16, 3>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 256) return segwarp_cfg<KB, PAIRS, 16, 4>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  return segwarp_cfg<KB, PAIRS, 16, 5>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
}

template <int KB, bool PAIRS, int FORM>
inline cudaError_t segmerge_form(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                                 unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  constexpr int V = SM_VT;
  if (seg_len <= 64 * V) return segmerge_cfg<KB, PAIRS, 64, FORM>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 128 * V) return segmerge_cfg<KB, PAIRS, 128, FORM>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 256 * V) return segmerge_cfg<KB, PAIRS, 256, FORM>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  return segmerge_cfg<KB, PAIRS, 512, FORM>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
}

template <int KB, bool PAIRS>
inline cudaError_t segmerge_any(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                                unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  if (xf == XF_FLOAT) return segmerge_form<KB, PAIRS, SM_FLOAT>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if constexpr (KB == 8 && PAIRS)
    if (xf == XF_CFLOAT) return segmerge_form<KB, PAIRS, SM_COMPLEX>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  return segmerge_form<KB, PAIRS, SM_INT>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
}

inline bool seg_merge_enabled()
{
  const char* e = std::getenv("B2S_SEG_MERGE");  // 0: rows above 512 stay on the radix kernel (comparisons)
  return e == nullptr || e[0] != '0';
}

template <int KB, bool PAIRS>
inline cudaError_t segsort_pairs(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len,
                                 unsigned long long nseg, int64_t index_offset, unsigned int* status, cudaStream_t stream)
{
  // Short rows go to the warp kernel (2^24 float32 keys with positions, against the one-CTA-per-row radix
  // and merge kernels they took before: rows of 2 19.2 ms -> 0.07 ms, of 32 1.31 -> 0.10, of 100 0.47 -> 0.17, of
  // 200 1.42 -> 0.15, of 512 0.34 -> 0.12).  One-byte rows of 65 to 128 stay with the radix kernel, which
  // needs a single pass for them whatever they hold.  2^24 uint8 keys in rows of 100, radix against warp kernel: spread
  // over 256 values 127 and 125 us, of three values 120 and 144, of one 45 and 74; the argsort 140 and 117, 132
  // and 137, 60 and 68.
  // Keys of a sort are mapped back from their images, which the complex64 image does not allow: those
  // rows are sorted with positions and the keys fetched through them.  So are keys below 4 bytes, whose
  // words have room for the position anyway.
  if constexpr (KB == 1)
    if (seg_len > 64 && seg_len <= 128)
      return segsort_cfg<KB, PAIRS, 32, 4>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= SW_MAX) {
    if constexpr (PAIRS || KB < 4) {
      return segwarp_any<KB, true>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
    } else {
      if (KB == 8 && xf == XF_CFLOAT) return segwarp_any<KB, true>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
      return segwarp_any<KB, false>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
    }
  }
  if constexpr (KB == 4 || KB == 8) {
    if (seg_merge_enabled()) {
      if constexpr (!PAIRS && KB == 8)
        if (xf == XF_CFLOAT) return segmerge_any<KB, true>(xf, in, out, nullptr, seg_len, nseg, index_offset, status, stream);
      return segmerge_any<KB, PAIRS>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
    }
  }
  if (seg_len <= 1024) return segsort_cfg<KB, PAIRS, 128, 8>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  if (seg_len <= 4096) return segsort_cfg<KB, PAIRS, 256, 16>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
  return segsort_cfg<KB, PAIRS, 512, 16>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);
}

#define B2S_INSTANTIATE_KEY_WIDTH(KB, HAS_FLOAT, HAS_CFLOAT)                                                          \
  template <>                                                                                             \
  cudaError_t launch_radix_1d<KB>(int xf, const void* in, void* out, int64_t* idx_out, unsigned int n,    \
                                  int64_t index_offset, unsigned char* ws, cudaStream_t stream, int idx32, \
                                  const uint32_t* idx_in, const unsigned int* hp, int hn)                 \
  {                                                                                                       \
    if (xf == XF_UNSIGNED) return radix_1d_xf<KB, XF_UNSIGNED>(in, out, idx_out, n, index_offset, ws, stream, idx32, idx_in, hp, hn); \
    if (xf == XF_SIGNED) return radix_1d_xf<KB, XF_SIGNED>(in, out, idx_out, n, index_offset, ws, stream, idx32, idx_in, hp, hn); \
    if (HAS_FLOAT && xf == XF_FLOAT)                                                                      \
      return radix_1d_xf<KB, (HAS_FLOAT ? XF_FLOAT : XF_UNSIGNED)>(in, out, idx_out, n, index_offset, ws, stream, idx32, idx_in, hp, hn); \
    if (HAS_CFLOAT && xf == XF_CFLOAT)                                                                    \
      return radix_1d_xf<KB, (HAS_CFLOAT ? XF_CFLOAT : XF_UNSIGNED)>(in, out, idx_out, n, index_offset, ws, stream, idx32, idx_in, hp, hn); \
    return cudaErrorInvalidValue;                                                                         \
  }                                                                                                       \
  template <>                                                                                             \
  cudaError_t launch_radix_seg<KB>(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len, \
                                   unsigned int nseg, int64_t index_offset, unsigned char* ws,           \
                                   cudaStream_t stream)                                                   \
  {                                                                                                       \
    if (xf == XF_UNSIGNED) return radix_seg_xf<KB, XF_UNSIGNED>(in, out, idx_out, seg_len, nseg, index_offset, ws, stream); \
    if (xf == XF_SIGNED) return radix_seg_xf<KB, XF_SIGNED>(in, out, idx_out, seg_len, nseg, index_offset, ws, stream); \
    if (HAS_FLOAT && xf == XF_FLOAT)                                                                      \
      return radix_seg_xf<KB, (HAS_FLOAT ? XF_FLOAT : XF_UNSIGNED)>(in, out, idx_out, seg_len, nseg, index_offset, ws, stream); \
    if (HAS_CFLOAT && xf == XF_CFLOAT)                                                                    \
      return radix_seg_xf<KB, (HAS_CFLOAT ? XF_CFLOAT : XF_UNSIGNED)>(in, out, idx_out, seg_len, nseg, index_offset, ws, stream); \
    return cudaErrorInvalidValue;                                                                         \
  }                                                                                                       \
  template <>                                                                                             \
  cudaError_t launch_segsort<KB>(int xf, const void* in, void* out, int64_t* idx_out, unsigned int seg_len, \
                                 unsigned long long nseg, int64_t index_offset, unsigned int* status,               \
                                 cudaStream_t stream)                                                     \
  {                                                                                                       \
    if ((!HAS_FLOAT && xf == XF_FLOAT) || (!HAS_CFLOAT && xf == XF_CFLOAT)) return cudaErrorInvalidValue; \
    if (idx_out != nullptr)                                                                               \
      return segsort_pairs<KB, true>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);    \
    return segsort_pairs<KB, false>(xf, in, out, idx_out, seg_len, nseg, index_offset, status, stream);     \
  }

}  // namespace b2s
