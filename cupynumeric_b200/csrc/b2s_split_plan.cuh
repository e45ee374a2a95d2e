// What a splitting sort (b2s_split.cuh) of given sizes needs: its levels and the memory of its tables.
#pragma once

#include "b2s_common.cuh"

namespace b2s {

constexpr unsigned int SPLIT_BINS = 256;       // buckets of a segment
constexpr unsigned int LEAF_MOST = 8192, LEAF_MOST_PAIRS = 6144;  // most keys of a leaf, without and with positions
constexpr unsigned int SPLIT_MAX_CELLS = 8192;
constexpr unsigned int FILL_CHUNK = 1u << 16;

// From a key's image to its cell.  Cell 0: below the sampled range; 1 .. CI: inside; CI + 1: above; float
// keys: the last cells hold the NaNs, of argsorts cut by position.
//   MAP_LIN  (image - lo) >> shift
//   MAP_POS  argsort of a small range of images: `mult` cells per image, cut by position
//   MAP_LOG  integers: exponent and leading bits of (image - lo) as a float32, for keys that crowd at the lower end
//   MAP_VAL  floats: (value - value of lo) * scale (the image itself is logarithmic)
//   MAP_TOP  sort of keys: MAP_LIN with a cell of its own for the image lo + top, of which there are many
enum : unsigned int { MAP_LIN = 0, MAP_POS = 1, MAP_LOG = 2, MAP_TOP = 3, MAP_VAL = 4 };
struct SplitMap {
  unsigned long long lo, range;  // images lo .. lo + range are inside
  unsigned long long top;        // MAP_VAL: the scale, as a double
  unsigned int mode;
  unsigned int shift;
  unsigned int mult;    // MAP_LOG: cell of 1, minus one
  unsigned int pscale;  // MAP_POS: position -> cell inside the image's own
  unsigned int nscale;  // position -> NaN cell
  unsigned int pad_;
  unsigned long long vmin;  // MAP_VAL: bits of the value of lo
};
struct SplitSeg {
  unsigned int begin, len, tile0;
  unsigned int drops;  // some of its keys are not moved
  SplitMap map;
};
// A bucket to be sorted (LEAF_BOUNDED: all of its images lie in lo .. lo + span; LEAF_COUNT: they are at most COUNT_SPAN + 1, and
// the keys may be more than `cap`), or (LEAF_FILL) `len` copies of the key `lo` to be written.
constexpr unsigned int LEAF_FILL = 1u << 31, LEAF_BOUNDED = 1u << 30, LEAF_COUNT = 1u << 29;
constexpr unsigned int LEAF_LEN   = LEAF_COUNT - 1;   // (two-split plans take fewer keys, rows are shorter)
constexpr unsigned int COUNT_SPAN = 2047;
// (one block counts a bucket: at this length, 96 keys per thread, it takes about as long as sending short rows back; 10^6 keys took
// it 1 ms while all others were done after 0.1)
constexpr unsigned int COUNT_MOST = 6;                // times `cap`
struct SplitLeaf {
  unsigned int begin, len;
  unsigned long long lo, span;
};

// Bit patterns among the float keys of a sort without positions whose image stands for several.
enum : unsigned int { MARK_ZERO = 1, MARK_NEG_ZERO = 2, MARK_NAN = 4 /* the canonical one */, MARK_MIXED = 8 /* several others */, MARK_OTHER = 16 /* others */ };
struct SplitMarks {
  unsigned long long nan;  // NaNs of another pattern; 0: none
  unsigned int flags;
};

// Shape of one split.
struct SplitShape {
  unsigned int nseg;   // most segments
  unsigned int cells, cap;
};

struct SplitPlan {
  bool ok;
  int levels;
  unsigned int radix_if;     // bit k: keys that differ in k bytes are left to the radix passes
  SplitShape lev[2];
  size_t zero_bytes;  // from the start: what has to be clear
  size_t off_marks, off_hist[2], off_segs[2], off_lut[2], off_cursor[2], off_tile_seg, off_leaves, total;
};

// nseg segments of seg_len keys; `room` bytes for the tables (the look-back tables of the radix passes, which are
// cleared anew if it comes to those).
inline SplitPlan split_plan(size_t seg_len, size_t nseg, bool pairs, size_t room)
{
  const unsigned int leaf_most = pairs ? LEAF_MOST_PAIRS : LEAF_MOST;
  SplitPlan p{};
  const size_t volume = seg_len * nseg;
  // Cells that hold a sixteenth of a bucket leave buckets about 15 / 16 full; 213 of the 256 are counted on.
  constexpr size_t FULL = 200;
  unsigned int cap = 2048;
  if (seg_len <= FULL * leaf_most) {
    if (seg_len > FULL * cap || seg_len * nseg > (size_t)148 * 4 * cap) cap = 4096;
    if (seg_len > FULL * cap) cap = leaf_most;
    p.levels = 1;
    unsigned int cells = 1024;
    while (cells < 4096 && cells < seg_len / cap * 16) cells <<= 1;
    p.lev[0] = SplitShape{(unsigned int)nseg, cells, cap};
  } else {
    if (nseg != 1) return p;
    p.levels = 2;
    // (the more keys, the more room for buckets that are not full, in numbers and in length)
    cap = seg_len <= (pairs ? 150ull * 150 * 4096 : 120ull * 120 * 4096) ? 4096 : leaf_most;
    if (seg_len > 230ull * 230 * leaf_most) return p;
    unsigned int b1 = 16;
    while ((size_t)b1 * b1 * cap * 15 / 16 < seg_len) ++b1;
    p.lev[0] = SplitShape{1u, b1 > 100 ? 8192u : 4096u, (unsigned int)(seg_len / b1)};
    p.lev[1] = SplitShape{2 * b1 + 2 < SPLIT_BINS ? 2 * b1 + 2 : SPLIT_BINS, b1 > 100 && !pairs ? 8192u : 4096u, cap};
  }
  p.off_marks = 0;
  size_t off  = 256;
  for (int l = 0; l < p.levels; ++l) {
    p.off_hist[l] = off;
    off += align_up((size_t)p.lev[l].nseg * p.lev[l].cells * 4, 256);
  }
  p.zero_bytes = off;
  for (int l = 0; l < p.levels; ++l) {
    p.off_segs[l] = off;
    off += align_up((size_t)p.lev[l].nseg * sizeof(SplitSeg), 256);
    p.off_lut[l] = off;
    off += align_up((size_t)p.lev[l].nseg * p.lev[l].cells * 2, 256);
    p.off_cursor[l] = off;
    off += align_up((size_t)p.lev[l].nseg * SPLIT_BINS * 4, 256);
  }
  p.off_tile_seg = off;
  if (p.levels == 2) off += align_up((volume / 4096 + p.lev[1].nseg + 1) * 2, 256);
  p.off_leaves = off;
  // a value to be filled in has more than cap / 4 copies, two neighbouring buckets between such values hold more than `cap` keys
  off += align_up((12 * volume / cap + 2 * ((size_t)p.lev[0].nseg + (p.levels == 2 ? p.lev[1].nseg : 0)) + volume / FILL_CHUNK + (p.levels == 2 ? SPLIT_BINS : 0) + 16) * sizeof(SplitLeaf), 256);
  p.total = off;
  p.ok    = off <= room;
  return p;
}

struct SplitJob {
  const void* in;
  void* out;            // keys, or
  int64_t* idx64;       // positions as int64 with index_offset added, or
  uint32_t* idx32;      // positions as they are
  const uint32_t* payload;  // takes the place of a position in the result; null: the position
  unsigned int seg_len, nseg;
  int64_t index_offset;
  void* tmp_keys[2];
  uint32_t* tmp_pos[2];
  unsigned char* tables;   // plan.total bytes, plan.zero_bytes of them clear
};

template <int KB>
cudaError_t launch_split(int xf, const SplitPlan& plan, const SplitJob& job, Ctrl* ctrl, cudaStream_t stream);

}  // namespace b2s
