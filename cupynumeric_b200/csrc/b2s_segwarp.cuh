// Segmented sort of short rows (up to 512 elements): a group of 1 to 32 threads of one warp sorts a row, a
// warp sorts 32 / group rows at a time, and nothing wider than the warp is ever waited for.  Every
// thread sorts its consecutive elements in registers with Batcher's odd-even merge network,
// then log2(group) rounds of merge-path merges run in the warp's own piece of shared memory.
//
// Keys travel as words that are ordered like the sort: the order-preserving image, with the element's
// position below it where positions are wanted (a 4-byte key and its position make one 64-bit word, a
// shorter key and its position one 32-bit word; 8-byte keys keep 16-bit positions beside them).  The
// position makes every word of a row unique, so the network, which is not stable, sorts stably.
//
// Rows above 64 elements go through the buckets of b2s_segmerge.cuh first, with the counters in the warp's
// own shared memory, and merge only where some row of the warp has its keys crowd.
//
// Bound: instruction issue, memory for the shortest rows.  A row per CTA, as the radix kernel takes them,
// leaves a short row's CTA waiting for its barriers and four counting passes.  2^24 float32 keys with
// positions, radix kernel -> merging here -> buckets: rows of 100 0.468 -> 0.220 -> 0.166 ms, of 200 1.42 -> 0.247
// -> 0.153, of 512 (merged by a block before) 0.339 -> 0.230 -> 0.116; float64 rows of 200 3.05 -> 0.310 -> 0.215.
// Rows whose keys crowd (heavy duplicates, an outlier) are merged; where counting cannot succeed it is left out, and
// where the threads' blocks come in order so are the merge rounds: 2^22 int64 keys of one value in rows of 100,
// argsort 89 -> 44 us (the radix kernel, which skips constant digits: 24), of three values 88 -> 78 (47).
// 16 elements per thread: the network costs 4 comparators per element, a merge round about 20 instructions,
// and 16 words are what the registers of 28 warps per SM hold.  Up to 64 elements two merge rounds cost no
// more than counting, scanning and placing.
#pragma once

#include "b2s_common.cuh"
#include "b2s_segmerge.cuh"

namespace b2s {

constexpr int SW_WARPS         = 4;    // warps per CTA, independent of each other
constexpr unsigned int SW_MAX  = 512;  // longest row: 32 threads of 16 elements

template <int KB, bool PAIRS> struct SegWarpWord {
  static constexpr bool PACK = PAIRS && KB < 8;
  static constexpr bool SIDE = PAIRS && KB == 8;
  static constexpr int BYTES = (KB == 8 || (PACK && KB == 4)) ? 8 : 4;
  static constexpr int SHIFT = KB == 4 ? 32 : 16;  // PACK: the image sits above this many bits of position
  using type                 = typename SmWord<BYTES>::type;
};

// A warp sorts 32 >> GL rows at a time, 1 << GL threads of VT elements per row; seg_len <= VT << GL.
// idx_out and out may each be null (not both).
template <int KB, bool PAIRS, int VT, int GL>
__global__ void __launch_bounds__(SW_WARPS * 32, KB == 8 ? (PAIRS ? 4 : 6) : PAIRS ? 7 : 8)
segwarp_kernel(const typename KeyOf<KB>::type* in, typename KeyOf<KB>::type* out,
               int64_t* idx_out, unsigned int seg_len, unsigned long long nseg, int xf, int64_t index_offset, unsigned int* status)
{
  using K  = typename KeyOf<KB>::type;
  using WD = SegWarpWord<KB, PAIRS>;
  using W  = typename WD::type;
  constexpr bool PACK = WD::PACK, SIDE = WD::SIDE;
  constexpr int G = 1 << GL, RT = G * VT, ROWS = 32 / G;
  constexpr int SPAN = 32 * (VT + 1);  // one spare word per thread: blocked accesses hit all banks
  constexpr W WMAX   = (W)~(W)0;
  __shared__ W sw_all[SW_WARPS * SPAN];
  __shared__ unsigned short sp_all[SIDE ? SW_WARPS * SPAN : 1];
  // rows long enough for it are sorted by buckets first (b2s_segmerge.cuh): two 16-bit counters per element
  constexpr bool BUCKETS = VT == 16 && GL >= 3;
  constexpr int NB       = 2 * RT;
  // 4-byte keys with positions are the form with the fewest registers to spare: leaving the counting out costs their
  // evenly spread rows 5 %, looking for rows in order 4 % above 128 elements (nothing up to there)
  constexpr bool FOUR_PAIRS = PAIRS && KB == 4;
  constexpr bool CHECKS     = BUCKETS && !(FOUR_PAIRS && GL > 3);
  constexpr int CNT      = BUCKETS ? 32 * VT + 32 * VT / 8 : 4;  // words per warp, four spare ones after every 32
  __shared__ __align__(16) unsigned int cnt_all[SW_WARPS * CNT];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g    = lane & (G - 1);          // my place in the row's group
  W* sw              = sw_all + warp * SPAN;
  unsigned short* sp = sp_all + (SIDE ? warp * SPAN : 0);
  auto at = [](int i) { return i + i / VT; };  // shared-memory index of a position of the warp's rows
  const int mine = lane * (VT + 1);
  const int row0 = (lane >> GL) * RT;          // first position of my row
  const bool gather = PAIRS && (KB >= 4 || xf == XF_FLOAT);  // keys come back through the positions

  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;  // nothing here waits, so nothing can time out
  const unsigned long long nblk = (nseg + ROWS - 1) / ROWS;
  for (unsigned long long blk = (unsigned long long)blockIdx.x * SW_WARPS + warp; blk < nblk;
       blk += (unsigned long long)gridDim.x * SW_WARPS) {
    const unsigned long long base = blk * ROWS;
    const int rows = (int)(nseg - base < (unsigned long long)ROWS ? nseg - base : ROWS);
    const K* src   = in + base * seg_len;
    // ---- load: consecutive lanes read consecutive elements; element j of a lane is in row j * 32 / RT ----
    int special = 0;
    K img[VT];
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      const int i = j * 32 + lane, r = i / RT, c = i % RT;
      img[j]      = r < rows && (unsigned int)c < seg_len ? src[r * seg_len + c] : (K)0;
    }
#pragma unroll
    for (int j = 0; j < VT; ++j) {
      const K raw = img[j];
      img[j]      = to_ordered_rt<KB>(raw, xf);
      if (!PAIRS && xf == XF_FLOAT) special |= sm_is_special<KB>(raw, xf) ? 1 : 0;  // (0 is not)
    }
    if (!PAIRS) special = __any_sync(0xFFFFFFFFu, special);
    auto word_of = [&](K o, int c) { return PACK ? (W)(((W)o << (PACK ? WD::SHIFT : 0)) | (W)(unsigned int)c) : (W)o; };
    W key[VT];
    unsigned int pay[SIDE ? VT : 1];
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
    auto read_words = [&](int first) {
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        key[j] = sw[at(first + j)];
        if (SIDE) pay[SIDE ? j : 0] = sp[at(first + j)];
      }
    };
    auto write_words = [&](int first) {
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        sw[at(first + j)] = key[j];
        if (SIDE) sp[at(first + j)] = (unsigned short)pay[SIDE ? j : 0];
      }
    };
    bool sorted = false;
    if constexpr (BUCKETS) {
      constexpr int PER = RT / 32;  // a lane's elements of one row
      unsigned char* cnt = reinterpret_cast<unsigned char*>(cnt_all + warp * CNT);
      for (int i = lane; i < CNT / 4; i += 32) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
      __syncwarp();
      unsigned int br[VT];  // where the bucket's counter is | rank in the bucket << 16
      int over = 0;
#pragma unroll
      for (int q = 0; q < ROWS; ++q) {
        if (q < rows) {
          auto mine_in = [&](int j) { return (unsigned int)((j * 32 + lane) % RT) < seg_len; };
          RowBuckets<KB, NB> rb;
          bool by_value = false;
          if constexpr (KB >= 4) by_value = xf == XF_FLOAT;
          if (by_value) {
            unsigned int lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
            for (int j = q * PER; j < (q + 1) * PER; ++j) {
              const unsigned int u = RowBuckets<KB, NB>::upper(img[j]);
              if (mine_in(j) && u - RowBuckets<KB, NB>::FIN_LO < RowBuckets<KB, NB>::FIN_N) {
                lo = min(lo, u);
                hi = max(hi, u);
              }
            }
            lo = __reduce_min_sync(0xFFFFFFFFu, lo);
            hi = __reduce_max_sync(0xFFFFFFFFu, hi);
            if constexpr (KB >= 4) rb.from_floats(lo, hi);
          } else {
            K lo = (K)~(K)0, hi = 0;
#pragma unroll
            for (int j = q * PER; j < (q + 1) * PER; ++j)
              if (mine_in(j)) {
                lo = img[j] < lo ? img[j] : lo;
                hi = img[j] > hi ? img[j] : hi;
              }
            if constexpr (KB < 8) {
              lo = (K)__reduce_min_sync(0xFFFFFFFFu, (unsigned int)lo);
              hi = (K)__reduce_max_sync(0xFFFFFFFFu, (unsigned int)hi);
            } else {
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) {
                const K l = __shfl_xor_sync(0xFFFFFFFFu, lo, o), h = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
                lo        = l < lo ? l : lo;
                hi        = h > hi ? h : hi;
              }
            }
            rb.from_images(lo, hi);
          }
          const bool counted = !PAIRS && rb.exact;  // a bucket holds equal keys, which need no order
          // fewer values than a ninth of the row: some bucket is too full, whatever the row holds (and a single
          // value would keep the counters waiting for each other)
          const bool full = !FOUR_PAIRS && rb.exact && (PAIRS ? (rb.range + 1) * SM_BUCKET < seg_len : rb.range == 0);
          if (!rb.ok || full) over = 1;
          else {
#pragma unroll
            for (int j = q * PER; j < (q + 1) * PER; ++j)
              if (mine_in(j)) {
                unsigned int b = 0;
                if constexpr (KB >= 4) b = by_value ? rb.bucket_float(img[j]) : rb.bucket_image(img[j]);
                else b = rb.bucket_image(img[j]);
                b += q * NB;
                const unsigned int place = b * 2 + (b >> 6) * 16;  // of the bucket's 16 bits
                const unsigned int h     = (b & 1u) * 16u;
                const unsigned int r     = (atomicAdd(reinterpret_cast<unsigned int*>(cnt + (place & ~3u)), 1u << h) >> h) & 0xFFFFu;
                over |= !counted && r >= (unsigned int)SM_BUCKET ? 1 : 0;
                br[j] = place | (r << 16);
              }
          }
        }
      }
      sorted = !__any_sync(0xFFFFFFFFu, over);
      __syncwarp();
      if (sorted) {
        // counts -> places: my 32 buckets, then the lanes of my row before me
        uint4* mine4     = reinterpret_cast<uint4*>(cnt) + 4 * lane + (lane >> 1);
        unsigned int sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 c = mine4[j];
          sum += c.x + c.y + c.z + c.w;  // two counts per word, added side by side
        }
        sum = (sum & 0xFFFFu) + (sum >> 16);
        unsigned int incl = sum;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, incl, o, G);
          if (g >= o) incl += t;
        }
        unsigned int run = incl - sum;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 c = mine4[j];
          auto place = [&](unsigned int& two) {
            const unsigned int first_n = two & 0xFFFFu, both = first_n + (two >> 16);
            two = run | ((run + first_n) << 16);
            run += both;
          };
          place(c.x);
          place(c.y);
          place(c.z);
          place(c.w);
          mine4[j] = c;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < VT; ++j) {
          const int i = j * 32 + lane, r = i / RT, c = i % RT;
          if (r < rows && (unsigned int)c < seg_len) {
            const int p = r * RT + *reinterpret_cast<const unsigned short*>(cnt + (br[j] & 0xFFFFu)) + (int)(br[j] >> 16);
            sw[at(p)]   = word_of(img[j], c);
            if (SIDE) sp[at(p)] = (unsigned short)c;
          } else {
            sw[at(i)] = WMAX;
            if (SIDE) sp[at(i)] = (unsigned short)c;
          }
        }
        __syncwarp();
        read_words(lane * VT);
        odd_even_merge_sort<VT, 1>(cmp_swap);
        write_words(lane * VT);
        __syncwarp();
        if (g < G - 1) {
          read_words(lane * VT + VT / 2);
          odd_even_merge_sort<VT, VT / 2>(cmp_swap);
          write_words(lane * VT + VT / 2);
        }
        __syncwarp();
        read_words(lane * VT);
      }
    }
    if (!sorted) {
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        const int i = j * 32 + lane, r = i / RT, c = i % RT;
        sw[at(i)]   = r < rows && (unsigned int)c < seg_len ? word_of(img[j], c) : WMAX;
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        key[j] = sw[mine + j];
        if (SIDE) pay[SIDE ? j : 0] = g * VT + j;
      }
      odd_even_merge_sort<VT, 1>(cmp_swap);
      if constexpr (CHECKS) {
        // rows of one value (which the buckets of floats and complex keys do not tell from crowded ones) and rows
        // whose blocks come in order need no merging
        sw[mine] = key[0];
        __syncwarp();
        sorted = !__any_sync(0xFFFFFFFFu, g < G - 1 && sw[mine + VT + 1] < key[VT - 1]);
      }
    }
    // ---- merge rounds: runs of `run` elements, pairwise; my VT outputs start at g * VT of the row ----
#pragma unroll 1
    for (int run = sorted ? RT : VT; run < RT; run <<= 1) {
      __syncwarp();
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        sw[mine + j] = key[j];
        if (SIDE) sp[mine + j] = (unsigned short)pay[SIDE ? j : 0];
      }
      __syncwarp();
      const int first = g * VT, pbase = first & ~(2 * run - 1), diag = first - pbase;
      const int a0 = row0 + pbase, b0 = a0 + run;
      int lo = max(0, diag - run), hi = min(diag, run);
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sw[at(a0 + mid)] <= sw[at(b0 + diag - 1 - mid)]) lo = mid + 1; else hi = mid;
      }
      int ia = lo, ib = diag - lo;
      W ka = ia < run ? sw[at(a0 + ia)] : WMAX, kb = ib < run ? sw[at(b0 + ib)] : WMAX;
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        // an exhausted run never wins; on equal words the lower run goes first
        const bool take_a = ib >= run || (ia < run && ka <= kb);
        key[j]            = take_a ? ka : kb;
        if (SIDE) pay[SIDE ? j : 0] = sp[at(take_a ? a0 + ia : b0 + ib)];
        ia += take_a ? 1 : 0;
        ib += take_a ? 0 : 1;
        const bool ok = take_a ? ia < run : ib < run;
        const W v     = ok ? sw[at(take_a ? a0 + ia : b0 + ib)] : WMAX;
        ka = take_a ? v : ka;
        kb = take_a ? kb : v;
      }
    }
    __syncwarp();
    // ---- results into shared memory, from there to memory with consecutive lanes on consecutive elements ----
    if (!PAIRS) {
#pragma unroll
      for (int j = 0; j < VT; ++j) sw[mine + j] = (W)sm_from_ordered<KB>((K)key[j], xf);
      if (special) {
        // some row of the warp holds a -0.0 or an unusual NaN, which the images fold: zeros and NaNs are
        // written again from the input, in input order
        const W zimg = (W)to_ordered_rt<KB>((K)0, xf);
        unsigned int z0 = 0, n0 = 0, cz = 0, cn = 0;
        K raw[VT];
#pragma unroll
        for (int j = 0; j < VT; ++j) {
          z0 += key[j] < zimg ? 1u : 0u;
          n0 += key[j] < WMAX ? 1u : 0u;
          const int c = g * VT + j;
          raw[j]      = (lane >> GL) < rows && (unsigned int)c < seg_len ? src[(lane >> GL) * seg_len + c] : (K)1;
          cz += sm_is_zero<KB>(raw[j]) ? 1u : 0u;
          cn += sm_is_nan<KB>(raw[j]) ? 1u : 0u;
        }
        const unsigned int start = z0 | (n0 << 16), count = cz | (cn << 16);
        unsigned int total = start, before = count;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          total += __shfl_xor_sync(0xFFFFFFFFu, total, o, G);
          const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, before, o, G);
          if (g >= o) before += t;
        }
        before -= count;
        int rz = (int)((total & 0xFFFFu) + (before & 0xFFFFu)), rn = (int)((total >> 16) + (before >> 16));
        __syncwarp();
#pragma unroll
        for (int j = 0; j < VT; ++j) {
          if (sm_is_zero<KB>(raw[j])) sw[at(row0 + rz++)] = (W)raw[j];
          if (sm_is_nan<KB>(raw[j])) sw[at(row0 + rn++)] = (W)raw[j];
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        if (SIDE) sp[mine + j] = (unsigned short)pay[SIDE ? j : 0];
        else sw[mine + j] = key[j];
      }
    }
    __syncwarp();
    K* dst = out != nullptr ? out + base * seg_len : nullptr;
    if (!PAIRS) {
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        const int i = j * 32 + lane, r = i / RT, c = i % RT;
        if (r < rows && (unsigned int)c < seg_len) dst[r * seg_len + c] = (K)sw[at(i)];
      }
    } else {
      unsigned int pos[VT];
#pragma unroll
      for (int j = 0; j < VT; ++j) {
        const int i = j * 32 + lane;
        pos[j]      = SIDE ? (unsigned int)sp[at(i)] : (unsigned int)sw[at(i)];
      }
      if (dst != nullptr) {
        // all keys of the warp's rows are read before any is written: the output may be the input
        K raw[VT];
#pragma unroll
        for (int j = 0; j < VT; ++j) {
          const int i = j * 32 + lane, r = i / RT, c = i % RT;
          if (r < rows && (unsigned int)c < seg_len) {
            if (gather) raw[j] = src[r * seg_len + (KB == 4 || SIDE ? pos[j] : (pos[j] & 0xFFFFu))];
            else raw[j] = sm_from_ordered<KB>((K)(pos[j] >> 16), xf);
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < VT; ++j) {
          const int i = j * 32 + lane, r = i / RT, c = i % RT;
          if (r < rows && (unsigned int)c < seg_len) dst[r * seg_len + c] = raw[j];
        }
      }
      if (idx_out != nullptr) {
        int64_t* idst = idx_out + base * seg_len;
#pragma unroll
        for (int j = 0; j < VT; ++j) {
          const int i = j * 32 + lane, r = i / RT, c = i % RT;
          if (r < rows && (unsigned int)c < seg_len)
            idst[r * seg_len + c] = (int64_t)(KB >= 4 ? pos[j] : (pos[j] & 0xFFFFu)) + index_offset;
        }
      }
    }
    __syncwarp();  // all reads of shared memory are done before the next rows' load
  }
}

}  // namespace b2s
