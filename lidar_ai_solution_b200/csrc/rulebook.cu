// Rulebook construction: coordinate hash table, submanifold neighbour map and
// strided-convolution map.  Integer work bound by L2 latency (small frames) or by the bytes of
// the maps (batches); every task reads its row count from device memory and strides, so
// launches never depend on host knowledge of the counts.
//
// Strided outputs are made unique and ordered without sorting: each candidate
// output cell sets one bit in a bitmap over the output grid, the popcounts of the words before
// it rank a set bit, and the rank is the output row.
//
// The steps of one rulebook are short (2-20 us) and several rulebooks are independent of one
// another, so they run as tasks of shared launches (RuleWave): a backbone of four strided and
// four SubM rulebooks takes 6 launches where one kernel per step took 24.
#include <limits.h>

#include <mutex>

#include "common.cuh"
#include "pdl.cuh"
#include "rulebook.hpp"

namespace spconvb {
namespace {

constexpr int kTaskThreads = 128;
constexpr int kTaskWarps = kTaskThreads / 32;
constexpr uint32_t kScanWords = kTaskThreads;  // bitmap words per scan block: one a thread

__device__ __forceinline__ uint32_t task_rows(const RuleTask& t) {
  return min(t.n_ptr ? load_in_order(t.n_ptr) : t.n_host, t.cap);
}

// v % s == 0 and v / s for v >= 0, without the integer division when the stride is a power
// of two (every strided layer of the lidar backbones has stride 1 or 2).
__device__ __forceinline__ bool stride_divides(int v, int s, int sh) {
  return sh >= 0 ? (v & (s - 1)) == 0 : v % s == 0;
}
__device__ __forceinline__ int stride_quotient(int v, int s, int sh) {
  return sh >= 0 ? v >> sh : v / s;
}
__host__ __device__ inline bool unit_dilation(const Kernel3& kr) {
  return kr.d[0] == 1 && kr.d[1] == 1 && kr.d[2] == 1;
}
__host__ __device__ inline bool is_k333(const Kernel3& kr) {
  return kr.k[0] == 3 && kr.k[1] == 3 && kr.k[2] == 3 && unit_dilation(kr);
}

// ---------------------------------------------------------------- the caller's rows
__device__ __forceinline__ void task_count(const RuleTask& t) {
  if (threadIdx.x != 0) return;
  const uint32_t n = t.n_ptr ? load_in_order(t.n_ptr) : t.n_host;
  if (n > t.cap) set_status(t.status, SPCONVB_ST_OVERFLOW, n);
  *t.n_out = min(n, t.cap);
}

// fp16 rows padded to 8 channels (the first layer of a lidar backbone: 4 or 5 point features in
// 16-byte rows): one thread per row, one 16-byte store.
__device__ __forceinline__ void task_pad8(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  for (uint32_t row = first; row < n; row += step) {
    const __half* src = (const __half*)t.feat + (size_t)row * t.channels;
    uint16_t h[8];
#pragma unroll
    for (int c = 0; c < 8; ++c)
      h[c] = c < t.channels ? __half_as_ushort(__ldg(src + c)) : (uint16_t)0;
    t.feat_out[row] = make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16,
                                 h[4] | (uint32_t)h[5] << 16, h[6] | (uint32_t)h[7] << 16);
  }
}

__device__ __forceinline__ void task_hash(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  if (first == 0 && t.n_ptr && *t.n_ptr > t.cap)
    set_status(t.status, SPCONVB_ST_OVERFLOW, *t.n_ptr);
  for (uint32_t row = first; row < n; row += step) {
    const int4 c = __ldg(t.coords + row);
    if ((unsigned)c.x >= (unsigned)t.gin.batch || (unsigned)c.y >= (unsigned)t.gin.g[0] ||
        (unsigned)c.z >= (unsigned)t.gin.g[1] || (unsigned)c.w >= (unsigned)t.gin.g[2]) {
      set_status(t.status, SPCONVB_ST_COORD_RANGE, row);
      continue;
    }
    hash_insert(t.table, t.mask, voxel_key(c.x, c.y, c.z, c.w, t.gin), row, t.status);
  }
}

// ------------------------------------------------------------------- SubM maps
// One thread per row: the row's coordinate is read once, its taps are walked in tap order, so
// a warp's stores of one tap land in one or two lines of map[k][.].
//
// Planes of a 3x3x3 kernel (9 taps of one k0): where the rows are few, a thread takes one plane of a
// row.  The lookups of a row are a chain of memory latencies, three planes in three threads are a
// third of it, and on a small frame there is room for them: 7.5 us for the map of 10 800 of the
// caller's rows, with a thread per row 13.9.  By rank as long as all planes run in one round (three
// rounds of 9 lookups cost what one of 27 does); by hash, whose probes are dearer, up to two rounds (a
// layer of 120 000 rows with its map 58.8 us, this way 56).
struct Planes {
  uint32_t n;  // items: rows, or three times the rows
  bool split;
};
__device__ __forceinline__ Planes planes_of(uint32_t rows, bool k333, uint32_t most) {
  Planes p;
  p.split = k333 && rows <= most;
  p.n = p.split ? 3u * rows : rows;
  return p;
}
// Row of an item, and the k0 it starts at and stops before.
__device__ __forceinline__ uint32_t plane_row(const Planes& p, uint32_t item, int& k0, int& k0_end) {
  k0 = 0;
  k0_end = 3;
  if (!p.split) return item;
  const uint32_t rows = p.n / 3u;
  k0 = item >= 2u * rows ? 2 : item >= rows ? 1 : 0;
  k0_end = k0 + 1;
  return item - (uint32_t)k0 * rows;
}

// ONE: plane `plane` only
template <bool K333, bool ONE, typename Lookup>
__device__ __forceinline__ void subm_row_taps(const int4 c, uint32_t row, int plane,
                                              const RuleTask& t, Lookup lookup) {
  const Grid3& g = t.gin;
  const Kernel3& kr = t.kr;
  const int K0 = K333 ? 3 : kr.k[0], K1 = K333 ? 3 : kr.k[1], K2 = K333 ? 3 : kr.k[2];
  const int D0 = K333 ? 1 : kr.d[0], D1 = K333 ? 1 : kr.d[1], D2 = K333 ? 1 : kr.d[2];
  const bool bok = (unsigned)c.x < (unsigned)g.batch;
  int32_t* dst = t.map + row + (size_t)(ONE ? plane * 9 : 0) * t.cap;
#pragma unroll
  for (int q = 0; q < (ONE ? 1 : K0); ++q) {
    const int k0 = ONE ? plane : q;
    const int p0 = c.y + (k0 - K0 / 2) * D0;
    const bool ok0 = bok && (unsigned)p0 < (unsigned)g.g[0];
#pragma unroll
    for (int k1 = 0; k1 < K1; ++k1) {
      const int p1 = c.z + (k1 - K1 / 2) * D1;
      const bool ok1 = ok0 && (unsigned)p1 < (unsigned)g.g[1];
#pragma unroll
      for (int k2 = 0; k2 < K2; ++k2) {
        const int p2 = c.w + (k2 - K2 / 2) * D2;
        int32_t r = -1;
        if (k0 == K0 / 2 && k1 == K1 / 2 && k2 == K2 / 2) r = (int32_t)row;
        else if (ok1 && (unsigned)p2 < (unsigned)g.g[2]) r = lookup(voxel_key(c.x, p0, p1, p2, g));
        *dst = r;
        dst += t.cap;
      }
    }
  }
}

// 3x3x3 lookups in the hash table.  A probe is a random L2 access of ~700 cycles and most find
// nothing, so what counts is how many are in flight: the first probes of the 9 taps of a plane
// are issued together and only then looked at (a probe loop per tap took its 27 latencies one
// after the other).  Taps whose first slot holds another cell go on probing one by one.
__device__ __forceinline__ void subm_hash_k333(const int4 c, uint32_t row, int k0_first, int k0_end,
                                               const RuleTask& t) {
  const Grid3& g = t.gin;
  const uint64_t* __restrict__ table = t.table;
  const bool bok = (unsigned)c.x < (unsigned)g.batch;
  int32_t* dst = t.map + row + (size_t)(k0_first * 9) * t.cap;
#pragma unroll 1
  for (int k0 = k0_first; k0 < k0_end; ++k0) {
    const int p0 = c.y + k0 - 1;
    const bool ok0 = bok && (unsigned)p0 < (unsigned)g.g[0];
    unsigned long long v[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int p1 = c.z + q / 3 - 1, p2 = c.w + q % 3 - 1;
      v[q] = 0ull;
      const bool centre = q == 4 && k0 == 1;
      if (ok0 && !centre && (unsigned)p1 < (unsigned)g.g[1] && (unsigned)p2 < (unsigned)g.g[2])
        v[q] = __ldg((const unsigned long long*)table +
                     hash_first_slot(voxel_key(c.x, p0, p1, p2, g), t.mask));
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      int32_t r = -1;
      if (q == 4 && k0 == 1) {
        r = (int32_t)row;  // the row itself, also where the table holds another row of its cell or none
      } else if (v[q] != 0ull) {
        const uint32_t key = voxel_key(c.x, p0, c.z + q / 3 - 1, c.w + q % 3 - 1, g);
        r = (uint32_t)(v[q] >> 32) == key + 1u ? (int32_t)(uint32_t)v[q]
                                               : hash_lookup_next(table, t.mask, key);
      }
      *dst = r;
      dst += t.cap;
    }
  }
}

__device__ __forceinline__ void task_subm_hash(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  const bool k333 = is_k333(t.kr);
  const Planes pl = planes_of(n, k333, step - step / 3u);
  for (uint32_t item = first; item < pl.n; item += step) {
    int k0, k0_end;
    const uint32_t row = plane_row(pl, item, k0, k0_end);
    const int4 c = __ldg(t.coords + row);
    if (k333)
      subm_hash_k333(c, row, k0, k0_end, t);
    else
      subm_row_taps<false, false>(
          c, row, 0, t, [&](uint32_t key) { return hash_lookup(t.table, t.mask, key); });
  }
}

// Rows in cell order: a warp's lookups of one tap fall into the same or adjacent bitmap words.
__device__ __forceinline__ void task_subm_rank(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  const bool k333 = is_k333(t.kr);
  auto look = [&](uint32_t key) { return rank_lookup(t.ws.bitmap, t.ws.prefix, key, t.cap); };
  const Planes pl = planes_of(n, k333, step / 3u);
  for (uint32_t item = first; item < pl.n; item += step) {
    int k0, k0_end;
    const uint32_t row = plane_row(pl, item, k0, k0_end);
    const int4 c = __ldg(t.coords + row);
    if (pl.split) subm_row_taps<true, true>(c, row, k0, t, look);
    else if (k333) subm_row_taps<true, false>(c, row, 0, t, look);
    else subm_row_taps<false, false>(c, row, 0, t, look);
  }
}

// ------------------------------------------------------------- strided maps: mark
// Visits the output cells one input row reaches: for every axis only the taps with
// (c + pad - k*dil) divisible by the stride and inside the output grid survive, so
// the nest below does ~14 divisions per row instead of 81, and `visit` runs once
// per (input row, tap) pair of the rulebook.
template <typename F>
__device__ __forceinline__ void for_each_output(const int4 c, const Grid3& gout, const Kernel3& kr,
                                                F visit) {
  for (int k0 = 0; k0 < kr.k[0]; ++k0) {
    const int v0 = c.y + kr.p[0] - k0 * kr.d[0];
    if (v0 < 0 || !stride_divides(v0, kr.s[0], kr.sh[0])) continue;
    const int o0 = stride_quotient(v0, kr.s[0], kr.sh[0]);
    if (o0 >= gout.g[0]) continue;
    for (int k1 = 0; k1 < kr.k[1]; ++k1) {
      const int v1 = c.z + kr.p[1] - k1 * kr.d[1];
      if (v1 < 0 || !stride_divides(v1, kr.s[1], kr.sh[1])) continue;
      const int o1 = stride_quotient(v1, kr.s[1], kr.sh[1]);
      if (o1 >= gout.g[1]) continue;
      for (int k2 = 0; k2 < kr.k[2]; ++k2) {
        const int v2 = c.w + kr.p[2] - k2 * kr.d[2];
        if (v2 < 0 || !stride_divides(v2, kr.s[2], kr.sh[2])) continue;
        const int o2 = stride_quotient(v2, kr.s[2], kr.sh[2]);
        if (o2 >= gout.g[2]) continue;
        visit((k0 * kr.k[1] + k1) * kr.k[2] + k2, voxel_key(c.x, o0, o1, o2, gout));
      }
    }
  }
}

// With dilation 1 the outputs an input coordinate c reaches along one axis are a range:
// tap k = c + pad - o * stride lies in [0, K) exactly for
// ceil((c + pad - K + 1) / stride) <= o <= floor((c + pad) / stride), clipped to the grid.
// No divisibility tests, no tap loop.  Nothing has checked the coordinate: none below -pad reaches a
// cell (the quotient would be rounded towards zero, to a cell and a tap that do not exist), and the
// sums stay inside an int for every value.
struct AxisRange { int lo, hi; };
__device__ __forceinline__ AxisRange output_range(int c, int a, const Grid3& gout,
                                                  const Kernel3& kr) {
  AxisRange r = {0, -1};
  if (c < -kr.p[a] || c > INT_MAX - kr.p[a]) return r;
  const int top = c + kr.p[a], t = top - kr.k[a] + 1;
  r.hi = min(stride_quotient(top, kr.s[a], kr.sh[a]), gout.g[a] - 1);
  if (t > 0) r.lo = stride_quotient(t - 1, kr.s[a], kr.sh[a]) + 1;
  return r;
}

// Up to kvol inputs reach the same cells: look before the atomic, most find them set.
__device__ __forceinline__ void mark_word(const DownWs& ws, uint32_t word, uint32_t bits) {
  uint32_t* p = ws.bitmap + word;
  if ((*(volatile uint32_t*)p & bits) != bits) atomicOr(p, bits);
}

__device__ __forceinline__ void task_mark_rows(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  const Kernel3& kr = t.kr;
  const bool unit = unit_dilation(kr) && kr.k[2] <= 32 * kr.s[2];
  for (uint32_t row = first; row < n; row += step) {
    const int4 c = __ldg(t.coords + row);
    if ((unsigned)c.x >= (unsigned)t.gin.batch) continue;
    if (unit) {
      // the reached cells are a box; its cells along the innermost axis are adjacent bits,
      // set with one atomic (two when the run crosses a word)
      const AxisRange r0 = output_range(c.y, 0, t.gout, kr), r1 = output_range(c.z, 1, t.gout, kr),
                      r2 = output_range(c.w, 2, t.gout, kr);
      if (r2.lo > r2.hi) continue;
      const uint32_t nbits = (uint32_t)(r2.hi - r2.lo + 1);
      for (int o0 = r0.lo; o0 <= r0.hi; ++o0)
        for (int o1 = r1.lo; o1 <= r1.hi; ++o1) {
          const uint32_t cell = voxel_key(c.x, o0, o1, r2.lo, t.gout);
          const unsigned long long run =
              (nbits >= 64u ? ~0ull : (1ull << nbits) - 1ull) << (cell & 31u);
          mark_word(t.ws, cell >> 5, (uint32_t)run);
          if (run >> 32) mark_word(t.ws, (cell >> 5) + 1, (uint32_t)(run >> 32));
        }
      continue;
    }
    for_each_output(c, t.gout, kr,
                    [&](int, uint32_t cell) { mark_word(t.ws, cell >> 5, 1u << (cell & 31)); });
  }
}

// 64 bits of a bitmap from cell `start` on, zero beyond its words (there is no cell 0xffffffff).
__device__ __forceinline__ unsigned long long line_bits64(const uint32_t* __restrict__ bitmap,
                                                          uint32_t words, uint32_t start) {
  const uint32_t w = start >> 5, off = start & 31u;
  const uint32_t a = w < words ? __ldg(bitmap + w) : 0u;
  const uint32_t b = w + 1 < words ? __ldg(bitmap + w + 1) : 0u;
  const uint32_t c = w + 2 < words ? __ldg(bitmap + w + 2) : 0u;
  const uint32_t low = __funnelshift_r(a, b, off), high = __funnelshift_r(b, c, off);
  return (unsigned long long)high << 32 | low;
}

// The mark step when the input rows were made by a strided rulebook themselves: the output
// bitmap is computed from the input's bitmap, 16 output cells of one line per thread.  Output
// cell o is set when any input cell of its window (o * stride - pad + [0, K) per axis, dilation
// 1) is set: the K0 x K1 input lines that matter are OR-ed as bit strings, then each output
// bit tests its K2-wide piece.  No rows are read, no two threads fight for a word (the two
// atomics per thread only merge neighbouring segments of a word).  Input cells whose rank is
// beyond the capacity of the input rows (an overflow the rulebook that made them has already
// reported) count as set.
constexpr int kMarkCells = 16;
__device__ __forceinline__ void task_mark_bitmap(const RuleTask& t, uint32_t first, uint32_t step) {
  const Grid3 &gin = t.gin, &gout = t.gout;
  const Kernel3& kr = t.kr;
  const uint32_t segs = (uint32_t)(gout.g[2] + kMarkCells - 1) / kMarkCells;
  const unsigned long long items =
      (unsigned long long)gout.batch * gout.g[0] * gout.g[1] * segs;
  const unsigned long long kmask = (1ull << kr.k[2]) - 1ull;
  for (unsigned long long item = first; item < items; item += step) {
    // fewer than 2^32 cells (checked by the callers), so 32-bit arithmetic holds
    const uint32_t line = (uint32_t)item / segs;
    const int ox0 = (int)((uint32_t)item - line * segs) * kMarkCells;
    const int ncell = min(kMarkCells, gout.g[2] - ox0);
    const uint32_t plane = line / (uint32_t)gout.g[1];
    const int o1 = (int)(line - plane * (uint32_t)gout.g[1]);
    const int b = (int)(plane / (uint32_t)gout.g[0]);
    const int o0 = (int)(plane - (uint32_t)b * (uint32_t)gout.g[0]);
    const int x0 = ox0 * kr.s[2] - kr.p[2];
    const int count = (ncell - 1) * kr.s[2] + kr.k[2];  // <= 64 (mark_from_bitmap)
    const int lo = max(x0, 0), hi = min(x0 + count - 1, gin.g[2] - 1);
    if (lo > hi) continue;
    unsigned long long win = 0ull;
    for (int k0 = 0; k0 < kr.k[0]; ++k0) {
      const int i0 = o0 * kr.s[0] - kr.p[0] + k0;
      if ((unsigned)i0 >= (unsigned)gin.g[0]) continue;
      for (int k1 = 0; k1 < kr.k[1]; k1 += 3) {
        // Three lines at once, without branches: nine loads in flight.  (A line after the other, each
        // behind its tests: 10 800 voxels 221.5 us the whole call, this way 216.8; BEVFusion's frame 261,
        // 258.)
        unsigned long long v[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int i1 = o1 * kr.s[1] - kr.p[1] + k1 + q;
          const bool in = k1 + q < kr.k[1] && (unsigned)i1 < (unsigned)gin.g[1];
          v[q] = line_bits64(t.in_ws.bitmap, t.in_ws.words,
                             in ? voxel_key(b, i0, i1, lo, gin) : 0xffffffffu);
        }
        win |= v[0] | v[1] | v[2];
      }
    }
    if (hi - lo < 63) win &= (1ull << (hi - lo + 1)) - 1ull;
    win <<= lo - x0;
    if (!win) continue;
    uint32_t r = 0;
#pragma unroll
    for (int i = 0; i < kMarkCells; ++i)
      if (i < ncell && ((win >> (i * kr.s[2])) & kmask)) r |= 1u << i;
    if (!r) continue;
    const uint32_t cell = line * (uint32_t)gout.g[2] + (uint32_t)ox0;
    const unsigned long long run = (unsigned long long)r << (cell & 31u);
    atomicOr(t.ws.bitmap + (cell >> 5), (uint32_t)run);
    if (run >> 32) atomicOr(t.ws.bitmap + (cell >> 5) + 1, (uint32_t)(run >> 32));
  }
}

// ------------------------------------------------------------- strided maps: emit
struct EmitShared {
  uint32_t before[kScanWords];  // set bits of the block's words before each
  uint32_t word[kScanWords];
  int4 cell[kScanWords];        // first cell of each word
  uint32_t blk;
  uint32_t warp_total[kTaskWarps];
  uint32_t back[kTaskWarps];
};

__device__ __forceinline__ void publish_bits(const RuleTask& t, uint32_t blk, uint32_t total) {
  atomicAdd(t.ws.scan_groups() + blk / kScanGroup, (1ull << 40) | total);
}

// Set bits of all blocks before `blk`.  Every block adds its count, with an arrival, to the total of
// its group of 16; a block needs the totals of the groups before its own, and counts the bits of the
// blocks before it in its group itself (at most 15 words a thread, from L2: counts of their own
// would make the workspace larger, and to wait for).  All totals are loaded at once (a
// batch of 8 frames has 21 000 blocks and 1 330 groups: 11 loads a thread); the chain of a look-back from block
// to block took 10 us on 2 700 blocks that start together.  What is waited for was drawn from the same
// counter before, so it is running or has finished; the wait is bounded like every other.
__device__ __forceinline__ uint32_t bits_before(const RuleTask& t, uint32_t blk, uint32_t total,
                                                EmitShared& sh) {
  unsigned long long* groups = t.ws.scan_groups();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, group = blk / kScanGroup;
  if (threadIdx.x == 0) publish_bits(t, blk, total);
  uint32_t sum = 0, spin = 0;
#pragma unroll 5
  for (uint32_t w = group * kScanGroup * kScanWords + threadIdx.x; w < blk * kScanWords; w += kTaskThreads)
    sum += (uint32_t)__popc(t.ws.bitmap[w]);
  for (uint32_t i = threadIdx.x; i < group; i += kTaskThreads) {
    unsigned long long v;
    while (((v = *(volatile unsigned long long*)(groups + i)) >> 40) != kScanGroup) {
      if (++spin < 1u << 21) {
        __nanosleep(32);
        continue;
      }
      set_status(t.status, SPCONVB_ST_TIMEOUT, 7u);
      break;
    }
    sum += (uint32_t)v;  // fewer than 2^32 cells
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) sh.back[warp] = sum;
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int w = 0; w < kTaskWarps; ++w) sum += sh.back[w];
  return sum;
}

// Ranks every set bit of one scan block: writes the rank of each word's first bit, the output
// coordinates and, for a map that is scattered into afterwards, the -1 of its rows; the last
// block publishes the count.  One pass over the bitmap; block numbers are drawn in the order blocks
// start, so that a wait can only be for a block that is running.
__device__ __forceinline__ void task_emit(const RuleTask& t, EmitShared& sh) {
  const DownWs& ws = t.ws;
  const Grid3& gout = t.gout;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sh.blk = atomicAdd(ws.scan_ticket(), 1u);
  __syncthreads();
  const uint32_t blk = sh.blk;
  const uint32_t w0 = blk * kScanWords + threadIdx.x;
  const uint32_t bits = w0 < ws.words ? ws.bitmap[w0] : 0u;
  uint32_t incl = (uint32_t)__popc(bits);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
    if ((int)lane >= d) incl += v;
  }
  if (lane == 31u) sh.warp_total[warp] = incl;
  __syncthreads();
  uint32_t total = 0, before = incl - (uint32_t)__popc(bits);
#pragma unroll
  for (int i = 0; i < kTaskWarps; ++i) {
    if (i < (int)warp) before += sh.warp_total[i];
    total += sh.warp_total[i];
  }
  if (total == 0u && blk != ws.blocks - 1) {
    // Nobody asks for ranks of words without bits: an empty block says so and makes room (the
    // 2 658 blocks of a first strided map are one and a half rounds of what runs at once; 10 800 voxels
    // 7.8 us, when they all waited for the blocks before them 13.8).
    if (threadIdx.x == 0) publish_bits(t, blk, 0u);
    return;
  }
  sh.before[threadIdx.x] = before;
  sh.word[threadIdx.x] = bits;
  if (bits) {
    uint32_t c = w0 << 5;
    uint32_t q = c / (uint32_t)gout.g[2];
    const int x = (int)(c - q * (uint32_t)gout.g[2]);
    c = q / (uint32_t)gout.g[1];
    const int y = (int)(q - c * (uint32_t)gout.g[1]);
    q = c / (uint32_t)gout.g[0];
    sh.cell[threadIdx.x] = make_int4((int)q, (int)(c - q * (uint32_t)gout.g[0]), y, x);
  }
  const uint32_t base = bits_before(t, blk, total, sh);
  if (threadIdx.x == 0 && blk == ws.blocks - 1) {
    if (base + total > t.cap) set_status(t.status, SPCONVB_ST_OVERFLOW, base + total);
    *t.n_out = min(base + total, t.cap);
  }
  if (w0 < ws.words) ws.prefix[w0] = base + before;
  // One thread per row: the row's word is the last one with at most that many bits before it,
  // its bit is found by halving.  The stores coalesce and a block takes as long as its rows,
  // which a lidar scene packs into few words: walking the words, a warp or a lane at a time, took
  // 30-90 us on the dense grids of the later stages, blocks of 512 words still 45.
  const uint32_t rows = base < t.cap ? min(total, t.cap - base) : 0u;
  const int kvol = t.map ? t.kr.k[0] * t.kr.k[1] * t.kr.k[2] : 0;
#pragma unroll 1
  for (uint32_t r = threadIdx.x; r < rows; r += kTaskThreads) {
    uint32_t w = 0;
#pragma unroll
    for (uint32_t half = kScanWords / 2; half > 0; half >>= 1)
      if (sh.before[w + half] <= r) w += half;
    uint32_t left = sh.word[w], nth = r - sh.before[w];
    int4 c = sh.cell[w];
#pragma unroll
    for (int half = 16; half > 0; half >>= 1) {
      const uint32_t low = (uint32_t)__popc(left & ((1u << half) - 1u));
      if (nth >= low) {
        nth -= low;
        left >>= half;
        c.w += half;
      }
    }
    while (c.w >= gout.g[2]) {
      c.w -= gout.g[2];
      if (++c.z >= gout.g[1]) {
        c.z = 0;
        if (++c.y >= gout.g[0]) { c.y = 0; ++c.x; }
      }
    }
    t.out_coords[base + r] = c;
    int32_t* m = t.map + base + r;
#pragma unroll 9
    for (int k = 0; k < kvol; ++k) {
      *m = -1;
      m += t.cap;
    }
  }
}

// ------------------------------------------------------------- strided maps: fill
// Input-stationary fill of the output-stationary map: every (input row, tap) pair finds its
// output row by rank and writes itself there.  The cells an input reaches were marked by it, so
// with dilation 1 nothing is tested: word and rank are loaded side by side.
__device__ __forceinline__ void task_scatter(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  const Kernel3& kr = t.kr;
  const uint32_t cap_out = t.map_cap;
  const bool unit = unit_dilation(kr);
  for (uint32_t row = first; row < n; row += step) {
    const int4 c = __ldg(t.coords + row);
    if ((unsigned)c.x >= (unsigned)t.gin.batch) continue;
    if (unit) {
      const AxisRange r0 = output_range(c.y, 0, t.gout, kr), r1 = output_range(c.z, 1, t.gout, kr),
                      r2 = output_range(c.w, 2, t.gout, kr);
      for (int o0 = r0.lo; o0 <= r0.hi; ++o0) {
        const int k0 = c.y + kr.p[0] - o0 * kr.s[0];
        for (int o1 = r1.lo; o1 <= r1.hi; ++o1) {
          const int k01 = k0 * kr.k[1] + (c.z + kr.p[1] - o1 * kr.s[1]);
#pragma unroll 2
          for (int o2 = r2.lo; o2 <= r2.hi; ++o2) {
            const int k = k01 * kr.k[2] + (c.w + kr.p[2] - o2 * kr.s[2]);
            const uint32_t cell = voxel_key(c.x, o0, o1, o2, t.gout);
            const uint32_t o = __ldg(t.ws.prefix + (cell >> 5)) +
                               __popc(__ldg(t.ws.bitmap + (cell >> 5)) & ((1u << (cell & 31u)) - 1u));
            if (o < cap_out) t.map[(size_t)k * cap_out + o] = (int32_t)row;
          }
        }
      }
      continue;
    }
    for_each_output(c, t.gout, kr, [&](int k, uint32_t cell) {
      const int32_t o = rank_lookup(t.ws.bitmap, t.ws.prefix, cell, cap_out);
      if (o >= 0) t.map[(size_t)k * cap_out + o] = (int32_t)row;
    });
  }
}

// Output-stationary form of the strided map, for inputs that were themselves made by a
// strided rulebook (their bitmap and ranks exist): one thread per output row walks the
// taps in tap order, finds the input cell of each (out * stride - pad + tap * dilation) and
// ranks it in the input's bitmap.  Every map entry is written exactly once, so there is no
// fill pass, and a warp's stores of one tap land in one or two lines of map[k][.].
template <bool K333, bool ONE>
__device__ __forceinline__ void gather_row(const int4 c, uint32_t row, int plane,
                                           const RuleTask& t) {
  const Grid3& gin = t.gin;
  const Kernel3& kr = t.kr;
  const int K0 = K333 ? 3 : kr.k[0], K1 = K333 ? 3 : kr.k[1], K2 = K333 ? 3 : kr.k[2];
  int32_t* dst = t.map + row + (size_t)(ONE ? plane * 9 : 0) * t.cap;
  const bool bok = (unsigned)c.x < (unsigned)gin.batch;
#pragma unroll
  for (int q = 0; q < (ONE ? 1 : K0); ++q) {
    const int k0 = ONE ? plane : q;
    const int p0 = c.y * kr.s[0] - kr.p[0] + k0 * (K333 ? 1 : kr.d[0]);
    const bool ok0 = bok && (unsigned)p0 < (unsigned)gin.g[0];
#pragma unroll
    for (int k1 = 0; k1 < K1; ++k1) {
      const int p1 = c.z * kr.s[1] - kr.p[1] + k1 * (K333 ? 1 : kr.d[1]);
      const bool ok1 = ok0 && (unsigned)p1 < (unsigned)gin.g[1];
#pragma unroll
      for (int k2 = 0; k2 < K2; ++k2) {
        const int p2 = c.w * kr.s[2] - kr.p[2] + k2 * (K333 ? 1 : kr.d[2]);
        int32_t r = -1;
        if (ok1 && (unsigned)p2 < (unsigned)gin.g[2])
          r = rank_lookup(t.in_ws.bitmap, t.in_ws.prefix, voxel_key(c.x, p0, p1, p2, gin),
                          t.other_cap);
        *dst = r;
        dst += t.cap;
      }
    }
  }
}

__device__ __forceinline__ void task_gather(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  const bool k333 = is_k333(t.kr);
  const Planes pl = planes_of(n, k333, step / 3u);
  for (uint32_t item = first; item < pl.n; item += step) {
    int k0, k0_end;
    const uint32_t row = plane_row(pl, item, k0, k0_end);
    const int4 c = __ldg(t.coords + row);
    if (pl.split) gather_row<true, true>(c, row, k0, t);
    else if (k333) gather_row<true, false>(c, row, 0, t);
    else gather_row<false, false>(c, row, 0, t);
  }
}

// Map of an inverse (transposed) convolution: it runs over the pairs of a strided rulebook with
// input and output swapped, so its outputs are that rulebook's input rows and map[k][i] is the
// strided output row that input row i reaches through tap k.  One thread per (row, tap), rows
// fastest: coalesced stores of map[k][row].
__device__ __forceinline__ void task_inverse(const RuleTask& t, uint32_t first, uint32_t step) {
  const uint32_t n = task_rows(t);
  const Kernel3& kr = t.kr;
  const int kvol = kr.k[0] * kr.k[1] * kr.k[2];
  const unsigned long long work = (unsigned long long)n * kvol;
  for (unsigned long long idx = first; idx < work; idx += step) {
    const int k = (int)(idx / n);
    const uint32_t row = (uint32_t)(idx - (unsigned long long)k * n);
    const int4 c = __ldg(t.coords + row);
    const int k2 = k % kr.k[2], k1 = (k / kr.k[2]) % kr.k[1], k0 = k / (kr.k[2] * kr.k[1]);
    const int v0 = c.y + kr.p[0] - k0 * kr.d[0], v1 = c.z + kr.p[1] - k1 * kr.d[1],
              v2 = c.w + kr.p[2] - k2 * kr.d[2];
    int32_t o = -1;
    if ((unsigned)c.x < (unsigned)t.gin.batch && v0 >= 0 && v1 >= 0 && v2 >= 0 &&
        stride_divides(v0, kr.s[0], kr.sh[0]) && stride_divides(v1, kr.s[1], kr.sh[1]) &&
        stride_divides(v2, kr.s[2], kr.sh[2])) {
      const int o0 = stride_quotient(v0, kr.s[0], kr.sh[0]),
                o1 = stride_quotient(v1, kr.s[1], kr.sh[1]),
                o2 = stride_quotient(v2, kr.s[2], kr.sh[2]);
      if (o0 < t.gout.g[0] && o1 < t.gout.g[1] && o2 < t.gout.g[2])
        o = rank_lookup(t.ws.bitmap, t.ws.prefix, voxel_key(c.x, o0, o1, o2, t.gout), t.other_cap);
    }
    t.map[(size_t)k * t.cap + row] = o;
  }
}

// ------------------------------------------------------------------------- launch
__global__ void __launch_bounds__(kTaskThreads, 12)
rule_wave_kernel(const __grid_constant__ RuleWave w) {
  __shared__ EmitShared sh;
  // No early trigger: the blocks of the next launch would take the places of this one's later
  // blocks and wait there (SubM map of 120 000 rows 22 us, with it 28).
  pdl_wait();
  uint32_t blk = blockIdx.x;
  int i = 0;
  while (blk >= w.t[i].blocks) {
    blk -= w.t[i].blocks;
    ++i;
  }
  // by value: its fields are read once, into registers.  Through a reference every use would be
  // a load from the parameter space again, after each store to the map (twice the time).
  const RuleTask t = w.t[i];
  const uint32_t first = blk * kTaskThreads + threadIdx.x, step = t.blocks * kTaskThreads;
  switch (t.kind) {
    case TASK_COUNT: task_count(t); break;
    case TASK_PAD8: task_pad8(t, first, step); break;
    case TASK_HASH: task_hash(t, first, step); break;
    case TASK_SUBM_HASH: task_subm_hash(t, first, step); break;
    case TASK_SUBM_RANK: task_subm_rank(t, first, step); break;
    case TASK_MARK_ROWS: task_mark_rows(t, first, step); break;
    case TASK_MARK_BITMAP: task_mark_bitmap(t, first, step); break;
    case TASK_EMIT: task_emit(t, sh); break;
    case TASK_SCATTER: task_scatter(t, first, step); break;
    case TASK_GATHER: task_gather(t, first, step); break;
    case TASK_INVERSE: task_inverse(t, first, step); break;
  }
}

uint32_t down_words(const int32_t og[3], int batch) {
  unsigned long long cells = (unsigned long long)batch * og[0] * og[1] * og[2];
  return (uint32_t)((cells + 31) / 32);
}
uint32_t scan_blocks(uint32_t words) { return (words + kScanWords - 1) / kScanWords; }

bool slots_ok(uint32_t cap, uint32_t slots) {
  return slots >= 8 && !(slots & (slots - 1)) && slots >= 2ull * cap;
}

}  // namespace

// (in 128 bits: the product of three extents and a batch may pass 2^64)
bool grid_fits(const int32_t g[3], int batch) {
  if (batch < 1 || g[0] < 1 || g[1] < 1 || g[2] < 1) return false;
  return (unsigned __int128)batch * g[0] * g[1] * g[2] < 0xffffffffull;
}

int check_hash(const int32_t grid[3], int batch, uint32_t cap, uint32_t slots) {
  if (!slots_ok(cap, slots)) return SPCONVB_E_ARG;
  return grid_fits(grid, batch) ? SPCONVB_OK : SPCONVB_E_RANGE;
}

int check_subm(const int32_t grid[3], int batch, const int32_t k[3], const int32_t d[3]) {
  if (!grid_fits(grid, batch)) return SPCONVB_E_RANGE;
  for (int a = 0; a < 3; ++a)
    if (k[a] < 1 || !(k[a] & 1) || d[a] < 1) return SPCONVB_E_ARG;
  return (long long)k[0] * k[1] * k[2] <= 65535 ? SPCONVB_OK : SPCONVB_E_ARG;
}

int check_strided(const int32_t grid[3], int batch, const int32_t k[3], const int32_t s[3],
                  const int32_t p[3], const int32_t d[3], int32_t og[3]) {
  if (!grid_fits(grid, batch)) return SPCONVB_E_RANGE;
  for (int a = 0; a < 3; ++a) {
    if (k[a] < 1 || s[a] < 1 || d[a] < 1 || p[a] < 0) return SPCONVB_E_ARG;
    og[a] = spconvb_out_extent(grid[a], k[a], s[a], p[a], d[a]);
    if (og[a] < 1) return SPCONVB_E_ARG;
  }
  if (!grid_fits(og, batch)) return SPCONVB_E_RANGE;
  return (long long)k[0] * k[1] * k[2] <= 65535 ? SPCONVB_OK : SPCONVB_E_ARG;
}

int launch_rule_wave(const RuleWave& w, cudaStream_t st) {
  uint32_t blocks = 0;
  for (int i = 0; i < w.count; ++i) blocks += w.t[i].blocks;
  if (!blocks) return SPCONVB_OK;
  SPCONVB_CUDA_TRY(launch_pdl(rule_wave_kernel, dim3(blocks), dim3(kTaskThreads), 0, st, w));
  return SPCONVB_OK;
}

// Blocks of a task that strides: one item per thread up to 12 blocks an SM, what fits on an empty
// GPU.  (6 an SM: SubM map of 120 000 rows 31.6 us instead of 27.1, of 234 910 ranked rows 18.2
// instead of 13.1.)
uint32_t task_blocks(unsigned long long items) {
  const unsigned long long b = (items + kTaskThreads - 1) / kTaskThreads, most = kSmCount * 12;
  return (uint32_t)(b < 1 ? 1 : b < most ? b : most);
}

// The maps of 3x3x3 kernels may take a thread per plane of a row.
uint32_t row_task_blocks(int32_t kind, unsigned long long rows) {
  const bool planes = kind == TASK_SUBM_HASH || kind == TASK_SUBM_RANK || kind == TASK_GATHER;
  return task_blocks(planes ? 3 * rows : rows);
}

uint32_t mark_bitmap_blocks(const int32_t og[3], int batch) {
  return task_blocks((unsigned long long)batch * og[0] * og[1] *
                     (unsigned long long)((og[2] + kMarkCells - 1) / kMarkCells));
}

Grid3 make_grid(const int32_t g[3], int batch) {
  Grid3 r;
  r.g[0] = g[0]; r.g[1] = g[1]; r.g[2] = g[2];
  r.batch = batch;
  return r;
}

Kernel3 make_kernel3(const int32_t k[3], const int32_t s[3], const int32_t p[3],
                     const int32_t d[3]) {
  Kernel3 kr;
  for (int a = 0; a < 3; ++a) {
    kr.k[a] = k[a];
    kr.s[a] = s ? s[a] : 1;
    kr.p[a] = p ? p[a] : 0;
    kr.d[a] = d[a];
    kr.sh[a] = -1;
    for (int b = 0; b < 16; ++b)
      if (kr.s[a] == (1 << b)) kr.sh[a] = b;
  }
  return kr;
}

DownWs down_ws(const int32_t og[3], int batch, const void* workspace) {
  DownWs ws;
  ws.words = down_words(og, batch);
  ws.blocks = scan_blocks(ws.words);
  ws.bitmap = (uint32_t*)workspace;
  ws.prefix = ws.bitmap + ws.words;
  ws.scan = (uint32_t*)(((uintptr_t)(ws.prefix + ws.words) + 7u) & ~(uintptr_t)7u);
  return ws;
}

// A thread's window of input cells has to fit 64 bits.
bool mark_from_bitmap(const Kernel3& kr) {
  return unit_dilation(kr) && kr.k[2] <= 32 && (kMarkCells - 1) * kr.s[2] + kr.k[2] <= 64;
}

// ------------------------------------------------- allocation-free variant
// Scratch for spconvb_down_map_static: part of the library image, so every GPU
// that loads the library holds these bytes until the process exits.
constexpr size_t kStaticScratchBytes = SPCONVB_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_down_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_down_scratch_ptr[kMaxDevices] = {};
static std::mutex g_down_scratch_mutex;

// The array's name is only a host-side handle; the address kernels can use
// comes from cudaGetSymbolAddress, asked once per device with that device current.
static int static_scratch_for_current_device(void** out) {
  int dev = -1;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) return (int)ce;
  if (dev < 0 || dev >= kMaxDevices) return SPCONVB_E_ARG;
  std::lock_guard<std::mutex> lock(g_down_scratch_mutex);
  if (!g_down_scratch_ptr[dev]) {
    void* p = nullptr;
    ce = cudaGetSymbolAddress(&p, g_down_scratch);
    if (ce != cudaSuccess) return (int)ce;
    if (!p) return SPCONVB_E_STATE;
    g_down_scratch_ptr[dev] = p;
  }
  *out = g_down_scratch_ptr[dev];
  return SPCONVB_OK;
}

}  // namespace spconvb

using namespace spconvb;

// One task as a launch of its own.
static int launch_task(const RuleTask& t, void* stream) {
  RuleWave w;
  w.add(t);
  return launch_rule_wave(w, (cudaStream_t)stream);
}

static RuleTask row_task(int32_t kind, const int32_t* coords, const uint32_t* n_ptr, uint32_t cap,
                         uint32_t launch_rows) {
  RuleTask t;
  t.kind = kind;
  t.coords = (const int4*)coords;
  t.n_ptr = n_ptr;
  t.cap = cap;
  t.blocks = row_task_blocks(kind, launch_rows == 0 || launch_rows > cap ? cap : launch_rows);
  return t;
}

extern "C" {

uint32_t spconvb_hash_slots(uint32_t cap_rows) {
  uint32_t s = 1024;
  while (s < 2u * cap_rows && s < 0x80000000u) s <<= 1;
  return s;
}

// Eight slots a row up to 8 MB (a table the L2 holds many times over): at half load every second
// lookup of an absent cell goes on to a second dependent probe or more.  120 000 rows: SubM map
// 68 us with 2^18 slots, 33 with 2^19, 22 with 2^20.
uint32_t spconvb_hash_slots_fast(uint32_t cap_rows) {
  uint32_t s = spconvb_hash_slots(cap_rows);
  while (s < 8u * cap_rows && s < (1u << 20)) s <<= 1;
  return s;
}

int32_t spconvb_out_extent(int32_t in, int32_t k, int32_t stride, int32_t pad, int32_t dilation) {
  int v = in + 2 * pad - dilation * (k - 1) - 1;
  if (v < 0 || stride < 1) return 0;
  return v / stride + 1;
}

int spconvb_hash_build(const int32_t* coords, const uint32_t* n_ptr, uint32_t cap,
                       uint32_t launch_rows, const int32_t grid[3], int32_t batch,
                       uint64_t* table, uint32_t slots, uint32_t flags, uint32_t* status,
                       void* stream) {
  if (!coords || !n_ptr || !table || !grid) return SPCONVB_E_ARG;
  const int rc = check_hash(grid, batch, cap, slots);
  if (rc != SPCONVB_OK) return rc;
  if (!(flags & SPCONVB_FLAG_PREZEROED))
    SPCONVB_CUDA_TRY(cudaMemsetAsync(table, 0, sizeof(uint64_t) * (size_t)slots,
                                     (cudaStream_t)stream));
  RuleTask t = row_task(TASK_HASH, coords, n_ptr, cap, launch_rows);
  t.gin = make_grid(grid, batch);
  t.table = table;
  t.mask = slots - 1;
  t.status = status;
  return launch_task(t, stream);
}

int spconvb_subm_map(const int32_t* coords, const uint32_t* n_ptr, uint32_t cap,
                     uint32_t launch_rows, const int32_t grid[3], int32_t batch,
                     const int32_t ksize[3], const int32_t dilation[3], const uint64_t* table,
                     uint32_t slots, int32_t* map, uint32_t* status, void* stream) {
  (void)status;
  if (!coords || !n_ptr || !table || !map || !grid || !ksize || !dilation) return SPCONVB_E_ARG;
  if (slots < 8 || (slots & (slots - 1))) return SPCONVB_E_ARG;
  const int rc = check_subm(grid, batch, ksize, dilation);
  if (rc != SPCONVB_OK) return rc;
  RuleTask t = row_task(TASK_SUBM_HASH, coords, n_ptr, cap, launch_rows);
  t.gin = make_grid(grid, batch);
  t.kr = make_kernel3(ksize, nullptr, nullptr, dilation);
  t.table = (uint64_t*)table;
  t.mask = slots - 1;
  t.map = map;
  return launch_task(t, stream);
}

int spconvb_subm_map_ranked(const int32_t* coords, const uint32_t* n_ptr, uint32_t cap,
                            uint32_t launch_rows, const int32_t grid[3], int32_t batch,
                            const int32_t ksize[3], const int32_t dilation[3],
                            const void* down_workspace, int32_t* map, uint32_t* status,
                            void* stream) {
  (void)status;
  if (!coords || !n_ptr || !down_workspace || !map || !grid || !ksize || !dilation)
    return SPCONVB_E_ARG;
  const int rc = check_subm(grid, batch, ksize, dilation);
  if (rc != SPCONVB_OK) return rc;
  RuleTask t = row_task(TASK_SUBM_RANK, coords, n_ptr, cap, launch_rows);
  t.gin = make_grid(grid, batch);
  t.kr = make_kernel3(ksize, nullptr, nullptr, dilation);
  t.ws = down_ws(grid, batch, down_workspace);
  t.map = map;
  return launch_task(t, stream);
}

int spconvb_inverse_map(const int32_t* coords, const uint32_t* n_ptr, uint32_t cap,
                        uint32_t launch_rows, const int32_t grid[3], int32_t batch,
                        const int32_t ksize[3], const int32_t stride[3], const int32_t pad[3],
                        const int32_t dilation[3], const void* down_workspace,
                        uint32_t cap_coarse, int32_t* map, uint32_t* status, void* stream) {
  (void)status;
  if (!coords || !n_ptr || !grid || !ksize || !stride || !pad || !dilation || !down_workspace ||
      !map)
    return SPCONVB_E_ARG;
  int32_t og[3];
  const int rc = check_strided(grid, batch, ksize, stride, pad, dilation, og);
  if (rc != SPCONVB_OK) return rc;
  const int kvol = ksize[0] * ksize[1] * ksize[2];
  RuleTask t = row_task(TASK_INVERSE, coords, n_ptr, cap, launch_rows);
  t.blocks = task_blocks((unsigned long long)(launch_rows == 0 || launch_rows > cap ? cap
                                                                                    : launch_rows) *
                         kvol);
  t.gin = make_grid(grid, batch);
  t.gout = make_grid(og, batch);
  t.kr = make_kernel3(ksize, stride, pad, dilation);
  t.ws = down_ws(og, batch, down_workspace);
  t.other_cap = cap_coarse;
  t.map = map;
  return launch_task(t, stream);
}

size_t spconvb_down_workspace_bytes(const int32_t out_grid[3], int32_t batch) {
  if (!out_grid || !grid_fits(out_grid, batch)) return 0;
  // The scan's state takes two words for 2 048 of the bitmap, one and what its alignment takes: inside
  // one word for 1 024 and 16.  (The size is part of the interface: it decides which grids
  // spconvb_down_map_static takes.)
  const size_t words = down_words(out_grid, batch);
  return sizeof(uint32_t) * (2 * words + (words + 1023) / 1024 + 16);
}

// Shared body of spconvb_down_map and spconvb_down_map_ranked.
static int down_map_impl(const int32_t* in_coords, const uint32_t* n_in_ptr, uint32_t cap_in,
                         uint32_t launch_rows, const int32_t in_grid[3], int32_t batch,
                         const int32_t ksize[3], const int32_t stride[3], const int32_t pad[3],
                         const int32_t dilation[3], const void* in_workspace, void* workspace,
                         int32_t* out_coords, uint32_t* n_out_ptr, uint32_t cap_out, int32_t* map,
                         uint64_t* out_table, uint32_t out_slots, uint32_t flags,
                         uint32_t* status, void* stream) {
  if (!in_coords || !n_in_ptr || !in_grid || !ksize || !stride || !pad || !dilation ||
      !workspace || !out_coords || !n_out_ptr || !map)
    return SPCONVB_E_ARG;
  if (out_table && !slots_ok(cap_out, out_slots)) return SPCONVB_E_ARG;
  int32_t og[3];
  int rc = check_strided(in_grid, batch, ksize, stride, pad, dilation, og);
  if (rc != SPCONVB_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;

  const DownWs ws = down_ws(og, batch, workspace);
  // PREZEROED speaks of the bitmap (and the table): the scan's state is this library's own and is
  // cleared on every call.  A stale ticket would number blocks past the end.
  SPCONVB_CUDA_TRY(cudaMemsetAsync(ws.scan, 0, sizeof(uint32_t) * scan_state_words(ws.blocks), st));
  if (!(flags & SPCONVB_FLAG_PREZEROED)) {
    SPCONVB_CUDA_TRY(cudaMemsetAsync(ws.bitmap, 0, sizeof(uint32_t) * (size_t)ws.words, st));
    if (out_table)
      SPCONVB_CUDA_TRY(cudaMemsetAsync(out_table, 0, sizeof(uint64_t) * (size_t)out_slots, st));
  }
  RuleTask mark = row_task(TASK_MARK_ROWS, in_coords, n_in_ptr, cap_in, launch_rows);
  mark.gin = make_grid(in_grid, batch);
  mark.gout = make_grid(og, batch);
  mark.kr = make_kernel3(ksize, stride, pad, dilation);
  mark.ws = ws;
  RuleTask fill = mark;
  if (in_workspace) mark.in_ws = fill.in_ws = down_ws(in_grid, batch, in_workspace);
  // rows made by a rulebook: their bitmap gives the outputs' bitmap directly
  if (in_workspace && mark_from_bitmap(mark.kr)) {
    mark.kind = TASK_MARK_BITMAP;
    mark.blocks = mark_bitmap_blocks(og, batch);
  }
  RuleTask emit;
  emit.kind = TASK_EMIT;
  emit.blocks = ws.blocks;
  emit.cap = cap_out;
  emit.gout = mark.gout;
  emit.kr = mark.kr;
  emit.ws = ws;
  emit.out_coords = (int4*)out_coords;
  emit.n_out = n_out_ptr;
  emit.map = in_workspace ? nullptr : map;
  emit.status = status;
  fill.map = map;
  if (in_workspace) {
    // the inputs can be ranked: every map entry is looked up from the output side
    fill.kind = TASK_GATHER;
    fill.coords = (const int4*)out_coords;
    fill.n_ptr = n_out_ptr;
    fill.cap = cap_out;
    fill.other_cap = cap_in;
    fill.blocks = row_task_blocks(TASK_GATHER, cap_out);
  } else {
    fill.kind = TASK_SCATTER;
    fill.map_cap = cap_out;
  }
  rc = launch_task(mark, stream);
  if (rc == SPCONVB_OK) rc = launch_task(emit, stream);
  if (rc != SPCONVB_OK) return rc;
  RuleWave last;
  last.add(fill);
  if (out_table) {  // the outputs' hash table, for callers that want one
    RuleTask hash = row_task(TASK_HASH, out_coords, n_out_ptr, cap_out, cap_out);
    hash.gin = mark.gout;
    hash.table = out_table;
    hash.mask = out_slots - 1;
    hash.status = status;
    last.add(hash);
  }
  return launch_rule_wave(last, st);
}

int spconvb_down_map(const int32_t* in_coords, const uint32_t* n_in_ptr, uint32_t cap_in,
                     uint32_t launch_rows, const int32_t in_grid[3], int32_t batch,
                     const int32_t ksize[3], const int32_t stride[3], const int32_t pad[3],
                     const int32_t dilation[3], const uint64_t* in_table, uint32_t in_slots,
                     void* workspace, int32_t* out_coords, uint32_t* n_out_ptr, uint32_t cap_out,
                     int32_t* map, uint64_t* out_table, uint32_t out_slots, uint32_t flags,
                     uint32_t* status, void* stream) {
  (void)in_table;
  (void)in_slots;
  return down_map_impl(in_coords, n_in_ptr, cap_in, launch_rows, in_grid, batch, ksize, stride,
                       pad, dilation, nullptr, workspace, out_coords, n_out_ptr, cap_out, map,
                       out_table, out_slots, flags, status, stream);
}

int spconvb_down_map_ranked(const int32_t* in_coords, const uint32_t* n_in_ptr, uint32_t cap_in,
                            uint32_t launch_rows, const int32_t in_grid[3], int32_t batch,
                            const int32_t ksize[3], const int32_t stride[3],
                            const int32_t pad[3], const int32_t dilation[3],
                            const void* in_workspace, void* workspace, int32_t* out_coords,
                            uint32_t* n_out_ptr, uint32_t cap_out, int32_t* map,
                            uint64_t* out_table, uint32_t out_slots, uint32_t flags,
                            uint32_t* status, void* stream) {
  if (!in_workspace) return SPCONVB_E_ARG;
  return down_map_impl(in_coords, n_in_ptr, cap_in, launch_rows, in_grid, batch, ksize, stride,
                       pad, dilation, in_workspace, workspace, out_coords, n_out_ptr, cap_out, map,
                       out_table, out_slots, flags, status, stream);
}

int spconvb_down_map_static(const int32_t* in_coords, const uint32_t* n_in_ptr, uint32_t cap_in,
                            uint32_t launch_rows, const int32_t in_grid[3], int32_t batch,
                            const int32_t ksize[3], const int32_t stride[3],
                            const int32_t pad[3], const int32_t dilation[3],
                            const uint64_t* in_table, uint32_t in_slots, int32_t* out_coords,
                            uint32_t* n_out_ptr, uint32_t cap_out, int32_t* map,
                            uint64_t* out_table, uint32_t out_slots, uint32_t flags,
                            uint32_t* status, void* stream) {
  // every argument check of spconvb_down_map that can fail comes first: nothing of the
  // caller's memory (the optional output table) is cleared for a call that is then refused
  if (!in_coords || !n_in_ptr || !in_grid || !ksize || !stride || !pad || !dilation ||
      !out_coords || !n_out_ptr || !map)
    return SPCONVB_E_ARG;
  if (out_table && !slots_ok(cap_out, out_slots)) return SPCONVB_E_ARG;
  int32_t og[3];
  int rc = check_strided(in_grid, batch, ksize, stride, pad, dilation, og);
  if (rc != SPCONVB_OK) return rc;
  const size_t need = spconvb_down_workspace_bytes(og, batch);
  if (need > kStaticScratchBytes) return SPCONVB_E_SCRATCH_LIMIT;
  void* scratch = nullptr;
  rc = static_scratch_for_current_device(&scratch);
  if (rc != SPCONVB_OK) return rc;
  // The array still holds the previous call's bitmap: it is cleared on every call, whatever the
  // caller says about its own buffers.
  cudaStream_t st = (cudaStream_t)stream;
  SPCONVB_CUDA_TRY(
      cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * (size_t)down_words(og, batch), st));
  if (out_table && !(flags & SPCONVB_FLAG_PREZEROED))
    SPCONVB_CUDA_TRY(cudaMemsetAsync(out_table, 0, sizeof(uint64_t) * (size_t)out_slots, st));
  return spconvb_down_map(in_coords, n_in_ptr, cap_in, launch_rows, in_grid, batch, ksize, stride,
                          pad, dilation, in_table, in_slots, scratch, out_coords, n_out_ptr,
                          cap_out, map, out_table, out_slots, flags | SPCONVB_FLAG_PREZEROED,
                          status, stream);
}


}  // extern "C"
