// Sparse convolution as an implicit GEMM on the sm_100a tensor cores, voxel rows on
// the N side of the MMA.
//
//   out[o, :] = epilogue( sum_k  W[:, k, :] . in[map[k][o], :] )
//
// is a GEMM between the weights [Cout x K] and a matrix [rows x K], K = kvol *
// Cin, that does not exist in memory: its row o is the concatenation of the
// feature rows of o's neighbours (zeros where a neighbour is absent).  A
// tcgen05.mma takes the same time whether its accumulator has 64 or 128 rows, and
// its time grows with its columns, so the voxel rows are put on the wide side: the
// weights are the M operand (128 accumulator rows = output channels, copied 128 / Cout
// times when Cout is smaller), a tile of up to 256 voxel rows is the N operand, and the
// accumulator in TMEM is the transposed output tile D[channel][row].  Copies of the
// weights let more epilogue warps share a tile.  The kernel is persistent (one CTA per
// SM) and warp-specialised:
//
//   warps 0-7   epilogue: warp w reads its lane quadrant (its channels) and its
//               share of the tile's rows from the accumulator with tcgen05.ld,
//               applies dequant + bias + activation (+ residual add) + requant
//               with per-lane scale and bias, and stores one element a lane: a
//               warp covers 32 contiguous channels of a row.  (Transposing 4x4
//               blocks for 4-byte stores took more instructions than it saved:
//               64 -> 64 with a residual 51.8 us, this way 45.9.)
//   warp  8     allocates TMEM; walks the chunks converged, one elected lane issues
//               tcgen05.mma (kind::i8 with int32 accumulators or kind::f16 with fp32)
//   warps 9-24  producers, two groups of as many warps as the tile has 32 rows that take
//               the chunks in turn (the work of a warp per chunk is a chain of dependent steps - wait for
//               the stage, neighbour indices, addresses, copies, arrival - that
//               takes longer than the tensor pipe needs for the chunk; two groups
//               give each warp two chunk periods for it).  Within a group each warp
//               owns 32 rows of the tile.  A thread loads the 8 neighbour indices
//               it needs for a chunk straight into registers (two 16-byte loads, two
//               of its chunks ahead) and gathers with 16-byte cp.async (8 lanes
//               per row, so a row is one contiguous request; zero-fill for missing
//               neighbours) straight into the 128-byte-swizzled K-major layout the
//               MMA reads.  A producer never waits for its copies: every thread lets
//               them arrive on the stage's mbarrier when they land, so all free
//               stages of the ring are in flight.
//   warp  25    streams the pre-swizzled weight chunks with bulk async copies into a
//               ring of their own, or keeps all of them there
//
// What bounds it.  On tall tiles the round trip of a stage - freed, gathered (a cp.async takes
// about a microsecond under load), multiplied, freed - over the number of stages in flight, and
// then shared memory: in isolation the MMAs of a 256-row chunk take 513 cycles, its gather 460
// (cp.async.cg; 640 with .ca, which keeps a copy in L1 that nothing reads again) and its weights
// 310, and they overlap, but with four stages of rows and weights together a chunk took 1000.
// Hence two rings that are sized to the tile's height in the kernel (256 rows: 5 stages of
// rows and 4 of weights; 160 rows: 6 and 6), and no work beside the MMAs in the issuing warp.
// Measured with both, int8, us: 208 071 rows 64 -> 64 49.2 to 41.3, 128 -> 128 86.9 to 69.3
// (730 cycles a chunk), fp16 181.6 to 158.1; 30 000 rows 128 -> 128 18.9 to 16.4.
//
// On low tiles the issuing warp is what a chunk waits for: 32-row tiles, 128 channels, 412 cycles a
// chunk in it, of which 74 are its look at the stage's barrier; 628 and 121 on 224 rows, where the
// MMAs fill the rest (clock counts of one CTA).  Close behind lies what a chunk brings into every SM,
// 16 KB of weights and 4 KB of rows: 50 bytes a cycle, the same weights 148 times over from L2.
//
// K is walked in chunks of 128 bytes (one swizzle atom per row): a chunk is 8
// taps of a 16-byte row, ..., 1 tap of a 128-byte row, or half a 256-byte row.
// The accumulator is double-buffered in TMEM (2 x 256 columns) so the epilogue of
// tile t overlaps the MMAs of tile t+1.
//
// Every wait is bounded: a wait that runs out sets SPCONVB_ST_TIMEOUT in the
// status block, raises a CTA-wide abort flag and all roles leave their loops,
// drain their copies and free TMEM.
#include "pdl.cuh"
#include "umma_common.cuh"

namespace spconvb {

using namespace umma_detail;

namespace {

constexpr int kTileRows = 256;  // most voxel rows per tile: the largest N of the MMA
constexpr int kEpiWarps = 8;
constexpr int kMmaWarp = 8;
constexpr int kProdWarp0 = 9;       // 9, 10, ... 24: four of them on every TMEM lane quadrant
constexpr int kWeightWarp = 25;
constexpr int kCtaThreads = 32 * 26;
constexpr uint32_t kTmemCols = 2 * kTileRows;
// 5 stages of 256 rows and 4 of weights: all a CTA can have.  No other block fits beside this one:
// 26 warps of 72 registers fill two of the SM's four register files.  With 64 registers and 12 KB
// less a rulebook block fits and the two do overlap, but the convolutions then take 3 % longer,
// which is what the overlap saves (batch of 8 frames 4.25 ms against 4.34).
constexpr uint32_t kRingBytes = 5 * kTileRows * kChunk + 4 * 128 * kChunk;
constexpr size_t kSmemBytes = kRingBytes + 1024 + 768;  // alignment slack, barriers

// ceil(2^32 / n): with it x / n = umulhi(x, .) for x < 2^29
__constant__ const uint32_t kReciprocal[9] = {0u,          0u,          0x80000000u,
                                              0x55555556u, 0x40000000u, 0x33333334u,
                                              0x2aaaaaabu, 0x24924925u, 0x20000000u};

// 32-bit instruction descriptor: [4,6) D format (1 = f32, 2 = s32), [7,10) A
// format, [10,13) B format (f16 kind: 0 = f16; i8 kind: 1 = signed), bits 15/16
// A/B major (0 = K), [17,23) N>>3, [24,29) M>>4.  M and N are added per launch.
template <bool INT8>
__device__ __forceinline__ constexpr uint32_t make_idesc() {
  return INT8 ? ((2u << 4) | (1u << 7) | (1u << 10)) : (1u << 4);
}

// Bytes or halves of 16 rows of one channel, `pitch` bytes apart; `n` rows exist.  The residual may be
// the output of the launch directly before, and neither its address nor the row count says so: both may
// be known before that launch is over.
template <bool I8>
__device__ __forceinline__ void load_rows16(const uint8_t* p, uint32_t pitch, uint32_t n,
                                            int32_t (&v)[16]) {
  if (n >= 16u) {
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i)
      v[i] = I8 ? load_in_order((const int8_t*)(p + i * pitch))
                : load_in_order((const uint16_t*)(p + i * pitch));
  } else {
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) {
      v[i] = 0;
      if (i < n)
        v[i] = I8 ? load_in_order((const int8_t*)(p + i * pitch))
                  : load_in_order((const uint16_t*)(p + i * pitch));
    }
  }
}

// ------------------------------------------------------------------- kernel
template <bool INT8, int RB, int COUT>
__global__ void __launch_bounds__(kCtaThreads, 1) conv_umma_kernel(const UmmaArgs a) {
  constexpr int OPC = RB <= kChunk ? kChunk / RB : 1;   // taps per chunk
  constexpr int SPO = RB <= kChunk ? RB / 16 : 8;       // 16-byte segments per tap per chunk
  constexpr int CPT = RB <= kChunk ? 1 : RB / kChunk;   // chunks per tap

  const int kbytes = a.kvol * RB;
  const int nchunk = (kbytes + kChunk - 1) / kChunk;
  const int last_ksteps = ((kbytes - (nchunk - 1) * kChunk) + 31) / 32;
  constexpr uint32_t kRep = 128 / COUT;            // copies of the weights along the accumulator rows
  constexpr uint32_t kWeightBytes = 128 * kChunk;  // one chunk of weights with its copies

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  uint64_t* bars = (uint64_t*)(smem + kRingBytes);
  uint32_t* tmem_holder = (uint32_t*)(bars + (kTileRows / 32 + 1) * kMaxStages + 4);
  volatile uint32_t* abort_flag = tmem_holder + 1;

  // "Stage empty", "accumulator full" and "empty", then "stage full" once for every tile height: how
  // many threads sign it depends on the height, and so on the row count.  All are made before that is
  // known.  (Made behind it, with their fences, they stood in the way of the first gather; one launch
  // after the other, waiting first, us: fp16 8 -> 16 of 28 000 rows 6.8 / 6.5, int8 16 -> 16 6.8 / 6.5.)
  const uint32_t bar_empty = smem_u32(bars);
  const uint32_t bar_tfull = bar_empty + 8 * kMaxStages;
  const uint32_t bar_tempty = bar_tfull + 16;
  const uint32_t bar_full0 = bar_tempty + 16;

  const int warp = threadIdx.x >> 5;
  const uint32_t lane = threadIdx.x & 31;
  // The row count, the first neighbour indices and the weights are fetched under the kernel before,
  // where that one has nothing to do with them; its results are waited for before the first gather
  // and the first drain.  (One launch after the other, all waiting here / waiting there, us: int8
  // 16 -> 16 of 14 000 rows 5.8 / 5.35, of 120 000 15.3 / 14.0; 128 -> 128 11.8 / 11.5, 41.5 / 40.7.)
  uint32_t n_out = 0;
  if (a.rules_ready) n_out = load_in_order(a.n_out_ptr);

  if (threadIdx.x < kTileRows / 32 * kMaxStages) {
    // a group of producers, as many warps as the tile has 32 rows, and the weights
    mbar_init(bar_full0 + 8 * threadIdx.x, 32u * (threadIdx.x / kMaxStages + 1u) + 1u);
    if (threadIdx.x < kMaxStages) mbar_init(bar_empty + 8 * threadIdx.x, 1);
    if (threadIdx.x < 2) {
      mbar_init(bar_tfull + 8 * threadIdx.x, 1);
      mbar_init(bar_tempty + 8 * threadIdx.x, kEpiWarps);
    }
    if (threadIdx.x == 0) *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  if (!a.rules_ready) {
    pdl_wait_and_trigger();
    n_out = load_in_order(a.n_out_ptr);
  }
  n_out = min(n_out, a.cap);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  // Tile height: the rows are dealt out in rounds over the CTAs, so a fixed 256-row tile
  // can leave most CTAs idle in the last round (227 tiles on 148 CTAs run as long as 296).
  // The height is instead the smallest multiple of 32 with which every CTA gets the same
  // number of tiles: per-CTA rows / rounds, rounded up.  Without integer divisions, which
  // would stand between the row count and the first index load of every launch; a quotient
  // that is off by one only makes another height.
  const uint32_t per_cta = max(1u, __umulhi(n_out + gridDim.x - 1, a.grid_inv));
  const uint32_t rounds = (per_cta + kTileRows - 1) / kTileRows;
  const uint32_t high =
      (uint32_t)(__fdividef((float)(per_cta + rounds - 1), (float)rounds) + 0.01f);
  const uint32_t tile_rows = min((uint32_t)kTileRows, (high + 31u) & ~31u);
  const uint32_t n32 = (n_out + 31u) >> 5, t32 = tile_rows >> 5;
  const uint32_t ntiles = t32 == 1u ? n32 : __umulhi(n32 + t32 - 1u, kReciprocal[t32]);
  // Two rings share the buffer: row stages as high as this launch's tile, and weight stages.
  // Low tiles get deeper rings: as many of both as fit, and what is left over goes to the rows.
  const uint32_t row_stage = tile_rows * kChunk;
  // Weights of which all chunks fit stay where they are after the first tile (a chunk in its own
  // stage): int8 16 -> 16, four chunks, 120 000 rows 16.1 / 14.9 us, with the copies above.  There are
  // never more weight stages than row stages: a chunk's weights are signed for on its row stage's
  // barrier as soon as their own stage is free, so a longer ring would sign a phase twice.
  const uint32_t fit = min((uint32_t)kMaxStages, kRingBytes / (kWeightBytes + row_stage));
  const bool resident = (uint32_t)nchunk <= fit;
  const uint32_t nwst = resident ? (uint32_t)nchunk : fit;
  const uint32_t nst = min((uint32_t)kMaxStages, (kRingBytes - nwst * kWeightBytes) / row_stage);
  const uint32_t sW = smem_u32(smem), sR = sW + nwst * kWeightBytes;
  // Only the producers that own rows of the tile take part, two groups of t32 warps.  (Warps that
  // only kept the barriers going cost low tiles a third of a chunk's time: fp16 128 -> 128 of 4 700
  // rows, 32 a tile, 18.2 to 15.0 us, int8 10.8 to 9.1.)
  const uint32_t bar_full = bar_full0 + 8 * kMaxStages * (t32 - 1u);

  const bool is_producer = warp > kMmaWarp && warp != kWeightWarp;
  // Who drains accumulators: the epilogue warps every tile of the CTA; the producers, which have
  // nothing left to gather by then, help with the last one.  It is the tail of every launch, and
  // on a small frame the only tile (128 channels, 224 rows: 6 200 cycles with 8 warps, with a
  // residual 15 000, beside 17 000 of MMAs).  A producer that is done knows that the MMAs are in
  // the last tile, or about to be, only if a tile has at least as many chunks as the ring.
  // With 16 channels a tile has 32 columns, a group of 16 for each of the epilogue's two sets of warps:
  // nothing to help with (fp16 16 -> 16 of 28 000 rows 7.6 us with the producers there, 7.2 without).
  const bool shared_tail = COUT > 16 && (uint32_t)nchunk >= nst;
  uint32_t drain_tile = blockIdx.x, drain_tl = 0;
  const uint32_t help_sets = t32 >> 1;  // sets of four warps, one a lane quadrant, among the producers
  bool drains = warp < kEpiWarps;
  if (warp == kWeightWarp) {
    // -------------------------------------------------------------- weights
    // One lane streams the chunks' pre-swizzled weight images, its ring may be shallower than
    // the rows': a weight stage is free when the chunk that used it last has been consumed.
    if (lane == 0) {
      uint32_t s = 0, ws = 0;    // row stage (whose barrier the copy signs), weight stage
      uint32_t os = 0, oph = 0;  // row stage and phase of the chunk `nwst` before
      uint32_t tile = blockIdx.x;
      int j = 0;
      auto fetch = [&]() {
        mbar_expect_tx(bar_full + 8 * s, kWeightBytes);
        // A bulk copy takes about 70 cycles of issue whatever its size (eight of 2 KB a chunk
        // instead of one of 16 KB: fp16 128 -> 128 of 4 700 rows 15.6 / 28.9 us), so the copies of
        // narrow weights are made in global memory where the caller can hold them: fp16 16 -> 16 of
        // 120 000 rows 20.4 / 19.2 us, 32 -> 32 29.7 / 26.7.
        const uint32_t dst = sW + ws * kWeightBytes;
        if (kRep > 1 && a.w_replicated) {
          bulk_g2s(dst, a.wpk + (size_t)j * kWeightBytes, kWeightBytes, bar_full + 8 * s);
        } else {
#pragma unroll
          for (uint32_t c = 0; c < kRep; ++c)
            bulk_g2s(dst + c * (COUT * kChunk), a.wpk + (size_t)j * (COUT * kChunk), COUT * kChunk,
                     bar_full + 8 * s);
        }
        if (++s == nst) s = 0;
        if (++ws == nwst) ws = 0;
        if (++j == nchunk) {
          j = 0;
          tile += gridDim.x;
        }
      };
#pragma unroll 1
      for (uint32_t n = 0; n < nwst && tile < ntiles; ++n) fetch();
      // No stage is freed before the rows are gathered, and the limit of a wait is for this launch,
      // not for what is left of the one before.
      pdl_wait();
      while (!resident && tile < ntiles) {
        // spinning: one lane, and every chunk waits for it (a launch of 4 736 rows 0.2 us less)
        if (!mbar_wait_spin(bar_empty + 8 * os, oph, abort_flag, a.status, 6u)) break;
        if (++os == nst) {
          os = 0;
          oph ^= 1u;
        }
        fetch();
      }
    }
    __syncwarp();
  } else if (is_producer) {
    // ------------------------------------------------------------ producers
    // Two groups of t32 warps take the chunks in turn (group g the chunks g, g + 2, ...), so a
    // warp has two chunk periods for the round trip of one chunk: wait for the stage, look
    // up the neighbours, issue the copies.  Within a group, warp w owns rows 32w..32w+31 of
    // the tile.  A chunk of the row tile is 256 rows x 8 segments of 16 bytes = 2048 copies,
    // 8 per thread: a thread copies segment `seg` of rows 32w + 8 slot + i, i = 0..7 (8
    // lanes per row, so the lanes that read the same neighbour row ask for one contiguous
    // piece of it).  Missing neighbours are zero-filled copies, so the 8 items are
    // branch-free and their address arithmetic and copies overlap.
    const uint32_t pw_all = (uint32_t)(warp - kProdWarp0);
    const uint32_t grp = pw_all >= t32 ? 1u : 0u, pw = grp ? pw_all - t32 : pw_all;
    const uint32_t seg = lane & 7u;        // 16-byte segment of the chunk this thread copies
    const uint32_t slot = lane >> 3;       // its 8 rows of the warp's 32
    // row R of the tile lives at (R / 8) * 1024 + (R % 8) * 128, its segments XOR-ed
    // with R % 8; here R / 8 = 4 pw + slot and R % 8 = i
    const uint32_t dst_base = (pw * 4u + slot) * 1024u;
    // tap (within the chunk) and byte offset (within the neighbour row) of `seg`
    const uint32_t seg_tap = RB <= kChunk ? seg / SPO : 0u;
    const uint32_t seg_byte = RB <= kChunk ? (seg % SPO) * 16u : seg * 16u;
    const uint32_t row_in_tile = pw * 32u + slot * 8u;
    // 16-byte index loads need the map rows 16-byte aligned and whole groups of 8 inside them
    const bool vec_ok = (a.cap & 7u) == 0u && ((uintptr_t)a.map & 15u) == 0u;

    // The 8 neighbour indices this thread needs for chunk j of a tile: its tap's map entries
    // of its 8 rows, straight from global memory into registers (two 16-byte loads; the 8
    // lanes of a row group that share a tap read the same 32 bytes).  Rows past the end,
    // taps past the kernel and tiles past the last give -1.
    auto load_idx = [&](uint32_t tile, int j, int32_t (&v)[8]) {
      const int k = RB <= kChunk ? j * OPC + (int)seg_tap : j / CPT;
      const uint32_t row = tile * tile_rows + row_in_tile;
      const bool live = tile < ntiles && k < a.kvol && row < n_out;
      const int32_t* src = a.map + (size_t)k * a.cap + row;
      if (live && vec_ok && row + 8u <= n_out) {
        const int4 lo = __ldg((const int4*)src), hi = __ldg((const int4*)src + 1);
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
        v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
      } else {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) v[i] = (live && row + i < n_out) ? __ldg(src + i) : -1;
      }
    };
    // This group's chunks: numbers it = grp, grp + 2, ... of the CTA's chunk sequence (tile
    // after tile, nchunk chunks each); chunk `it` uses stage it % nst.
    auto advance2 = [&](uint32_t& tile, int& j) {  // two chunks on
      j += 2;
      while (j >= nchunk) {
        j -= nchunk;
        tile += gridDim.x;
      }
    };
    uint32_t tile = pw < t32 ? blockIdx.x : ntiles;  // a warp without rows has no chunks
    int j = grp == 1u ? 1 : 0;
    while (j >= nchunk) {
      j -= nchunk;
      tile += gridDim.x;
    }
    uint32_t tiles_done = 0;  // (of use where no step passes a tile: nchunk > 1)
    uint32_t ntile = tile;  // the chunk whose indices are loaded next
    int nj = j;
    uint32_t it = grp, s = grp % nst, ph = (grp / nst) & 1u;
    const uint32_t first_thread = 32u * (kProdWarp0 + grp * t32);  // of this group
    // One chunk: its rows go from the indices in `idx` into the stage, and `idx` is then
    // refilled for the chunk after next.  Two register sets take turns and are never copied,
    // so the load has a whole chunk of the group's time to arrive.
    auto step = [&](int32_t (&idx)[8]) -> bool {
      if (tile >= ntiles) return false;
      // every lane polls: one shared-memory word, no divergence, no broadcast afterwards
      if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, a.status, 1u)) return false;
      // segments of the last chunk that lie in K steps past the kernel's last tap are never
      // read by an MMA: nothing to copy, nothing to zero
      const bool dead_seg = j == nchunk - 1 && (int)(seg >> 1) >= last_ksteps;
      if (!dead_seg) {
        const uint8_t* src = a.in + seg_byte + (RB > kChunk ? (uint32_t)(j % CPT) * kChunk : 0u);
        const uint32_t stage_addr = sR + s * row_stage + dst_base;
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
          const int32_t sr = idx[i];
          cp_async16(stage_addr + i * 128u + ((seg ^ i) << 4),
                     src + (int64_t)sr * RB, sr < 0 ? 0u : 16u);
        }
      }
      if (!(a.wait_test > 0 && it + 1u >= (uint32_t)a.wait_test))
        cp_async_arrive_noinc(bar_full + 8 * s);
      // the weights' arrival, where they are there already
      if (resident && tile != blockIdx.x && threadIdx.x == first_thread) mbar_arrive(bar_full + 8 * s);
      load_idx(ntile, nj, idx);
      advance2(ntile, nj);
      const uint32_t was = tile;
      advance2(tile, j);
      if (tile != was) ++tiles_done;
      it += 2;
      s += 2;
      if (s >= nst) {
        s -= nst;
        ph ^= 1u;
      }
      return true;
    };
    int32_t idx_a[8], idx_b[8];
    load_idx(ntile, nj, idx_a);
    advance2(ntile, nj);
    load_idx(ntile, nj, idx_b);
    advance2(ntile, nj);
    pdl_wait_and_trigger();
    while (step(idx_a) && step(idx_b)) {
    }
    cp_async_wait_all();  // nothing of this thread may still be writing when the CTA exits
    __syncwarp();
    // As one warp: where a launch gives up, some lanes may have left at a stage that came too late for
    // them and others not, and the drain exchanges between all 32.
    if (__all_sync(0xffffffffu, shared_tail && (pw_all >> 2) < help_sets && tile >= ntiles &&
                                    tiles_done > 0u)) {
      drains = true;
      drain_tile = tile - gridDim.x;
      drain_tl = tiles_done - 1u;
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issue
    // The whole warp walks the chunks and one elected lane issues, by predicate: the loop's values stay
    // warp-uniform, so an MMA costs its own time (measured in isolation, M = 128, N = 256: 513
    // cycles per chunk against 583 when a single lane runs the loop, whose descriptors are moved
    // to uniform registers one MMA after the other).
    //
    // MMAs are queued: what a chunk costs here is the issue of its instructions, and with up to 24 other
    // warps around every one takes tens of cycles.  So the loop carries addresses and nothing
    // else, and a chunk is four MMAs, a commit and one test of the next stage's barrier.
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc<INT8>() | ((tile_rows >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t wdesc0 = make_smem_desc(sW);  // M operand: weights
    const uint64_t rdesc0 = make_smem_desc(sR);  // N operand: gathered rows
    // 32-bit arithmetic only: the descriptors differ in their low word (the address)
    const uint32_t desc_hi = (uint32_t)(wdesc0 >> 32);
    const uint32_t w_step = kWeightBytes >> 4, r_step = row_stage >> 4;
    const uint32_t w_lo0 = (uint32_t)wdesc0, r_lo0 = (uint32_t)rdesc0;
    const uint32_t w_end = w_lo0 + nwst * w_step, bar_end = bar_full + 8 * nst;
    const uint32_t to_empty = bar_empty - bar_full;  // from a stage's full barrier to its empty one
    uint32_t bar = bar_full, rd = r_lo0, wd = w_lo0, ph = 0, tl = 0;
    auto next_stage = [&]() {
      bar += 8;
      rd += r_step;
      if (bar == bar_end) {
        bar = bar_full;
        rd = r_lo0;
        ph ^= 1u;
      }
      wd += w_step;
      if (wd == w_end) wd = w_lo0;
    };
    // A lane that gives up walks on without waiting, and the issuing one without issuing: the lanes
    // never part, so none asks about a stage a whole ring behind another (whose phase it would take
    // for the one after), and none waits at a warp barrier for one that has left.
    bool alive = true;
    auto stage_full = [&]() {
      alive = alive && (mbar_test_wait(bar, ph) || mbar_wait_spin(bar, ph, abort_flag, a.status, 3u));
      __syncwarp();  // (a wait that runs out may part them)
    };
    pdl_wait();  // no stage fills before; the limit of a wait is for this launch, as above
    // The loop is entered with the current chunk's stage known to be full.
    if (blockIdx.x < ntiles) stage_full();
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++tl) {
      const uint32_t buf = tl & 1u;
      alive = alive && mbar_wait_spin(bar_tempty + 8 * buf, ((tl >> 1) & 1u) ^ 1u, abort_flag, a.status, 2u);
      tc_fence_after();  // the epilogue's reads of this accumulator come before these MMAs
      const uint32_t d_tmem = tmem_base + buf * kTileRows;
      // The rows of a stage are written by cp.async, through the generic proxy, and read by the MMAs
      // through the async proxy: the stage's mbarrier orders the threads, the fence the proxies.  (It
      // costs nothing that shows: 120 000 voxels 638.7 us without, 638.8 with it.)
      uint32_t accumulate = 0u;
#pragma unroll 1
      for (int j = nchunk - 1; j > 0; --j) {
        const uint32_t issue = leader && alive ? 1u : 0u;
        fence_proxy_async();
        umma_if<INT8>(issue, d_tmem, wd, rd, desc_hi, idesc, accumulate);
        umma_if<INT8>(issue, d_tmem, wd + 2u, rd + 2u, desc_hi, idesc, 1u);
        umma_if<INT8>(issue, d_tmem, wd + 4u, rd + 4u, desc_hi, idesc, 1u);
        umma_if<INT8>(issue, d_tmem, wd + 6u, rd + 6u, desc_hi, idesc, 1u);
        tc_commit_if(issue, bar + to_empty);
        accumulate = 1u;
        next_stage();
        stage_full();
      }
      const uint32_t issue = leader && alive ? 1u : 0u;
      fence_proxy_async();
      for (int ks = 0; ks < last_ksteps; ++ks) {
        umma_if<INT8>(issue, d_tmem, wd + 2u * ks, rd + 2u * ks, desc_hi, idesc, accumulate);
        accumulate = 1u;
      }
      tc_commit_if(issue, bar + to_empty);
      tc_commit_if(issue, bar_tfull + 8 * buf);
      next_stage();
      if (tile + gridDim.x < ntiles) stage_full();
    }
    __syncwarp();
  }
  if (drains) {
    // ------------------------------------------------------------- epilogue
    // Same arithmetic as common.cuh:epilogue_value, written so that the per-element
    // work is a handful of instructions: ReLU as a max with 0 or -inf, float -> int8
    // as one saturating round-to-nearest-even convert, and the layer-wide switches
    // hoisted out of the element loops.
    const Epilogue ep = a.ep;
    pdl_wait();  // residual rows are read, and rows written that the kernel before may still read
    // Accumulator row m (TMEM lane m) holds channel m % COUT of weight copy m / COUT.  Copy c
    // owns cols_rep rows of the tile from c * cols_rep on, and the warps of a lane quadrant take
    // its groups of 16 rows in turn: two warps, and where the producers help with the last tile one more
    // for every 64 rows of its height (2 to 6).
    const uint32_t q = (uint32_t)warp & 3u;        // TMEM lane quadrant of this warp
    const uint32_t part = is_producer ? 2u + (((uint32_t)warp - kProdWarp0) >> 2) : (uint32_t)warp >> 2;
    const uint32_t acc_row = 32u * q + lane, acc_row0 = 32u * q;
    const uint32_t ch = acc_row % COUT;            // this lane's channel
    const uint32_t cols_rep = (tile_rows + 32u * kRep - 1u) / (32u * kRep) * 32u;
    // first row (of the tile) of this lane's copy, and of lane 0's: they differ only for COUT = 16,
    // where the two halves of a warp belong to different copies
    constexpr bool split_warp = COUT == 16;
    const uint32_t copy_lane = (acc_row / COUT) * cols_rep, copy_warp = (acc_row0 / COUT) * cols_rep;
    // columns of lane 0's copy that lie inside the tile
    const uint32_t cols = copy_warp < tile_rows ? min(cols_rep, tile_rows - copy_warp) : 0u;
    const float sc = (INT8 && a.scale) ? __ldg(a.scale + ch) : 1.f;
    const float bi = a.bias ? __ldg(a.bias + ch) : 0.f;
    const float lo = ep.act == SPCONVB_ACT_RELU ? 0.f : -INFINITY;
    const float lo2 = ep.res_relu ? 0.f : -INFINITY;
    const bool res_i8 = ep.res_kind == SPCONVB_I8;
    // A lane owns a channel, so a group of 16 rows is 16 loads or stores of one element each, at
    // constant distances; the 32 lanes of a warp cover a contiguous piece of every row.
    constexpr uint32_t kRow8 = COUT, kRow16 = 2 * COUT;  // bytes of an int8 / fp16 row
    auto load_res = [&](uint32_t row, uint32_t n, int32_t (&r)[16]) {
      if (res_i8) load_rows16<true>(a.res + (size_t)row * kRow8 + ch, kRow8, n, r);
      else load_rows16<false>(a.res + (size_t)row * kRow16 + 2u * ch, kRow16, n, r);
    };
    // rows of this lane's group of 16 that exist: a group lies inside the tile or not as a whole
    // (the tile height is a multiple of 32); rows past the tile belong to the next one
    auto rows_of = [&](uint32_t row, uint32_t col) -> uint32_t {
      return col < tile_rows && row < n_out ? min(16u, n_out - row) : 0u;
    };
    uint32_t tl = drain_tl;
    for (uint32_t tile = drain_tile; tile < ntiles; tile += gridDim.x, ++tl) {
      const uint32_t buf = tl & 1u;
      const uint32_t step = shared_tail && tile + gridDim.x >= ntiles ? (2u + help_sets) * 16u : 2u * 16u;
      const uint32_t trow0 = tile * tile_rows;
      uint32_t col = 16u * part;  // of the copy
      // the first residual rows are fetched before the accumulator is waited for; after that
      // the loads run one group of 16 rows ahead of the arithmetic
      int32_t rnext[16];
      if (ep.has_res && col < cols)
        load_res(trow0 + copy_lane + col, rows_of(trow0 + copy_lane + col, copy_lane + col), rnext);
      uint32_t ok = 1u;
      if (lane == 0) {
        ok = mbar_wait(bar_tfull + 8 * buf, (tl >> 1) & 1u, abort_flag, a.status, 4u) ? 1u : 0u;
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((32u * q) << 16) + buf * kTileRows + copy_warp;
      auto release = [&]() {  // no more reads of this accumulator by this warp
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && !is_producer) mbar_arrive(bar_tempty + 8 * buf);
      };
      if (col >= cols) release();
#pragma unroll 1
      for (; col < cols; col += step) {
        const uint32_t row0 = trow0 + copy_lane + col;
        const uint32_t rows = rows_of(row0, copy_lane + col);
        uint32_t v[16];
        tmem_ld16(taddr + col, v);
        if (split_warp) {
          // the upper half of the warp belongs to the next copy: its rows are one copy's
          // worth of columns further on
          uint32_t vm[16];
          tmem_ld16(taddr + cols_rep + col, vm);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = lane >= 16u ? vm[i] : v[i];
        } else {
          tmem_ld_wait();
        }
        if (col + step >= cols) release();
        float y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (INT8) y[i] = fmaxf(fmaf((float)(int)v[i], sc, bi), lo);
          else y[i] = fmaxf(__fadd_rn(__uint_as_float(v[i]), bi), lo);
        }
        if (ep.has_res) {
          // the conv result as it would have been stored (mid), plus the residual
          if (ep.mid_kind == SPCONVB_I8) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              y[i] = __fmul_rn((float)cvt_sat_s8(__fmul_rn(y[i], ep.mid_inv_scale)), ep.mid_scale);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) y[i] = __half2float(__float2half_rn(y[i]));
          }
          if (res_i8) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              y[i] = fmaxf(__fadd_rn(y[i], __fmul_rn((float)rnext[i], ep.res_scale)), lo2);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              y[i] = fmaxf(__fadd_rn(y[i], __half2float(__ushort_as_half((uint16_t)rnext[i]))), lo2);
          }
          if (col + step < cols)
            load_res(row0 + step, rows_of(row0 + step, copy_lane + col + step), rnext);
        }
        if (ep.out_kind == SPCONVB_I8) {
          int8_t* o = (int8_t*)a.out + (size_t)row0 * kRow8 + ch;
          if (rows == 16u) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              o[i * kRow8] = (int8_t)cvt_sat_s8(__fmul_rn(y[i], ep.inv_out_scale));
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (i < (int)rows) o[i * kRow8] = (int8_t)cvt_sat_s8(__fmul_rn(y[i], ep.inv_out_scale));
          }
        } else {
          __half* o = (__half*)a.out + (size_t)row0 * COUT + ch;
          if (rows == 16u) {
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i * COUT] = __float2half_rn(y[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (i < (int)rows) o[i * COUT] = __float2half_rn(y[i]);
          }
        }
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies already issued a bounded time to land before the CTA exits
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 50000ull) {
    }
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
}

template <bool INT8, int RB, int COUT>
int launch_one(const UmmaArgs& args, uint32_t launch_rows, cudaStream_t st) {
  static bool attr_done[64] = {};
  int dev = 0;
  SPCONVB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !attr_done[dev]) {
    SPCONVB_CUDA_TRY(cudaFuncSetAttribute(conv_umma_kernel<INT8, RB, COUT>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kSmemBytes));
    if (dev >= 0 && dev < 64) attr_done[dev] = true;
  }
  uint32_t tiles = (launch_rows + 31) / 32;  // the kernel picks the tile height per launch
  const int grid = (int)(tiles < (uint32_t)kSmCount ? (tiles ? tiles : 1u) : (uint32_t)kSmCount);
  UmmaArgs with_grid = args;
  with_grid.grid_inv = grid > 1 ? 0xffffffffu / (uint32_t)grid + 1u : 0xffffffffu;
  SPCONVB_CUDA_TRY(launch_pdl(conv_umma_kernel<INT8, RB, COUT>, dim3(grid), dim3(kCtaThreads),
                              kSmemBytes, st, with_grid));
  return SPCONVB_OK;
}

template <bool INT8, int RB>
int launch_cout(int cout, const UmmaArgs& args, uint32_t launch_rows, cudaStream_t st) {
  switch (cout) {
    case 16: return launch_one<INT8, RB, 16>(args, launch_rows, st);
    case 32: return launch_one<INT8, RB, 32>(args, launch_rows, st);
    case 64: return launch_one<INT8, RB, 64>(args, launch_rows, st);
    case 128: return launch_one<INT8, RB, 128>(args, launch_rows, st);
  }
  return SPCONVB_E_UNSUPPORTED;
}

template <bool INT8>
int launch_rb(int rb, int cout, const UmmaArgs& args, uint32_t launch_rows, cudaStream_t st) {
  switch (rb) {
    case 16: return launch_cout<INT8, 16>(cout, args, launch_rows, st);
    case 32: return launch_cout<INT8, 32>(cout, args, launch_rows, st);
    case 64: return launch_cout<INT8, 64>(cout, args, launch_rows, st);
    case 128: return launch_cout<INT8, 128>(cout, args, launch_rows, st);
    case 256: return launch_cout<INT8, 256>(cout, args, launch_rows, st);
  }
  return SPCONVB_E_UNSUPPORTED;
}

}  // namespace

int conv_umma_kernel_launch(const UmmaArgs& a, bool int8, int rb, int cout, uint32_t launch_rows,
                            cudaStream_t st) {
  return int8 ? launch_rb<true>(rb, cout, a, launch_rows, st)
              : launch_rb<false>(rb, cout, a, launch_rows, st);
}

}  // namespace spconvb
