// Rulebook work as tasks: what the kernel-level entry points (rulebook.cu) and the engine
// (engine.cpp) put together into launches.  Tasks that do not depend on one another go into one
// wave, which is one kernel launch whose blocks are dealt out to its tasks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "grid3.hpp"

namespace spconvb {

struct Kernel3 {
  int32_t k[3];
  int32_t s[3];
  int32_t p[3];
  int32_t d[3];
  int32_t sh[3];  // log2 of the stride when it is a power of two (1, 2, 4, ...), else -1
};

// Workspace of a strided rulebook (32-bit words):
//   [0, W)        bitmap over the output grid                     (zero before the mark task)
//   [W, 2W)       rank of the word's first set bit (after the emit task)
//   [2W, ...)     state of the emit task's scan                    (zero before the emit task):
//                 totals of groups of 16 scan blocks of 128 words (64 bits each, from the next
//                 8-byte boundary on: the workspace may start at any word), a counter of the blocks
//                 started
constexpr uint32_t kScanGroup = 16;
struct DownWs {
  uint32_t* bitmap;
  uint32_t* prefix;
  uint32_t* scan;
  uint32_t words;
  uint32_t blocks;
#ifdef __CUDACC__
  __device__ unsigned long long* scan_groups() const { return (unsigned long long*)scan; }
  __device__ uint32_t* scan_ticket() const {
    return scan + 2 * ((blocks + kScanGroup - 1) / kScanGroup);
  }
#endif
};
inline size_t scan_state_words(uint32_t blocks) {
  return 2 * (size_t)((blocks + kScanGroup - 1) / kScanGroup) + 1;
}

enum RuleTaskKind : int32_t {
  TASK_COUNT,        // the caller's row count, clamped, into the engine's word
  TASK_PAD8,         // fp16 rows of <= 8 channels into 16-byte rows
  TASK_HASH,         // rows into the hash table
  TASK_SUBM_HASH,    // SubM map of the caller's rows
  TASK_SUBM_RANK,    // SubM map of rows a strided rulebook made
  TASK_MARK_ROWS,    // output bitmap of a strided rulebook from the input rows
  TASK_MARK_BITMAP,  // the same from the bitmap of input rows a strided rulebook made
  TASK_EMIT,         // ranks, output coordinates and count from the bitmap
  TASK_SCATTER,      // strided map from the input side (over entries the emit task set to -1)
  TASK_GATHER,       // strided map from the output side, input rows made by a strided rulebook
  TASK_INVERSE,      // map of an inverse convolution
};

struct RuleTask {
  int32_t kind = 0;
  uint32_t blocks = 1;
  // rows the task walks: n = min(n_ptr ? *n_ptr : n_host, cap)
  const int4* coords = nullptr;
  const uint32_t* n_ptr = nullptr;
  uint32_t n_host = 0;
  uint32_t cap = 0;
  Grid3 gin{}, gout{};
  Kernel3 kr{};
  DownWs ws{}, in_ws{};
  int32_t* map = nullptr;      // EMIT: set to -1 for the rows it emits when not null
  uint32_t map_cap = 0;        // row stride of map where it is not `cap`
  uint32_t other_cap = 0;      // rows the other side of the map may hold
  uint64_t* table = nullptr;
  uint32_t mask = 0;
  int4* out_coords = nullptr;
  uint32_t* n_out = nullptr;   // EMIT, COUNT
  uint32_t* status = nullptr;
  const void* feat = nullptr;  // PAD8
  uint4* feat_out = nullptr;
  int32_t channels = 0;
};

constexpr int kMaxWaveTasks = 8;
struct RuleWave {
  RuleTask t[kMaxWaveTasks];
  int32_t count = 0;
  void add(const RuleTask& x) { t[count++] = x; }
  bool full() const { return count == kMaxWaveTasks; }
};

#ifdef __CUDACC__
// Row of a cell from the bitmap and its ranks, -1 if the cell is empty or lies beyond the
// capacity.
__device__ __forceinline__ int32_t rank_lookup(const uint32_t* __restrict__ bitmap,
                                               const uint32_t* __restrict__ prefix,
                                               uint32_t cell, uint32_t cap) {
  const uint32_t bits = __ldg(bitmap + (cell >> 5));
  const uint32_t b = cell & 31u;
  if (!((bits >> b) & 1u)) return -1;
  const uint32_t row = __ldg(prefix + (cell >> 5)) + __popc(bits & ((1u << b) - 1u));
  return row < cap ? (int32_t)row : -1;
}
#endif

// One launch for the wave's tasks; an empty wave launches nothing.
int launch_rule_wave(const RuleWave& w, cudaStream_t st);

// What a rulebook is refused for, by the kernel-level entry points and by the engine alike (its
// waves are made of tasks, which check nothing).  A cell's number has to fit 32 bits: in a larger
// grid different cells would share one.
bool grid_fits(const int32_t g[3], int batch);
int check_hash(const int32_t grid[3], int batch, uint32_t cap, uint32_t slots);
int check_subm(const int32_t grid[3], int batch, const int32_t k[3], const int32_t d[3]);
// and the output grid
int check_strided(const int32_t grid[3], int batch, const int32_t k[3], const int32_t s[3],
                  const int32_t p[3], const int32_t d[3], int32_t out_grid[3]);

// Task makers: arguments already checked.
DownWs down_ws(const int32_t out_grid[3], int batch, const void* workspace);
Grid3 make_grid(const int32_t g[3], int batch);
Kernel3 make_kernel3(const int32_t k[3], const int32_t s[3], const int32_t p[3], const int32_t d[3]);
bool mark_from_bitmap(const Kernel3& kr);  // the bitmap-to-bitmap mark covers this geometry
uint32_t task_blocks(unsigned long long items);
uint32_t row_task_blocks(int32_t kind, unsigned long long rows);
uint32_t mark_bitmap_blocks(const int32_t out_grid[3], int batch);

}  // namespace spconvb
