// Point cloud -> voxels (mean of the first P points of every voxel), with a
// result that does not depend on thread scheduling:
//   * a voxel's first point is the smallest point index that reached its hash slot; the
//     up to P - 1 kept points after it are found with a cascade of atomicMin over slots (slot
//     s ends up holding the (s+2)-th smallest index), and all are summed in ascending order;
//   * voxel ids are the ranks of the voxels' first points, from a two-level
//     exclusive scan over the points.
// This is what the reference's three kernels compute when points are processed
// one after another; run in parallel they return an arbitrary voxel order and,
// for crowded voxels, an arbitrary subset of points.
//
// A sweep is a few megabytes: what it costs is launches and dependent L2 accesses.  One clear and
// three kernels; a slot holds key and first point in one word, so that most voxels (nine of ten
// hold one point) take one compare-and-swap and nothing else.  271 156 fp16 points: 40 us of kernels
// with a counter of voxels that every first point drew from, a separate array of ids and a
// cascade for every point.
#include "common.cuh"
#include "pdl.cuh"

namespace spconvb {

constexpr int kVoxThreads = 256;
constexpr int kVoxScanThreads = 512;
constexpr uint32_t kNoPoint = 0xffffffffu;

struct VoxWs {
  unsigned long long* table;  // [slots]   (key + 1) << 32 | first point, 0 = empty  (zeroed per call)
  uint32_t* block_sums;       // [blocks]  voxels that begin in each scan block
  uint32_t* pslot;            // [points]  slot of a point, kNoPoint if outside
  uint32_t* pprefix;          // [points]  rank of a first point inside its scan block, else kNoPoint
  uint32_t* kept;             // [points][P - 1]  at a voxel's first point: the next smallest ones
  uint32_t slots;
  uint32_t blocks;
};

__host__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

__host__ inline uint32_t vox_slots(uint32_t max_points) {
  uint32_t s = 1024;
  while (s < 2u * max_points && s < 0x80000000u) s <<= 1;
  return s;
}

__host__ inline VoxWs vox_layout(void* base, const spconvb_voxel_params& p, uint32_t max_points,
                                 size_t* zero_bytes, size_t* total_bytes) {
  VoxWs w;
  w.slots = vox_slots(max_points);
  w.blocks = (max_points + kVoxScanThreads - 1) / kVoxScanThreads;
  if (w.blocks < 1) w.blocks = 1;
  uint8_t* b = (uint8_t*)base;
  // the table's 64-bit slots start at the next 8-byte boundary: the workspace may start at any word
  size_t off = (8u - ((uintptr_t)base & 7u)) & 7u;
  w.table = (unsigned long long*)(b + off); off += align_up(sizeof(uint64_t) * (size_t)w.slots, 256);
  if (zero_bytes) *zero_bytes = off;
  w.block_sums = (uint32_t*)(b + off); off += align_up(sizeof(uint32_t) * (size_t)w.blocks, 256);
  w.pslot = (uint32_t*)(b + off); off += align_up(sizeof(uint32_t) * (size_t)max_points, 256);
  w.pprefix = (uint32_t*)(b + off); off += align_up(sizeof(uint32_t) * (size_t)max_points, 256);
  w.kept = (uint32_t*)(b + off);
  off += align_up(sizeof(uint32_t) * (size_t)max_points * (p.max_points_per_voxel - 1), 256);
  if (total_bytes) *total_bytes = off + 256;  // (room for that)
  return w;
}

__device__ __forceinline__ float point_feat(const void* points, int kind, size_t i) {
  return kind ? __half2float(((const __half*)points)[i]) : ((const float*)points)[i];
}

__device__ __forceinline__ int3 voxel_of(float px, float py, float pz,
                                         const spconvb_voxel_params& p) {
  return make_int3((int)floorf(__fdiv_rn(__fsub_rn(px, p.range_min[0]), p.voxel_size[0])),
                   (int)floorf(__fdiv_rn(__fsub_rn(py, p.range_min[1]), p.voxel_size[1])),
                   (int)floorf(__fdiv_rn(__fsub_rn(pz, p.range_min[2]), p.voxel_size[2])));
}

// Pass 1: every in-range point goes to its voxel's slot, which keeps the smallest index.
__global__ void __launch_bounds__(kVoxThreads)
vox_hash_kernel(const void* __restrict__ points, uint32_t n, spconvb_voxel_params p, VoxWs w,
                uint32_t* status) {
  const uint32_t i = blockIdx.x * kVoxThreads + threadIdx.x;
  float px = 0.f, py = 0.f, pz = 0.f;
  if (i < n) {
    px = point_feat(points, p.points_kind, (size_t)i * p.num_features);
    py = point_feat(points, p.points_kind, (size_t)i * p.num_features + 1);
    pz = point_feat(points, p.points_kind, (size_t)i * p.num_features + 2);
  }
  // the block's share of `kept`, while the points are on their way
  {
    const uint32_t per = (uint32_t)p.max_points_per_voxel - 1u;
    const size_t first = (size_t)blockIdx.x * kVoxThreads * per;
    const uint32_t words = min((uint32_t)kVoxThreads, n - blockIdx.x * kVoxThreads) * per;
    for (uint32_t k = threadIdx.x; k < words; k += kVoxThreads) w.kept[first + k] = kNoPoint;
  }
  if (i >= n) return;
  uint32_t slot = kNoPoint;
  if (px >= p.range_min[0] && px < p.range_max[0] && py >= p.range_min[1] &&
      py < p.range_max[1] && pz >= p.range_min[2] && pz < p.range_max[2]) {
    const int3 v = voxel_of(px, py, pz, p);
    if (v.x >= 0 && v.x < p.grid[0] && v.y >= 0 && v.y < p.grid[1] && v.z >= 0 && v.z < p.grid[2]) {
      const uint32_t key = ((uint32_t)v.z * p.grid[1] + v.y) * p.grid[0] + v.x;
      const unsigned long long entry = ((unsigned long long)(key + 1u) << 32) | i;
      const uint32_t mask = w.slots - 1;
      uint32_t s = hash32(key) & mask;
      for (uint32_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long old = atomicCAS(w.table + s, 0ull, entry);
        if (old == 0ull || (uint32_t)(old >> 32) == key + 1u) {
          if (old > entry) atomicMin(w.table + s, entry);
          slot = s;
          break;
        }
        s = (s + 1) & mask;
      }
      if (slot == kNoPoint) set_status(status, SPCONVB_ST_HASH_FULL, i);
    }
  }
  w.pslot[i] = slot;
}

// Pass 2: ranks the first points (exclusive scan inside a block of points); the others look for
// a place among the P - 1 smallest after the first.
__global__ void __launch_bounds__(kVoxScanThreads) vox_scan_kernel(uint32_t n, int per, VoxWs w) {
  __shared__ uint32_t warp_sums[kVoxScanThreads / 32];
  pdl_wait();
  const uint32_t i = blockIdx.x * kVoxScanThreads + threadIdx.x;
  uint32_t flag = 0, first = 0;
  bool later = false;
  if (i < n) {
    const uint32_t slot = w.pslot[i];
    if (slot != kNoPoint) {
      first = (uint32_t)w.table[slot];
      flag = first == i ? 1u : 0u;
      later = !flag && per > 0;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t ballot = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) warp_sums[warp] = __popc(ballot);
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int k = 0; k < kVoxScanThreads / 32; ++k) {
    if (k < warp) before += warp_sums[k];
    total += warp_sums[k];
  }
  if (threadIdx.x == 0) w.block_sums[blockIdx.x] = total;
  if (i < n)
    w.pprefix[i] = flag ? before + __popc(ballot & ((1u << lane) - 1u)) : kNoPoint;
  if (later) {
    uint32_t* k = w.kept + (size_t)first * per;
    uint32_t v = i;
    // what a full row keeps only gets smaller: most points of a crowded voxel end here
    if (*(volatile uint32_t*)(k + per - 1) < v) return;
    for (int s = 0; s < per; ++s) {
      const uint32_t old = atomicMin(k + s, v);
      v = max(old, v);
      if (v == kNoPoint) break;
    }
  }
}

// Pass 3: the first point of a voxel writes the voxel: its index and the mean of the kept points,
// summed in ascending point order in fp32.  With `clear_tail` the rows after the last voxel become
// zero.
__global__ void __launch_bounds__(kVoxScanThreads)
vox_emit_kernel(const void* __restrict__ points, uint32_t n, spconvb_voxel_params p, VoxWs w,
                __half* __restrict__ features, int4* __restrict__ indices,
                uint32_t* n_voxels_ptr, uint32_t* status, int clear_tail) {
  __shared__ uint32_t red[2][kVoxScanThreads / 32];
  pdl_wait();
  const uint32_t i = blockIdx.x * kVoxScanThreads + threadIdx.x;
  const uint32_t pre = i < n ? w.pprefix[i] : kNoPoint;
  const int F = p.num_features, per = p.max_points_per_voxel - 1;
  const uint32_t next = pre != kNoPoint && per > 0 ? w.kept[(size_t)i * per] : kNoPoint;
  float sum[8];
#pragma unroll
  for (int f = 0; f < 8; ++f)
    sum[f] = f < F && pre != kNoPoint ? point_feat(points, p.points_kind, (size_t)i * F + f) : 0.f;
  uint32_t part = 0, all = 0;
  for (uint32_t b = threadIdx.x; b < w.blocks; b += kVoxScanThreads) {
    const uint32_t v = w.block_sums[b];
    all += v;
    if (b < blockIdx.x) part += v;
  }
  part = __reduce_add_sync(0xffffffffu, part);
  all = __reduce_add_sync(0xffffffffu, all);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = part;
    red[1][threadIdx.x >> 5] = all;
  }
  __syncthreads();
  uint32_t base = 0, total = 0;
#pragma unroll
  for (int k = 0; k < kVoxScanThreads / 32; ++k) {
    base += red[0][k];
    total += red[1][k];
  }
  const uint32_t most = (uint32_t)p.max_voxels, count = min(total, most);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (total > most) set_status(status, SPCONVB_ST_OVERFLOW, total);
    *n_voxels_ptr = count;
  }
  if (clear_tail) {
    const size_t from = (size_t)count * F, to = (size_t)most * F;
    for (size_t k = from + i; k < to; k += (size_t)gridDim.x * kVoxScanThreads)
      features[k] = __ushort_as_half(0);
    for (size_t k = count + (size_t)i; k < most; k += (size_t)gridDim.x * kVoxScanThreads)
      indices[k] = make_int4(0, 0, 0, 0);
  }
  if (pre == kNoPoint || base + pre >= most) return;
  const uint32_t id = base + pre;
  const int3 v = voxel_of(sum[0], sum[1], sum[2], p);
  int cnt = 1;
#pragma unroll
  for (int f = 0; f < 8; ++f) sum[f] = __fadd_rn(0.f, sum[f]);  // sums start at 0: a lone -0 gives +0
  if (next != kNoPoint) {
    const uint32_t* k = w.kept + (size_t)i * per;
    for (int s = 0; s < per; ++s) {
      const uint32_t q = k[s];
      if (q == kNoPoint) break;
      ++cnt;
#pragma unroll
      for (int f = 0; f < 8; ++f)
        if (f < F) sum[f] = __fadd_rn(sum[f], point_feat(points, p.points_kind, (size_t)q * F + f));
    }
  }
#pragma unroll
  for (int f = 0; f < 8; ++f)
    if (f < F) features[(size_t)id * F + f] = __float2half_rn(__fdiv_rn(sum[f], (float)cnt));
  indices[id] = p.order == 0 ? make_int4(0, v.z, v.y, v.x) : make_int4(0, v.x, v.y, v.z);
}

}  // namespace spconvb

using namespace spconvb;

extern "C" {

size_t spconvb_voxelize_workspace_bytes(const spconvb_voxel_params* p, uint32_t max_points) {
  if (!p || max_points < 1 || p->max_points_per_voxel < 1) return 0;
  size_t total = 0;
  vox_layout(nullptr, *p, max_points, nullptr, &total);
  return total;
}

int spconvb_voxelize(const spconvb_voxel_params* p, const void* points, uint32_t num_points,
                     void* workspace, void* features, int32_t* indices, uint32_t* n_voxels_ptr,
                     uint32_t* status, void* stream) {
  return spconvb_voxelize_flags(p, points, num_points, workspace, features, indices, n_voxels_ptr,
                                0, status, stream);
}

int spconvb_voxelize_flags(const spconvb_voxel_params* p, const void* points, uint32_t num_points,
                           void* workspace, void* features, int32_t* indices,
                           uint32_t* n_voxels_ptr, uint32_t flags, uint32_t* status,
                           void* stream) {
  if (!p || !points || !workspace || !features || !indices || !n_voxels_ptr)
    return SPCONVB_E_ARG;
  if (p->num_features < 3 || p->num_features > 8 || p->max_points_per_voxel < 1 ||
      p->max_points_per_voxel > 16 || p->max_voxels < 1)
    return SPCONVB_E_ARG;
  unsigned long long cells = (unsigned long long)p->grid[0] * p->grid[1] * p->grid[2];
  if (p->grid[0] < 1 || p->grid[1] < 1 || p->grid[2] < 1 || cells >= 0xffffffffull)
    return SPCONVB_E_RANGE;
  cudaStream_t st = (cudaStream_t)stream;
  const int clear_tail = (flags & SPCONVB_FLAG_CLEAR_TAIL) != 0;
  if (num_points == 0) {
    SPCONVB_CUDA_TRY(cudaMemsetAsync(n_voxels_ptr, 0, sizeof(uint32_t), st));
    if (clear_tail) {
      const size_t rows = (size_t)p->max_voxels;
      SPCONVB_CUDA_TRY(cudaMemsetAsync(features, 0, sizeof(__half) * rows * p->num_features, st));
      SPCONVB_CUDA_TRY(cudaMemsetAsync(indices, 0, sizeof(int4) * rows, st));
    }
    return SPCONVB_OK;
  }
  size_t zero_bytes = 0, total = 0;
  VoxWs w = vox_layout(workspace, *p, num_points, &zero_bytes, &total);
  SPCONVB_CUDA_TRY(cudaMemsetAsync(workspace, 0, zero_bytes, st));
  const int blocks = (num_points + kVoxThreads - 1) / kVoxThreads;
  vox_hash_kernel<<<blocks, kVoxThreads, 0, st>>>(points, num_points, *p, w, status);
  SPCONVB_LAUNCH_CHECK();
  SPCONVB_CUDA_TRY(launch_pdl(vox_scan_kernel, dim3(w.blocks), dim3(kVoxScanThreads), 0, st,
                              num_points, p->max_points_per_voxel - 1, w));
  SPCONVB_CUDA_TRY(launch_pdl(vox_emit_kernel, dim3(w.blocks), dim3(kVoxScanThreads), 0, st, points,
                              num_points, *p, w, (__half*)features, (int4*)indices, n_voxels_ptr,
                              status, clear_tail));
  return SPCONVB_OK;
}

}  // extern "C"
