// CenterPoint head decode + rotated-box NMS, entirely on the device.
//
// Stage replaced: PostProcessCuda and the per-task host loop of CUDA-CenterPoint
// (src/postprocess_kernels.cu:28-403, src/centerpoint.cpp:163-216), which per task copies the
// candidate list to the host, sorts it there, copies it back, copies the suppression mask to
// the host and scans it there: three stream synchronisations per task, six tasks per frame.
//
// Here one call enqueues a clear and three kernels for all tasks together (blockIdx selects the
// task); a few hundred boxes leave the GPU idle, so what counts is the number of dependent steps:
//   candidates  one thread per heat-map cell: class arg-max of the sigmoid, score and centre
//               range filters; survivors append a 64-bit key (score bits | cell | label) and are
//               counted in a histogram of their scores
//   rank        16 CTAs per task: the histogram tells which scores the max_det best can have; the
//               rank of a key is the number of greater keys among those, counted by a warp per
//               key, so nothing is sorted; the box parameters (exp, atan2), corners and the
//               trigonometry are evaluated for the ranked cells only
//   mask        pairwise rotated IoU >= threshold below the diagonal, in tiles of 16 x 64
//               pairs: cheap upper bounds queue the pairs whose IoU can reach the threshold, then
//               the queue is spread over full warps; the last CTA of a task walks the ranking, 64
//               boxes at a time, and the last task packs all boxes into the caller's list
//
// This file is compiled without multiply-add contraction so that every product and sum rounds
// as in the reference's expression order on a CPU; only the library functions (expf, sinf,
// cosf, atan2f) may differ from a host libm by a few ulp.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "pdl.cuh"
#include "spconvb.h"
#include "spconvb_centerpoint.h"

namespace spconvb {
namespace {

constexpr int kDet = 11;         // floats per detection
constexpr int kBoxStride = 16;   // floats per prepared NMS box (struct BoxRec)
constexpr int kMaxDet = 1024;
constexpr int kMaskWords = 16;   // 64-bit words per mask row: 1024 / 64
// Scores by their leading bits: bin 0 up to 2^-5, then 512 bins an octave (sigmoids end at 1).
constexpr uint32_t kScoreBase = 0x3d000000u;  // bits of 2^-5
constexpr int kScoreShift = 14;
constexpr int kScoreBins = 2560;
__device__ __forceinline__ uint32_t score_bin(uint32_t bits) {
  return bits <= kScoreBase ? 0u : min((bits - kScoreBase) >> kScoreShift, (uint32_t)kScoreBins - 1u);
}

struct TaskBuffers {
  uint32_t* n_cand;
  uint32_t* n_det;
  uint32_t* n_kept;
  unsigned long long* cand;  // [H*W]
  float* det;                // [max_det][11]
  float* box;                // [max_det][16], BoxRec
  unsigned long long* mask;  // [max_det][16]: bit i of row j = the earlier box i suppresses box j
  uint32_t* kept;            // [post_max] ranks of the boxes that stay
  uint32_t* hist;            // [kScoreBins]
  uint32_t* ticket;          // mask CTAs that are done
};

struct PostArgs {
  spconvb_cp_head head[SPCONVB_CP_MAX_TASKS];
  TaskBuffers buf[SPCONVB_CP_MAX_TASKS];
  spconvb_cp_params p;
  int num_tasks;
  uint32_t* ticket;
  float* out_boxes;
  uint32_t* out_count;
  uint32_t* out_count_host;  // may be null
};

struct Layout {
  size_t counters_bytes;  // zeroed before every call
  size_t per_task;
  size_t cand, det, box, mask, kept;
  size_t total;
};

__host__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

__host__ Layout layout_of(const spconvb_cp_params& p, int tasks) {
  Layout l{};
  l.counters_bytes = align_up(
      sizeof(uint32_t) * (1 + 4 * (size_t)SPCONVB_CP_MAX_TASKS + kScoreBins * (size_t)tasks), 256);
  size_t off = 0;
  l.cand = off; off += align_up(sizeof(unsigned long long) * (size_t)p.H * p.W, 256);
  l.det = off;  off += align_up(sizeof(float) * kDet * (size_t)p.max_det, 256);
  l.box = off;  off += align_up(sizeof(float) * kBoxStride * (size_t)p.max_det, 256);
  l.mask = off; off += align_up(sizeof(unsigned long long) * kMaskWords * (size_t)p.max_det, 256);
  l.kept = off; off += align_up(sizeof(uint32_t) * (size_t)p.nms_post_max, 256);
  l.per_task = off;
  l.total = l.counters_bytes + l.per_task * (size_t)tasks;
  return l;
}

__host__ void bind_buffers(const Layout& l, void* workspace, int tasks, PostArgs& a) {
  char* base = (char*)workspace;
  uint32_t* counters = (uint32_t*)base;
  a.ticket = counters;
  for (int t = 0; t < tasks; ++t) {
    char* tb = base + l.counters_bytes + l.per_task * (size_t)t;
    a.buf[t].n_cand = counters + 1 + 4 * t;
    a.buf[t].n_det = counters + 2 + 4 * t;
    a.buf[t].n_kept = counters + 3 + 4 * t;
    a.buf[t].ticket = counters + 4 + 4 * t;
    a.buf[t].hist = counters + 1 + 4 * SPCONVB_CP_MAX_TASKS + kScoreBins * t;
    a.buf[t].cand = (unsigned long long*)(tb + l.cand);
    a.buf[t].det = (float*)(tb + l.det);
    a.buf[t].box = (float*)(tb + l.box);
    a.buf[t].mask = (unsigned long long*)(tb + l.mask);
    a.buf[t].kept = (uint32_t*)(tb + l.kept);
  }
}

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float ldh(const void* p, int i) {
  return __half2float(((const __half*)p)[i]);
}

// ------------------------------------------------------------------ candidates
__global__ void cp_candidates_kernel(const PostArgs a) {
  const int task = blockIdx.y;
  const spconvb_cp_head& hd = a.head[task];
  const int HW = a.p.H * a.p.W;
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= HW) return;
  const int h = cell / a.p.W, w = cell % a.p.W;
  int label = 0;
  float score = sigmoid_f(ldh(hd.hm, cell));
  for (int c = 1; c < hd.num_classes; ++c) {
    const float s = sigmoid_f(ldh(hd.hm, c * HW + cell));
    if (s > score) {
      score = s;
      label = c;
    }
  }
  if (score < a.p.score_threshold) return;
  float xs = ldh(hd.reg, cell) + (float)w;
  float ys = ldh(hd.reg, HW + cell) + (float)h;
  xs = xs * a.p.out_size_factor * a.p.voxel_size[0] + a.p.pc_range[0];
  ys = ys * a.p.out_size_factor * a.p.voxel_size[1] + a.p.pc_range[1];
  const float zs = ldh(hd.height, cell);
  const float* r = a.p.post_center_range;
  if (xs < r[0] || xs > r[3] || ys < r[1] || ys > r[4] || zs < r[2] || zs > r[5]) return;
  // positive floats order like their bit patterns; a smaller cell index ranks first on ties
  const unsigned long long key = ((unsigned long long)__float_as_uint(score) << 32) |
                                 ((unsigned long long)(0xFFFFFFu - (uint32_t)cell) << 8) |
                                 (unsigned long long)label;
  const uint32_t slot = atomicAdd(a.buf[task].n_cand, 1u);
  a.buf[task].cand[slot] = key;  // at most one key per cell, so slot < H*W
  atomicAdd(a.buf[task].hist + score_bin(__float_as_uint(score)), 1u);
}

// ------------------------------------------------------------------ rotated overlap
struct Pt { float x, y; };

// A box as the overlap test wants it: centre, extents, the rotation by -angle used by the
// corner-inside-box test, and the four corners turned by +angle about the centre.
struct BoxRec {
  float x, y, dx, dy;
  float cos_neg, sin_neg;
  Pt corner[4];
  float angle, reach;  // reach: half the diagonal, the farthest any point of the box is from its centre
};
static_assert(sizeof(BoxRec) == sizeof(float) * kBoxStride, "BoxRec layout");

__device__ __forceinline__ void prepare_box(const float* box, BoxRec& r) {
  r.x = box[0]; r.y = box[1]; r.dx = box[3]; r.dy = box[4];
  r.angle = box[6];
  r.reach = 0.5f * sqrtf(box[3] * box[3] + box[4] * box[4]);
  r.cos_neg = cosf(-box[6]);
  r.sin_neg = sinf(-box[6]);
  const float hx = box[3] / 2, hy = box[4] / 2;
  const float x1 = box[0] - hx, y1 = box[1] - hy, x2 = box[0] + hx, y2 = box[1] + hy;
  const float co = cosf(box[6]), si = sinf(box[6]);
  const float rx[4] = {x1, x2, x2, x1}, ry[4] = {y1, y1, y2, y2};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    r.corner[k].x = (rx[k] - box[0]) * co + (ry[k] - box[1]) * (-si) + box[0];
    r.corner[k].y = (rx[k] - box[0]) * si + (ry[k] - box[1]) * co + box[1];
  }
}

__device__ __forceinline__ float cross3(Pt p1, Pt p2, Pt p0) {
  return (p1.x - p0.x) * (p2.y - p0.y) - (p2.x - p0.x) * (p1.y - p0.y);
}

__device__ __forceinline__ bool inside_with_margin(const BoxRec& box, Pt p) {
  const float margin = 1e-2f;
  const float rx = (p.x - box.x) * box.cos_neg + (p.y - box.y) * (-box.sin_neg);
  const float ry = (p.x - box.x) * box.sin_neg + (p.y - box.y) * box.cos_neg;
  return fabsf(rx) < box.dx / 2 + margin && fabsf(ry) < box.dy / 2 + margin;
}

__device__ __forceinline__ bool segments_cross(Pt p1, Pt p0, Pt q1, Pt q0, Pt& ans) {
  if (!(fminf(p0.x, p1.x) <= fmaxf(q0.x, q1.x) && fminf(q0.x, q1.x) <= fmaxf(p0.x, p1.x) &&
        fminf(p0.y, p1.y) <= fmaxf(q0.y, q1.y) && fminf(q0.y, q1.y) <= fmaxf(p0.y, p1.y)))
    return false;
  const float s1 = cross3(q0, p1, p0);
  const float s2 = cross3(p1, q1, p0);
  const float s3 = cross3(p0, q1, q0);
  const float s4 = cross3(q1, p1, q0);
  if (!(s1 * s2 > 0 && s3 * s4 > 0)) return false;
  const float s5 = cross3(q1, p1, p0);
  if ((double)fabsf(s5 - s1) > 1e-8) {
    ans.x = (s5 * q0.x - s1 * q1.x) / (s5 - s1);
    ans.y = (s5 * q0.y - s1 * q1.y) / (s5 - s1);
  } else {
    const float a0 = p0.y - p1.y, b0 = p1.x - p0.x, c0 = p0.x * p1.y - p1.x * p0.y;
    const float a1 = q0.y - q1.y, b1 = q1.x - q0.x, c1 = q0.x * q1.y - q1.x * q0.y;
    const float D = a0 * b1 - a1 * b0;
    ans.x = (b0 * c1 - b1 * c0) / D;
    ans.y = (a1 * c0 - a0 * c1) / D;
  }
  return true;
}

__device__ float rotated_iou(const BoxRec& A, const BoxRec& B) {
  // Boxes farther apart than their reaches (plus far more than the 1e-2 margin of the corner
  // test and any rounding) share no edge crossing and no corner: the full computation below
  // would find no point and return 0 as well.
  {
    const float ddx = A.x - B.x, ddy = A.y - B.y, far = A.reach + B.reach + 0.1f;
    if (ddx * ddx + ddy * ddy > far * far) return 0.f;
  }
  Pt pts[16];
  float ang[16];
  int cnt = 0;
  Pt centre = {0.f, 0.f};
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      Pt x;
      if (segments_cross(A.corner[(i + 1) & 3], A.corner[i], B.corner[(j + 1) & 3], B.corner[j], x)) {
        centre.x = centre.x + x.x;
        centre.y = centre.y + x.y;
        pts[cnt++] = x;
      }
    }
  for (int k = 0; k < 4; ++k) {
    if (inside_with_margin(A, B.corner[k])) {
      centre.x = centre.x + B.corner[k].x;
      centre.y = centre.y + B.corner[k].y;
      pts[cnt++] = B.corner[k];
    }
    if (inside_with_margin(B, A.corner[k])) {
      centre.x = centre.x + A.corner[k].x;
      centre.y = centre.y + A.corner[k].y;
      pts[cnt++] = A.corner[k];
    }
  }
  if (cnt == 0) return 0.f;
  centre.x /= (float)cnt;
  centre.y /= (float)cnt;
  // stable ascending order of the polar angle about the centre
  for (int k = 0; k < cnt; ++k) ang[k] = atan2f(pts[k].y - centre.y, pts[k].x - centre.x);
  for (int k = 1; k < cnt; ++k) {
    const Pt p = pts[k];
    const float ak = ang[k];
    int j = k - 1;
    while (j >= 0 && ang[j] > ak) {
      pts[j + 1] = pts[j];
      ang[j + 1] = ang[j];
      --j;
    }
    pts[j + 1] = p;
    ang[j + 1] = ak;
  }
  float area = 0.f;
  for (int k = 0; k + 1 < cnt; ++k) {
    const float ax = pts[k].x - pts[0].x, ay = pts[k].y - pts[0].y;
    const float bx = pts[k + 1].x - pts[0].x, by = pts[k + 1].y - pts[0].y;
    area += ax * by - ay * bx;
  }
  const float overlap = fabsf(area) / 2.0f;
  const float sa = A.dx * A.dy, sb = B.dx * B.dy;
  return overlap / fmaxf(sa + sb - overlap, 1e-8f);
}

__global__ void rotated_iou_pairs_kernel(const float* a, const float* b, int n, float* iou) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  BoxRec A, B;
  prepare_box(a + (size_t)i * 7, A);
  prepare_box(b + (size_t)i * 7, B);
  iou[i] = rotated_iou(A, B);
}

// ------------------------------------------------------------------ rank
constexpr int kRankParts = 16;
constexpr int kRankThreads = 512;
constexpr int kRankList = 2048;  // keys a CTA compares with

// The K-th largest key, most significant byte first (keys are distinct): for frames where so many
// scores are equal to within a histogram bin that the list would not hold them.
__device__ unsigned long long select_kth(const unsigned long long* cand, uint32_t n, uint32_t K,
                                         uint32_t* hist, unsigned long long* s_prefix,
                                         uint32_t* s_need) {
  const int tid = threadIdx.x;
  if (tid == 0) { *s_prefix = 0ull; *s_need = K; }
  for (int shift = 56; shift >= 0; shift -= 8) {
    if (tid < 256) hist[tid] = 0u;
    __syncthreads();
    const unsigned long long prefix = *s_prefix;
    const unsigned long long hi = shift == 56 ? 0ull : (~0ull << (shift + 8));
    for (uint32_t base = 0; base < n; base += kRankThreads) {
      // keys of one score share their upper bytes: lanes with the same digit add once
      const uint32_t i = base + tid;
      const unsigned long long k = i < n ? cand[i] : 0ull;
      const bool live = i < n && ((k ^ prefix) & hi) == 0ull;
      const uint32_t digit = live ? ((uint32_t)(k >> shift) & 255u) : 256u;
      const uint32_t peers = __match_any_sync(0xffffffffu, digit);
      if (live && (tid & 31) == __ffs(peers) - 1) atomicAdd(&hist[digit], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (tid < 32) {
      // lane l owns bins 8l..8l+7; the digit is the highest bin whose count, together with
      // everything above it, reaches what is still needed
      uint32_t mine[8], sum = 0u;
#pragma unroll
      for (int k = 0; k < 8; ++k) { mine[k] = hist[tid * 8 + k]; sum += mine[k]; }
      uint32_t incl = sum;  // becomes the count in this lane's bins and in all higher lanes
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_down_sync(0xffffffffu, incl, d);
        if (tid + d < 32) incl += v;
      }
      const uint32_t above = incl - sum, need = *s_need;
      if (above < need && incl >= need) {  // exactly one lane
        uint32_t acc = above;
        int k = 7;
        for (; k > 0; --k) {
          if (acc + mine[k] >= need) break;
          acc += mine[k];
        }
        *s_need = need - acc;
        *s_prefix = prefix | ((unsigned long long)(tid * 8 + k) << shift);
      }
    }
    __syncthreads();
  }
  return *s_prefix;
}

// The detection and the prepared box of a ranked cell.
__device__ __forceinline__ void rank_write(const PostArgs& a, const spconvb_cp_head& hd,
                                           const TaskBuffers& b, unsigned long long key,
                                           uint32_t rank, int HW) {
  const int cell = (int)(0xFFFFFFu - (uint32_t)((key >> 8) & 0xFFFFFFull));
  const int label = (int)(key & 0xFFull);
  const float score = __uint_as_float((uint32_t)(key >> 32));
  const int h = cell / a.p.W, w = cell % a.p.W;
  float xs = ldh(hd.reg, cell) + (float)w;
  float ys = ldh(hd.reg, HW + cell) + (float)h;
  xs = xs * a.p.out_size_factor * a.p.voxel_size[0] + a.p.pc_range[0];
  ys = ys * a.p.out_size_factor * a.p.voxel_size[1] + a.p.pc_range[1];
  const float zs = ldh(hd.height, cell);
  const float dx = expf(ldh(hd.dim, cell));
  const float dy = expf(ldh(hd.dim, HW + cell));
  const float dz = expf(ldh(hd.dim, 2 * HW + cell));
  const float vx = ldh(hd.vel, cell), vy = ldh(hd.vel, HW + cell);
  const float rs = atan2f(ldh(hd.rot, cell), ldh(hd.rot, HW + cell));
  float* d = b.det + (size_t)rank * kDet;
  d[0] = xs; d[1] = ys; d[2] = zs; d[3] = dx; d[4] = dy; d[5] = dz;
  d[6] = vx; d[7] = vy; d[8] = rs; d[9] = (float)label; d[10] = score;
  // the box NMS sees: length and width swapped, yaw turned into the lidar frame
  const float nms_box[7] = {xs, ys, zs, dy, dx, dz, (float)(-(double)rs - 3.141592653 * 0.5)};
  prepare_box(nms_box, *(BoxRec*)(b.box + (size_t)rank * kBoxStride));
}

__global__ void __launch_bounds__(kRankThreads) cp_rank_kernel(const PostArgs a) {
  const int task = blockIdx.y, part = blockIdx.x, tid = threadIdx.x;
  const uint32_t lane = tid & 31u, warp = tid >> 5;
  const TaskBuffers& b = a.buf[task];
  const spconvb_cp_head& hd = a.head[task];
  const int HW = a.p.H * a.p.W;
  __shared__ unsigned long long list[kRankList], own[kRankList];
  __shared__ uint16_t rank_of[kRankList];
  __shared__ uint32_t hist[256];
  __shared__ unsigned long long s_prefix;
  __shared__ uint32_t s_need, s_list, s_own;
  pdl_wait();

  const uint32_t n = min(load_in_order(b.n_cand), (uint32_t)HW);
  const uint32_t K = min(n, (uint32_t)a.p.max_det);
  if (part == 0 && tid == 0) *b.n_det = K;
  if (tid == 0) { s_list = 0u; s_own = 0u; s_need = 0u; }
  __syncthreads();
  unsigned long long least = 0ull;  // keys below cannot be among the K best
  if (n > (uint32_t)kMaxDet) {
    // the bin in which the K-th best score lies: every thread sums kBinsEach bins, the sums are
    // scanned from the top
    constexpr int kBinsEach = kScoreBins / kRankThreads;
    static_assert(kBinsEach * kRankThreads == kScoreBins, "bins per thread");
    uint32_t mine[kBinsEach], sum = 0u;
#pragma unroll
    for (int k = 0; k < kBinsEach; ++k) {
      mine[k] = b.hist[tid * kBinsEach + k];
      sum += mine[k];
    }
    uint32_t incl = sum;  // the bins of this lane and of all higher lanes of the warp
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_down_sync(0xffffffffu, incl, d);
      if (lane + d < 32u) incl += v;
    }
    if (lane == 0) hist[warp] = incl;
    __syncthreads();
    uint32_t above = incl - sum;
    for (uint32_t w = warp + 1; w < kRankThreads / 32; ++w) above += hist[w];
    if (above < K && above + sum >= K) {  // exactly one thread
      uint32_t acc = above;
      int k = kBinsEach - 1;
      for (; k > 0; --k) {
        if (acc + mine[k] >= K) break;
        acc += mine[k];
      }
      const uint32_t bin = (uint32_t)(tid * kBinsEach + k);
      s_prefix = bin == 0u ? 0ull
                           : (unsigned long long)(kScoreBase + (bin << kScoreShift)) << 32;
      s_need = acc + mine[k];  // keys from that bin on
    }
    __syncthreads();
    least = s_prefix;
    if (s_need > (uint32_t)kRankList) {
      __syncthreads();
      least = select_kth(b.cand, n, K, hist, &s_prefix, &s_need);
    }
  }
  // the keys that count, in any order; this part ranks those at positions 32 part, 32 (part +
  // 16), ... of the candidates
  constexpr int kAtOnce = 8;
  auto is_mine = [&](uint32_t base) {
    return (((base >> 5) + warp) % kRankParts) == (uint32_t)part;
  };
  for (uint32_t base = 0; base < n; base += kAtOnce * kRankThreads) {
    unsigned long long k[kAtOnce];
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const uint32_t i = base + u * kRankThreads + tid;
      k[u] = i < n ? b.cand[i] : 0ull;  // no key is 0
    }
    uint32_t vote[kAtOnce], all = 0, mine = 0;
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      vote[u] = __ballot_sync(0xffffffffu, k[u] != 0ull && k[u] >= least);
      all += (uint32_t)__popc(vote[u]);
      if (is_mine(base + u * kRankThreads)) mine += (uint32_t)__popc(vote[u]);
    }
    if (all == 0u) continue;
    uint32_t at = 0, own_at = 0;
    if (lane == 0) {
      at = atomicAdd(&s_list, all);
      if (mine) own_at = atomicAdd(&s_own, mine);
    }
    at = __shfl_sync(0xffffffffu, at, 0);
    own_at = __shfl_sync(0xffffffffu, own_at, 0);
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const uint32_t off = __popc(vote[u] & ((1u << lane) - 1u));
      const bool in = (vote[u] >> lane) & 1u;
      if (in && at + off < (uint32_t)kRankList) list[at + off] = k[u];
      at += (uint32_t)__popc(vote[u]);
      if (is_mine(base + u * kRankThreads)) {
        if (in && own_at + off < (uint32_t)kRankList) own[own_at + off] = k[u];
        own_at += (uint32_t)__popc(vote[u]);
      }
    }
  }
  __syncthreads();
  const uint32_t count = min(s_list, (uint32_t)kRankList), owned = min(s_own, (uint32_t)kRankList);
  // a warp takes four keys through the list together
  for (uint32_t o = warp * 4u; o < owned; o += kRankThreads / 32 * 4u) {
    unsigned long long k[4];
    uint32_t greater[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) k[u] = own[min(o + u, owned - 1u)];
#pragma unroll 4
    for (uint32_t i = lane; i < count; i += 32) {
      const unsigned long long other = list[i];
#pragma unroll
      for (int u = 0; u < 4; ++u) greater[u] += other > k[u] ? 1u : 0u;
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      greater[u] = __reduce_add_sync(0xffffffffu, greater[u]);
      if (lane == 0 && o + u < owned) rank_of[o + u] = (uint16_t)greater[u];
    }
  }
  __syncthreads();
  for (uint32_t o = tid; o < owned; o += kRankThreads) {
    const uint32_t r = rank_of[o];
    if (r >= K) continue;
    rank_write(a, hd, b, own[o], r, HW);
  }
}

// ------------------------------------------------------------------ mask
constexpr int kMaskRows = 16;  // ranked boxes per tile; divides 64, so a tile's rows share a word
constexpr int kMaskCtasPerTask = 98;  // six tasks: one wave of four CTAs an SM
constexpr int kMaskThreads = 256;
constexpr int kMaskSlots = 6;  // tiles of a CTA: a task has at most 2 * 16 * 17 = 544
static_assert(kMaskSlots * kMaskCtasPerTask >= 544, "tiles of a task");

// The greedy walk over one task's ranking, by one CTA.  64 boxes at a time: four threads a box
// look whether an earlier kept box suppresses it, then the first warp decides among the 64: a box stays when every box of them that
// suppresses it is out, and is out when one of them stays, so the rounds are as many as the
// longest chain of suppressions and not as the boxes.  Boxes after the first nms_post_max
// survivors cannot reach the output.
constexpr int kNearWords = 6;
struct WalkShared {
  unsigned long long word[kNearWords * 64][kNearWords];
};
__device__ void walk_ranking(const PostArgs& a, const TaskBuffers& b, int m, WalkShared& sh) {
  __shared__ unsigned long long s_keep[kMaskWords], s_inner[64];
  __shared__ uint32_t s_gone[2], s_kept;
  const int tid = threadIdx.x, box = tid >> 2, quarter = tid & 3;
  const uint32_t lane = tid & 31u;
  const int words = (m + 63) / 64;
  if (tid == 0) s_kept = 0u;
  // the walk usually ends within the first few hundred boxes: their words are fetched together
  const int near = min(words, kNearWords);
#pragma unroll
  for (int k = tid; k < kNearWords * 64 * kNearWords; k += kMaskThreads) {
    const int j = k / kNearWords, word = k % kNearWords;
    sh.word[j][word] = j < m && word <= j / 64 ? __ldcg(b.mask + (size_t)j * kMaskWords + word) : 0ull;
  }
  __syncthreads();
  for (int w = 0; w < words; ++w) {
    if (tid < 2) s_gone[tid] = 0u;
    __syncthreads();
    const uint32_t kept = s_kept;
    if (kept >= (uint32_t)a.p.nms_post_max) break;
    const int j = w * 64 + box;
    bool gone = j >= m;
#pragma unroll
    for (int v = 0; v < kMaskWords / 4; ++v) {
      const int word = 4 * v + quarter;
      if (word > w || j >= m) continue;
      const unsigned long long bits =
          w < near ? sh.word[j][word] : __ldcg(b.mask + (size_t)j * kMaskWords + word);
      if (word < w) gone = gone || (bits & s_keep[word]) != 0ull;
      else s_inner[box] = bits;
    }
    if (gone) atomicOr(&s_gone[box >> 5], 1u << (box & 31));
    __syncthreads();
    if (tid < 32) {
      // lane l decides boxes l and 32 + l
      const unsigned long long in0 = s_inner[lane], in1 = s_inner[lane + 32];
      unsigned long long open = ~((unsigned long long)s_gone[0] | (unsigned long long)s_gone[1] << 32);
      unsigned long long keep = 0ull;
      while (open) {
        const bool o0 = (open >> lane) & 1ull, o1 = (open >> (lane + 32)) & 1ull;
        const bool k0 = o0 && (in0 & (open | keep)) == 0ull, k1 = o1 && (in1 & (open | keep)) == 0ull;
        const bool d0 = o0 && (in0 & keep) != 0ull, d1 = o1 && (in1 & keep) != 0ull;
        const unsigned long long nk = (unsigned long long)__ballot_sync(0xffffffffu, k0) |
                                      (unsigned long long)__ballot_sync(0xffffffffu, k1) << 32;
        const unsigned long long nd = (unsigned long long)__ballot_sync(0xffffffffu, d0) |
                                      (unsigned long long)__ballot_sync(0xffffffffu, d1) << 32;
        keep |= nk;
        open &= ~(nk | nd);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t bit = lane + 32u * h;
        const uint32_t at = kept + (uint32_t)__popcll(keep & ((1ull << bit) - 1ull));
        if (((keep >> bit) & 1ull) && at < (uint32_t)a.p.nms_post_max)
          b.kept[at] = (uint32_t)w * 64u + bit;
      }
      if (lane == 0) {
        s_keep[w] = keep;
        s_kept = kept + (uint32_t)__popcll(keep);
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (tid == 0) *b.n_kept = min(s_kept, (uint32_t)a.p.nms_post_max);
}

// The last task to get here packs every task's boxes into the caller's list, in task order.
constexpr int kPackBoxes = 1024;
struct PackShared {
  const float* from[kPackBoxes];
  int offset[kPackBoxes];
};
__device__ void pack_boxes(const PostArgs& a, PackShared& sh) {
  __shared__ bool s_last_task;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last_task = atomicAdd(a.ticket, 1u) == (uint32_t)(a.num_tasks - 1);
  __syncthreads();
  if (!s_last_task) return;
  __threadfence();
  uint32_t first[SPCONVB_CP_MAX_TASKS + 1];
  first[0] = 0;
#pragma unroll
  for (int t = 0; t < SPCONVB_CP_MAX_TASKS; ++t)
    first[t + 1] = first[t] + (t < a.num_tasks ? __ldcg(a.buf[t].n_kept) : 0u);
  const uint32_t total = first[SPCONVB_CP_MAX_TASKS];
  if (threadIdx.x == 0) {
    *a.out_count = total;
    if (a.out_count_host) *a.out_count_host = total;  // seen by the host when the kernel has ended
  }
  // where the boxes stand, then their values in the order of the list (coalesced both ways)
  for (uint32_t base = 0; base < total; base += kPackBoxes) {
    const uint32_t boxes = min(total - base, (uint32_t)kPackBoxes);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < boxes; k += kMaskThreads) {
      const uint32_t* kept = a.buf[0].kept + base + k;
      const float* det = a.buf[0].det;
      int offset = a.head[0].label_offset;
#pragma unroll
      for (int q = 1; q < SPCONVB_CP_MAX_TASKS; ++q)
        if (q < a.num_tasks && base + k >= first[q]) {
          kept = a.buf[q].kept + (base + k - first[q]);
          det = a.buf[q].det;
          offset = a.head[q].label_offset;
        }
      sh.from[k] = det + (size_t)__ldcg(kept) * kDet;
      sh.offset[k] = offset;
    }
    __syncthreads();
    // eight values a thread in flight (the stores may not be moved past loads, so by hand)
    constexpr uint32_t kAtOnce = 8;
    for (uint32_t e0 = threadIdx.x; e0 < boxes * kDet; e0 += kAtOnce * kMaskThreads) {
      float v[kAtOnce];
#pragma unroll
      for (uint32_t u = 0; u < kAtOnce; ++u) {
        const uint32_t e = min(e0 + u * kMaskThreads, boxes * kDet - 1u), k = e / kDet;
        v[u] = __ldcg(sh.from[k] + (e - k * kDet));
      }
#pragma unroll
      for (uint32_t u = 0; u < kAtOnce; ++u) {
        const uint32_t e = e0 + u * kMaskThreads, k = e / kDet;
        if (e >= boxes * kDet) break;
        a.out_boxes[(size_t)base * kDet + e] =
            e - k * kDet == 9u ? (float)(sh.offset[k] + (int)v[u]) : v[u];
      }
    }
  }
}

// Whether the IoU of two boxes is certain to stay below the threshold: the common part lies inside
// the bounding box, along A's axes (and along B's), of what both cover there.  Half the pairs in
// reach of one another are decided by this.  The margin covers the 1e-2 by which corners outside a
// box still count as inside, and the rounding of corners and crossings where positions and extents
// are below kBoundLimit, within which the bound is taken (at 10 000 m a float's step is 0.001; random
// pairs show none decided wrongly up to 100 000 m, some from 1 000 000 m on).
constexpr float kBoundLimit = 1e4f;
struct BoxBounds { float x, y, dx, dy, c, s; };
__device__ __forceinline__ float cover_along(const BoxBounds& A, const BoxBounds& B) {
  const float ddx = B.x - A.x, ddy = B.y - A.y;
  const float rx = ddx * A.c - ddy * A.s, ry = ddx * A.s + ddy * A.c;
  const float co = fabsf(A.c * B.c + A.s * B.s), si = fabsf(A.s * B.c - A.c * B.s);
  const float ex = 0.5f * (co * B.dx + si * B.dy), ey = 0.5f * (si * B.dx + co * B.dy);
  const float hx = 0.5f * A.dx, hy = 0.5f * A.dy;
  const float wx = fminf(hx, rx + ex) - fmaxf(-hx, rx - ex) + 0.1f;
  const float wy = fminf(hy, ry + ey) - fmaxf(-hy, ry - ey) + 0.1f;
  return fmaxf(wx, 0.f) * fmaxf(wy, 0.f);
}
__device__ __forceinline__ bool surely_below(const BoxBounds& A, const BoxBounds& B, float threshold) {
  const float cover = fminf(cover_along(A, B), cover_along(B, A)) * 1.02f + 1e-3f;
  const float most = fmaxf(fmaxf(fmaxf(fabsf(A.x), fabsf(A.y)), fmaxf(fabsf(B.x), fabsf(B.y))),
                           fmaxf(fmaxf(A.dx, A.dy), fmaxf(B.dx, B.dy)));
  return threshold > 0.f && most <= kBoundLimit &&
         cover < threshold * 0.999f * (A.dx * A.dy + B.dx * B.dy - cover);
}

// rotated_iou(A, B) >= threshold by a whole warp: lane e < 16 looks for the crossing of edge e / 4
// of A and e % 4 of B, lanes 16..23 at the corners, in the order in which the serial code appends
// its points; sums run in that order and in the order of the angles, so every bit is the same.
// Angles that are not numbers have no order: there the serial insertion decides which points end up
// where (boxes of 1e12 m and more, whose crossings overflow: some of their overlaps are infinite).
struct IouScratch {
  Pt point[24];  // in the order of the serial code, then of the angles
  float value[24];
};
__device__ __forceinline__ bool iou_reaches(const BoxRec& A, const BoxRec& B, float threshold,
                                            IouScratch& sh) {
  const uint32_t lane = threadIdx.x & 31u;
  Pt p = {0.f, 0.f};
  bool have = false;
  if (lane < 16u) {
    const int i = lane >> 2, j = lane & 3;
    have = segments_cross(A.corner[(i + 1) & 3], A.corner[i], B.corner[(j + 1) & 3], B.corner[j], p);
  } else if (lane < 24u) {
    const int k = (lane - 16u) >> 1;
    p = (lane & 1u) ? A.corner[k] : B.corner[k];
    have = (lane & 1u) ? inside_with_margin(B, p) : inside_with_margin(A, p);
  }
  const uint32_t set = __ballot_sync(0xffffffffu, have);
  const int cnt = __popc(set);
  float iou = 0.f;
  if (cnt != 0) {
    // lane k goes on with point k; what is summed in order goes through shared memory
    __syncwarp();
    if (have) sh.point[__popc(set & ((1u << lane) - 1u))] = p;
    __syncwarp();
    Pt centre = {0.f, 0.f};
#pragma unroll 4
    for (int k = 0; k < cnt; ++k) {
      centre.x = centre.x + sh.point[k].x;
      centre.y = centre.y + sh.point[k].y;
    }
    centre.x /= (float)cnt;
    centre.y /= (float)cnt;
    const bool mine = (int)lane < cnt;
    if (mine) p = sh.point[lane];
    const float ang = mine ? atan2f(p.y - centre.y, p.x - centre.x) : 0.f;
    if (mine) sh.value[lane] = ang;
    // a vote orders no memory: this orders the angles before their readers below, and the reads of
    // the points above before the points are put in their places
    __syncwarp();
    if (!__any_sync(0xffffffffu, ang != ang)) {
      // place in the stable ascending order of the angles
      int place = 0;
#pragma unroll 4
      for (int k = 0; k < cnt; ++k) {
        const float other = sh.value[k];
        if (other < ang || (other == ang && k < (int)lane)) ++place;
      }
      if (mine) sh.point[place] = p;
    } else if (lane == 0) {
      for (int k = 1; k < cnt; ++k) {
        const Pt pk = sh.point[k];
        const float ak = sh.value[k];
        int j = k - 1;
        for (; j >= 0 && sh.value[j] > ak; --j) {
          sh.point[j + 1] = sh.point[j];
          sh.value[j + 1] = sh.value[j];
        }
        sh.point[j + 1] = pk;
        sh.value[j + 1] = ak;
      }
    }
    __syncwarp();
    if ((int)lane + 1 < cnt) {
      const Pt p0 = sh.point[0], pk = sh.point[lane], pn = sh.point[lane + 1];
      const float ax = pk.x - p0.x, ay = pk.y - p0.y, bx = pn.x - p0.x, by = pn.y - p0.y;
      sh.value[lane] = ax * by - ay * bx;
    }
    __syncwarp();
    float area = 0.f;
#pragma unroll 4
    for (int k = 0; k + 1 < cnt; ++k) area += sh.value[k];
    const float overlap = fabsf(area) / 2.0f;
    const float sa = A.dx * A.dy, sb = B.dx * B.dy;
    iou = overlap / fmaxf(sa + sb - overlap, 1e-8f);
  }
  return iou >= threshold;
}

// One tile = 16 boxes x 64 earlier ones; a CTA takes all its tiles (up to six) through each pass
// together.  Pass 1: every thread tests pairs for reach, bounds the IoU of the others and queues
// what is left: 3 to 10 of a tile's 1 024, at most 30 in the benchmark's heads, so that what
// counts is how long one pair takes and not how many there are.  Pass 2: a warp per queued pair.
// The CTA that finishes a task's last tile walks that task's ranking.
__global__ void __launch_bounds__(kMaskThreads) cp_mask_kernel(const PostArgs a) {
  const int task = blockIdx.y;
  const TaskBuffers& b = a.buf[task];
  const int tid = threadIdx.x;
  constexpr int kBoxes = 64 + kMaskRows;
  // 17 words a box: the lanes of a warp read the same field of 32 boxes
  struct PaddedBox { BoxRec rec; float pad; };
  __shared__ union {
    struct {
      PaddedBox box[kMaskSlots][kBoxes];
      uint16_t near[kMaskSlots * kMaskRows * 64];  // pairs in reach; those left go to its front
    } tiles;
    WalkShared walk;
    PackShared pack;
  } sh;
  __shared__ int s_first[kMaskSlots][2];
  __shared__ unsigned long long words[kMaskSlots][kMaskRows];
  __shared__ IouScratch scratch[kMaskThreads / 32];
  __shared__ uint32_t in_reach;
  __shared__ uint32_t queued;
  __shared__ bool s_last;
  pdl_wait();
  const int m = (int)load_in_order(b.n_det);
  const float threshold = a.p.nms_iou_threshold;
  // tiles on or below the diagonal: 4 row groups of 16 in block row G, G + 1 tiles each
  const int groups = (m + kMaskRows - 1) / kMaskRows, whole = groups / 4;
  const int tiles = 2 * whole * (whole + 1) + (groups - 4 * whole) * (whole + 1);
  // CTAs without a tile leave at once and are not waited for (one stays to walk an empty ranking)
  const int ctas = max(1, min((int)gridDim.x, tiles));
  if ((int)blockIdx.x >= ctas) return;
  const int slots = max(0, (tiles - (int)blockIdx.x + ctas - 1) / ctas);
  if (tid < slots) {
    const int tile = blockIdx.x + tid * ctas;
    int G = 0;
    while (2 * (G + 1) * (G + 2) <= tile) ++G;
    const int in = tile - 2 * G * (G + 1);
    s_first[tid][0] = (4 * G + in / (G + 1)) * kMaskRows;
    s_first[tid][1] = in % (G + 1) * 64;
  }
  if (tid < kMaskSlots * kMaskRows) words[tid / kMaskRows][tid % kMaskRows] = 0ull;
  if (tid == 0) in_reach = queued = 0u;
  __syncthreads();
  {
    float4 v[kMaskSlots * kBoxes * 4 / kMaskThreads + 1];  // all in flight together
#pragma unroll
    for (int u = 0; u < kMaskSlots * kBoxes * 4 / kMaskThreads + 1; ++u) {
      const int k = tid + u * kMaskThreads, slot = k / (kBoxes * 4), at = k / 4 % kBoxes;
      if (slot >= slots) break;
      const int box = min(at < 64 ? s_first[slot][1] + at : s_first[slot][0] + at - 64, m - 1);
      v[u] = __ldcg((const float4*)(b.box + (size_t)box * kBoxStride) + (k & 3));
    }
#pragma unroll
    for (int u = 0; u < kMaskSlots * kBoxes * 4 / kMaskThreads + 1; ++u) {
      const int k = tid + u * kMaskThreads, slot = k / (kBoxes * 4), at = k / 4 % kBoxes;
      if (slot >= slots) break;
      float* to = (float*)&sh.tiles.box[slot][at] + (k & 3) * 4;
      to[0] = v[u].x; to[1] = v[u].y; to[2] = v[u].z; to[3] = v[u].w;
    }
  }
  __syncthreads();
  for (int slot = 0; slot < slots; ++slot) {
    // a thread keeps its column and takes every fourth row
    const int c = tid & 63, i = s_first[slot][1] + c;
    const BoxRec& A = sh.tiles.box[slot][c].rec;
    const float x = A.x, y = A.y, reach = A.reach;
#pragma unroll
    for (int u = 0; u < kMaskRows / 4; ++u) {
      const int r = (tid >> 6) + 4 * u, j = s_first[slot][0] + r;
      const BoxRec& B = sh.tiles.box[slot][64 + r].rec;
      const float ddx = x - B.x, ddy = y - B.y, far = reach + B.reach + 0.1f;
      // the same test rotated_iou starts with
      if (j < m && i < j && !(ddx * ddx + ddy * ddy > far * far))
        sh.tiles.near[atomicAdd(&in_reach, 1u)] = (uint16_t)(slot << 10 | r << 6 | c);
    }
  }
  __syncthreads();
  const uint32_t n_reach = in_reach;
  for (uint32_t q0 = 0; q0 < n_reach; q0 += kMaskThreads) {
    const uint32_t q = q0 + tid;
    bool stays = false;
    uint16_t pair = 0;
    if (q < n_reach) {
      pair = sh.tiles.near[q];
      const BoxRec& A = sh.tiles.box[pair >> 10][pair & 63].rec;
      const BoxRec& B = sh.tiles.box[pair >> 10][64 + ((pair >> 6) & (kMaskRows - 1))].rec;
      stays = !surely_below({A.x, A.y, A.dx, A.dy, A.cos_neg, A.sin_neg},
                            {B.x, B.y, B.dx, B.dy, B.cos_neg, B.sin_neg}, threshold);
    }
    __syncthreads();  // this round's pairs are read; fewer than that are kept
    if (stays) sh.tiles.near[atomicAdd(&queued, 1u)] = pair;
  }
  __syncthreads();
  const uint32_t n_pairs = queued;
  for (uint32_t q = tid >> 5; q < n_pairs; q += kMaskThreads / 32) {
    const int pair = sh.tiles.near[q], slot = pair >> 10, r = (pair >> 6) & (kMaskRows - 1);
    const int c = pair & 63;
    // the earlier box first
    if (iou_reaches(sh.tiles.box[slot][c].rec, sh.tiles.box[slot][64 + r].rec, threshold,
                    scratch[tid >> 5]) &&
        (tid & 31) == 0)
      atomicOr(&words[slot][r], 1ull << c);
  }
  __syncthreads();
  for (int k = tid; k < slots * kMaskRows; k += kMaskThreads) {
    const int slot = k / kMaskRows, row = s_first[slot][0] + k % kMaskRows;
    if (row < m)
      b.mask[(size_t)row * kMaskWords + s_first[slot][1] / 64] = words[slot][k % kMaskRows];
  }
  __threadfence();  // every thread's words are visible device-wide before the ticket is taken
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(b.ticket, 1u) == (uint32_t)ctas - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  walk_ranking(a, b, m, sh.walk);
  pack_boxes(a, sh.pack);
}

bool params_ok(const spconvb_cp_params* p) {
  return p && p->H >= 1 && p->W >= 1 && (size_t)p->H * p->W <= 0xFFFFFFu && p->max_det >= 1 &&
         p->max_det <= kMaxDet && p->nms_post_max >= 1 && p->nms_post_max <= p->max_det;
}

}  // namespace
}  // namespace spconvb

using namespace spconvb;

extern "C" {

void spconvb_cp_default_params(spconvb_cp_params* p) {
  if (!p) return;
  p->H = 180; p->W = 180;
  p->out_size_factor = 8.f;
  p->voxel_size[0] = p->voxel_size[1] = 0.075f;
  p->pc_range[0] = p->pc_range[1] = -54.f;
  p->score_threshold = 0.1f;
  const float r[6] = {-61.2f, -61.2f, -10.0f, 61.2f, 61.2f, 10.0f};
  for (int i = 0; i < 6; ++i) p->post_center_range[i] = r[i];
  p->nms_iou_threshold = 0.2f;
  p->max_det = 1000;
  p->nms_post_max = 83;
}

size_t spconvb_cp_workspace_bytes(const spconvb_cp_params* p, int32_t num_tasks) {
  if (!params_ok(p) || num_tasks < 1 || num_tasks > SPCONVB_CP_MAX_TASKS) return 0;
  return layout_of(*p, num_tasks).total;
}

int spconvb_cp_postprocess(const spconvb_cp_head* heads, int32_t num_tasks,
                           const spconvb_cp_params* p, void* workspace, size_t workspace_bytes,
                           float* out_boxes, uint32_t* out_count, void* stream) {
  return spconvb_cp_postprocess_host(heads, num_tasks, p, workspace, workspace_bytes, out_boxes,
                                     out_count, nullptr, stream);
}

int spconvb_cp_postprocess_host(const spconvb_cp_head* heads, int32_t num_tasks,
                                const spconvb_cp_params* p, void* workspace,
                                size_t workspace_bytes, float* out_boxes, uint32_t* out_count,
                                uint32_t* out_count_host, void* stream) {
  if (!heads || !params_ok(p) || !workspace || !out_boxes || !out_count || num_tasks < 1 ||
      num_tasks > SPCONVB_CP_MAX_TASKS || ((uintptr_t)workspace & 255u))
    return SPCONVB_E_ARG;
  const Layout l = layout_of(*p, num_tasks);
  if (workspace_bytes < l.total) return SPCONVB_E_NOMEM;
  PostArgs a{};
  for (int t = 0; t < num_tasks; ++t) {
    const spconvb_cp_head& h = heads[t];
    if (!h.reg || !h.height || !h.dim || !h.rot || !h.vel || !h.hm || h.num_classes < 1 ||
        h.num_classes > 256)
      return SPCONVB_E_ARG;
    a.head[t] = h;
  }
  a.p = *p;
  a.num_tasks = num_tasks;
  a.out_boxes = out_boxes;
  a.out_count = out_count;
  a.out_count_host = out_count_host;
  bind_buffers(l, workspace, num_tasks, a);
  cudaStream_t st = (cudaStream_t)stream;
  SPCONVB_CUDA_TRY(cudaMemsetAsync(workspace, 0, l.counters_bytes, st));
  const int HW = p->H * p->W;
  cp_candidates_kernel<<<dim3((HW + 255) / 256, num_tasks), 256, 0, st>>>(a);
  SPCONVB_LAUNCH_CHECK();
  SPCONVB_CUDA_TRY(launch_pdl(cp_rank_kernel, dim3(kRankParts, num_tasks), dim3(kRankThreads), 0,
                              st, a));
  SPCONVB_CUDA_TRY(launch_pdl(cp_mask_kernel, dim3(kMaskCtasPerTask, num_tasks), dim3(kMaskThreads),
                              0, st, a));
  return SPCONVB_OK;
}

int spconvb_cp_task_detections(const spconvb_cp_params* p, int32_t num_tasks,
                               const void* workspace, int32_t task, const float** detections,
                               const uint32_t** n_det) {
  if (!params_ok(p) || !workspace || num_tasks < 1 || num_tasks > SPCONVB_CP_MAX_TASKS ||
      task < 0 || task >= num_tasks)
    return SPCONVB_E_ARG;
  PostArgs a{};
  bind_buffers(layout_of(*p, num_tasks), (void*)workspace, num_tasks, a);
  if (detections) *detections = a.buf[task].det;
  if (n_det) *n_det = a.buf[task].n_det;
  return SPCONVB_OK;
}

int spconvb_cp_rotated_iou(const float* boxes_a, const float* boxes_b, int32_t n, float* iou,
                           void* stream) {
  if (!boxes_a || !boxes_b || !iou || n < 0) return SPCONVB_E_ARG;
  if (n == 0) return SPCONVB_OK;
  rotated_iou_pairs_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(boxes_a, boxes_b, n,
                                                                              iou);
  SPCONVB_LAUNCH_CHECK();
  return SPCONVB_OK;
}

}  // extern "C"
