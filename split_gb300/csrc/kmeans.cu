// k-means for the segmentation path: assignment over packed or planar pixel
// features with the centroids in shared memory, and a deterministic FP32
// centroid update, fused in one persistent cooperative kernel per call.
//
// Restates split/src/split/device/kmeans/{cluster,label,centroids,
// propagation}.cu (see the per-function notes) without the N x K distance
// matrix, the radix sort per iteration or the host round trip per iteration.
//
// Work decomposition (fixed per image, so a result never depends on what else
// shares the launch): an image is cut into warp spans of 64 columns by 2, 4, 8
// or 16 rows (an eighth of the tuning table's unit height).
// Every warp accumulates (x - c_label) over its span's pixel batches in FP32
// registers and a warp-private shared-memory slot (warp butterfly sums per
// distinct label); at the end of the span the slots are rounded to multiples
// of 2^-24 and added, as integers, into the block's shared sums
// (warp_to_fix).  A span whose candidate mask names one cluster adds the
// exact integer sum of its pixels' features instead (add_span_sums).  The
// block adds its integer sums into per-image accumulators as 96-bit fixed
// point (64-bit atomics on a low and a high word).  Integer addition does not
// depend on order, so the image total is the same whatever blocks took which
// spans and whatever else shares the launch.
//
// Iterations: a block goes through its share of spans, warp by warp
// (span_pass), and adds its integer sums into the image accumulators once.
// The first iteration keeps every fast span's exact feature sum, where the
// workspace has room; in later ones a span with one candidate then needs none
// of its pixels.  The grid barrier that ends the iteration publishes the sums;
// then c_new = c + S / n is formed in FP32 from the exact sum
// (form_centroids) by every block that works on the image, from the same
// inputs (bit-identical), one of them publishing it.  The sums are kept in
// three slots by iteration, so that one can clear the slot of the iteration
// after next while the current slot fills and the last one is read.
#include <limits.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "f32x2.cuh"
#include "fixsum.cuh"
#include "pixels.cuh"

namespace sg {
namespace km {

// Resident blocks per SM the register budget is set for: 2 (up to 128
// registers a thread) keeps the span passes free of spills; at 3 (80
// registers) they spill.
#ifndef SG_KM_MINBLOCKS
#define SG_KM_MINBLOCKS 2
#endif
constexpr int kBatchMinBlocks = 2;
// Costs of a batch's partition: a span that needs its pixels against one that
// does not, and taking up an image (in spans, and in clocks).
constexpr int kPixelCost = 20;
constexpr int kImageSpans = 32, kImageClocks = 20000;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
// A unit is a tile of unit_rows x kTile pixels (unit_rows = 16 to 128, per
// image from the tuning table); warp w owns rows [w * r, (w + 1) * r) of it,
// r = unit_rows / 8.
constexpr int kTile = 64;
constexpr int kMaxK = 64;
constexpr int kMaxDim = 5;
constexpr int kSpanSums = 8;   // words of a span's entry in Image::span_sum (kMaxDim used)
constexpr int kHeavyCap = 512; // deferred spans a block lists per iteration
// Span sums are added into the image accumulators as multiples of 2^-24; a
// span's FP32 sum must stay below 2^38 in magnitude (a span holds at most
// 1024 pixels, so |x - c| below 2.6e8 everywhere).  Beyond it the call
// reports SPLIT_ERR_OVERFLOW.
constexpr float kFixScale = 16777216.0f;   // 2^24
constexpr float kFixLimit = 274877906944.0f;   // 2^38

enum Mode { kCluster = 0, kUpdateOnly = 1, kAssignOnly = 2 };

struct Image {
  const void* points;
  int unit_range;           // colour features known to lie in [0, 1]
  int any_width;            // RGB8: fast spans at any width and alignment
  int64_t npoints;
  int width;
  float xy_scale;
  float* centroids;         // user array, dim x K planar (in/out)
  int32_t* labels;          // output labels (cluster / assign modes)
  const int32_t* labels_in; // update-only mode
  int K;
  int max_iter;
  float threshold;
  int32_t* d_iterations;
  int nspans;               // warp spans: ceil(height / (unit_rows / kWarps)) * ntx
  int scatter;              // batches: a step coprime to nspans, about 0.618 of it
  int first_cost;           // batches: cost of the first iteration, in spans
  int height;               // rows (ceil(npoints / width))
  int ntx;                  // tiles per row of tiles
  int unit_rows;            // rows of a unit (kTile or 2 * kTile, from the tuning table)
  int ref_shift;            // SPLIT_KMEANS_REFERENCE_SHIFT (D = 3, K >= 3)
  // Exact feature sums of the fast spans (kSpanSums words each), written in
  // the first iteration of a call (null: none kept).  A fast span's slot is
  // (first row / span rows) * span_cols + tile column.
  long long* span_sum;
  int span_cols;            // width / kTile: tile columns of full width
};

// Of a batch's image: the centroid shift after iteration i - 1 in slot i & 1,
// (slot 0) the iteration at whose start it stopped (0: still running), and what
// iteration i cost (cost_at).
struct ImageState {
  float delta;
  int done;
  int cost[2];
};

struct Params {
  Image img0;            // used when nimages == 1
  const Image* images;   // device array when nimages > 1
  int nimages;
  int total_spans;
  int max_iter;
  // sums of iteration i live in slot i % 3 (see form_centroids)
  unsigned long long* acc_lo;  // [3][nimages][kMaxK * kMaxDim] low 32-bit words of the sums
  unsigned long long* acc_hi;  // [3][nimages][kMaxK * kMaxDim] high words (signed)
  unsigned* acc_cnt;           // [3][nimages][kMaxK] member counts
  float* cur;                  // [2][nimages][kMaxK * 8]: centroids of iteration i in i & 1
  ImageState* state;     // [2][nimages] (batches)
  WsHeader* hdr;
  int blocks_per_sm;     // 0: as many as fit (host side only)
  // grid barriers: polls before a wait gives up, and a block that leaves
  // without arriving (-1: none); see split_kmeans_set_wait_test
  unsigned wait_limit;
  int wait_skip;
};

constexpr int cstride(int dim) { return dim == 3 ? 4 : 8; }

__device__ __forceinline__ const Image& image_of(const Params& p, int i) {
  return p.images ? p.images[i] : p.img0;
}

__device__ __forceinline__ size_t acc_slot(const Params& p, int slot, int img) {
  return (size_t)slot * p.nimages + img;
}

// Where iteration i adds up an image's cost: one of three words, by i mod 3.
__device__ __forceinline__ int* cost_at(const Params& p, int img, int i) {
  const int slot = i % 3;
  return &p.state[acc_slot(p, slot >> 1, img)].cost[slot & 1];
}

// Pixel feature loader.  dim == 5 appends xy_scale * (column, row).
template <int LAYOUT, int DIM>
struct Loader {
  const void* pts;
  int64_t n;
  float xy;
  __device__ __forceinline__ void load(int64_t i, int row, int col,
                                       float (&f)[DIM]) const {
    if (LAYOUT == SPLIT_LAYOUT_PLANAR) {
      const float* p = static_cast<const float*>(pts);
#pragma unroll
      for (int d = 0; d < DIM; ++d) f[d] = __ldg(p + d * n + i);
      return;
    } else if (LAYOUT == SPLIT_LAYOUT_FLOAT4) {
      float4 v = __ldg(static_cast<const float4*>(pts) + i);
      f[0] = v.x;
      f[1] = v.y;
      f[2] = v.z;
    } else {
      const uint8_t* p = static_cast<const uint8_t*>(pts) + 3 * i;
#pragma unroll
      for (int c = 0; c < 3; ++c) f[c] = __fdiv_rn((float)__ldg(p + c), 255.0f);
    }
    if (DIM == 5) {
      f[3] = __fmul_rn(xy, (float)col);
      f[4] = __fmul_rn(xy, (float)row);
    }
  }
};

// Order-preserving float -> int key (for warp min/max reductions).
__device__ __forceinline__ int fkey(float x) {
  const int i = __float_as_int(x);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float fkey_inv(int k) {
  return __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
}

// Candidate clusters of a 32-pixel batch whose features lie in the box
// [lo, hi]: lane l bounds clusters l and l + 32.  For every cluster,
// LB = squared distance from the centroid to the box (a lower bound of each
// pixel's distance) and UB = squared distance to the farthest box corner (an
// upper bound).  A cluster whose LB exceeds the smallest UB by more than the
// 1e-4 relative margin is strictly farther than the winner from every pixel
// of the batch even after FP32 rounding (a few ulp), so skipping it leaves
// every argmin - ties included - unchanged.
template <int DIM>
__device__ __forceinline__ unsigned long long candidates(const float (&lo)[DIM],
                                                         const float (&hi)[DIM],
                                                         const float* __restrict__ cs, int K) {
  constexpr int CS = cstride(DIM);
  const int lane = threadIdx.x & 31;
  float lb[2], ubm = INFINITY;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = lane + 32 * h;
    // a slot past K compares false even against an infinite thr (a box
    // with an infinite feature)
    lb[h] = __int_as_float(0x7fffffff);
    if (k < K) {
      float l = 0.0f, u = 0.0f;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        const float c = cs[k * CS + d];
        const float g = fmaxf(fmaxf(lo[d] - c, c - hi[d]), 0.0f);
        const float e = fmaxf(c - lo[d], hi[d] - c);
        l = __fmaf_rn(g, g, l);
        u = __fmaf_rn(e, e, u);
      }
      lb[h] = l;
      ubm = fminf(ubm, u);
    }
  }
  // UB >= 0: its bit pattern orders like the value
  const float ub = __int_as_float(__reduce_min_sync(0xffffffffu, __float_as_int(ubm)));
  const float thr = ub * 1.0001f;
  const unsigned m0 = __ballot_sync(0xffffffffu, lb[0] <= thr);
  const unsigned m1 = __ballot_sync(0xffffffffu, lb[1] <= thr);
  return ((unsigned long long)m1 << 32) | m0;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct Smem {
  alignas(16) float cent[kMaxK * 8];
  float acc[kWarps][kMaxK * kMaxDim];
  int cnt[kWarps][kMaxK];
  // the sums of the spans processed since the last flush, in 64-bit fixed
  // point (each span's converted on its own, then added as integers); two
  // words, because shared memory adds 32 bits in one operation
  unsigned fix_lo[kMaxK * kMaxDim], fix_hi[kMaxK * kMaxDim];
  int fixn[kMaxK];
  // classification of spans with xy features: the colour part of a centroid's
  // bounds over the unit cube (lower, upper) and its xy
  float4 bound[kMaxK];
  // n * c * 2^24 of every centroid value, n the pixels of a whole span
  long long nc[kMaxK * kMaxDim];
  // spans deferred to the second pass of an iteration (see span_pass)
  int heavy[kHeavyCap];
  unsigned long long heavy_mask[kHeavyCap];   // their candidates
  unsigned finite[2];   // bit k: centroid k has no infinity and no NaN
  int nheavy;
  int next_heavy;
  int counted;   // spans of the pass that needed their pixels (batches)
  // centroid forming: squared shifts, the last shift, the decisions
  float sdiff[kMaxK * kMaxDim];
  float delta;
  int stopped, more;
};

// sum idx += v (64 bits, wrapping)
__device__ __forceinline__ void fix_add(Smem& sm, int idx, long long v) {
  const unsigned lo = (unsigned)v;
  const unsigned old = atomicAdd(&sm.fix_lo[idx], lo);
  const unsigned hi = (unsigned)((unsigned long long)v >> 32) + (old + lo < old ? 1u : 0u);
  if (hi) atomicAdd(&sm.fix_hi[idx], hi);
}

// acc[d] += x[d] - c[d] for every dimension, in IEEE single precision: the
// pairs (0, 1) and (3, 4) on the packed pipe (per-lane results, the same bits
// as the scalar operations).
template <int DIM>
__device__ __forceinline__ void add_centered(const float (&x)[DIM], const float* c,
                                             float (&acc)[DIM]) {
  const float2 a01 = fadd2(make_float2(acc[0], acc[1]),
                           fsub2(make_float2(x[0], x[1]), make_float2(c[0], c[1])));
  acc[0] = a01.x;
  acc[1] = a01.y;
  acc[2] = __fadd_rn(acc[2], __fsub_rn(x[2], c[2]));
  if (DIM == 5) {
    constexpr int X = DIM == 5 ? 3 : 0, Y = DIM == 5 ? 4 : 0;
    const float2 a34 = fadd2(make_float2(acc[X], acc[Y]),
                             fsub2(make_float2(x[X], x[Y]), make_float2(c[X], c[Y])));
    acc[X] = a34.x;
    acc[Y] = a34.y;
  }
}

constexpr int kLanesPerRow = kTile / kPx;  // 16 lanes cover a tile row
constexpr int kBatchRows = 32 / kLanesPerRow;
static_assert((kTile / kWarps) % kBatchRows == 0, "whole batches per warp span");

// Nearest centroid among `mask` for the lane's pixels; the distance is the
// fma chain of (x - c)^2 in dimension order, strict < in ascending k (ties to
// the lowest k; label.cu:23-32, :98-105), evaluated on pixel pairs with the
// packed f32x2 pipe.  NB batches share the walk over the mask.
template <int DIM, int NB>
__device__ __forceinline__ void nearest_px(const float (&f)[NB][kPx][DIM],
                                           const float* __restrict__ cs,
                                           unsigned long long mask, int (&lab)[NB][kPx]) {
  constexpr int CS = cstride(DIM);
  float best[NB][kPx];
#pragma unroll
  for (int i = 0; i < NB; ++i)
#pragma unroll
    for (int j = 0; j < kPx; ++j) {
      best[i][j] = INFINITY;
      lab[i][j] = 0;
    }
  // ascending k over the two 32-bit halves of the mask
  unsigned m = (unsigned)mask, hi = (unsigned)(mask >> 32);
  int base = 0;
  for (;;) {
    if (!m) {
      if (!hi) break;
      m = hi;
      hi = 0;
      base = 32;
    }
    const int k = base + __ffs(m) - 1;
    m &= m - 1;
    const float4 c0 = *reinterpret_cast<const float4*>(cs + k * CS);
    const float cc[5] = {c0.x, c0.y, c0.z, c0.w, DIM == 5 ? cs[k * CS + 4] : 0.0f};
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int q = 0; q < kPx / 2; ++q) {
        const int a = 2 * q, b = 2 * q + 1;
        float2 t = fsub2(make_float2(f[i][a][0], f[i][b][0]), make_float2(cc[0], cc[0]));
        float2 d = fmul2(t, t);
#pragma unroll
        for (int dd = 1; dd < DIM; ++dd) {
          t = fsub2(make_float2(f[i][a][dd], f[i][b][dd]), make_float2(cc[dd], cc[dd]));
          d = ffma2(t, t, d);
        }
        if (d.x < best[i][a]) {
          best[i][a] = d.x;
          lab[i][a] = k;
        }
        if (d.y < best[i][b]) {
          best[i][b] = d.y;
          lab[i][b] = k;
        }
      }
  }
}

// Sums of N (4, 8 or 16) per-lane values over the warp, each in the butterfly
// order of warp_sum (so the same bits): at each level a lane keeps half of its
// values and sends the others, which takes N - 1 shuffles and a few instead of
// 5 N.  Lane l returns the sum of value l / (32 / N).
template <int N>
__device__ __forceinline__ float warp_sums(float (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i >= h) continue;
      const float send = upper ? v[i] : v[i + h];
      const float keep = upper ? v[i + h] : v[i];
      v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, o));
    }
  }
#pragma unroll
  for (int q = 32 / N / 2; q >= 1; q >>= 1)
    v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], q));
  return v[0];
}

// Warp-collective: add the per-lane sums `acc` (label l, warp-uniform) to the
// warp's shared slot.
template <int DIM>
__device__ __forceinline__ void flush_acc(Smem& sm, int warp, int l, const float (&acc)[DIM],
                                          int n) {
  constexpr int N = DIM == 3 ? 4 : 8;
  const int lane = threadIdx.x & 31;
  float v[N];
#pragma unroll
  for (int d = 0; d < N; ++d) v[d] = d < DIM ? acc[d < DIM ? d : 0] : 0.0f;
  v[DIM] = (float)n;
  const float s = warp_sums<N>(v);
  const int d = lane / (32 / N);
  __syncwarp();   // the slots may have been written by other lanes
  if (lane % (32 / N) == 0) {
    if (d < DIM)
      sm.acc[warp][l * kMaxDim + d] = __fadd_rn(sm.acc[warp][l * kMaxDim + d], s);
    else if (d == DIM)
      sm.cnt[warp][l] += (int)s;
  }
}

// A span's FP32 sum into the block's integer sums.
__device__ __forceinline__ void sum_to_fix(Smem& sm, int idx, float v, int* status) {
  if (!(fabsf(v) < kFixLimit)) set_status(status, SPLIT_ERR_OVERFLOW);
  fix_add(sm, idx, __float2ll_rn(__fmul_rn(v, kFixScale)));
}

// The end of a span: the warp's FP32 sums (its slots, one per label it met)
// rounded to fixed point and added into the block's integer sums, the slots
// cleared.  Each span's sums are converted on their own, so the totals do not
// depend on which block or pass took the span, nor in what order.
template <int DIM>
__device__ __forceinline__ void warp_to_fix(Smem& sm, int warp, int K, int* status) {
  __syncwarp();   // the lanes' slot updates are visible to the warp
  for (int k = threadIdx.x & 31; k < K; k += 32) {
    const int c = sm.cnt[warp][k];
    if (c == 0) continue;
    sm.cnt[warp][k] = 0;
    atomicAdd(&sm.fixn[k], c);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const float v = sm.acc[warp][k * kMaxDim + d];
      if (v == 0.0f) continue;
      sm.acc[warp][k * kMaxDim + d] = 0.0f;
      sum_to_fix(sm, k * kMaxDim + d, v, status);
    }
  }
  __syncwarp();
}

// The sums of a span whose pixels all carry one of two labels, straight into
// the block's integer sums: what flush_acc into empty slots and warp_to_fix
// would give.
template <int DIM>
__device__ __forceinline__ void pair_to_fix(Smem& sm, int ka, int kb, const float (&acc)[DIM],
                                            int n, const float (&acc2)[DIM], int n2,
                                            int* status) {
  constexpr int NV = DIM + 1;
  constexpr int N = 2 * NV <= 8 ? 8 : 16;
  const int lane = threadIdx.x & 31;
  float v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = 0.0f;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    v[d] = acc[d];
    v[NV + d] = acc2[d];
  }
  v[DIM] = (float)n;
  v[NV + DIM] = (float)n2;
  const float s = warp_sums<N>(v);
  const int i = lane / (32 / N);
  if (lane % (32 / N) != 0 || i >= 2 * NV || s == 0.0f) return;
  const int k = i < NV ? ka : kb, d = i < NV ? i : i - NV;
  if (d < DIM)
    sum_to_fix(sm, k * kMaxDim + d, s, status);
  else
    atomicAdd(&sm.fixn[k], (int)s);
}

// Accumulate one batch of x - c_label; labels below 0 mark pixels outside the
// image.  A batch of one label adds to the lanes' running sums; otherwise the
// batch's labels, in groups, are summed over the warp into their slots.
template <int DIM>
__device__ __forceinline__ void accumulate(Smem& sm, int warp, int K, const float (&f)[kPx][DIM],
                                           const int (&lab)[kPx], int& acc_l, int& acc_n,
                                           float (&acc)[DIM]) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  constexpr int CS = cstride(DIM);
  // the labels of the batch
  unsigned m0 = 0, m1 = 0;
#pragma unroll
  for (int j = 0; j < kPx; ++j) {
    const unsigned bit = 1u << (lab[j] & 31);
    if (lab[j] >= 0 && lab[j] < 32) m0 |= bit;
    if (lab[j] >= 32) m1 |= bit;
  }
  m0 = __reduce_or_sync(full, m0);
  if (K > 32) m1 = __reduce_or_sync(full, m1);
  const int nlab = __popc(m0) + __popc(m1);
  if (nlab == 0) return;
  if (nlab == 1) {
    const int l = m0 ? __ffs(m0) - 1 : 31 + __ffs(m1);
    if (l != acc_l) {
      if (acc_l >= 0) flush_acc<DIM>(sm, warp, acc_l, acc, acc_n);
      acc_l = l;
      acc_n = 0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) acc[d] = 0.0f;
    }
    float c[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) c[d] = sm.cent[l * CS + d];
#pragma unroll
    for (int j = 0; j < kPx; ++j) {
      if (lab[j] >= 0) {
        add_centered<DIM>(f[j], c, acc);
        ++acc_n;
      }
    }
    return;
  }
  if (acc_l >= 0) flush_acc<DIM>(sm, warp, acc_l, acc, acc_n);
  acc_l = -1;
  // each pixel's x - c_label
  float t[kPx][DIM];
#pragma unroll
  for (int j = 0; j < kPx; ++j) {
    const float* c = sm.cent + max(lab[j], 0) * CS;
#pragma unroll
    for (int d = 0; d < DIM; ++d) t[j][d] = __fsub_rn(f[j][d], c[d]);
  }
  constexpr int NV = DIM + 1;    // the sums and the count of a label
  constexpr int G = 16 / NV;     // labels of a group
  const int i = lane >> 1, g = i / NV, d = i - g * NV;   // what this lane receives
  while (m0 | m1) {
    float v[16];
    int mine = -1;
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = 0.0f;
#pragma unroll
    for (int q = 0; q < G; ++q) {
      int l = -2;
      if (m0) {
        l = __ffs(m0) - 1;
        m0 &= m0 - 1;
      } else if (m1) {
        l = 31 + __ffs(m1);
        m1 &= m1 - 1;
      }
      if (g == q) mine = l;
#pragma unroll
      for (int j = 0; j < kPx; ++j) {
        if (lab[j] == l) {
#pragma unroll
          for (int dd = 0; dd < DIM; ++dd) v[q * NV + dd] = __fadd_rn(v[q * NV + dd], t[j][dd]);
          v[q * NV + DIM] += 1.0f;
        }
      }
    }
    const float s = warp_sums<16>(v);
    __syncwarp();   // the slots may have been written by other lanes
    if ((lane & 1) == 0 && g < G && mine >= 0) {
      if (d < DIM)
        sm.acc[warp][mine * kMaxDim + d] = __fadd_rn(sm.acc[warp][mine * kMaxDim + d], s);
      else
        sm.cnt[warp][mine] += (int)s;
    }
  }
}

// ---- asynchronous copies into shared memory (no registers hold the data)
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Staging of the float4 fast path: per warp kStages batches of kPx x 32
// float4, pixel j of lane l at [j][l] (conflict-free copies and reads).  Four
// hold a whole span of a 64-row unit: its loads are all under way at once.
constexpr int kStages = 4;
constexpr int kStageFloat4 = kWarps * kStages * 4 * 32;   // float4 elements per block
constexpr size_t kStageBytes = (size_t)kStageFloat4 * 16;

// The lane's pixels when the candidates are exactly ka < kb: labels by the
// same distances, in the same order and with the same comparisons, as
// nearest_px over a two-bit mask, and each pixel's differences (those of its
// distance) added to the sums of its label, in pixel order.
template <int DIM>
__device__ __forceinline__ void pair_px(const float (&f)[kPx][DIM], const float* __restrict__ cs,
                                        int ka, int kb, int (&lab)[kPx], float (&acc)[DIM],
                                        int& acc_n, float (&acc2)[DIM], int& acc2_n) {
  constexpr int CS = cstride(DIM);
  float ca[DIM], cb[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    ca[d] = cs[ka * CS + d];
    cb[d] = cs[kb * CS + d];
  }
#pragma unroll
  for (int q = 0; q < kPx / 2; ++q) {
    float2 ta[DIM], tb[DIM], da, db;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const float2 x = make_float2(f[2 * q][d], f[2 * q + 1][d]);
      ta[d] = fsub2(x, make_float2(ca[d], ca[d]));
      tb[d] = fsub2(x, make_float2(cb[d], cb[d]));
      da = d == 0 ? fmul2(ta[0], ta[0]) : ffma2(ta[d], ta[d], da);
      db = d == 0 ? fmul2(tb[0], tb[0]) : ffma2(tb[d], tb[d], db);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float xa = h ? da.y : da.x, xb = h ? db.y : db.x;
      const bool finite = xa < INFINITY;
      const bool second = xb < (finite ? xa : INFINITY);
      const int l = second ? kb : finite ? ka : 0;
      lab[2 * q + h] = l;
      if (l == ka) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) acc[d] = __fadd_rn(acc[d], h ? ta[d].y : ta[d].x);
        ++acc_n;
      } else {
#pragma unroll
        for (int d = 0; d < DIM; ++d) acc2[d] = __fadd_rn(acc2[d], h ? tb[d].y : tb[d].x);
        ++acc2_n;
      }
    }
  }
}

// Labels of a whole fast span set to k (lane rows and columns as in a batch).
__device__ __forceinline__ void write_span_labels(const Image& im, int row_first, int col,
                                                  int nbatches, int k, bool vec_labels) {
  const int64_t step = (int64_t)kBatchRows * im.width;
  int64_t px0 = (int64_t)row_first * im.width + col;
  for (int b = 0; b < nbatches; ++b, px0 += step) {
    if (vec_labels) {
      *reinterpret_cast<int4*>(im.labels + px0) = make_int4(k, k, k, k);
    } else {
#pragma unroll
      for (int j = 0; j < kPx; ++j) im.labels[px0 + j] = k;
    }
  }
}

// Adds a single-candidate span's pixels to cluster k's sums of the unit, as
// the exact fixed-point sum of (x - c_k): S (the span's exact feature words,
// lane d holding dimension d) minus n * c_k * 2^24, rounded once (Smem::nc: a
// fast span always has the same n).  The same integers whether S was just summed from the pixels or
// kept from the first iteration, so a call's result does not depend on
// which; integer adds, so not on their order either.
template <int DIM>
__device__ __forceinline__ void add_span_sums(Smem& sm, int k, long long s_lane, int n) {
  const int lane = threadIdx.x & 31;
  if (lane < DIM) {
    fix_add(sm, k * kMaxDim + lane, s_lane - sm.nc[k * kMaxDim + lane]);
  } else if (lane == DIM) {
    atomicAdd(&sm.fixn[k], n);
  }
}

// Exact feature words of a span (2^-24 units): colour from the lanes' pixel
// sums `qc`, the xy features from the geometry (each lane's kPx columns in
// every batch row it covers); summed over the warp, lane d returns
// dimension d.
template <int DIM>
__device__ __forceinline__ long long span_words(const long long (&qc)[3], const float (&fx)[kPx],
                                                float xy_scale, int row_first, int nbatches) {
  const int lane = threadIdx.x & 31;
  long long w[DIM];
  w[0] = qc[0];
  w[1] = qc[1];
  w[2] = qc[2];
  if (DIM == 5) {
    long long qx = 0, qy = 0;
#pragma unroll
    for (int j = 0; j < kPx; ++j) qx += __float2ll_rn(__fmul_rn(fx[j], kFixScale));
    for (int b = 0; b < nbatches; ++b)
      qy += __float2ll_rn(
          __fmul_rn(__fmul_rn(xy_scale, (float)(row_first + b * kBatchRows)), kFixScale));
    w[DIM == 5 ? 3 : 0] = qx * nbatches;
    w[DIM == 5 ? 4 : 0] = qy * kPx;
  }
  long long mine = 0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      w[d] += (long long)__shfl_xor_sync(0xffffffffu, (unsigned long long)w[d], o);
    if (lane == d) mine = w[d];
  }
  return mine;
}

// How a span's candidate mask is used: one cluster (every pixel's label
// outright), two clusters with finite centroids (two running sums per lane),
// or any other mask (per-batch reduction by label).
enum SpanKind { kSpanSingle = 0, kSpanPair = 1, kSpanAny = 2 };

// The batches of a fast span (see fast_span).  For kSpanPair every pixel's
// label is ka or kb (finite features and centroids), so `acc` runs for ka
// and a second per-lane sum for kb, reduced once at the end of the span
// however often the two labels mix within its batches.
//
// A single-candidate span of a clustering adds its pixels' exact feature
// words instead of running FP32 sums, and keeps them in `entry` (if any);
// any other span given an `entry` (the first iteration's) also sums and keeps
// its words, besides its FP32 sums.
template <int LAYOUT, int DIM, int MODE, int KIND, bool FIRST>
__device__ __forceinline__ void span_batches(const Image& im, Smem& sm, int warp, int row_first,
                                             int col, int nbatches, unsigned long long mask,
                                             int ka, int kb, bool write_labels, bool vec_labels,
                                             int& acc_l, int& acc_n, float (&acc)[DIM],
                                             long long* entry, int* status) {
  constexpr int CS = cstride(DIM);
  constexpr bool kFixSingle = KIND == kSpanSingle && MODE == kCluster;
  // the first iteration also keeps the words of spans with several candidates
  const bool keep = MODE == kCluster && FIRST && KIND != kSpanSingle && entry != nullptr;
  long long qc[3] = {0, 0, 0};
  const int64_t step = (int64_t)kBatchRows * im.width;
  int64_t px0 = (int64_t)row_first * im.width + col;
  float acc2[DIM];
  int acc2_n = 0;
  if (KIND == kSpanPair) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) acc2[d] = 0.0f;
  }
  float fx[kPx];
#pragma unroll
  for (int j = 0; j < kPx; ++j) fx[j] = __fmul_rn(im.xy_scale, (float)(col + j));
  // float4: the next batch is copied into shared memory while this one runs.
  // Lane l copies batch pixels l + 32 j (each copy a contiguous 512 bytes of
  // one row) and reads its own pixels 4 l + j; slots are swizzled so that
  // both are free of bank conflicts.
  extern __shared__ float4 km_stage[];
  const int ln = threadIdx.x & 31;
  float4* stage = km_stage + warp * (kStages * kPx * 32);
  const int64_t gw = (int64_t)im.width;
  // batch pixel q = 64 r + c of the batch's first row (row_first - lrow)
  const float4* gb0 = static_cast<const float4*>(im.points) + (px0 - (int64_t)(ln / kLanesPerRow) * gw
                                                               - (ln % kLanesPerRow) * kPx);
  // slot(q) = (q & ~7) | ((q + (q >> 3)) & 7), in closed form for the lane's
  // copies (q = ln + 32 j) and reads (q = 4 ln + j)
  const int cs0 = (ln & ~7) + ((ln + (ln >> 3)) & 7), cs1 = cs0 ^ 4;
  const int rs0 = 8 * (ln >> 1), rt = (4 * ln + (ln >> 1)) & 7;
  // batch b into buffer b % kStages (an empty group past the end, so that
  // the groups in flight count batches)
  auto fetch = [&](int b) {
    if (b < nbatches) {
      const float4* g = gb0 + (int64_t)b * step + ln;
      float4* dst = stage + (b % kStages) * (kPx * 32);
      cp_async16(dst + cs0, g);
      cp_async16(dst + 32 + cs1, g + 32);
      cp_async16(dst + 64 + cs0, g + gw);
      cp_async16(dst + 96 + cs1, g + gw + 32);
    }
    cp_async_commit();
  };
  // RGB8: the next batches' words in registers, moved up as they are used
  RawPx<SPLIT_LAYOUT_RGB8, DIM> raw[kStages];
  if (LAYOUT == SPLIT_LAYOUT_FLOAT4) {
#pragma unroll
    for (int b = 0; b < kStages; ++b) fetch(b);
  } else {
#pragma unroll
    for (int b = 0; b < kStages; ++b) raw[b].load(im.points, im.npoints, px0 + b * step, b < nbatches ? kPx : 0);
  }
  for (int b = 0; b < nbatches; ++b, px0 += step) {
    float f[kPx][DIM];
    if (LAYOUT == SPLIT_LAYOUT_FLOAT4) {
      cp_async_wait<kStages - 1>();
      // the copies of the other lanes must have landed too
      __syncwarp();
      const float4* src = stage + (b % kStages) * (kPx * 32);
#pragma unroll
      for (int j = 0; j < kPx; ++j) {
        const float4 v = src[rs0 + ((rt + j) & 7)];
        f[j][0] = v.x;
        f[j][1] = v.y;
        f[j][2] = v.z;
      }
      __syncwarp();   // every lane has read the buffer that is refilled now
      fetch(b + kStages);
    } else {
      raw[0].features(0.0f, 0, 0, f);
#pragma unroll
      for (int i = 0; i + 1 < kStages; ++i) raw[i] = raw[i + 1];
      raw[kStages - 1].load(im.points, im.npoints, px0 + kStages * step, b + kStages < nbatches ? kPx : 0);
    }
    if (DIM == 5) {
      const float fy = __fmul_rn(im.xy_scale, (float)(row_first + b * kBatchRows));
#pragma unroll
      for (int j = 0; j < kPx; ++j) {
        f[j][3] = fx[j];
        f[j][4] = fy;
      }
    }
    if (kFixSingle || keep) {
#pragma unroll
      for (int j = 0; j < kPx; ++j)
#pragma unroll
        for (int c = 0; c < 3; ++c) qc[c] += __float2int_rn(__fmul_rn(f[j][c], kFixScale));
    }
    int lab[kPx];
    if (KIND == kSpanSingle) {
      // one candidate for the whole span: every pixel's argmin, no distances
#pragma unroll
      for (int j = 0; j < kPx; ++j) lab[j] = ka;
    } else if (KIND == kSpanPair) {
      // the distances, and the sums from the same differences
      pair_px<DIM>(f, sm.cent, ka, kb, lab, acc, acc_n, acc2, acc2_n);
    } else {
      nearest_px<DIM, 1>(reinterpret_cast<const float(&)[1][kPx][DIM]>(f), sm.cent, mask,
                         reinterpret_cast<int(&)[1][kPx]>(lab));
    }
    if (write_labels) {
      if (vec_labels) {
        *reinterpret_cast<int4*>(im.labels + px0) = make_int4(lab[0], lab[1], lab[2], lab[3]);
      } else {
#pragma unroll
        for (int j = 0; j < kPx; ++j) im.labels[px0 + j] = lab[j];
      }
    }
    if (MODE != kAssignOnly) {
      if (KIND == kSpanSingle) {
        // a clustering's single spans are summed exactly (after the loop)
        if (!kFixSingle) {
          const float* c = sm.cent + ka * CS;
#pragma unroll
          for (int j = 0; j < kPx; ++j) add_centered<DIM>(f[j], c, acc);
          acc_n += kPx;
        }
      } else if (KIND == kSpanAny) {
        accumulate<DIM>(sm, warp, im.K, f, lab, acc_l, acc_n, acc);
      }
    }
  }
  if (MODE != kAssignOnly && KIND == kSpanPair)
    pair_to_fix<DIM>(sm, ka, kb, acc, acc_n, acc2, acc2_n, status);
  if (kFixSingle || keep) {
    const long long w = span_words<DIM>(qc, fx, im.xy_scale, row_first, nbatches);
    if (FIRST && entry && (threadIdx.x & 31) < DIM) __stcg(entry + (threadIdx.x & 31), w);
    if (kFixSingle) add_span_sums<DIM>(sm, ka, w, 32 * kPx * nbatches);
  }
}


// A warp span that lies wholly inside the image, with packed features (float4,
// or RGB8 read as the up to four 32-bit words that hold 4 pixels) and a candidate mask known
// for the whole span: no per-pixel bounds checks, one pointer step per batch,
// the column feature hoisted.  Results equal the general path's labels; the
// sums are the same pixels' in a fixed, data-dependent order.  Returns whether
// those sums have gone into the block's (kSpanAny leaves its in the slots).
//
// In a clustering, `entry` is the span's slot of kept feature words (or
// null).  Iteration 0 writes it for every span; in later iterations a span
// with one candidate reads it back instead of its pixels: its labels are
// that candidate's (written when asked) and its sums are exact integers, so
// nothing else needs the pixels.
template <int LAYOUT, int DIM, int MODE, bool FIRST>
__device__ __forceinline__ bool fast_span(const Image& im, Smem& sm, int warp, int row_first,
                                          int col, int nbatches, unsigned long long mask,
                                          bool write_labels, bool vec_labels, int& acc_l,
                                          int& acc_n, float (&acc)[DIM], long long* entry,
                                          int* status) {
  constexpr int CS = cstride(DIM);
  // A mask with one cluster names every pixel's nearest centroid outright:
  // the span's box excludes all others for every pixel it holds (and the
  // features of this path lie in the unit cube, so none is NaN).
  int kind = kSpanAny, ka = -1, kb = -1;
  if (mask != 0ull && (mask & (mask - 1ull)) == 0ull) {
    kind = kSpanSingle;
    ka = __ffsll((long long)mask) - 1;
  } else if (MODE != kAssignOnly && __popcll((long long)mask) == 2) {
    const int a = __ffsll((long long)mask) - 1, b = 63 - __clzll((long long)mask);
    const bool fin = ((sm.finite[a >> 5] >> (a & 31)) & (sm.finite[b >> 5] >> (b & 31)) & 1u) != 0u;
    if (fin) {
      kind = kSpanPair;
      ka = a;
      kb = b;
    }
  }
  if (MODE == kCluster && !FIRST && kind == kSpanSingle && entry) {
    const int lane = threadIdx.x & 31;
    add_span_sums<DIM>(sm, ka, lane < DIM ? __ldcg(entry + lane) : 0ll, 32 * kPx * nbatches);
    if (write_labels) write_span_labels(im, row_first, col, nbatches, ka, vec_labels);
    return true;
  }
  if (kind == kSpanSingle)
    span_batches<LAYOUT, DIM, MODE, kSpanSingle, FIRST>(im, sm, warp, row_first, col, nbatches, mask, ka,
                                                 kb, write_labels, vec_labels, acc_l, acc_n, acc,
                                                 entry, status);
  else if (kind == kSpanPair)
    span_batches<LAYOUT, DIM, MODE, kSpanPair, FIRST>(im, sm, warp, row_first, col, nbatches, mask, ka,
                                               kb, write_labels, vec_labels, acc_l, acc_n, acc,
                                               entry, status);
  else
    span_batches<LAYOUT, DIM, MODE, kSpanAny, FIRST>(im, sm, warp, row_first, col, nbatches, mask, ka,
                                              kb, write_labels, vec_labels, acc_l, acc_n, acc,
                                              entry, status);
  return MODE == kCluster && kind != kSpanAny;
}

// Whether the features are xy ones with colour known to lie in [0, 1].  A batch
// reads byte / 255 features from the bytes, and its float4 ones (Lab + beta) do
// not lie there.
template <int LAYOUT, int DIM, bool BATCH>
__device__ __forceinline__ bool unit_features(const Image& im) {
  return DIM == 5 && (LAYOUT == SPLIT_LAYOUT_RGB8 ||
                      (LAYOUT == SPLIT_LAYOUT_FLOAT4 && !BATCH && im.unit_range));
}

// Whether a warp span takes the fast path: unit features and the whole span inside
// the image.  Plain RGB8 asks for 4-pixel-aligned rows too: the loads take any
// alignment, but which spans are summed exactly decides that layout's last bits.
// It depends only on the geometry and the layout, so a span is fast in every
// iteration or in none.
template <int LAYOUT, int DIM, int MODE, bool BATCH>
__device__ __forceinline__ bool fast_geometry(const Image& im, int row0, int col0, int wrows,
                                              bool vec_labels) {
  return MODE != kUpdateOnly && unit_features<LAYOUT, DIM, BATCH>(im) && row0 + wrows <= im.height &&
         col0 + kTile <= im.width &&
         (LAYOUT == SPLIT_LAYOUT_FLOAT4 ||
          (LAYOUT == SPLIT_LAYOUT_RGB8 &&
           (im.any_width ||
            (vec_labels && (reinterpret_cast<uintptr_t>(im.points) & 3) == 0))));
}

// The candidate mask of a span with xy features and colour in [0, 1]: the
// box is exact without the pixels.
template <int DIM>
__device__ __forceinline__ unsigned long long unit_box_mask(const Image& im, const Smem& sm,
                                                            int row0, int col0, int rows_in,
                                                            int cols_in) {
  float lo[DIM], hi[DIM];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = 0.0f;
    hi[d] = 1.0f;
  }
  lo[DIM == 5 ? 3 : 0] = __fmul_rn(im.xy_scale, (float)col0);
  hi[DIM == 5 ? 3 : 0] = __fmul_rn(im.xy_scale, (float)(col0 + cols_in - 1));
  lo[DIM == 5 ? 4 : 0] = __fmul_rn(im.xy_scale, (float)row0);
  hi[DIM == 5 ? 4 : 0] = __fmul_rn(im.xy_scale, (float)(row0 + rows_in - 1));
  return candidates<DIM>(lo, hi, sm.cent, im.K);
}

// One warp span: rows srow * wrows .. + wrows of tile column tx (wrows =
// unit_rows / kWarps; a unit, a 64-column tile of unit_rows rows, is the
// spans of its kWarps warps): assign (unless update-only) and accumulate the
// calling warp's sums of (x - c_label).  A batch is 2 rows x 64 columns, each
// lane holding kPx consecutive pixels of a row.
//
// Candidate clusters: with xy features and colour features known to lie in
// [0, 1] the box of the warp's span is exact without touching the pixels, so
// one candidate mask serves all its batches.  Otherwise the colour box of
// every batch is measured (warp min / max) and joined with the batch's xy
// extent.
//
// While consecutive batches carry one label, every lane keeps a register
// running sum; a batch with several labels is reduced label by label in
// ascending order.  All orders depend only on the data.  The span's sums end
// in the block's integer sums (warp_to_fix).
//
// Returns whether the span needs its pixels in later iterations too (as long
// as its candidates stay the same).
// listed: span_mask is the span's candidate mask already (list_spans).
template <int LAYOUT, int DIM, int MODE, bool FIRST, bool BATCH>
__device__ __forceinline__ bool process_span(const Image& im, int srow, int tx, Smem& sm,
                                             bool write_labels, int* status,
                                             unsigned long long span_mask, bool listed) {
  const unsigned full = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int CS = cstride(DIM);
  constexpr bool kXY = DIM == 5 && LAYOUT != SPLIT_LAYOUT_PLANAR;
  const int wrows = im.unit_rows / kWarps;
  const int row0 = srow * wrows;
  const int col0 = tx * kTile;
  if (row0 >= im.height) return false;
  const int lrow = lane / kLanesPerRow, lcol = (lane % kLanesPerRow) * kPx;
  const int rows_in = min(wrows, im.height - row0);
  const int cols_in = min(kTile, im.width - col0);
  const bool unit_box = unit_features<LAYOUT, DIM, BATCH>(im);
  const bool vec_labels =
      (reinterpret_cast<uintptr_t>(MODE == kUpdateOnly ? im.labels_in : im.labels) & 15) == 0 &&
      (im.width % kPx) == 0;
  // (labels are stored one by one where a row's start is not 16-byte aligned)
  const bool fast = fast_geometry<LAYOUT, DIM, MODE, BATCH>(im, row0, col0, wrows, vec_labels);
  // slot (srow, tx) of a fast span's kept sums
  long long* entry = (fast && MODE == kCluster && im.span_sum)
                         ? im.span_sum + ((size_t)srow * im.span_cols + tx) * kSpanSums
                         : nullptr;

  if (MODE != kUpdateOnly && unit_box && !listed)
    span_mask = unit_box_mask<DIM>(im, sm, row0, col0, rows_in, cols_in);

  int acc_l = -1, acc_n = 0;
  float acc[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) acc[d] = 0.0f;

  bool direct = false;   // the sums are in the block's already
  if (fast)
    direct = fast_span<LAYOUT, DIM, MODE, FIRST>(im, sm, warp, row0 + lrow, col0 + lcol, wrows / kBatchRows,
                                 span_mask, write_labels, vec_labels, acc_l, acc_n, acc,
                                        entry, status);
  // the lane's pixels inside the image in the span's rows
  auto valid_px = [&](int row) {
    const int64_t left = im.npoints - ((int64_t)row * im.width + col0 + lcol);
    return row < im.height ? (int)max((int64_t)0, min((int64_t)min(kPx, im.width - col0 - lcol), left))
                           : 0;
  };
  // Three-dimensional features: two batches per step share the box, the
  // candidates and the walk over them, whose latencies (box 0.2 us, candidates
  // 0.2 us, 0.1 us a candidate) are most of a step; more dimensions do not fit
  // the registers.  The next step's loads go out before this one is examined.
  constexpr int NB = DIM == 3 ? 2 : 1;
  const int nb = fast ? 0 : (rows_in + kBatchRows - 1) / kBatchRows;
  const int col = col0 + lcol;
  RawPx<LAYOUT, DIM> raw[NB];
  int valid_next[NB];
  auto load = [&](int b) {
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int row = row0 + (b + i) * kBatchRows + lrow;
      valid_next[i] = b + i < nb ? valid_px(row) : 0;
      raw[i].load(im.points, im.npoints, (int64_t)row * im.width + col, valid_next[i]);
    }
  };
  if (!fast) load(0);
  for (int b = 0; b < nb; b += NB) {
    float f[NB][kPx][DIM];
    int valid[NB], lab[NB][kPx];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      valid[i] = valid_next[i];
      raw[i].features(im.xy_scale, row0 + (b + i) * kBatchRows + lrow, col, f[i]);
    }
    if (b + NB < nb) load(b + NB);
    if (MODE == kUpdateOnly) {
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int64_t px0 = (int64_t)(row0 + (b + i) * kBatchRows + lrow) * im.width + col;
        if (valid[i] == kPx && vec_labels) {
          const int4 v = __ldg(reinterpret_cast<const int4*>(im.labels_in + px0));
          lab[i][0] = v.x; lab[i][1] = v.y; lab[i][2] = v.z; lab[i][3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < kPx; ++j) lab[i][j] = j < valid[i] ? __ldg(im.labels_in + px0 + j) : -1;
        }
#pragma unroll
        for (int j = 0; j < kPx; ++j)
          if (j >= valid[i] || lab[i][j] < 0 || lab[i][j] >= im.K) lab[i][j] = -1;
      }
    } else {
      unsigned long long mask = span_mask;
      if (!unit_box) {
        // Box of the step's pixels.  fminf / fmaxf skip NaN: a NaN pixel gets
        // label 0 whatever the mask (every distance compares false), and the
        // box still bounds all other pixels.
        float lo[DIM], hi[DIM];
        constexpr int kBoxDims = kXY ? 3 : DIM;
#pragma unroll
        for (int d = 0; d < kBoxDims; ++d) {
          float a = INFINITY, z = -INFINITY;
#pragma unroll
          for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int j = 0; j < kPx; ++j) {
              if (j < valid[i]) {
                a = fminf(a, f[i][j][d]);
                z = fmaxf(z, f[i][j][d]);
              }
            }
          lo[d] = fkey_inv(__reduce_min_sync(full, fkey(a)));
          hi[d] = fkey_inv(__reduce_max_sync(full, fkey(z)));
        }
        if (kXY) {
          const int r0 = row0 + b * kBatchRows;
          lo[3] = __fmul_rn(im.xy_scale, (float)col0);
          hi[3] = __fmul_rn(im.xy_scale, (float)(col0 + cols_in - 1));
          lo[4] = __fmul_rn(im.xy_scale, (float)r0);
          hi[4] = __fmul_rn(im.xy_scale, (float)min(r0 + NB * kBatchRows - 1, im.height - 1));
        }
        mask = candidates<DIM>(lo, hi, sm.cent, im.K);
      }
      if (unit_box && mask != 0ull && (mask & (mask - 1ull)) == 0ull) {
        // one candidate for the span names every pixel's label (features in
        // the unit cube: none is NaN), as on the fast path
        const int k1 = __ffsll((long long)mask) - 1;
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
          for (int j = 0; j < kPx; ++j) lab[i][j] = k1;
      } else {
        nearest_px<DIM, NB>(f, sm.cent, mask, lab);
      }
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int64_t px0 = (int64_t)(row0 + (b + i) * kBatchRows + lrow) * im.width + col;
        if (write_labels) {
          if (valid[i] == kPx && vec_labels) {
            *reinterpret_cast<int4*>(im.labels + px0) =
                make_int4(lab[i][0], lab[i][1], lab[i][2], lab[i][3]);
          } else {
#pragma unroll
            for (int j = 0; j < kPx; ++j)
              if (j < valid[i]) im.labels[px0 + j] = lab[i][j];
          }
        }
#pragma unroll
        for (int j = 0; j < kPx; ++j)
          if (j >= valid[i]) lab[i][j] = -1;
      }
    }
    if (MODE == kAssignOnly) continue;
#pragma unroll
    for (int i = 0; i < NB; ++i)
      accumulate<DIM>(sm, warp, im.K, f[i], lab[i], acc_l, acc_n, acc);
  }
  if (MODE != kAssignOnly && !direct) {
    if (acc_l >= 0) flush_acc<DIM>(sm, warp, acc_l, acc, acc_n);
    warp_to_fix<DIM>(sm, warp, im.K, status);
  }
  return !entry || (span_mask & (span_mask - 1ull)) != 0ull;
}

// Adds the block's integer sums into the image accumulators (96-bit fixed
// point: low 32 bits and the signed rest in two 64-bit words) and clears
// them.
__device__ void block_to_accum(Smem& sm, const Params& p, int img, int K, int dim, int slot) {
  __syncthreads();
  if (threadIdx.x == 0) {
    sm.nheavy = 0;
    sm.next_heavy = 0;
  }
  unsigned long long* lo = p.acc_lo + acc_slot(p, slot, img) * (kMaxK * kMaxDim);
  unsigned long long* hi = p.acc_hi + acc_slot(p, slot, img) * (kMaxK * kMaxDim);
  for (int idx = threadIdx.x; idx < K * kMaxDim; idx += blockDim.x) {
    const unsigned wlo = sm.fix_lo[idx], whi = sm.fix_hi[idx];
    if ((wlo | whi) == 0u) continue;
    const long long q = (long long)(((unsigned long long)whi << 32) | wlo);
    sm.fix_lo[idx] = 0u;
    sm.fix_hi[idx] = 0u;
    if ((idx % kMaxDim) < dim) {
      atomicAdd(lo + idx, (unsigned long long)q & 0xffffffffull);
      atomicAdd(hi + idx, (unsigned long long)(q >> 32));
    }
  }
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const int c = sm.fixn[k];
    sm.fixn[k] = 0;
    if (c) atomicAdd(p.acc_cnt + acc_slot(p, slot, img) * kMaxK + k, (unsigned)c);
  }
}

// n * c * 2^24 rounded once: n = span rows * kTile is a power of two, so the
// product is exact in FP32 (FP64 runs at two lanes per clock here)
__device__ __forceinline__ long long span_centre(const Image& im, float c) {
  return __float2ll_rn(__fmul_rn(c, (float)(im.unit_rows / kWarps * kTile) * kFixScale));
}

// Smem::bound and Smem::finite of centroid k < kMaxK (two whole warps call
// this): the first three steps of the fma chains of candidates() over lo = 0,
// hi = 1, and the centroid's xy.
__device__ __forceinline__ void set_bounds(Smem& sm, int k, int K, const float* src, int stride) {
  bool fin = false;
  if (k < K) {
    float c[5], l = 0.0f, u = 0.0f;
    fin = true;
#pragma unroll
    for (int d = 0; d < 5; ++d) {
      c[d] = src[k * stride + d];
      fin = fin && isfinite(c[d]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float g = fmaxf(fmaxf(0.0f - c[d], c[d] - 1.0f), 0.0f);
      const float e = fmaxf(c[d] - 0.0f, 1.0f - c[d]);
      l = __fmaf_rn(g, g, l);
      u = __fmaf_rn(e, e, u);
    }
    sm.bound[k] = make_float4(l, u, c[3], c[4]);
  }
  const unsigned m = __ballot_sync(0xffffffffu, fin);
  if ((k & 31) == 0) sm.finite[k >> 5] = m;
}

// The centroids of slot `src` into shared memory (strides cstride(DIM) there,
// 8 in the slot).
template <int DIM>
__device__ __forceinline__ void load_centroids(const Image& im, const float* src, Smem& sm) {
  constexpr int CS = cstride(DIM);
  for (int idx = threadIdx.x; idx < im.K * CS; idx += blockDim.x) {
    const int k = idx / CS, d = idx % CS;
    const float c = d < DIM ? __ldcg(src + k * 8 + d) : 0.0f;
    sm.cent[idx] = c;
    if (d < DIM) sm.nc[k * kMaxDim + d] = span_centre(im, c);
  }
  if (DIM == 5 && threadIdx.x < kMaxK) set_bounds(sm, threadIdx.x, im.K, src, 8);
}

// The squared "centroid shift" as the reference's cluster() measures it
// (cluster.cu:40-50, :73-87): it keeps the previous centroids at float
// offset 2N of its workspace, but within the same iteration label_points
// writes its N x K distance matrix from offset 0 (label.cu:80-88, entry
// i * K + c = distance of point i to centroid c, Norm2 at label.cu:23-32) and
// calculate_centroids writes its K reciprocal cluster sizes at offset 2N
// (centroids.cu:40-63).  So the words it compares the new centroids with
// (planar, entry j = d * K + k) are
//   j < K:  1 / n_j (the reciprocal size of cluster j, FP32 division);
//   j >= K: the distance of point (2N + j) / K to centroid (2N + j) % K of
//           the iteration's input, sum of squares in dimension order;
// and the shift is the FP32 sum of (c_new[j] - word[j])^2 in j order.  Only
// the reference's 3-D case is defined, and only for K >= 3 (smaller K would
// read words no call of the iteration wrote).
template <int LAYOUT, int DIM>
__device__ float reference_shift(const Image& im, const float* cent, const float* c_old,
                                 const unsigned* cnt) {
  constexpr int CS = cstride(DIM);
  Loader<LAYOUT, DIM> ld{im.points, im.npoints, im.xy_scale};
  const int64_t base = 2 * im.npoints;
  float acc = 0.0f;
  for (int j = 0; j < im.K * 3; ++j) {
    const int d = j / im.K, k = j % im.K;
    float word;
    if (j < im.K) {
      word = __fdiv_rn(1.0f, (float)__ldcg(cnt + j));
    } else {
      const int64_t e = base + j;
      const int64_t px = e / im.K;
      const int c = (int)(e % im.K);
      float f[DIM];
      ld.load(px, 0, 0, f);
      const float a0 = __fsub_rn(f[0], __ldcg(c_old + c * 8 + 0));
      const float a1 = __fsub_rn(f[1], __ldcg(c_old + c * 8 + 1));
      const float a2 = __fsub_rn(f[2], __ldcg(c_old + c * 8 + 2));
      word = __fadd_rn(__fadd_rn(__fmul_rn(a0, a0), __fmul_rn(a1, a1)), __fmul_rn(a2, a2));
    }
    const float t = __fsub_rn(cent[k * CS + d], word);
    acc = __fadd_rn(acc, __fmul_rn(t, t));
  }
  return acc;
}

// Centroids of iteration i >= 1 of an image, c(i) = c(i-1) + S(i-1) / n
// (empty cluster: unchanged; cluster.cu:71-88), formed after the grid barrier
// that ended iteration i - 1, and the convergence test of that iteration.
//
// Its inputs are not written during iteration i, so every block that calls it
// gets bit-identical centroids and the same decision.  Of a single image
// (LOCAL) every block calls it every iteration, and c(i-1) and the last shift
// are where the last call left them, in shared memory: one round of loads
// (the sums) is all it waits for.  Of a batch the blocks that work on the
// image call it, and read those from the slots of iteration i - 1 (c(i-1) in
// cur[(i-1) & 1], the shift in state[(i-1) & 1]).  The sums are in slot
// (i-1) % 3.  The owner publishes: c(i) to cur[i & 1], the shift to state[i &
// 1], zeros for sums slot (i+1) % 3 (read for the last time in iteration i-1,
// written again in iteration i+1), and on convergence the caller's centroids
// and iteration count.  Returns whether the image runs iteration i (uniform
// in the block); its centroids are left in sm.cent (stride cstride(DIM)).
template <int LAYOUT, int DIM, int MODE, bool LOCAL>
__device__ bool form_centroids(const Params& p, int img, const Image& im, int i, Smem& sm,
                               bool owner) {
  constexpr int CS = cstride(DIM);
  ImageState* next = p.state + acc_slot(p, i & 1, img);
  const size_t sb = acc_slot(p, (i - 1) % 3, img);
  const unsigned long long* lo = p.acc_lo + sb * (kMaxK * kMaxDim);
  const unsigned long long* hi = p.acc_hi + sb * (kMaxK * kMaxDim);
  const unsigned* cnt = p.acc_cnt + sb * kMaxK;
  const float* c_old = p.cur + acc_slot(p, (i - 1) & 1, img) * (kMaxK * 8);
  float* c_new = p.cur + acc_slot(p, i & 1, img) * (kMaxK * 8);
  if (!LOCAL && threadIdx.x == kThreads - 1) {
    sm.delta = __ldcg(&p.state[acc_slot(p, (i - 1) & 1, img)].delta);
    sm.stopped = __ldcg(&p.state[img].done);
  }
  for (int idx = threadIdx.x; idx < im.K * DIM; idx += blockDim.x) {
    const int k = idx / DIM, d = idx % DIM, a = k * kMaxDim + d;
    const unsigned n = __ldcg(cnt + k);
    const unsigned long long l = __ldcg(lo + a), h = __ldcg(hi + a);
    const float c = LOCAL ? sm.cent[k * CS + d] : __ldcg(c_old + k * 8 + d);
    float cn = c;
    if (n > 0) {
      // S = (hi * 2^32 + lo) * 2^-24: one FP64 rounding of the exact sum,
      // one to FP32 (the scaling by 2^-24 is exact); then c + S / n in FP32
      // (every block forms all K x D values, so the FP64 pipe is kept to the
      // conversion: a division there costs the iteration about a microsecond)
      const double S64 = __fma_rn((double)(long long)h, 4294967296.0, (double)l);
      const float S = __fmul_rn(__double2float_rn(S64), 1.0f / 16777216.0f);
      cn = __fadd_rn(c, __fdiv_rn(S, (float)n));
    }
    sm.cent[k * CS + d] = cn;
    sm.nc[a] = span_centre(im, cn);
    const float df = __fsub_rn(cn, c);
    sm.sdiff[idx] = __fmul_rn(df, df);
  }
  __syncthreads();
  if (!LOCAL && sm.stopped) {
    __syncthreads();
    return false;
  }
  if (DIM == 5 && threadIdx.x >= kThreads - kMaxK)
    set_bounds(sm, (int)threadIdx.x - (kThreads - kMaxK), im.K, sm.cent, CS);
  if (owner && threadIdx.x >= 32) {
    const size_t zb = acc_slot(p, (i + 1) % 3, img);
    const int t = (int)threadIdx.x - 32, nt = (int)blockDim.x - 32;
    for (int idx = t; idx < im.K * DIM; idx += nt)
      __stcg(c_new + (idx / DIM) * 8 + idx % DIM, sm.cent[(idx / DIM) * CS + idx % DIM]);
    for (int idx = t; idx < im.K * kMaxDim; idx += nt) {
      __stcg(p.acc_lo + zb * (kMaxK * kMaxDim) + idx, 0ull);
      __stcg(p.acc_hi + zb * (kMaxK * kMaxDim) + idx, 0ull);
    }
    for (int k = t; k < im.K; k += nt) __stcg(p.acc_cnt + zb * kMaxK + k, 0u);
    if (!LOCAL && t == 0) __stcg(cost_at(p, img, i + 1), 0);
  }
  if (threadIdx.x < 32) {
    // squared centroid shift, summed in a fixed order
    float acc = 0.0f;
    for (int idx = threadIdx.x; idx < im.K * DIM; idx += 32) acc = __fadd_rn(acc, sm.sdiff[idx]);
    acc = warp_sum(acc);
    if (DIM == 3 && im.ref_shift && threadIdx.x == 0)
      acc = reference_shift<LAYOUT, DIM>(im, sm.cent, c_old, cnt);
    if (threadIdx.x == 0) {
      const float delta = sqrtf(acc);
      bool more = i < im.max_iter && fabsf(delta - sm.delta) > im.threshold;
      if (MODE == kUpdateOnly) more = false;
      sm.more = more ? 1 : 0;
      sm.delta = delta;
      if (owner) {
        next->delta = delta;
        if (!more) p.state[img].done = i;
        if (im.d_iterations && !more) *im.d_iterations = i;
      }
    }
  }
  __syncthreads();
  const bool more = sm.more != 0;
  if (!more) {
    // final centroids back to the caller's planar array
    if (owner)
      for (int idx = threadIdx.x; idx < im.K * DIM; idx += blockDim.x)
        im.centroids[(idx % DIM) * im.K + idx / DIM] = sm.cent[(idx / DIM) * CS + idx % DIM];
    __syncthreads();
  }
  return more;
}

// The spans a block takes of an image in an iteration: place j < count is
// span first + j * step of the image (mod nspans when SCATTER; from the other
// end when `back`).
template <bool SCATTER>
struct SpanShare {
  int first, step, count;
  bool back;
  int nspans, ntx;
  __device__ __forceinline__ void at(int j, int& srow, int& tx) const {
    int v = SCATTER ? (int)(((long long)first + (long long)j * step) % nspans) : first + j * step;
    if (back) v = nspans - 1 - v;
    srow = v / ntx;
    tx = v - srow * ntx;
  }
};
// Places [w0, w1) of the block's share after the first iteration, a lane each:
// classified from the geometry alone (the bounds and the test of candidates(),
// one centroid after the other, so that a warp bounds 32 spans at a time).  A
// span with one candidate is finished: its kept words are added and, when
// asked, its labels written.  The others are listed.  With a warp per span
// this took 4.5 us of a 4K iteration, now 2.1.
template <int LAYOUT, int DIM, int MODE, bool BATCH>
__device__ __forceinline__ void list_spans(Smem& sm, const Image& im,
                                           const SpanShare<BATCH>& share, int w0, int w1,
                                           bool wl) {
  constexpr unsigned full = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wrows = im.unit_rows / kWarps;
  const int rows = wrows / kBatchRows;
  const int lrow = lane / kLanesPerRow, lcol = (lane % kLanesPerRow) * kPx;
  const bool vec_labels = (reinterpret_cast<uintptr_t>(im.labels) & 15) == 0 && (im.width % kPx) == 0;
  const int per = (w1 - w0 + kWarps - 1) / kWarps;
  const int end = min(w0 + (warp + 1) * per, w1);
  for (int j0 = w0 + warp * per; j0 < end; j0 += 32) {
    const int j = j0 + lane;
    const bool mine = j < end;
    int sr = 0, tx = 0;
    if (mine) share.at(j, sr, tx);
    int k = -1;   // a light span's cluster
    unsigned long long mask = 0;
    if (mine) {
      const int row0 = sr * wrows, col0 = tx * kTile;
      const int rows_in = min(wrows, im.height - row0), cols_in = min(kTile, im.width - col0);
      const float lo3 = __fmul_rn(im.xy_scale, (float)col0);
      const float hi3 = __fmul_rn(im.xy_scale, (float)(col0 + cols_in - 1));
      const float lo4 = __fmul_rn(im.xy_scale, (float)row0);
      const float hi4 = __fmul_rn(im.xy_scale, (float)(row0 + rows_in - 1));
      float ub = INFINITY;
      for (int q = 0; q < im.K; ++q) {
        const float4 c = sm.bound[q];
        const float e3 = fmaxf(c.z - lo3, hi3 - c.z), e4 = fmaxf(c.w - lo4, hi4 - c.w);
        ub = fminf(ub, __fmaf_rn(e4, e4, __fmaf_rn(e3, e3, c.y)));
      }
      const float thr = ub * 1.0001f;
      for (int q = 0; q < im.K; ++q) {
        const float4 c = sm.bound[q];
        const float g3 = fmaxf(fmaxf(lo3 - c.z, c.z - hi3), 0.0f);
        const float g4 = fmaxf(fmaxf(lo4 - c.w, c.w - hi4), 0.0f);
        if (__fmaf_rn(g4, g4, __fmaf_rn(g3, g3, c.x)) <= thr) mask |= 1ull << q;
      }
      if (mask != 0ull && (mask & (mask - 1ull)) == 0ull &&
          fast_geometry<LAYOUT, DIM, MODE, BATCH>(im, row0, col0, wrows, vec_labels))
        k = __ffsll((long long)mask) - 1;
    }
    if (k >= 0) {
      const long long* e = im.span_sum + ((size_t)sr * im.span_cols + tx) * kSpanSums;
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        fix_add(sm, k * kMaxDim + d, __ldcg(e + d) - sm.nc[k * kMaxDim + d]);
      atomicAdd(&sm.fixn[k], wrows * kTile);
    }
    if (wl) {
      for (unsigned m = __ballot_sync(full, k >= 0); m; m &= m - 1) {
        const int g = __ffs(m) - 1;
        write_span_labels(im, __shfl_sync(full, sr, g) * wrows + lrow,
                          __shfl_sync(full, tx, g) * kTile + lcol, rows, __shfl_sync(full, k, g),
                          vec_labels);
      }
    }
    const unsigned heavy = __ballot_sync(full, mine && k < 0);
    if (heavy) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&sm.nheavy, __popc(heavy));
      base = __shfl_sync(full, base, 0);
      if ((heavy >> lane) & 1u) {
        const int slot = base + __popc(heavy & ((1u << lane) - 1u));
        sm.heavy[slot] = sr * im.ntx + tx;
        sm.heavy_mask[slot] = mask;
      }
    }
  }
}

// One iteration of the block's share of an image's spans.  There is no block
// barrier and no global traffic per span: warps take places j = warp, warp +
// kWarps, ..., each span's contribution is added to the block's integer sums,
// and those go to the image accumulators once, at the end.  A span's
// contribution does not depend on who takes it, so neither does the result.
//
// After the first iteration, where the fast spans' sums are kept, most spans
// need none of their pixels (one candidate: labels and sums known): the warps
// finish those at once and list the others; the block's warps then take the
// listed spans one at a time.
template <int LAYOUT, int DIM, int MODE, bool BATCH>
__device__ __forceinline__ void span_pass(const Params& p, Smem& sm, const Image& im, int img,
                                          const SpanShare<BATCH>& share, int it) {
  constexpr unsigned full = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool wl = MODE == kAssignOnly ||
                  (MODE == kCluster && (im.threshold >= 0.0f || it == im.max_iter - 1));
  int* status = &p.hdr->status;
  if (MODE != kCluster || it == 0) {
    int counted = 0;
    for (int j = warp; j < share.count; j += kWarps) {
      int sr, tx;
      share.at(j, sr, tx);
      counted += process_span<LAYOUT, DIM, MODE, true, BATCH>(im, sr, tx, sm, wl, status, 0ull,
                                                              false);
    }
    if (BATCH) {
      // what the next iteration may cost: spans, and those that need pixels
      if (lane == 0 && counted) atomicAdd(&sm.counted, counted);
      __syncthreads();
      if (threadIdx.x == 0) {
        atomicAdd(cost_at(p, img, it), kPixelCost * sm.counted + share.count);
        sm.counted = 0;
      }
    }
  } else {
    // (with at most one span per warp nothing is gained by listing)
    const bool light =
        unit_features<LAYOUT, DIM, BATCH>(im) && im.span_sum && share.count > kWarps;
    for (int w0 = 0; w0 < share.count;) {
      const int w1 = light ? min(share.count, w0 + kHeavyCap) : share.count;
      if (light) {
        list_spans<LAYOUT, DIM, MODE, BATCH>(sm, im, share, w0, w1, wl);
        __syncthreads();
      }
      const int n = light ? sm.nheavy : w1;
      for (int own = warp;; own += kWarps) {
        int idx = own;
        if (light) {
          if (lane == 0) idx = atomicAdd(&sm.next_heavy, 1);
          idx = __shfl_sync(full, idx, 0);
        }
        if (idx >= n) break;
        int sr, tx;
        if (light) {
          const int s = sm.heavy[idx];
          sr = s / im.ntx;
          tx = s - sr * im.ntx;
        } else {
          share.at(idx, sr, tx);
        }
        process_span<LAYOUT, DIM, MODE, false, BATCH>(im, sr, tx, sm, wl, status,
                                               light ? sm.heavy_mask[idx] : 0ull, light);
      }
      w0 = w1;
      if (w0 < share.count) {   // another window
        __syncthreads();
        if (threadIdx.x == 0) sm.nheavy = sm.next_heavy = 0;
        __syncthreads();
      }
    }
  }
  if (MODE != kAssignOnly) block_to_accum(sm, p, img, im.K, DIM, it % 3);
}

__device__ __forceinline__ void clear_sums(Smem& sm) {
  for (int i = threadIdx.x; i < kWarps * kMaxK * kMaxDim; i += blockDim.x)
    (&sm.acc[0][0])[i] = 0.0f;
  for (int i = threadIdx.x; i < kWarps * kMaxK; i += blockDim.x) (&sm.cnt[0][0])[i] = 0;
  for (int i = threadIdx.x; i < kMaxK * kMaxDim; i += blockDim.x) sm.fix_lo[i] = sm.fix_hi[i] = 0u;
  for (int i = threadIdx.x; i < kMaxK; i += blockDim.x) sm.fixn[i] = 0;
  if (threadIdx.x == 0) {
    sm.nheavy = 0;
    sm.next_heavy = 0;
    sm.counted = 0;
    sm.delta = 0.0f;
  }
}

// A single image.  Block b takes the spans b, b + grid, ...; every block
// forms the centroids, so one grid barrier ends an iteration.
template <int LAYOUT, int DIM, int MODE>
__global__ void __launch_bounds__(kThreads, SG_KM_MINBLOCKS) kmeans_kernel(Params p) {
  __shared__ Smem sm;
  const Image& im = p.img0;
  clear_sums(sm);
  load_centroids<DIM>(im, p.cur, sm);
  __syncthreads();
  SpanShare<false> share;
  share.first = (int)blockIdx.x;
  share.step = (int)gridDim.x;
  share.count = (im.nspans - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  share.nspans = im.nspans;
  share.ntx = im.ntx;
  unsigned nbar = 0;   // grid barriers passed (every block passes the same ones)
  for (int it = 0; it < p.max_iter; ++it) {
    if (MODE != kAssignOnly && it > 0 &&
        !form_centroids<LAYOUT, DIM, MODE, true>(p, 0, im, it, sm, blockIdx.x == 0))
      return;   // converged: the same decision in every block
    // odd iterations go backwards: they start on what the last one left in L2
    share.back = (it & 1) != 0;
    span_pass<LAYOUT, DIM, MODE, false>(p, sm, im, 0, share, it);
    if (MODE == kAssignOnly) return;
    // the barrier publishes every block's sums (fire-and-forget adds ordered
    // by the block barrier before the arrival's release)
    if (!grid_barrier_counted(p.hdr, ++nbar, p.wait_limit, p.wait_skip)) return;
  }
  // centroids after the last iteration
  if (blockIdx.x == 0)
    form_centroids<LAYOUT, DIM, MODE, true>(p, 0, im, p.max_iter, sm, true);
}

// A batch.  In every iteration the running images, end to end, are cut into
// one range per block, equal in cost: an image costs a unit per span and
// kPixelCost more for each that needed its pixels in the iteration before.  A
// range meets few images, and its block forms their centroids itself, so one
// grid barrier ends an iteration here too.  A range's spans are scattered over
// the image (steps of about 0.618 nspans), so that it gets its share of the
// busy regions.
//
// What bounds it: an iteration waits for the block with the most spans that need
// their pixels, each one warp's pass (48 images, 54.7 Mpix, with the other
// stages: 3.0 ms).
constexpr int kSegCap = 128;   // images of a range listed at a time
struct RangeList {
  int n;
  int img[kSegCap + 2], begin[kSegCap + 2], end[kSegCap + 2];
  long long sums[kWarps];
  int count;
};

template <int LAYOUT, int DIM>
__global__ void __launch_bounds__(kThreads, kBatchMinBlocks) kmeans_batch_kernel(Params p) {
  __shared__ Smem sm;
  __shared__ RangeList rl;
  __shared__ Image im;
  clear_sums(sm);
  __syncthreads();
  auto take_image = [&](int img) {
    const int* src = reinterpret_cast<const int*>(p.images + img);
    if (threadIdx.x < sizeof(Image) / 4) reinterpret_cast<int*>(&im)[threadIdx.x] = src[threadIdx.x];
    __syncthreads();
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned nbar = 0;
  for (int it = 0;; ++it) {
    // the centroids of images whose last iteration was it - 1
    if (it > 0)
      for (int img = (int)blockIdx.x; img < p.nimages; img += gridDim.x) {
        if (p.images[img].max_iter != it) continue;
        take_image(img);
        form_centroids<LAYOUT, DIM, kCluster, false>(p, img, im, it, sm, true);
      }
    if (it >= p.max_iter) return;
    // the running images' cost up to each thread's images
    const int per = (p.nimages + kThreads - 1) / kThreads;
    const int i0 = min(p.nimages, (int)threadIdx.x * per), i1 = min(p.nimages, i0 + per);
    // (what a block pays to take up an image comes first: a range that holds the
    // end of one image and the start of another gets less of both)
    const long long fixed = it < 2 ? kImageSpans : kImageClocks >> 8;
    auto cost_of = [&](int img) -> long long {
      if (p.images[img].max_iter <= it) return 0;
      // stopped at the start of an iteration before this one (one that stops
      // in this iteration still has its spans in the ranges)
      const int done = __ldcg(&p.state[img].done);
      if (done != 0 && done < it) return 0;
      return fixed + (it == 0 ? p.images[img].first_cost : max(1, __ldcg(cost_at(p, img, it - 1))));
    };
    long long mine = 0;
    for (int i = i0; i < i1; ++i) mine += cost_of(i);
    long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) rl.sums[warp] = incl;
    if (threadIdx.x == 0) rl.count = 0;
    __syncthreads();
    long long before = incl - mine, total = 0;
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) before += rl.sums[w];
      total += rl.sums[w];
    }
    const long long p0 = total * blockIdx.x / gridDim.x;
    const long long p1 = total * (blockIdx.x + 1) / gridDim.x;
    // the images of the range; more than the list holds (many tiny images):
    // the range in windows that meet fewer
    long long window = p1 - p0;
    {
      int met = 0;
      long long x = before;
      for (int i = i0; i < i1 && x < p1; ++i) {
        const long long c = cost_of(i);
        met += c > 0 && x + c > p0;
        x += c;
      }
      if (met) atomicAdd(&rl.count, met);
      __syncthreads();
      if (rl.count > kSegCap) window = kSegCap;
    }
    for (long long w0 = p0; w0 < p1; w0 += window) {
      const long long w1 = min(p1, w0 + window);
      if (threadIdx.x == 0) rl.n = 0;
      __syncthreads();
      long long x = before;
      for (int i = i0; i < i1 && x < w1; ++i) {
        const long long c = cost_of(i);
        if (c > 0 && x + c > w0) {
          const long long n = p.images[i].nspans;
          // where the range cuts the image's spans
          auto cut = [&](long long w) {
            const long long in = min(max(w - x - fixed, 0ll), c - fixed);
            return (int)(in * n / (c - fixed));
          };
          const int a = cut(w0), b = cut(w1);
          if (a < b) {
            const int k = atomicAdd(&rl.n, 1);
            rl.img[k] = i;
            rl.begin[k] = a;
            rl.end[k] = b;
          }
        }
        x += c;
      }
      __syncthreads();
      const int nseg = rl.n;
      for (int k = 0; k < nseg; ++k) {
        const int img = rl.img[k];
        take_image(img);
        bool more = true;
        if (it > 0) {
          more = form_centroids<LAYOUT, DIM, kCluster, false>(p, img, im, it, sm,
                                                             rl.begin[k] == 0);
        } else {
          load_centroids<DIM>(im, p.cur + (size_t)img * (kMaxK * 8), sm);
          __syncthreads();
        }
        if (!more) continue;
        SpanShare<true> share;
        share.first = (int)((long long)rl.begin[k] * im.scatter % im.nspans);
        share.step = im.scatter;
        share.count = rl.end[k] - rl.begin[k];
        share.back = false;
        share.nspans = im.nspans;
        share.ntx = im.ntx;
        const unsigned began = clock();
        span_pass<LAYOUT, DIM, kCluster, true>(p, sm, im, img, share, it);
        if (it > 0 && threadIdx.x == 0)
          atomicAdd(cost_at(p, img, it), 1 + (int)(((unsigned)clock() - began) >> 8));
        __syncthreads();   // the image is replaced next
      }
    }
    if (!grid_barrier_counted(p.hdr, ++nbar, p.wait_limit, p.wait_skip)) return;
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct Layout {
  unsigned long long* acc_lo;
  unsigned long long* acc_hi;
  unsigned* acc_cnt;
  float* cur;
  ImageState* state;
  Image* images;
  long long* span_sum;   // single image: kept span feature words (after the rest)
  WsHeader* hdr;
  size_t bytes;
};

inline int height_of(int64_t n, int width) { return (int)((n + width - 1) / width); }
inline int tiles_x(int width) { return (width + kTile - 1) / kTile; }
// warp spans at a unit height of `rows`
inline int spans_of(int64_t n, int width, int rows) {
  const int wrows = rows / kWarps;
  return tiles_x(width) * ((height_of(n, width) + wrows - 1) / wrows);
}
// Fast spans of an image: full kTile-wide tile columns times full span-row
// slices at the smallest span height (2 rows, 16-row units), which bounds
// every unit height the tuning table may choose.
inline int64_t span_slots(int64_t n, int width) {
  return (int64_t)(width / kTile) * (height_of(n, width) / 2);
}

// The workspace holds per-image state (accumulators, centroids, counters),
// whose size does not depend on the image sizes, and optionally a single
// image's kept span sums (kSpanSums words per fast span, after the rest: a
// workspace without them runs the same clustering, reading every pixel in
// every iteration).
static Layout carve(void* ws, int nimages, int64_t span_entries = 0) {
  Carver c(ws);
  Layout l;
  l.hdr = c.take<WsHeader>(1);
  l.acc_lo = c.take<unsigned long long>((size_t)3 * nimages * kMaxK * kMaxDim);
  l.acc_hi = c.take<unsigned long long>((size_t)3 * nimages * kMaxK * kMaxDim);
  l.acc_cnt = c.take<unsigned>((size_t)3 * nimages * kMaxK);
  l.cur = c.take<float>((size_t)2 * nimages * kMaxK * 8);
  l.state = c.take<ImageState>((size_t)2 * nimages);
  l.images = nimages > 1 ? c.take<Image>((size_t)nimages) : nullptr;
  l.span_sum = span_entries > 0 ? c.take<long long>((size_t)span_entries * kSpanSums) : nullptr;
  l.bytes = c.size();
  return l;
}

// Header words used by the barrier and the work counters and all three
// accumulator slots start every call at zero (a call that stopped early, or
// a workspace used by another call, may have left data there).
static int reset_counters(const Layout& l, int nimages, cudaStream_t st) {
  (void)nimages;
  SG_CUDA_TRY(cudaMemsetAsync(reinterpret_cast<char*>(l.hdr) + sizeof(int), 0,
                              sizeof(unsigned) * 4, st));
  SG_CUDA_TRY(cudaMemsetAsync(l.acc_lo, 0, reinterpret_cast<char*>(l.cur) -
                                               reinterpret_cast<char*>(l.acc_lo), st));
  return SPLIT_OK;
}

// Per-image iteration state (cluster.cu:65-68: the shift starts at 0).
__global__ void init_kernel(Params p) {
  pdl_wait();
  for (int img = blockIdx.x * blockDim.x + threadIdx.x; img < p.nimages;
       img += gridDim.x * blockDim.x) {
    const Image& im = image_of(p, img);
    p.state[img] = ImageState{0.0f, 0, {0, 0}};
    p.state[p.nimages + img] = ImageState{0.0f, 0, {0, 0}};
    if (im.d_iterations && im.max_iter <= 0) *im.d_iterations = 0;
  }
}

// Per-call setup of a single-image clustering in one launch: the header's
// barrier and work counters and all three accumulator slots to zero
// (`zero` .. `zero` + zero_words: the slots and the counts), the iteration
// state (cluster.cu:65-68), and the caller's planar centroids into slot 0.  It is
// a composite call's first launch that writes to a stage's workspace.
template <int DIM>
__global__ void setup_kernel(Params p, unsigned* zero, int zero_words, StageHeaders own) {
  pdl_wait();
  const Image& im = p.img0;
  // (read at once, used at the end: nothing here waits for it)
  const unsigned long long last = threadIdx.x == 0 && own.hdr ? own.hdr->stamp : own.stamp;
  if (threadIdx.x == 0) {
    p.hdr->barrier_count = 0u;
    p.hdr->barrier_gen = 0u;
    p.hdr->stamp = kStampDirty;
    if (im.d_iterations && im.max_iter <= 0) *im.d_iterations = 0;
  }
  for (int i = threadIdx.x; i < zero_words; i += blockDim.x) zero[i] = 0u;
  for (int idx = threadIdx.x; idx < im.K * DIM; idx += blockDim.x) {
    const int k = idx / DIM, d = idx % DIM;
    p.cur[k * 8 + d] = im.centroids[d * im.K + k];
  }
  if (threadIdx.x == 0) enter_stages(own, last);
}

template <int DIM>
__global__ void load_user_centroids(Params p) {
  pdl_wait();
  for (int img = blockIdx.x; img < p.nimages; img += gridDim.x) {
    const Image& im = image_of(p, img);
    float* c0 = p.cur + (size_t)img * (kMaxK * 8);
    for (int idx = threadIdx.x; idx < im.K * DIM; idx += blockDim.x) {
      const int k = idx / DIM, d = idx % DIM;
      c0[k * 8 + d] = im.centroids[d * im.K + k];
    }
  }
}

// ---- tuning table (host side) ----------------------------------------------
// Per image size class: the unit height and the resident blocks per SM of
// the cooperative launch.  A unit height is chosen from the image's own pixel
// count, so an image gets the same reduction tree alone and in a batch.
struct TuneTable {
  std::mutex m;
  std::vector<split_tune_entry> e;
};
static TuneTable& tune_table() {
  static TuneTable t;
  return t;
}
split_tune_entry tuned(int64_t npix) {
  TuneTable& t = tune_table();
  std::lock_guard<std::mutex> g(t.m);
  for (const split_tune_entry& x : t.e)
    if (npix <= x.max_pixels) return x;
  return split_tune_entry{INT64_MAX, kTile, 0};
}

// The float4 kernels stage features in kStageBytes of dynamic shared memory,
// above the default 48 KB limit with their static part: the attribute is set
// once per device, before any launch (no stream work, so a graph capture may be
// under way).  A batch stages nothing (unit_features).
static int stage_attributes() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  SG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return SPLIT_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return SPLIT_OK;
  const void* kerns[] = {
      (const void*)kmeans_kernel<SPLIT_LAYOUT_FLOAT4, 5, kCluster>,
      (const void*)kmeans_kernel<SPLIT_LAYOUT_FLOAT4, 5, kAssignOnly>};
  for (const void* k : kerns)
    SG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kStageBytes));
  done[dev] = true;
  return SPLIT_OK;
}

template <int LAYOUT, int DIM, int MODE>
static int launch(Params& p, cudaStream_t st) {
  DeviceInfo di;
  SG_TRY(device_info(&di));
  auto kern = kmeans_kernel<LAYOUT, DIM, MODE>;
  if constexpr (MODE == kCluster)
    if (p.images) kern = kmeans_batch_kernel<LAYOUT, DIM>;
  // (3-D features never take the fast path, a batch's float4 ones neither)
  const size_t dyn =
      LAYOUT == SPLIT_LAYOUT_FLOAT4 && DIM == 5 && MODE != kUpdateOnly && !p.images ? kStageBytes
                                                                                    : 0;
  if (dyn) SG_TRY(stage_attributes());
  int per_sm = 0;
  SG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, dyn));
  if (per_sm < 1) return SPLIT_ERR_UNSUPPORTED;
  if (p.blocks_per_sm > 0 && p.blocks_per_sm < per_sm) per_sm = p.blocks_per_sm;
  int grid = di.sm_count * per_sm;
  // a block has kWarps warps, each taking spans
  grid = std::max(1, std::min(grid, (p.total_spans + kWarps - 1) / kWarps));
  if (MODE == kAssignOnly) {
    kern<<<grid, kThreads, dyn, st>>>(p);
    return launch_status();
  }
  void* args[] = {&p};
  SG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kThreads),
                                          args, dyn, st));
  return launch_status();
}

template <int MODE>
static int dispatch(int layout, int dim, Params& p, cudaStream_t st) {
#define SG_KM_CASE(L, D) \
  if (layout == L && dim == D) return launch<L, D, MODE>(p, st);
  SG_KM_CASE(SPLIT_LAYOUT_PLANAR, 3)
  SG_KM_CASE(SPLIT_LAYOUT_PLANAR, 5)
  SG_KM_CASE(SPLIT_LAYOUT_FLOAT4, 3)
  SG_KM_CASE(SPLIT_LAYOUT_FLOAT4, 5)
  SG_KM_CASE(SPLIT_LAYOUT_RGB8, 3)
  SG_KM_CASE(SPLIT_LAYOUT_RGB8, 5)
#undef SG_KM_CASE
  return SPLIT_ERR_INVALID;
}

static bool valid_features(const void* points, int layout, int dim, int64_t n,
                           int width, int K) {
  layout &= ~(SPLIT_FEATURES_UNIT_RANGE | SPLIT_KMEANS_REFERENCE_SHIFT);
  if (!points || n <= 0 || n > 0x7fffffffLL || K < 1 || K > kMaxK) return false;
  if (dim != 3 && dim != 5) return false;
  if (layout < SPLIT_LAYOUT_PLANAR || layout > SPLIT_LAYOUT_RGB8) return false;
  if (width < 1) return false;
  if (layout == SPLIT_LAYOUT_FLOAT4 && (reinterpret_cast<uintptr_t>(points) & 15)) return false;
  return true;
}

// Test setting of the grid barriers of single-image launches
// (split_kmeans_set_wait_test): poll limit (0: kSpinLimit) and skipping block.
static std::atomic<unsigned> g_wait_limit{0};
static std::atomic<int> g_wait_skip{-1};
static void wait_test(unsigned* limit, int* skip) {
  const unsigned l = g_wait_limit.load(std::memory_order_relaxed);
  *limit = l ? l : kSpinLimit;
  *skip = g_wait_skip.load(std::memory_order_relaxed);
}

static int run(int mode, const void* points, int layout, int dim, int64_t n,
               int width, float xy_scale, float* centroids,
               const float* centroids_in, int K, int32_t* labels,
               const int32_t* labels_in, void* ws, size_t ws_bytes, int max_iter,
               float threshold, int32_t* d_iter, cudaStream_t st, bool any_width = false,
               const StageHeaders& own = StageHeaders{}) {
  if (!valid_features(points, layout, dim, n, width, K)) return SPLIT_ERR_INVALID;
  const int unit_range = (layout & SPLIT_FEATURES_UNIT_RANGE) ? 1 : 0;
  const int ref_shift = (layout & SPLIT_KMEANS_REFERENCE_SHIFT) ? 1 : 0;
  layout &= ~(SPLIT_FEATURES_UNIT_RANGE | SPLIT_KMEANS_REFERENCE_SHIFT);
  // the reference's shift is defined for its own case only: 3-D clustering
  // with every word it reads inside the N x K distance matrix
  if (ref_shift && (mode != kCluster || dim != 3 || K < 3 || n * (K - 2) < 3 * (int64_t)K))
    return SPLIT_ERR_INVALID;
  const split_tune_entry te = tuned(n);
  const int spans = spans_of(n, width, te.kmeans_unit_rows);
  Layout l = carve(nullptr, 1);
  if (!ws || ws_bytes < l.bytes || (reinterpret_cast<uintptr_t>(ws) & 255))
    return SPLIT_ERR_WORKSPACE;
  // span sums for a clustering of more than one iteration, where the
  // workspace holds them
  const int64_t slots = span_slots(n, width);
  const bool keep = mode == kCluster && max_iter > 1 && slots > 0 &&
                    ws_bytes >= carve(nullptr, 1, slots).bytes;
  l = carve(ws, 1, keep ? slots : 0);
  Params p{};
  Image& im = p.img0;
  im.points = points;
  im.unit_range = unit_range;
  im.any_width = any_width;
  im.npoints = n;
  im.width = width;
  im.xy_scale = xy_scale;
  im.centroids = centroids;
  im.labels = labels;
  im.labels_in = labels_in;
  im.K = K;
  im.max_iter = max_iter;
  im.threshold = threshold;
  im.d_iterations = d_iter;
  im.nspans = spans;
  im.height = height_of(n, width);
  im.ntx = tiles_x(width);
  im.unit_rows = te.kmeans_unit_rows;
  im.ref_shift = ref_shift;
  im.span_sum = l.span_sum;
  im.span_cols = width / kTile;
  p.blocks_per_sm = te.kmeans_blocks_per_sm;
  wait_test(&p.wait_limit, &p.wait_skip);
  p.nimages = 1;
  p.images = nullptr;
  p.total_spans = spans;
  p.max_iter = max_iter;
  p.acc_lo = l.acc_lo;
  p.acc_hi = l.acc_hi;
  p.acc_cnt = l.acc_cnt;
  p.cur = l.cur;
  p.state = l.state;
  p.hdr = l.hdr;
  (void)centroids_in;
  // counters, accumulator slots, state and centroids in one launch (the
  // slots and counts lie between acc_lo and cur, 256-byte aligned pieces)
  unsigned* zero = reinterpret_cast<unsigned*>(l.acc_lo);
  const int zero_words = (int)((reinterpret_cast<char*>(l.cur) -
                                reinterpret_cast<char*>(l.acc_lo)) / sizeof(unsigned));
  if (dim == 3) launch_pdl(setup_kernel<3>, dim3(1), dim3(256), 0, st, p, zero, zero_words, own);
  else launch_pdl(setup_kernel<5>, dim3(1), dim3(256), 0, st, p, zero, zero_words, own);
  SG_TRY(launch_status());
  if (max_iter <= 0) return SPLIT_OK;
  if (mode == kCluster) return dispatch<kCluster>(layout, dim, p, st);
  if (mode == kUpdateOnly) return dispatch<kUpdateOnly>(layout, dim, p, st);
  return dispatch<kAssignOnly>(layout, dim, p, st);
}

}  // namespace km
}  // namespace sg

using namespace sg;

namespace sg {
namespace kmw {
// more clusters than the persistent kernel holds (kmeans_wide.cu)
int run(bool cluster, const void* points, int layout, int dim, int64_t n, int width,
        float xy_scale, float* centroids, const float* cent_in, int K, int32_t* labels,
        void* ws, size_t ws_bytes, int max_iter, float threshold, int32_t* d_iter,
        cudaStream_t st, const StageHeaders& own = StageHeaders{});
size_t workspace_bytes(int K, int dim);
}  // namespace kmw
}  // namespace sg

extern "C" void split_kmeans_set_wait_test(unsigned spin_limit, int skip_block) {
  km::g_wait_limit.store(spin_limit, std::memory_order_relaxed);
  km::g_wait_skip.store(skip_block < 0 ? -1 : skip_block, std::memory_order_relaxed);
}

extern "C" size_t split_kmeans_cluster_workspace_size_2d(int64_t npoints, int width,
                                                         int nclusters, int dim) {
  if (npoints <= 0 || width < 1) return 0;
  if (nclusters > km::kMaxK) {
    if (dim != 3 && dim != 5) dim = 5;
    return kmw::workspace_bytes(nclusters, dim);
  }
  // with the kept span sums of a clustering
  return km::carve(nullptr, 1, km::span_slots(npoints, width)).bytes;
}

extern "C" size_t split_kmeans_cluster_workspace_size(int64_t npoints, int nclusters, int dim) {
  // without the image width: room for the span sums at any width
  // ((width / 64) * (height / 2) <= npoints / 64 + 1)
  if (npoints <= 0) return 0;
  if (nclusters > km::kMaxK) return split_kmeans_cluster_workspace_size_2d(npoints, 1, nclusters, dim);
  return km::carve(nullptr, 1, npoints / 64 + 1).bytes;
}

extern "C" int split_kmeans_cluster(const void* points, int layout, int dim, int64_t npoints,
                                    int width, float xy_scale, float* centroids, int nclusters,
                                    int32_t* labels, void* workspace, size_t workspace_bytes,
                                    int max_iter, float threshold, int32_t* d_iterations,
                                    void* stream) {
  if (!centroids || !labels) return SPLIT_ERR_INVALID;
  if (nclusters > km::kMaxK)
    return kmw::run(true, points, layout, dim, npoints, width, xy_scale, centroids, centroids,
                    nclusters, labels, workspace, workspace_bytes, max_iter, threshold,
                    d_iterations, as_stream(stream));
  return km::run(km::kCluster, points, layout, dim, npoints, width, xy_scale, centroids,
                 centroids, nclusters, labels, nullptr, workspace, workspace_bytes, max_iter,
                 threshold, d_iterations, as_stream(stream));
}

// A composite call's clustering (`own`: its stage headers).  With `bytes`
// byte / 255 features straight from RGB8, with the results of
// split_kmeans_cluster on the packed float4 ones (unit range): the same values
// and, at any image width, the same fast spans.
namespace sg {
int kmeans_cluster_stage(const void* points, int layout, bool bytes, int dim, int64_t n, int width,
                         float xy_scale, float* centroids, int K, int32_t* labels, void* ws,
                         size_t ws_bytes, int max_iter, float threshold, const StageHeaders& own,
                         cudaStream_t st) {
  if (K > km::kMaxK)
    return kmw::run(true, points, layout, dim, n, width, xy_scale, centroids, centroids, K, labels,
                    ws, ws_bytes, max_iter, threshold, nullptr, st, own);
  return km::run(km::kCluster, points, layout, dim, n, width, xy_scale, centroids, centroids, K,
                 labels, nullptr, ws, ws_bytes, max_iter, threshold, nullptr, st, bytes, own);
}
}  // namespace sg

extern "C" size_t split_kmeans_assign_workspace_size(int64_t npoints, int nclusters) {
  // one assignment keeps no span sums
  if (npoints <= 0) return 0;
  if (nclusters > km::kMaxK) return split_kmeans_cluster_workspace_size(npoints, nclusters, 5);
  return km::carve(nullptr, 1).bytes;
}

extern "C" int split_kmeans_assign(const void* points, int layout, int dim, int64_t npoints,
                                   int width, float xy_scale, const float* centroids,
                                   int nclusters, int32_t* labels, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  if (!centroids || !labels) return SPLIT_ERR_INVALID;
  if (nclusters > km::kMaxK)
    return kmw::run(false, points, layout, dim, npoints, width, xy_scale, nullptr, centroids,
                    nclusters, labels, workspace, workspace_bytes, 1, -1.0f, nullptr,
                    as_stream(stream));
  return km::run(km::kAssignOnly, points, layout, dim, npoints, width, xy_scale,
                 const_cast<float*>(centroids), centroids, nclusters, labels, nullptr,
                 workspace, workspace_bytes, 1, -1.0f, nullptr, as_stream(stream));
}

namespace sg {
namespace segm {
int run(const int32_t* labels, const void* points, int layout, int dim, int64_t n, int width,
        float xy_scale, float* centroids, int K, void* ws, size_t ws_bytes, cudaStream_t st);
size_t workspace_bytes(int K, int dim);
}  // namespace segm
}  // namespace sg

extern "C" size_t split_kmeans_update_workspace_size(int64_t npoints, int nclusters, int dim) {
  // more clusters than the k-means kernel holds in shared memory: per-cluster
  // accumulators (16 B per feature value + a count)
  if (nclusters > km::kMaxK) {
    if (npoints <= 0 || dim < 1) return 0;
    return segm::workspace_bytes(nclusters, dim);
  }
  if (npoints <= 0) return 0;
  return km::carve(nullptr, 1).bytes;
}

extern "C" int split_kmeans_update(const int32_t* labels, const void* points, int layout,
                                   int dim, int64_t npoints, int width, float xy_scale,
                                   float* centroids, int nclusters, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  if (!centroids || !labels) return SPLIT_ERR_INVALID;
  if (nclusters > km::kMaxK)
    return segm::run(labels, points, layout, dim, npoints, width, xy_scale, centroids,
                     nclusters, workspace, workspace_bytes, as_stream(stream));
  return km::run(km::kUpdateOnly, points, layout, dim, npoints, width, xy_scale, centroids,
                 centroids, nclusters, nullptr, labels, workspace, workspace_bytes, 1, -1.0f,
                 nullptr, as_stream(stream));
}

namespace {
// Bound by the stores.  Four pixels per thread where rows of n floats keep the
// alignment (equal neighbours share one look-up): 2 Mpx to three rows, 33 MB,
// 12.6 us a pixel at a time, 8.4 us four at a time.
__device__ __forceinline__ float centroid_of(const float* row, int K, int l) {
  return l >= 0 && l < K ? __ldg(row + l) : 0.0f;
}

template <bool VEC>
__global__ void __launch_bounds__(256)
propagate_kernel(const int32_t* __restrict__ labels, int64_t n, const float* __restrict__ cent,
                 int K, int dim, float* __restrict__ out) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (VEC) {
    for (; i < n / 4; i += step) {
      const int4 l = __ldg(reinterpret_cast<const int4*>(labels) + i);
#pragma unroll 3
      for (int d = 0; d < dim; ++d) {
        const float* const row = cent + (int64_t)d * K;
        float4 v;
        v.x = centroid_of(row, K, l.x);
        v.y = l.y == l.x ? v.x : centroid_of(row, K, l.y);
        v.z = l.z == l.y ? v.y : centroid_of(row, K, l.z);
        v.w = l.w == l.z ? v.z : centroid_of(row, K, l.w);
        reinterpret_cast<float4*>(out + d * n)[i] = v;
      }
    }
    return;
  }
  for (; i < n; i += step) {
    const int l = __ldg(labels + i);
    for (int d = 0; d < dim; ++d) out[d * n + i] = centroid_of(cent + (int64_t)d * K, K, l);
  }
}
}  // namespace

extern "C" int split_kmeans_propagate(const int32_t* labels, int64_t npoints,
                                      const float* centroids, int nclusters, int dim,
                                      float* out, void* stream) {
  if (!labels || !centroids || !out || npoints <= 0 || nclusters < 1 || dim < 1)
    return SPLIT_ERR_INVALID;
  DeviceInfo di;
  SG_TRY(device_info(&di));
  const bool vec = npoints % 4 == 0 && ((reinterpret_cast<uintptr_t>(labels) |
                                         reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  int64_t blocks = ((vec ? npoints / 4 : npoints) + 255) / 256;
  const int64_t cap = (int64_t)di.sm_count * 8;
  if (blocks > cap) blocks = cap;
  (vec ? propagate_kernel<true> : propagate_kernel<false>)
      <<<(int)blocks, 256, 0, as_stream(stream)>>>(labels, npoints, centroids, nclusters, dim,
                                                   out);
  return launch_status();
}

// ---------------------------------------------------------------------------
// Allocation-free clustering.  Some callers cannot allocate device memory at
// the point where they cluster: a latency-critical serving loop (cudaMalloc
// and cudaFree synchronise the device), and host plugins whose device memory
// is owned by a pool they may not touch.  This variant keeps its scratch in
// one file-scope device array of fixed size, so a call needs no workspace.
//
// Limits and sharing rules:
//   - the array holds the state of one image, whatever its size: three
//     accumulator slots, two centroid slots and the iteration state for up
//     to kMaxK (64) clusters of up to kMaxDim (5) dimensions, 20736 bytes.
//     K above 64, or D other than 3 and 5, is rejected with
//     SPLIT_ERR_INVALID before anything is queued, as the workspace entry
//     point does;
//   - every GPU that loads the library holds the array until the process
//     exits; its device address is looked up once per device, on the first
//     call made with that device current.  A cudaDeviceReset of that device
//     unloads the module and may move the array, so the cached address is
//     stale afterwards: a process that resets a device must not call this
//     entry point on it again;
//   - all calls share the array: two calls whose work overlaps on the GPU
//     (different streams, or different host threads without ordering) race
//     and corrupt each other's results.  Order them on one stream.
// ---------------------------------------------------------------------------
#include <mutex>

namespace sg {
namespace km {

// Size of carve(ws, 1), evaluated at compile time (every piece starts on a
// 256-byte boundary).
constexpr size_t round256(size_t v) { return (v + 255) & ~size_t(255); }
constexpr size_t kStaticBytes =
    round256(round256(round256(round256(round256(round256(sizeof(WsHeader)) +
                                                 (size_t)3 * kMaxK * kMaxDim * 8) +
                                        (size_t)3 * kMaxK * kMaxDim * 8) +
                               (size_t)3 * kMaxK * 4) +
                      (size_t)2 * kMaxK * 8 * 4) +
             (size_t)2 * sizeof(ImageState));

static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

// Device address of g_static_scratch on the current device (looked up once).
static int static_scratch(void** out) {
  static std::mutex mu;
  static void* addr[64] = {nullptr};
  int dev = 0;
  SG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return SPLIT_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || !p) return SPLIT_ERR_CUDA;
    addr[dev] = p;
  }
  *out = addr[dev];
  return SPLIT_OK;
}

}  // namespace km
}  // namespace sg

extern "C" int split_kmeans_cluster_noalloc(const void* points, int layout, int dim,
                                            int64_t npoints, int width, float xy_scale,
                                            float* centroids, int nclusters, int32_t* labels,
                                            int max_iter, float threshold,
                                            int32_t* d_iterations, int32_t* d_status,
                                            void* stream) {
  using namespace sg::km;
  if (!centroids || !labels || npoints <= 0 || width < 1) return SPLIT_ERR_INVALID;
  // K, D and the layout first: nothing is queued for a call run() would refuse
  if (!valid_features(points, layout, dim, npoints, width, nclusters)) return SPLIT_ERR_INVALID;
  // one image's state, for any image size, always fits the array
  if (carve(nullptr, 1).bytes > kStaticBytes) return SPLIT_ERR_WORKSPACE;
  void* ws = nullptr;
  SG_TRY(static_scratch(&ws));
  cudaStream_t st = as_stream(stream);
  // The array keeps the previous call's contents: the status word starts at
  // zero here (run() clears the barrier words, counters and accumulators).
  Layout l = carve(ws, 1);
  SG_CUDA_TRY(cudaMemsetAsync(l.hdr, 0, sizeof(WsHeader), st));
  SG_TRY(run(kCluster, points, layout, dim, npoints, width, xy_scale, centroids, centroids,
             nclusters, labels, nullptr, ws, kStaticBytes, max_iter, threshold, d_iterations,
             st));
  if (d_status)
    SG_CUDA_TRY(cudaMemcpyAsync(d_status, &l.hdr->status, sizeof(int), cudaMemcpyDeviceToDevice,
                                st));
  return SPLIT_OK;
}

// ---------------------------------------------------------------------------
// Batches: one cooperative launch clusters every image of a batch (per-image
// K, iteration count and threshold); each image keeps its own tiles, groups,
// reduction tree and convergence test, so its result does not depend on what
// else shares the launch.
// ---------------------------------------------------------------------------
#include "kmeans_batch.h"

namespace sg {

// Kept span sums of a batch's images (those clustered more than once).
static int64_t batch_span_slots(const KmBatchImage* imgs, int nimages) {
  int64_t t = 0;
  for (int i = 0; i < nimages; ++i)
    if (imgs[i].iters > 1) t += km::span_slots(imgs[i].npoints, imgs[i].width);
  return t;
}

size_t kmeans_batch_workspace(const KmBatchImage* imgs, int nimages) {
  return km::carve(nullptr, nimages > 1 ? nimages : 2, batch_span_slots(imgs, nimages)).bytes;
}

int kmeans_batch_prepare(const KmBatchImage* imgs, int nimages, int layout, int dim,
                         float xy_scale, bool any_width, void* ws, size_t ws_bytes,
                         cudaStream_t st, KmBatchPlan* plan) {
  using namespace km;
  if (!imgs || nimages < 1 || (dim != 3 && dim != 5)) return SPLIT_ERR_INVALID;
  // single images only (see unit_features)
  if (layout & (SPLIT_KMEANS_REFERENCE_SHIFT | SPLIT_FEATURES_UNIT_RANGE)) return SPLIT_ERR_INVALID;
  const int slots = nimages > 1 ? nimages : 2;
  Layout l = carve(nullptr, slots);
  if (!ws || ws_bytes < l.bytes || (reinterpret_cast<uintptr_t>(ws) & 255))
    return SPLIT_ERR_WORKSPACE;
  // the images' kept span sums, where the workspace holds them
  const int64_t span_total = batch_span_slots(imgs, nimages);
  const bool keep = span_total > 0 && ws_bytes >= carve(nullptr, slots, span_total).bytes;
  l = carve(ws, slots, keep ? span_total : 0);
  int64_t span_off = 0;
  std::vector<Image> host(nimages);
  int64_t spans = 0;
  int max_iter = 0;
  for (int i = 0; i < nimages; ++i) {
    const KmBatchImage& b = imgs[i];
    if (!valid_features(b.points, layout, dim, b.npoints, b.width, b.nclusters) || !b.centroids ||
        !b.labels)
      return SPLIT_ERR_INVALID;
    Image& im = host[i];
    memset(&im, 0, sizeof(im));
    im.points = b.points;
    im.any_width = any_width;
    im.npoints = b.npoints;
    im.width = b.width;
    im.xy_scale = xy_scale;
    im.centroids = b.centroids;
    im.labels = b.labels;
    im.K = b.nclusters;
    im.max_iter = b.iters;
    im.threshold = b.threshold;
    im.unit_rows = tuned(b.npoints).kmeans_unit_rows;
    im.nspans = spans_of(b.npoints, b.width, im.unit_rows);
    im.scatter = std::max(1, (int)(0.6180339887 * im.nspans));
    while (std::gcd(im.scatter, im.nspans) != 1) ++im.scatter;
    // Every span reads its pixels in the first iteration; one with several
    // candidates costs about five times as much.  Their share, from the size
    // of a cluster's cell against a span's 64 + 8: sqrt(K) 72 / sqrt(W H)
    // (0.13 for K = 4 at 1000 x 1200, 0.40 for K = 32 at 1300 x 800).
    const double several =
        dim == 5 ? std::min(1.0, 72.0 * std::sqrt((double)b.nclusters / (double)b.npoints)) : 1.0;
    im.first_cost = (int)(im.nspans * (1.0 + 4.0 * several));
    spans += im.nspans;
    im.height = height_of(b.npoints, b.width);
    im.ntx = tiles_x(b.width);
    im.span_cols = b.width / kTile;
    if (keep && b.iters > 1) {
      im.span_sum = l.span_sum + span_off * kSpanSums;
      span_off += span_slots(b.npoints, b.width);
    }
    max_iter = max_iter > b.iters ? max_iter : b.iters;
  }
  SG_CUDA_TRY(cudaMemcpyAsync(l.images, host.data(), sizeof(Image) * nimages,
                              cudaMemcpyHostToDevice, st));
  // the host copy must outlive the transfer
  SG_CUDA_TRY(cudaStreamSynchronize(st));
  plan->nimages = nimages;
  if (spans > INT_MAX) return SPLIT_ERR_INVALID;
  plan->spans = (int)spans;
  plan->max_iter = max_iter;
  plan->layout = layout;
  plan->dim = dim;
  // the tuning table's residency is measured on single images, whose kernel
  // instance differs: a batch runs as many blocks as fit
  plan->blocks_per_sm = 0;
  return SPLIT_OK;
}

int kmeans_batch_run(const KmBatchPlan& plan, void* ws, cudaStream_t st) {
  using namespace km;
  const int slots = plan.nimages > 1 ? plan.nimages : 2;
  Layout l = carve(ws, slots);
  Params p{};
  p.nimages = plan.nimages;
  p.images = l.images;  // a one-image batch reads its descriptor from the table too
  p.total_spans = plan.spans;
  p.max_iter = plan.max_iter;
  p.acc_lo = l.acc_lo;
  p.acc_hi = l.acc_hi;
  p.acc_cnt = l.acc_cnt;
  p.cur = l.cur;
  p.state = l.state;
  p.hdr = l.hdr;
  p.blocks_per_sm = plan.blocks_per_sm;
  p.wait_limit = kSpinLimit;   // the wait test applies to single images only
  p.wait_skip = -1;
  SG_TRY(reset_counters(l, plan.nimages, st));
  launch_pdl(init_kernel, dim3((plan.nimages + 255) / 256), dim3(256), 0, st, p);
  SG_TRY(launch_status());
  // one block per image (the kernel strides over images past 1024)
  const int cb = plan.nimages < 1024 ? plan.nimages : 1024;
  if (plan.dim == 3) launch_pdl(load_user_centroids<3>, dim3(cb), dim3(64), 0, st, p);
  else launch_pdl(load_user_centroids<5>, dim3(cb), dim3(64), 0, st, p);
  SG_TRY(launch_status());
  if (plan.max_iter <= 0) return SPLIT_OK;
  return dispatch<kCluster>(plan.layout, plan.dim, p, st);
}

}  // namespace sg

// ---------------------------------------------------------------------------
// Tuning table C API
// ---------------------------------------------------------------------------
extern "C" int split_tune_set(const split_tune_entry* entries, int n) {
  if (n < 0 || n > SPLIT_TUNE_MAX_ENTRIES || (n > 0 && !entries)) return SPLIT_ERR_INVALID;
  for (int i = 0; i < n; ++i) {
    const split_tune_entry& e = entries[i];
    if (e.max_pixels <= 0 || (i > 0 && e.max_pixels <= entries[i - 1].max_pixels))
      return SPLIT_ERR_INVALID;
    if (e.kmeans_unit_rows != 16 && e.kmeans_unit_rows != 32 && e.kmeans_unit_rows != 64 &&
        e.kmeans_unit_rows != 128)
      return SPLIT_ERR_INVALID;
    if (e.kmeans_blocks_per_sm < 0 || e.kmeans_blocks_per_sm > 8) return SPLIT_ERR_INVALID;
  }
  sg::km::TuneTable& t = sg::km::tune_table();
  std::lock_guard<std::mutex> g(t.m);
  t.e.assign(entries, entries + n);
  return SPLIT_OK;
}

extern "C" int split_tune_get(split_tune_entry* out, int capacity) {
  sg::km::TuneTable& t = sg::km::tune_table();
  std::lock_guard<std::mutex> g(t.m);
  const int n = (int)t.e.size();
  for (int i = 0; i < n && i < capacity && out; ++i) out[i] = t.e[i];
  return n;
}

// ---------------------------------------------------------------------------
// Centroids of many clusters (K > kMaxK): calculate_centroids on segment
// labels (samples/src/main.cu:293-294, :306-307 call it with K = the number
// of segments).  Per-cluster sums of the member features in the same 96-bit
// fixed point as the k-means update (each feature rounded to a multiple of
// 2^-24, low and high words added with 64-bit atomics), so the result is the
// same whatever order pixels are added in.  Means in FP64, rounded to FP32; a
// cluster without members keeps its input centroid.
// ---------------------------------------------------------------------------
namespace sg {
namespace segm {

constexpr int kThreads = 256;

struct Layout {
  WsHeader* hdr;
  unsigned long long* lo;   // [K][dim]
  unsigned long long* hi;   // [K][dim]
  unsigned* cnt;            // [K]
  size_t bytes;
};

inline Layout carve(void* ws, int K, int dim) {
  Carver c(ws);
  Layout l;
  l.hdr = c.take<WsHeader>(1);
  l.lo = c.take<unsigned long long>((size_t)K * dim);
  l.hi = c.take<unsigned long long>((size_t)K * dim);
  l.cnt = c.take<unsigned>((size_t)K);
  l.bytes = c.size();
  return l;
}

// the features of pixel i
template <int LAYOUT, int DIM>
__device__ __forceinline__ void pixel_features(const void* points, int64_t n, int64_t i, int width,
                                               float xy_scale, float (&f)[DIM]) {
  if (LAYOUT == SPLIT_LAYOUT_FLOAT4) {
    const float4 v = __ldg(static_cast<const float4*>(points) + i);
    f[0] = v.x;
    f[1] = v.y;
    f[2] = v.z;
  } else if (LAYOUT == SPLIT_LAYOUT_RGB8) {
    const uint8_t* p = static_cast<const uint8_t*>(points) + 3 * i;
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] = __fdiv_rn((float)__ldg(p + c), 255.0f);
  } else {
    const float* p = static_cast<const float*>(points);
#pragma unroll
    for (int d = 0; d < DIM; ++d) f[d] = __ldg(p + (int64_t)d * n + i);
  }
  if (DIM == 5 && LAYOUT != SPLIT_LAYOUT_PLANAR) {
    const int64_t row = i / width;
    f[3] = __fmul_rn(xy_scale, (float)(i - row * width));
    f[4] = __fmul_rn(xy_scale, (float)row);
  }
}

// A run's word of one dimension into the sums: below 2^32, or any 64-bit one.
__device__ __forceinline__ void add_word(const Layout& L, size_t s, unsigned q) {
  atomicAdd(L.lo + s, (unsigned long long)q);
}
__device__ __forceinline__ void add_word(const Layout& L, size_t s, long long q) {
  atomicAdd(L.lo + s, (unsigned long long)q & 0xffffffffull);
  if (q >> 32) atomicAdd(L.hi + s, (unsigned long long)(q >> 32));
}
__device__ __forceinline__ unsigned shfl_down(unsigned v, int o) {
  return __shfl_down_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ long long shfl_down(long long v, int o) {
  return (long long)fix::shfl_down_u64((unsigned long long)v, o);
}

// Adds a run of pixels of one label.
template <int DIM, typename W>
__device__ __forceinline__ void add_run(const Layout& L, int l, const W (&q)[DIM],
                                        unsigned count) {
#pragma unroll
  for (int d = 0; d < DIM; ++d) add_word(L, (size_t)l * DIM + d, q[d]);
  atomicAdd(L.cnt + l, count);
}

// Bound by the reductions of runs and the atomics that they end in.  Four
// consecutive pixels per thread: it adds the runs that end inside them as they
// are, and its last run takes part in a segmented reduction over the lanes, whose
// run heads add.  A warp whose features all lie in [0, 1] (colours do) has words
// of at most 2^24, so the sums of its 128 pixels fit 32 bits; one with features
// below 2^32 has 64-bit sums; others add 96-bit words, a pixel of every lane at a
// time.  2 Mpx in 24 thousand segments, planar colours: 15.4 us.
constexpr int kPer = 4;

// the runs of the warp's pixels, words as W; `word` gives pixel j's
template <int DIM, typename W, class F>
__device__ __forceinline__ void add_runs(const Layout& L, const int (&l)[kPer], F&& word) {
  const int lane = threadIdx.x & 31;
  W q[DIM];
  unsigned c = 0u;
  int cur = l[0];
#pragma unroll
  for (int d = 0; d < DIM; ++d) q[d] = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (j > 0 && l[j] != cur) {
      if (cur >= 0) add_run<DIM, W>(L, cur, q, c);
      cur = l[j];
      c = 0u;
#pragma unroll
      for (int d = 0; d < DIM; ++d) q[d] = 0;
    }
    ++c;
#pragma unroll
    for (int d = 0; d < DIM; ++d) q[d] += word(j, d);
  }
  // the lanes' last runs: a lane adds from lane + o while that lane is in its
  // run; a lane that began its run with fewer than four pixels is a head, its
  // label not the lane's before (or cut off by the runs already added)
  const int before = __shfl_up_sync(0xffffffffu, cur, 1);
  const unsigned heads =
      __ballot_sync(0xffffffffu, lane == 0 || cur != before || c != (unsigned)kPer);
  const unsigned after = heads & ~(0xffffffffu >> (31 - lane));
  const int run_end = after ? __ffs(after) - 1 : 32;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const bool in_run = lane + o < run_end;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const W a = shfl_down(q[d], o);
      if (in_run) q[d] += a;
    }
    const unsigned a = __shfl_down_sync(0xffffffffu, c, o);
    if (in_run) c += a;
  }
  if (cur >= 0 && (heads >> lane & 1u)) add_run<DIM, W>(L, cur, q, c);
}

template <int LAYOUT, int DIM>
__global__ void __launch_bounds__(kThreads)
accumulate_kernel(const int32_t* __restrict__ labels, const void* __restrict__ points,
                  int64_t n, int width, float xy_scale, int K, Layout L, bool vec) {
  if (blockIdx.x == 0 && threadIdx.x == 0) L.hdr->stamp = kStampDirty;
  const int lane = threadIdx.x & 31;
  const int64_t i0 = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * kPer;
  int l[kPer];
  float f[kPer][DIM];
  if (vec && i0 + kPer <= n) {   // n is a multiple of kPer
    const int4 v = __ldg(reinterpret_cast<const int4*>(labels + i0));
    l[0] = v.x; l[1] = v.y; l[2] = v.z; l[3] = v.w;
  } else {
#pragma unroll
    for (int j = 0; j < kPer; ++j) l[j] = i0 + j < n ? __ldg(labels + i0 + j) : -1;
  }
#pragma unroll
  for (int j = 0; j < kPer; ++j)
    if (l[j] >= K) l[j] = -1;
  if (LAYOUT == SPLIT_LAYOUT_PLANAR && vec) {
    const float* p = static_cast<const float*>(points);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const float4 v = i0 < n ? __ldg(reinterpret_cast<const float4*>(p + (int64_t)d * n + i0))
                              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      f[0][d] = v.x; f[1][d] = v.y; f[2][d] = v.z; f[3][d] = v.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) f[j][d] = 0.0f;
      if (l[j] >= 0) pixel_features<LAYOUT, DIM>(points, n, i0 + j, width, xy_scale, f[j]);
    }
  }
  // (false for NaN)
  bool unit = true, small = true;
#pragma unroll
  for (int j = 0; j < kPer; ++j)
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      unit &= l[j] < 0 || (f[j][d] >= 0.0f && f[j][d] <= 1.0f);
      small &= l[j] < 0 || fabsf(f[j][d]) < 4294967296.0f;
    }
  if (__all_sync(0xffffffffu, unit)) {
    add_runs<DIM, unsigned>(
        L, l, [&](int j, int d) { return __float2uint_rn(__fmul_rn(f[j][d], fix::kScale)); });
  } else if (__all_sync(0xffffffffu, small)) {
    add_runs<DIM, long long>(
        L, l, [&](int j, int d) { return __float2ll_rn(__fmul_rn(f[j][d], fix::kScale)); });
  } else {
    // neighbouring pixels in neighbouring lanes again
    const int64_t w0 = i0 - (int64_t)lane * kPer;
    for (int j = 0; j < kPer; ++j) {
      const int64_t i = w0 + 32 * j + lane;
      int lj = i < n ? __ldg(labels + i) : -1;
      if (lj < 0 || lj >= K) lj = -1;
      float g[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) g[d] = 0.0f;
      if (lj >= 0) pixel_features<LAYOUT, DIM>(points, n, i, width, xy_scale, g);
      unsigned long long qlo[DIM], qhi[DIM];
      fix::quantize<DIM>(g, lj, &L.hdr->status, qlo, qhi);
      fix::warp_add<DIM>(lj, qlo, qhi, L.lo, L.hi, L.cnt);
    }
  }
}

__global__ void __launch_bounds__(kThreads)
finish_kernel(Layout L, int K, int dim, float* __restrict__ centroids) {
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < (int64_t)K * dim;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(idx / dim), d = (int)(idx - (int64_t)k * dim);
    const unsigned nk = L.cnt[k];
    if (nk == 0) continue;
    centroids[(int64_t)d * K + k] = fix::mean(L.lo[idx], L.hi[idx], nk);
  }
}

size_t workspace_bytes(int K, int dim) { return carve(nullptr, K, dim).bytes; }

int run(const int32_t* labels, const void* points, int layout, int dim, int64_t n, int width,
        float xy_scale, float* centroids, int K, void* ws, size_t ws_bytes, cudaStream_t st) {
  layout &= ~SPLIT_FEATURES_UNIT_RANGE;
  if (!labels || !points || !centroids || n <= 0 || n > 0x7fffffffLL || K < 1 || width < 1)
    return SPLIT_ERR_INVALID;
  if ((dim != 3 && dim != 5) || layout < SPLIT_LAYOUT_PLANAR || layout > SPLIT_LAYOUT_RGB8)
    return SPLIT_ERR_INVALID;
  if (layout == SPLIT_LAYOUT_FLOAT4 && (reinterpret_cast<uintptr_t>(points) & 15))
    return SPLIT_ERR_INVALID;
  Layout l = carve(nullptr, K, dim);
  if (!ws || ws_bytes < l.bytes || (reinterpret_cast<uintptr_t>(ws) & 255))
    return SPLIT_ERR_WORKSPACE;
  l = carve(ws, K, dim);
  SG_CUDA_TRY(cudaMemsetAsync(l.lo, 0, l.bytes - sizeof(WsHeader), st));
  DeviceInfo di;
  SG_TRY(device_info(&di));
  // whole vectors of labels and, planar, of every feature row
  const bool vec = n % kPer == 0 && ((reinterpret_cast<uintptr_t>(labels) |
                                      (layout == SPLIT_LAYOUT_PLANAR
                                           ? reinterpret_cast<uintptr_t>(points) : 0)) & 15) == 0;
#define SG_SEG_CASE(LY, D)                                                                 \
  if (layout == LY && dim == D) {                                                          \
    accumulate_kernel<LY, D><<<(int)((n + kThreads * kPer - 1) / (kThreads * kPer)),       \
                               kThreads, 0, st>>>(labels, points, n, width, xy_scale, K,  \
                                                  l, vec);                                 \
  }
  SG_SEG_CASE(SPLIT_LAYOUT_PLANAR, 3)
  SG_SEG_CASE(SPLIT_LAYOUT_PLANAR, 5)
  SG_SEG_CASE(SPLIT_LAYOUT_FLOAT4, 3)
  SG_SEG_CASE(SPLIT_LAYOUT_FLOAT4, 5)
  SG_SEG_CASE(SPLIT_LAYOUT_RGB8, 3)
  SG_SEG_CASE(SPLIT_LAYOUT_RGB8, 5)
#undef SG_SEG_CASE
  SG_TRY(launch_status());
  const int64_t cap = (int64_t)di.sm_count * 8;
  int64_t fb = ((int64_t)K * dim + kThreads - 1) / kThreads;
  if (fb > cap) fb = cap;
  finish_kernel<<<(int)fb, kThreads, 0, st>>>(l, K, dim, centroids);
  return launch_status();
}

}  // namespace segm
}  // namespace sg
