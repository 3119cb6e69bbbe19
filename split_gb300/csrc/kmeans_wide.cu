// k-means with more clusters than the persistent kernel keeps in shared
// memory (64 < K <= 2^20): label_points (split/src/split/device/kmeans/
// label.cu:74-106) and cluster (cluster.cu:27-93), which set no limit on K.
//
// Assignment (assign_kernel): a block takes a tile of 1024 pixels at a time (64 x
// 16 of most images), a warp 128 of them (4 consecutive ones per lane, measured as
// two packed FP32x2 pairs).  The centroids come in shared-memory chunks of 32 KB (1024
// centroids of 5 dimensions, 2048 of 3).  The block prunes a chunk exactly
// with bounds over its tile's feature box to a list, each warp the list over
// its own pixels' box, and measures the survivors.  The squared distance is
// the reference's sum of (x - c)^2 in dimension order (label.cu:23-32) with
// one rounding per operation, and ties go to the lowest cluster index (strict
// < in ascending k, as the reference's argmin over the distance row,
// label.cu:98-105).  In a clustering the same pass adds every pixel's
// features to its cluster's fixed-point sums (fixsum.cuh), so the update reads
// no pixel again; a tile's sums are added up in shared memory first where the
// image has many tiles.
//
// Clustering: per iteration one assignment launch and one forming launch
// (form_kernel), all max_iter pairs queued at once, each launch a
// programmatic dependent of the one before.  The forming launch turns the
// sums into means (FP64 division of the exact sum, rounded once to FP32; a
// cluster without members keeps its centroid), measures the centroid shift,
// and decides on the device whether the next iteration runs (|delta -
// old_delta| > threshold, cluster.cu:65-88).  After the stop, the launches
// still queued return at once.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "common.cuh"
#include "f32x2.cuh"
#include "fixsum.cuh"
#include "pixels.cuh"

namespace sg {
namespace kmw {

constexpr int kMinK = 65;                 // smaller K runs in the persistent kernel
constexpr int kMaxClusters = 1 << 20;
constexpr int kThreads = 256;
constexpr int kPix = kPx;                 // pixels per thread (two pairs)
constexpr int kTilePxLog2 = 10;           // a block's pixels, whole rows of lanes' four
constexpr int kTileWLog2 = 6;             // 64 x 16 of them, see tile_width_log2
constexpr int kWarps = kThreads / 32;
static_assert(1 << kTilePxLog2 == kThreads * kPix && kPix == 4, "one lane each");
constexpr int kSlots = 128;               // clusters of a tile summed in shared memory
constexpr int kDirectTiles = 32;          // up to this many tiles add to the global sums
constexpr int kChunkF4 = 2048;            // float4 slots of one centroid chunk (32 KB)
constexpr int kFormSlots = 1024;          // strided partials of the shift
constexpr int kFormThreads = 256, kFormBlocks = 16;
constexpr int kFormMaxThreads = 1024;     // one block, up to kFormFew values
constexpr int kFormFew = 512;

struct State {
  float delta;   // shift of the last formed iteration (0 before the first)
  int iters;     // iterations formed
  int done;      // no further iteration runs
  unsigned arrived;   // forming blocks that have finished their share
};

struct Layout {
  WsHeader* hdr;
  State* state;
  float* cur;                // [2][DIM][K] planar: input centroids of odd / even iterations
  unsigned long long* lo;    // [K][DIM] low words of the fixed-point sums
  unsigned long long* hi;    // [K][DIM] high words (signed)
  unsigned* cnt;             // [K] member counts
  float* word;               // [3K] squared terms of the reference's shift
  float* part;               // [kFormSlots] partials of the L2 shift
  size_t bytes;
};

inline Layout carve(void* ws, int K, int dim) {
  Carver c(ws);
  Layout l;
  l.hdr = c.take<WsHeader>(1);
  l.state = c.take<State>(1);
  l.cur = c.take<float>((size_t)2 * dim * K);
  l.lo = c.take<unsigned long long>((size_t)K * dim);
  l.hi = c.take<unsigned long long>((size_t)K * dim);
  l.cnt = c.take<unsigned>((size_t)K);
  l.word = c.take<float>((size_t)3 * K);
  l.part = c.take<float>(kFormSlots);
  l.bytes = c.size();
  return l;
}

struct Points {
  const void* pts;
  int64_t n;
  int width;
  float xy;      // xy_scale: dimension 3 and 4 of 5-D packed features
};

// Features of pixel i (i < n): RGB8 channels / 255, packed float4 .xyz or
// planar rows; 5-D packed features append xy * (column, row) of an image
// `width` pixels wide.
template <int LAYOUT, int DIM>
__device__ __forceinline__ void load_px(const Points& P, int64_t i, float (&f)[DIM]) {
  if (LAYOUT == SPLIT_LAYOUT_PLANAR) {
    const float* p = static_cast<const float*>(P.pts);
#pragma unroll
    for (int d = 0; d < DIM; ++d) f[d] = __ldg(p + d * P.n + i);
    return;
  }
  if (LAYOUT == SPLIT_LAYOUT_FLOAT4) {
    const float4 v = __ldg(static_cast<const float4*>(P.pts) + i);
    f[0] = v.x;
    f[1] = v.y;
    f[2] = v.z;
  } else {
    const uint8_t* p = static_cast<const uint8_t*>(P.pts) + 3 * i;
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] = __fdiv_rn((float)__ldg(p + c), 255.0f);
  }
  if (DIM == 5) {
    const int row = (int)i / P.width;
    const int col = (int)i - row * P.width;
    f[DIM == 5 ? 3 : 0] = __fmul_rn(P.xy, (float)col);
    f[DIM == 5 ? 4 : 0] = __fmul_rn(P.xy, (float)row);
  }
}

struct AssignArgs {
  Points P;
  int K;
  const float* cent;        // [DIM][K] planar
  int32_t* labels;
  const State* state;       // clustering: the launch returns once done is set
  unsigned long long* lo;
  unsigned long long* hi;
  unsigned* cnt;
  int* status;
  int tile_w_log2;          // a tile is 2^tile_w_log2 pixels wide
};

// Order-preserving float -> int key (warp min / max of the box).
__device__ __forceinline__ int fkey(float x) {
  const int i = __float_as_int(x);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float fkey_inv(int k) {
  return __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
}

// Squared distances of the pixel pair (p, q) to one centroid (c.x, c.y, c.z,
// c.w, c4), the reference's sum in dimension order, kept where it is below
// the pair's best so far (ties keep the lower index seen first).
template <int DIM>
__device__ __forceinline__ void closer(const float (&fp)[DIM], const float (&fq)[DIM],
                                       const float4 c, float c4, int k, float& bp, float& bq,
                                       int& kp, int& kq) {
  float2 t = fsub2(make_float2(fp[0], fq[0]), make_float2(c.x, c.x));
  float2 dd = fmul2(t, t);
  t = fsub2(make_float2(fp[1], fq[1]), make_float2(c.y, c.y));
  dd = ffma2(t, t, dd);
  t = fsub2(make_float2(fp[2], fq[2]), make_float2(c.z, c.z));
  dd = ffma2(t, t, dd);
  if (DIM == 5) {
    constexpr int X = DIM == 5 ? 3 : 0, Y = DIM == 5 ? 4 : 0;
    t = fsub2(make_float2(fp[X], fq[X]), make_float2(c.w, c.w));
    dd = ffma2(t, t, dd);
    t = fsub2(make_float2(fp[Y], fq[Y]), make_float2(c4, c4));
    dd = ffma2(t, t, dd);
  }
  if (dd.x < bp) {
    bp = dd.x;
    kp = k;
  }
  if (dd.y < bq) {
    bq = dd.y;
    kq = k;
  }
}

// Exact pruning over a box [lo, hi] of pixels' features: for a centroid, LB =
// squared distance to the box (below every pixel's distance) and UB = squared
// distance to the farthest corner (above it).  thr = the smallest UB seen so
// far (over this chunk and the ones before) bounds every pixel's best
// distance, so a centroid whose LB exceeds thr by more than the 1e-4 relative
// margin is strictly farther than another centroid from every pixel, even
// after FP32 rounding (a few ulp), and is skipped: every argmin, ties
// included, is unchanged.
template <int DIM>
__device__ __forceinline__ float upper_bound(const float* c, const float (&lo)[DIM],
                                             const float (&hi)[DIM]) {
  float u = 0.0f;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const float e = fmaxf(c[d] - lo[d], hi[d] - c[d]);
    u = __fmaf_rn(e, e, u);
  }
  return u;
}
template <int DIM>
__device__ __forceinline__ float lower_bound(const float* c, const float (&lo)[DIM],
                                             const float (&hi)[DIM]) {
  float l = 0.0f;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const float g = fmaxf(fmaxf(lo[d] - c[d], c[d] - hi[d]), 0.0f);
    l = __fmaf_rn(g, g, l);
  }
  return l;
}

// The tile's sums per list entry (64-bit fixed point in two words).
template <int DIM>
struct TileSums {
  unsigned lo[kSlots * DIM], hi[kSlots * DIM];
  unsigned cnt[kSlots];
};

template <int DIM>
__device__ __forceinline__ void tile_add(TileSums<DIM>& ts, int idx, unsigned long long v) {
  const unsigned lo = (unsigned)v;
  const unsigned old = atomicAdd(&ts.lo[idx], lo);
  const unsigned hi = (unsigned)(v >> 32) + (old + lo < old ? 1u : 0u);
  if (hi) atomicAdd(&ts.hi[idx], hi);
}

// Adds the warp's pixels (features in [0, 2^14)) to the sums of their list
// entries `at` (below 0: none), entry by entry: the lanes' words split at bit
// 24, so that each half's warp sum fits the 32-bit warp reduction.
template <int LAYOUT, int DIM>
__device__ __forceinline__ void warp_to_tile(TileSums<DIM>& ts, const float (&f)[kPix][DIM],
                                             const int (&at)[kPix]) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  unsigned long long q[kPix][DIM];
#pragma unroll
  for (int j = 0; j < kPix; ++j)
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      q[j][d] = (unsigned long long)__float2ll_rn(__fmul_rn(f[j][d], fix::kScale));
  int left = -1;   // entries up to this one are done
  for (;;) {
    unsigned next = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < kPix; ++j)
      if (at[j] > left) next = min(next, (unsigned)at[j]);
    const unsigned p = __reduce_min_sync(full, next);
    if (p == 0xffffffffu) break;
    left = (int)p;
    unsigned n = 0;
    unsigned long long mine = 0;
#pragma unroll
    for (int j = 0; j < kPix; ++j) n += at[j] == left ? 1u : 0u;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      unsigned long long s = 0;
#pragma unroll
      for (int j = 0; j < kPix; ++j) s += at[j] == left ? q[j][d] : 0ull;
      unsigned long long total;
      if (LAYOUT == SPLIT_LAYOUT_RGB8 && d < 3)   // values up to 1: at most 2^31 in all
        total = __reduce_add_sync(full, (unsigned)s);
      else
        total = ((unsigned long long)__reduce_add_sync(full, (unsigned)(s >> 24)) << 24) +
                __reduce_add_sync(full, (unsigned)s & 0xffffffu);
      if (lane == d) mine = total;
    }
    n = __reduce_add_sync(full, n);
    if (lane < DIM) tile_add(ts, left * DIM + lane, mine);
    if (lane == DIM) atomicAdd(&ts.cnt[left], n);
  }
}

// What bounds it: instruction issue (a pixel's labels and sums are a few
// bytes).  Bounding every centroid against every 128 pixels and sending each
// warp's sums to global memory took 120 us an iteration at 2560 x 1440, K =
// 256, 5-D (75 without the sums); with the tile's list and sums in shared
// memory 56 (54 for the labels alone).
//
// TW: log2 of the tile's width; 0: as given at run time (tile_w_log2).
template <int LAYOUT, int DIM, bool ACC, int TW>
__global__ void __launch_bounds__(kThreads, 3) assign_kernel(AssignArgs a) {
  constexpr int CS = DIM == 5 ? 2 : 1;          // float4 slots per centroid
  constexpr int kChunk = kChunkF4 / CS;         // centroids per chunk
  constexpr unsigned full = 0xffffffffu;
  __shared__ float4 cs[kChunkF4];
  __shared__ unsigned short list[kChunk];       // the tile's candidates, ascending
  __shared__ TileSums<DIM> sums;   // (clusterings only)
  __shared__ float boxes[kWarps][2 * DIM], box[2 * DIM], least[kWarps];
  __shared__ int counts[kWarps];
  __shared__ int stop;
  pdl_wait();
  if (ACC) {
    if (threadIdx.x == 0) stop = __ldcg(&a.state->done);
    __syncthreads();
    if (stop) return;
  }
  const int K = a.K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nchunks = (K + kChunk - 1) / kChunk;
  float* csf = reinterpret_cast<float*>(cs);
  const int W = a.P.width;
  const int H = (int)((a.P.n + W - 1) / W);
  const int tw = TW ? TW : a.tile_w_log2, th = kTilePxLog2 - tw;
  const int tiles_x = ((W - 1) >> tw) + 1;
  const int tiles = tiles_x * (((H - 1) >> th) + 1);
  // a warp's 128 pixels, 32 x 4 where the tile allows it: its place in the tile
  // and the lane's four pixels in it
  const int sw = tw > 8 ? tw - 3 : min(tw, 5);
  const int wrow = (warp >> (tw - sw) << (7 - sw)) + (lane >> (sw - 2));
  const int wcol = ((warp & ((1 << (tw - sw)) - 1)) << sw) + ((lane & ((1 << (sw - 2)) - 1)) << 2);

  auto load_chunk = [&](int ch) {
    const int k0 = ch * kChunk;
    const int kc = min(kChunk, K - k0);
    __syncthreads();
    for (int idx = threadIdx.x; idx < kc * DIM; idx += kThreads) {
      const int d = idx / kc, k = idx - d * kc;
      csf[k * (4 * CS) + d] = __ldg(a.cent + (int64_t)d * K + k0 + k);
    }
    __syncthreads();
  };
  if (nchunks == 1) load_chunk(0);
  // A few tiles hardly meet at the global sums, and a way through shared memory
  // only adds to the one tile that their blocks wait for: 100 x 80, K = 128, 3-D,
  // 35 us an iteration through the tile's sums, 29 without.
  const bool tile_sums = ACC && nchunks == 1 && tiles > kDirectTiles;
  if (ACC && tile_sums) {
    for (int i = threadIdx.x; i < kSlots * DIM; i += kThreads) sums.lo[i] = sums.hi[i] = 0u;
    for (int i = threadIdx.x; i < kSlots; i += kThreads) sums.cnt[i] = 0u;
  }

  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int ty = tile / tiles_x, tx = tile - ty * tiles_x;
    // (64 bits where the last tile of a long row or column may reach past 2^31)
    using Coord = std::conditional_t<TW == kTileWLog2, int, int64_t>;
    const Coord row = ((Coord)ty << th) + wrow, col = ((Coord)tx << tw) + wcol;
    const int64_t px0 = (int64_t)row * W + col;
    const int valid =
        row < H ? (int)max((int64_t)0, min((int64_t)min((Coord)kPix, W - col), a.P.n - px0)) : 0;
    RawPx<LAYOUT, DIM> raw;
    raw.load(a.P.pts, a.P.n, px0, valid);
    float f[kPix][DIM];
    raw.features(a.P.xy, (int)row, (int)col, f);
    // box of the warp's pixels; fminf / fmaxf skip NaN (a NaN pixel's
    // distances all compare false, so it keeps label 0 whatever is skipped)
    float lo[DIM], hi[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      float x = INFINITY, z = -INFINITY;
#pragma unroll
      for (int j = 0; j < kPix; ++j) {
        if (j < valid) {
          x = fminf(x, f[j][d]);
          z = fmaxf(z, f[j][d]);
        }
      }
      lo[d] = fkey_inv(__reduce_min_sync(full, fkey(x)));
      hi[d] = fkey_inv(__reduce_max_sync(full, fkey(z)));
      if (lane == 0) {
        boxes[warp][d] = lo[d];
        boxes[warp][DIM + d] = hi[d];
      }
    }
    __syncthreads();
    if (threadIdx.x < 2 * DIM) {
      float v = boxes[0][threadIdx.x];
      for (int w = 1; w < kWarps; ++w)
        v = threadIdx.x < DIM ? fminf(v, boxes[w][threadIdx.x]) : fmaxf(v, boxes[w][threadIdx.x]);
      box[threadIdx.x] = v;
    }
    __syncthreads();
    float blo[DIM], bhi[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      blo[d] = box[d];
      bhi[d] = box[DIM + d];
    }
    float best[kPix];
    int bk[kPix];   // with one chunk the list entry, otherwise the cluster
#pragma unroll
    for (int j = 0; j < kPix; ++j) {
      best[j] = INFINITY;
      bk[j] = -1;   // (no distance compares: label 0)
    }
    float tile_ub = INFINITY, ub_min = INFINITY;
    int nlist = 0;
    for (int ch = 0; ch < nchunks; ++ch) {
      if (nchunks > 1) load_chunk(ch);
      const int k0 = ch * kChunk;
      const int kc = min(kChunk, K - k0);
      // the tile's candidates of the chunk
      float um = tile_ub;
      for (int k = threadIdx.x; k < kc; k += kThreads)
        um = fminf(um, upper_bound<DIM>(csf + k * (4 * CS), blo, bhi));
      // UB >= 0: its bit pattern orders like the value
      um = __int_as_float(__reduce_min_sync(full, __float_as_int(um)));
      if (lane == 0) least[warp] = um;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < kWarps; ++w) tile_ub = fminf(tile_ub, least[w]);
      const float tile_thr = tile_ub * 1.0001f;
      nlist = 0;
      for (int g = 0; g < kc; g += kThreads) {
        const int k = g + (int)threadIdx.x;
        const bool in = k < kc && lower_bound<DIM>(csf + k * (4 * CS), blo, bhi) <= tile_thr;
        const unsigned m = __ballot_sync(full, in);
        if (lane == 0) counts[warp] = __popc(m);
        __syncthreads();
        int before = nlist;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          if (w < warp) before += counts[w];
          nlist += counts[w];
        }
        if (in) list[before + __popc(m & ((1u << lane) - 1u))] = (unsigned short)k;
        __syncthreads();
      }
      // the warp's, 32 list entries at a time
      um = ub_min;
      for (int i = lane; i < nlist; i += 32)
        um = fminf(um, upper_bound<DIM>(csf + list[i] * (4 * CS), lo, hi));
      ub_min = __int_as_float(__reduce_min_sync(full, __float_as_int(um)));
      const float thr = ub_min * 1.0001f;
      for (int g = 0; g < nlist; g += 32) {
        const int i = g + lane;
        const bool in = i < nlist && lower_bound<DIM>(csf + list[i] * (4 * CS), lo, hi) <= thr;
        unsigned m = __ballot_sync(full, in);
        // two at a time: both are read before the first is measured
        while (m) {
          const int p = g + __ffs(m) - 1;
          m &= m - 1;
          const int q = m ? g + __ffs(m) - 1 : p;
          const int kp = list[p], kq = list[q];
          const float4 c = cs[kp * CS], e = cs[kq * CS];
          const float c4 = DIM == 5 ? cs[kp * CS + (CS - 1)].x : 0.0f;
          const float e4 = DIM == 5 ? cs[kq * CS + (CS - 1)].x : 0.0f;
          const int np = nchunks == 1 ? p : k0 + kp, nq = nchunks == 1 ? q : k0 + kq;
          closer<DIM>(f[0], f[1], c, c4, np, best[0], best[1], bk[0], bk[1]);
          closer<DIM>(f[2], f[3], c, c4, np, best[2], best[3], bk[2], bk[3]);
          if (!m) break;
          m &= m - 1;
          closer<DIM>(f[0], f[1], e, e4, nq, best[0], best[1], bk[0], bk[1]);
          closer<DIM>(f[2], f[3], e, e4, nq, best[2], best[3], bk[2], bk[3]);
        }
      }
    }
    int lab[kPix];
#pragma unroll
    for (int j = 0; j < kPix; ++j)
      lab[j] = bk[j] < 0 ? 0 : nchunks == 1 ? (int)list[bk[j]] : bk[j];
    if (valid == kPix && (W & 3) == 0 && (reinterpret_cast<uintptr_t>(a.labels) & 15) == 0) {
      *reinterpret_cast<int4*>(a.labels + px0) = make_int4(lab[0], lab[1], lab[2], lab[3]);
    } else {
#pragma unroll
      for (int j = 0; j < kPix; ++j)
        if (j < valid) a.labels[px0 + j] = lab[j];
    }
    if constexpr (ACC) {
      // Features in [0, 2^14) whose clusters fit the tile's sums (the common
      // case by far); below 2^32, the narrow fixed-point form straight into
      // the global sums; otherwise the general form.  A pixel that no distance
      // named (all infinite or NaN) belongs to cluster 0, which the list may
      // not hold: not for the tile's sums either.
      bool tiled = tile_sums && nlist <= kSlots, small = true;
#pragma unroll
      for (int j = 0; j < kPix; ++j) {
        tiled = tiled && (j >= valid || bk[j] >= 0);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          tiled = tiled && (j >= valid || (f[j][d] >= 0.0f && f[j][d] < 16384.0f));
          small = small && (j >= valid || fabsf(f[j][d]) < 4294967296.0f);
        }
      }
      if (__all_sync(full, tiled)) {
        int at[kPix];
#pragma unroll
        for (int j = 0; j < kPix; ++j) at[j] = j < valid ? bk[j] : -1;
        warp_to_tile<LAYOUT, DIM>(sums, f, at);
      } else if (__all_sync(full, small)) {
        // where every lane's four pixels carry one label (or lie outside), the
        // lane adds them first
        bool one = valid == kPix;
#pragma unroll
        for (int j = 1; j < kPix; ++j) one = one && lab[j] == lab[0];
        if (__all_sync(full, one || valid == 0)) {
          long long q[DIM];
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            q[d] = 0;
#pragma unroll
            for (int j = 0; j < kPix; ++j)
              if (valid) q[d] += __float2ll_rn(__fmul_rn(f[j][d], fix::kScale));
          }
          fix::warp_add_narrow<DIM>(valid ? lab[0] : -1, q, kPix, a.lo, a.hi, a.cnt);
        } else {
#pragma unroll
          for (int j = 0; j < kPix; ++j) {
            const int l = j < valid ? lab[j] : -1;
            long long q[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
              q[d] = l >= 0 ? __float2ll_rn(__fmul_rn(f[j][d], fix::kScale)) : 0ll;
            fix::warp_add_narrow<DIM>(l, q, 1u, a.lo, a.hi, a.cnt);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < kPix; ++j) {
          unsigned long long qlo[DIM], qhi[DIM];
          const int l = j < valid ? lab[j] : -1;
          fix::quantize<DIM>(f[j], l, a.status, qlo, qhi);
          fix::warp_add<DIM>(l, qlo, qhi, a.lo, a.hi, a.cnt);
        }
      }
      // the tile's sums into the global ones (a block has few tiles: the list
      // changes with the tile)
      __syncthreads();
      const int used = tile_sums ? min(nlist, kSlots) : 0;
      for (int i = threadIdx.x; i < used * DIM; i += kThreads) {
        const unsigned wl = sums.lo[i], wh = sums.hi[i];
        if ((wl | wh) == 0u) continue;
        sums.lo[i] = sums.hi[i] = 0u;
        const size_t s = (size_t)list[i / DIM] * DIM + i % DIM;
        atomicAdd(a.lo + s, (unsigned long long)wl);
        if (wh) atomicAdd(a.hi + s, (unsigned long long)wh);
      }
      for (int i = threadIdx.x; i < used; i += kThreads) {
        const unsigned n = sums.cnt[i];
        if (n == 0u) continue;
        sums.cnt[i] = 0u;
        atomicAdd(a.cnt + list[i], n);
      }
    }
    __syncthreads();   // the list and the boxes are the next tile's
  }
}

// Initial state, the caller's centroids into cur[0], zero sums.
__global__ void setup_kernel(Layout L, int K, int dim, const float* __restrict__ cent,
                             int32_t* d_iter, int max_iter, StageHeaders own) {
  pdl_wait();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nt = (int64_t)gridDim.x * blockDim.x;
  if (t == 0) {
    enter_stages(own, own.hdr ? own.hdr->stamp : 0ull);
    State s;
    s.delta = 0.0f;
    s.iters = 0;
    s.done = max_iter <= 0;
    s.arrived = 0u;
    *L.state = s;
    L.hdr->stamp = kStampDirty;
    if (d_iter && max_iter <= 0) *d_iter = 0;
  }
  const int64_t kd = (int64_t)K * dim;
  for (int64_t i = t; i < kd; i += nt) {
    L.cur[i] = cent[i];
    L.lo[i] = 0ull;
    L.hi[i] = 0ull;
  }
  for (int64_t k = t; k < K; k += nt) L.cnt[k] = 0u;
}

struct FormArgs {
  Layout L;
  Points P;
  int K;
  int i;                    // iteration being formed (1-based)
  int max_iter;
  float threshold;
  int ref_shift;            // the reference's shift measure (3-D only)
  float* centroids;         // the caller's [DIM][K], written when the run stops
  int32_t* d_iter;
};

// Centroids of iteration i from the sums of its assignment, the shift, the
// decision.  Every sum is read once and cleared for the next iteration.  The
// L2 shift is summed in a fixed order (kFormSlots strided partials, then a
// fixed tree), so it does not vary between runs.  FP64 runs at two lanes per
// clock and SM, and the means divide in FP64: one block took 10.4 us for K =
// 256, so the slots are spread over kFormBlocks blocks and the last to finish
// measures the shift and decides.
//
// With ref_shift the shift is the reference's own measure (cluster.cu:40-50,
// :73-87): it compares the new planar centroids, entry j = d * K + k, with
// the words its workspace holds at float offset 2N at that point, which are
//   j < K:  1 / n_j (centroids.cu:40-63 writes the reciprocal sizes there);
//   j >= K: the distance of point (2N + j) / K to centroid (2N + j) % K of
//           the iteration's input (label.cu:80-88 writes the N x K distance
//           matrix from offset 0), sum of squares in dimension order;
// and sums (c_new[j] - word[j])^2 in FP32 in j order.
template <int LAYOUT, int DIM>
__global__ void __launch_bounds__(kFormMaxThreads) form_kernel(FormArgs a) {
  __shared__ float part[kFormSlots];
  __shared__ int stop, last, more;
  pdl_wait();
  if (threadIdx.x == 0) stop = __ldcg(&a.L.state->done);
  __syncthreads();
  if (stop) return;
  const int K = a.K;
  const int64_t kd = (int64_t)K * DIM;
  const float* c_old = a.L.cur + (size_t)((a.i - 1) & 1) * kd;
  float* c_new = a.L.cur + (size_t)(a.i & 1) * kd;
  const int nt = (int)blockDim.x;
  for (int slot = (int)(blockIdx.x + threadIdx.x * gridDim.x); slot < kFormSlots;
       slot += (int)gridDim.x * nt) {
    float acc = 0.0f;
    for (int64_t idx = slot; idx < kd; idx += kFormSlots) {
      const int d = (int)(idx / K), k = (int)(idx - (int64_t)d * K);
      const float c = __ldcg(c_old + idx);
      const unsigned n = __ldcg(a.L.cnt + k);
      const size_t s = (size_t)k * DIM + d;
      const float cn = n ? fix::mean(__ldcg(a.L.lo + s), __ldcg(a.L.hi + s), n) : c;
      a.L.lo[s] = 0ull;
      a.L.hi[s] = 0ull;
      __stcg(c_new + idx, cn);
      const float df = __fsub_rn(cn, c);
      acc = __fadd_rn(acc, __fmul_rn(df, df));
    }
    if (gridDim.x == 1) part[slot] = acc;
    else __stcg(a.L.part + slot, acc);
  }
  if (gridDim.x > 1) {
    // the block that finishes last has every block's words
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&a.L.state->arrived, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < kFormSlots; i += nt) part[i] = __ldcg(a.L.part + i);
  } else {
    __syncthreads();   // (the shift's words read other threads' centroids)
  }
  if (DIM == 3 && a.ref_shift) {
    const int64_t base = 2 * a.P.n;
    for (int64_t j = threadIdx.x; j < 3 * (int64_t)K; j += nt) {
      float word;
      if (j < K) {
        word = __fdiv_rn(1.0f, (float)__ldcg(a.L.cnt + j));
      } else {
        const int64_t e = base + j;
        const int64_t px = e / K;
        const int c = (int)(e - px * K);
        float f[DIM];
        load_px<LAYOUT, DIM>(a.P, px, f);
        float w = 0.0f;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          const float t = __fsub_rn(f[d], __ldcg(c_old + (int64_t)d * K + c));
          w = d == 0 ? __fmul_rn(t, t) : __fadd_rn(w, __fmul_rn(t, t));
        }
        word = w;
      }
      const float t = __fsub_rn(__ldcg(c_new + j), word);
      a.L.word[j] = __fmul_rn(t, t);
    }
  }
  __syncthreads();
  for (int s = kFormSlots / 2; s > 0; s >>= 1) {
    for (int i = threadIdx.x; i < s; i += nt) part[i] = __fadd_rn(part[i], part[i + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    float sq = part[0];
    if (DIM == 3 && a.ref_shift) {
      sq = 0.0f;
      for (int64_t j = 0; j < 3 * (int64_t)K; ++j) sq = __fadd_rn(sq, a.L.word[j]);
    }
    const float delta = sqrtf(sq);
    const float old_delta = a.L.state->delta;
    const bool m = a.i < a.max_iter && fabsf(delta - old_delta) > a.threshold;
    a.L.state->delta = delta;
    a.L.state->iters = a.i;
    a.L.state->arrived = 0u;
    if (!m) {
      a.L.state->done = 1;
      if (a.d_iter) *a.d_iter = a.i;
    }
    more = m ? 1 : 0;
  }
  __syncthreads();
  if (!more)
    for (int64_t idx = threadIdx.x; idx < kd; idx += nt)
      a.centroids[idx] = __ldcg(c_new + idx);
  for (int k = threadIdx.x; k < K; k += nt) a.L.cnt[k] = 0u;
}

size_t workspace_bytes(int K, int dim) { return carve(nullptr, K, dim).bytes; }

// The width of the tiles (as a power of two) and their number.  64 x 16 pixels
// keep the candidates of an image few; where that shape leaves much of its tiles
// outside the image (rows or columns shorter than a tile's), the shape with the
// fewest tiles is taken instead, and features that do not depend on the place
// (`xy` false) are taken as one long row.  400 thousand points in one row, K =
// 1500, 3-D: 64 x 16 tiles 3.4 ms an iteration, 1024 x 1 0.26.  From 1024
// clusters on a place-independent tile prunes less, and the line lies lower (641
// x 479, a tenth more tiles: K = 1500 218 against 194 us, K = 512 96 against 112).
static int tile_width_log2(Points& P, int K, bool xy, int64_t* tiles) {
  auto count = [&](int tw) {
    const int64_t w = 1 << tw, h = 1 << (kTilePxLog2 - tw);
    const int64_t rows = (P.n + P.width - 1) / P.width;
    return (P.width + w - 1) / w * ((rows + h - 1) / h);
  };
  int best = kTileWLog2;
  *tiles = count(best);
  const int64_t least = (P.n + (1 << kTilePxLog2) - 1) >> kTilePxLog2;
  const int64_t over = xy || K < 1024 ? 8 : 16;   // an eighth, or a sixteenth, more
  if (*tiles * over <= least * (over + 1)) return best;
  if (!xy) {
    P.width = (int)P.n;
    *tiles = least;
    return kTilePxLog2;
  }
  for (int tw = 2; tw <= kTilePxLog2; ++tw)
    if (count(tw) < *tiles) {
      best = tw;
      *tiles = count(tw);
    }
  return best;
}

template <int LAYOUT, int DIM>
static int queue(bool cluster, Points P, int K, const float* cent, float* centroids,
                 int32_t* labels, const Layout& L, int max_iter, float threshold, int ref_shift,
                 int32_t* d_iter, const StageHeaders& own, cudaStream_t st) {
  DeviceInfo di;
  SG_TRY(device_info(&di));
  int per_sm = 0;
  constexpr bool kXY = LAYOUT != SPLIT_LAYOUT_PLANAR && DIM == 5;
  constexpr int kOther = kXY ? 0 : kTilePxLog2;
  int64_t blocks;
  const int tw = tile_width_log2(P, K, kXY, &blocks);
  auto ak = tw == kTileWLog2 ? cluster ? assign_kernel<LAYOUT, DIM, true, kTileWLog2>
                                       : assign_kernel<LAYOUT, DIM, false, kTileWLog2>
            : cluster        ? assign_kernel<LAYOUT, DIM, true, kOther>
                             : assign_kernel<LAYOUT, DIM, false, kOther>;
  SG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ak, kThreads, 0));
  if (per_sm < 1) return SPLIT_ERR_UNSUPPORTED;
  const int64_t cap = (int64_t)di.sm_count * per_sm;
  if (blocks > cap) blocks = cap;
  AssignArgs aa{};
  aa.P = P;
  aa.tile_w_log2 = tw;
  aa.K = K;
  aa.labels = labels;
  aa.state = L.state;
  aa.lo = L.lo;
  aa.hi = L.hi;
  aa.cnt = L.cnt;
  aa.status = &L.hdr->status;
  if (!cluster) {
    aa.cent = cent;
    SG_CUDA_TRY(launch_pdl(ak, dim3((unsigned)blocks), dim3(kThreads), 0, st, aa));
    return launch_status();
  }
  int64_t sb = ((int64_t)K * DIM + 255) / 256;
  if (sb > di.sm_count * 4) sb = di.sm_count * 4;
  SG_CUDA_TRY(launch_pdl(setup_kernel, dim3((unsigned)sb), dim3(256), 0, st, L, K, DIM, cent,
                         d_iter, max_iter, own));
  SG_TRY(launch_status());
  FormArgs fa{};
  fa.L = L;
  fa.P = P;
  fa.K = K;
  fa.max_iter = max_iter;
  fa.threshold = threshold;
  fa.ref_shift = ref_shift;
  fa.centroids = centroids;
  fa.d_iter = d_iter;
  const size_t kd = (size_t)K * DIM;
  // few values: one block's divisions take less than the blocks' meeting
  const bool few = kd <= kFormFew;
  for (int i = 1; i <= max_iter; ++i) {
    aa.cent = L.cur + (size_t)((i - 1) & 1) * kd;
    SG_CUDA_TRY(launch_pdl(ak, dim3((unsigned)blocks), dim3(kThreads), 0, st, aa));
    SG_TRY(launch_status());
    fa.i = i;
    SG_CUDA_TRY(launch_pdl(form_kernel<LAYOUT, DIM>, dim3(few ? 1 : kFormBlocks),
                           dim3(few ? kFormMaxThreads : kFormThreads), 0, st, fa));
    SG_TRY(launch_status());
  }
  return SPLIT_OK;
}

int run(bool cluster, const void* points, int layout, int dim, int64_t n, int width,
        float xy_scale, float* centroids, const float* cent_in, int K, int32_t* labels,
        void* ws, size_t ws_bytes, int max_iter, float threshold, int32_t* d_iter,
        cudaStream_t st, const StageHeaders& own) {
  const int ref_shift = (layout & SPLIT_KMEANS_REFERENCE_SHIFT) ? 1 : 0;
  layout &= ~(SPLIT_FEATURES_UNIT_RANGE | SPLIT_KMEANS_REFERENCE_SHIFT);
  if (!points || !cent_in || !labels || n <= 0 || n > 0x7fffffffLL || width < 1)
    return SPLIT_ERR_INVALID;
  if (K < kMinK || K > kMaxClusters || (dim != 3 && dim != 5)) return SPLIT_ERR_INVALID;
  if (layout < SPLIT_LAYOUT_PLANAR || layout > SPLIT_LAYOUT_RGB8) return SPLIT_ERR_INVALID;
  if (layout == SPLIT_LAYOUT_FLOAT4 && (reinterpret_cast<uintptr_t>(points) & 15))
    return SPLIT_ERR_INVALID;
  // the reference's shift: 3-D clustering, every word it reads inside the
  // N x K distance matrix
  if (ref_shift && (!cluster || dim != 3 || n * (K - 2) < 3 * (int64_t)K))
    return SPLIT_ERR_INVALID;
  Layout l = carve(nullptr, K, dim);
  if (!ws || ws_bytes < l.bytes || (reinterpret_cast<uintptr_t>(ws) & 255))
    return SPLIT_ERR_WORKSPACE;
  l = carve(ws, K, dim);
  const Points P{points, n, width, xy_scale};
  if (cluster && max_iter <= 0) max_iter = 0;
#define SG_KMW_CASE(LY, D)                                                                  \
  if (layout == LY && dim == D)                                                             \
    return queue<LY, D>(cluster, P, K, cent_in, centroids, labels, l, max_iter, threshold,  \
                        ref_shift, d_iter, own, st);
  SG_KMW_CASE(SPLIT_LAYOUT_PLANAR, 3)
  SG_KMW_CASE(SPLIT_LAYOUT_PLANAR, 5)
  SG_KMW_CASE(SPLIT_LAYOUT_FLOAT4, 3)
  SG_KMW_CASE(SPLIT_LAYOUT_FLOAT4, 5)
  SG_KMW_CASE(SPLIT_LAYOUT_RGB8, 3)
  SG_KMW_CASE(SPLIT_LAYOUT_RGB8, 5)
#undef SG_KMW_CASE
  return SPLIT_ERR_INVALID;
}

}  // namespace kmw
}  // namespace sg
