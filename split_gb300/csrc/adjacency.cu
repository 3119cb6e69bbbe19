// Segment adjacency: the edge list of pixels that border another segment
// (8-neighbourhood) and the sorted list of distinct (segment, neighbouring
// segment) pairs.
//
// Restates split/src/split/device/ccl/segment_adjacency.cu:
//   segment_adjacency_edges (:170-254): for every pixel i in index order and
//     every in-image neighbour j in the order NW, N, NE, W, E, SW, S, SE
//     (NeighbourKeys, :112-142) with labels[i] != labels[j] (the remove_if
//     at :239-243 keeps the survivors in order), one edge (i, j); the m
//     sources go to edges[0, m), the targets to edges[m, 2m) (:249-251).
//   segment_adjacency (:256-289): the label pairs (labels[i], labels[j]) of
//     those edges, sorted by key then value (:279-284), without repeats
//     (:286).
//
// No N x 16 edge array and no comparison sort of the edges: the edges are
// written by an order-preserving compaction (per-block counts, one scan, a
// write pass that recomputes each item's outputs).  The pairs need no order
// before the sort, and a boundary repeats its pair at every pixel: each tile
// keeps its distinct pairs in a shared-memory set and appends those (a 1080p
// labelling of 400 segments and 4000 single pixels: 12 to 20 thousand keys to
// sort for 0.9 million edges).  One cooperative launch sorts the keys, 64 bits,
// and keeps one of each: a few by their ranks in sorted tiles, more by a stable
// LSD radix sort (8-bit digits; a digit equal in every key is skipped).
// Counts come back through device words.
#include <algorithm>

#include "common.cuh"

namespace sg {
namespace adj {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;                    // items per thread
constexpr int kTile = kThreads * kItems;      // items per block
constexpr int kScanThreads = 1024;
// 16 n edge words must stay addressable with int32 (as in the reference)
constexpr int64_t kMaxPixels = (1ll << 27) - 1;

struct Layout {
  WsHeader* hdr;
  int* block_sum;                   // [blocks + 1]: per-block counts, then their prefix
  int* total;                       // [2]: keys to sort
  unsigned long long* bits;         // [2]: OR and AND of every pair key
  unsigned long long* keys[2];      // [8 n] each, whole rank tiles: pair keys, sort ping-pong
  unsigned* hist;                   // [256 * sort blocks + 256]: digit counts, then offsets;
                                    // the digits' totals
  size_t bytes;
};

__host__ __device__ inline int blocks_of(int64_t items) {
  return (int)((items + kTile - 1) / kTile);
}

// Up to kFewKeys keys are ranked, more are sorted by digits.  Ranking costs
// every key a search in every tile of kRankTile keys and three barriers; a
// digit pass three barriers and two passes over the keys, six to eight times.
constexpr int64_t kFewKeys = 1 << 17;
constexpr int kRankBits = 10, kRankTile = 1 << kRankBits;

static Layout carve(void* ws, int64_t n, bool pairs) {
  Carver c(ws);
  Layout l{};
  l.hdr = c.take<WsHeader>(1);
  const int64_t items = pairs ? 8 * n : n;
  l.block_sum = c.take<int>((size_t)blocks_of(items) + 1);
  l.total = c.take<int>(2);
  l.bits = c.take<unsigned long long>(2);
  if (pairs) {
    const size_t cap = (size_t)((8 * n + kRankTile - 1) / kRankTile * kRankTile);
    l.keys[0] = c.take<unsigned long long>(cap);
    l.keys[1] = c.take<unsigned long long>(cap);
    l.hist = c.take<unsigned>((size_t)256 * blocks_of(8 * n) + 256);
  }
  l.bytes = c.size();
  return l;
}

// neighbour d of pixel (x, y) in the reference's order, or -1 outside
__device__ __forceinline__ int neighbour(int x, int y, int w, int h, int d) {
  const int dx = (d == 0 || d == 3 || d == 5) ? -1 : (d == 2 || d == 4 || d == 7) ? 1 : 0;
  const int dy = d < 3 ? -1 : d > 4 ? 1 : 0;
  const int nx = x + dx, ny = y + dy;
  return (nx >= 0 && nx < w && ny >= 0 && ny < h) ? ny * w + nx : -1;
}

// A pair key whose unsigned order is the (key, value) order of signed ints.
__device__ __forceinline__ unsigned long long pair_key(int a, int b) {
  return ((unsigned long long)((unsigned)a ^ 0x80000000u) << 32) |
         (unsigned long long)((unsigned)b ^ 0x80000000u);
}

// ---- stable LSD radix sort bookkeeping ---------------------------------------
// Pass p sorts on bits [8 p, 8 p + 8).  A pass whose digit is equal in every
// key is skipped; the buffer a pass reads is keys[q & 1], q the number of
// passes before it that were not skipped.
__device__ __forceinline__ bool pass_runs(const unsigned long long* bits, int p) {
  return (((bits[0] ^ bits[1]) >> (8 * p)) & 0xffull) != 0ull;
}
__device__ __forceinline__ int pass_parity(const unsigned long long* bits, int p) {
  int q = 0;
  for (int k = 0; k < p; ++k) q += pass_runs(bits, k);
  return q & 1;
}

// the neighbours of pixel i that border another segment, a bit each
__device__ __forceinline__ unsigned edge_mask(const int32_t* lab, int w, int h, int i) {
  const int x = i % w, y = i / w, v = __ldg(lab + i);
  unsigned m = 0;
#pragma unroll
  for (int d = 0; d < 8; ++d) {
    const int j = neighbour(x, y, w, h, d);
    if (j >= 0 && __ldg(lab + j) != v) m |= 1u << d;
  }
  return m;
}

// Edges per tile of pixels (contiguous kItems per thread).
__global__ void __launch_bounds__(kThreads) count_kernel(const int32_t* __restrict__ lab, int w,
                                                          int h, int* block_sum) {
  pdl_wait();
  const int n = w * h;
  __shared__ int ws[kWarps];
  int c = 0;
  for (int k = 0; k < kItems; ++k) {
    const int i = blockIdx.x * kTile + threadIdx.x * kItems + k;
    if (i < n) c += __popc(edge_mask(lab, w, h, i));
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int k = 0; k < kWarps; ++k) s += ws[k];
    block_sum[blockIdx.x] = s;
  }
}

// Exclusive scan of one value per thread over the block; the total to every
// thread.
template <int THREADS, typename T>
__device__ T scan_threads(T v, T& total) {
  __shared__ T part[THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += u;
  }
  __syncthreads();
  if (lane == 31) part[warp] = s;
  __syncthreads();
  T before = 0, all = 0;
#pragma unroll
  for (int k = 0; k < THREADS / 32; ++k) {
    if (k == warp) before = all;
    all += part[k];
  }
  total = all;
  return before + s - v;
}

// Exclusive scan of `count` words in place by one block, in tiles of THREADS
// with a carried prefix; returns the grand total.
template <int THREADS, typename T>
__device__ T block_scan(T* a, int count) {
  T carry = 0;
  for (int t0 = 0; t0 < count; t0 += THREADS) {
    const int i = t0 + threadIdx.x;
    T total;
    const T before = scan_threads<THREADS, T>(i < count ? a[i] : 0, total);
    if (i < count) a[i] = carry + before;
    carry += total;
  }
  return carry;
}

// Prefix of the block totals (their total to *total).
__global__ void __launch_bounds__(kScanThreads) scan_blocks_kernel(int count, int* block_sum,
                                                                   int* total, WsHeader* hdr) {
  pdl_wait();
  if (threadIdx.x == 0) hdr->stamp = kStampDirty;
  const int all = block_scan<kScanThreads>(block_sum, count);
  if (threadIdx.x == 0) *total = all;
}

// Writes every pixel's edges at their place in the order of the pixels (a
// block-wide exclusive scan of the threads' counts, plus the tile's prefix).
__global__ void __launch_bounds__(kThreads) write_kernel(const int32_t* __restrict__ lab, int w,
                                                          int h, const int* block_sum,
                                                          const int* total, int32_t* edges) {
  pdl_wait();
  const int n = w * h;
  const int first = blockIdx.x * kTile + threadIdx.x * kItems;
  int c = 0;
  for (int k = 0; k < kItems; ++k)
    if (first + k < n) c += __popc(edge_mask(lab, w, h, first + k));
  int all;
  int at = block_sum[blockIdx.x] + scan_threads<kThreads>(c, all);
  const int m = *total;
  for (int k = 0; k < kItems; ++k) {
    const int i = first + k;
    if (i >= n) break;
    const int x = i % w, y = i / w;
    for (unsigned mask = edge_mask(lab, w, h, i); mask; mask &= mask - 1) {
      edges[at] = i;
      edges[m + at] = neighbour(x, y, w, h, __ffs(mask) - 1);
      ++at;
    }
  }
}

// ---- the keys to sort ----------------------------------------------------------
// no keys and no pairs yet, the OR / AND of none, and the sort's barrier
__global__ void reset_kernel(const Layout l, int* d_count) {
  pdl_wait();
  if (threadIdx.x == 0) {
    *d_count = 0;
    l.hdr->barrier_count = 0u;
    l.hdr->stamp = kStampDirty;
    l.total[0] = 0;
    l.bits[0] = 0ull;
    l.bits[1] = ~0ull;
  }
}

// The distinct pair keys of one tile of pixels, appended to keys[0] in any
// order.  A pair borders both ways, so four of the eight neighbours (east,
// south-west, south, south-east) find it and both its keys are appended; a
// pair that the set has no room for within a short probe is appended as it is
// (the sort brings the copies together), after a shorter one from then on: in
// noise nearly every pair fails, and a failed probe takes as long as 16 loads.  A key is never 0: its two labels
// differ.  Every pair appended has an edge of its own, at most 4 n there are,
// so 8 n keys hold all.  The pixels that have an edge go to a list first, which
// the block walks densely.  1080p, 400 segments and 4000 single pixels: 23 us
// with all eight neighbours at every pixel, 14 us.
constexpr int kPixH = 32, kPixW = 64, kHaloW = kPixW + 2, kHaloH = kPixH + 1;
constexpr int kSetBits = 10, kSetProbes = 16;
constexpr int kFullProbes = 4;   // once a pair has found no room
static_assert(kPixH * kPixW <= 1 << 11 && kThreads % kPixW == 0, "list entries; whole rows");
__global__ void __launch_bounds__(kThreads) pair_kernel(const int32_t* __restrict__ lab, int w,
                                                         int h, const Layout l) {
  __shared__ int tile[kHaloH * kHaloW];
  __shared__ unsigned long long set[1 << kSetBits];
  __shared__ unsigned short todo[kPixH * kPixW];   // local pixel, then its edges in 4 bits
  __shared__ int ntodo, found, base, full;
  pdl_wait();
  const int tiles_x = (w + kPixW - 1) / kPixW;
  const int x0 = (int)(blockIdx.x % tiles_x) * kPixW, y0 = (int)(blockIdx.x / tiles_x) * kPixH;
  if (threadIdx.x == 0) ntodo = found = full = 0;
  // pixels outside the image take the nearest inside: the pixel itself or
  // another of its neighbours, so no pair is added
  for (int q = threadIdx.x; q < kHaloH * kHaloW; q += kThreads) {
    const int y = min(y0 + q / kHaloW, h - 1);
    const int x = min(max(x0 - 1 + q % kHaloW, 0), w - 1);
    tile[q] = __ldg(lab + (size_t)y * w + x);
  }
  for (int i = threadIdx.x; i < (1 << kSetBits); i += kThreads) set[i] = 0ull;
  __syncthreads();
  const int lane = threadIdx.x & 31, lx = threadIdx.x % kPixW;
#pragma unroll
  for (int r = 0; r < kPixH; r += kThreads / kPixW) {
    const int ly = threadIdx.x / kPixW + r;
    const int* c = tile + ly * kHaloW + lx + 1;
    const int v = c[0];
    unsigned m = 0u;
    if (x0 + lx < w && y0 + ly < h)
      m = (c[1] != v ? 1u : 0u) | (c[kHaloW - 1] != v ? 2u : 0u) | (c[kHaloW] != v ? 4u : 0u) |
          (c[kHaloW + 1] != v ? 8u : 0u);
    const unsigned any = __ballot_sync(0xffffffffu, m != 0u);
    if (any) {
      int at = lane == 0 ? atomicAdd(&ntodo, __popc(any)) : 0;
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(any & ((1u << lane) - 1u));
      if (m) todo[at] = (unsigned short)((ly * kPixW + lx) << 4 | m);
    }
  }
  __syncthreads();
  const int nt = ntodo;
  if (nt == 0) return;
  unsigned long long o_or = 0ull, o_and = ~0ull;
  auto append = [&](unsigned long long key, int at) {
    const unsigned long long back = key << 32 | key >> 32;
    l.keys[0][at] = key;
    l.keys[0][at + 1] = back;
    o_or |= key | back;
    o_and &= key & back;
  };
  for (int q0 = (int)threadIdx.x - lane; q0 < nt; q0 += kThreads) {   // whole warps
    const int q = q0 + lane;
    const unsigned item = q < nt ? todo[q] : 0u, m = item & 15u, px = item >> 4;
    const int* c = tile + (px / kPixW) * kHaloW + px % kPixW + 1;
    const int v = *c;
    const int t[4] = {c[1], c[kHaloW - 1], c[kHaloW], c[kHaloW + 1]};
    const int probes = *(volatile int*)&full ? kFullProbes : kSetProbes;
    unsigned out = 0u;   // pairs that found no room
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      bool add = m >> a & 1u;
#pragma unroll
      for (int b = 0; b < a; ++b) add = add && t[b] != t[a];
      if (!add) continue;
      const unsigned long long key = pair_key(min(v, t[a]), max(v, t[a]));
      unsigned s = (unsigned)((key * 0x9E3779B97F4A7C15ull) >> (64 - kSetBits));
      bool in = false;
      for (int probe = 0; probe < probes && !in; ++probe, s = (s + 1) & ((1 << kSetBits) - 1)) {
        unsigned long long k = *(volatile unsigned long long*)&set[s];
        if (k == 0ull) k = atomicCAS(&set[s], 0ull, key);
        in = k == 0ull || k == key;
      }
      if (!in) out |= 1u << a;
    }
    __syncwarp();
    if (!__any_sync(0xffffffffu, out != 0u)) continue;
    *(volatile int*)&full = 1;
    // one place in the list per warp
    const int mine = 2 * __popc(out);
    int at = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += u;
    }
    int first = lane == 31 ? atomicAdd(l.total, at) : 0;
    first = __shfl_sync(0xffffffffu, first, 31);
    at += first - mine;
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if (out >> a & 1u) {
        append(pair_key(min(v, t[a]), max(v, t[a])), at);
        at += 2;
      }
  }
  __syncthreads();
  // the set's keys, with one place in the list per block
  constexpr int kMine = (1 << kSetBits) / kThreads;
  int mine = 0;
#pragma unroll
  for (int k = 0; k < kMine; ++k) mine += set[threadIdx.x + k * kThreads] != 0ull;
  int at = mine ? atomicAdd(&found, 2 * mine) : 0;
  __syncthreads();
  if (threadIdx.x == 0) base = found ? atomicAdd(l.total, found) : 0;
  __syncthreads();
  at += base;
#pragma unroll
  for (int k = 0; k < kMine; ++k) {
    const unsigned long long key = set[threadIdx.x + k * kThreads];
    if (key == 0ull) continue;
    append(key, at);
    at += 2;
  }
  // digits that differ between keys (a digit equal in all is not sorted on)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    o_or |= __shfl_xor_sync(0xffffffffu, o_or, o);
    o_and &= __shfl_xor_sync(0xffffffffu, o_and, o);
  }
  if (lane == 0 && (o_or != 0ull || o_and != ~0ull)) {
    atomicOr(l.bits, o_or);
    atomicAnd(l.bits + 1, o_and);
  }
}

// ---- distinct keys in order, by their ranks -----------------------------------
// Tiles of kRankTile keys are sorted in shared memory; a key that no earlier
// tile holds (and that is the first of its run in its own) goes out, at the
// number of such keys below it in all tiles: one binary search per tile, whose
// loads meet in the caches, the keys of a warp being neighbours in order.
// Bound by the barriers and the searches' latency, kWide tiles in flight.
// 12 thousand keys (12 tiles): 28 us, of which the three barriers are 7.

// places of `key` in the kWide tiles from t0 on (tiles past the last repeat it)
constexpr int kWide = 16;
__device__ __forceinline__ void lower_bounds(const unsigned long long* a, int t0, int tiles,
                                             unsigned long long key, int (&at)[kWide]) {
  int base[kWide];
#pragma unroll
  for (int g = 0; g < kWide; ++g) {
    base[g] = min(t0 + g, tiles - 1) * kRankTile;
    at[g] = 0;
  }
#pragma unroll
  for (int step = kRankTile / 2; step > 0; step >>= 1)
#pragma unroll
    for (int g = 0; g < kWide; ++g)
      if (a[base[g] + at[g] + step - 1] < key) at[g] += step;
#pragma unroll
  for (int g = 0; g < kWide; ++g)
    if (a[base[g] + at[g]] < key) ++at[g];
}

// Bitonic sort of a block's kRankTile keys, kPer per thread: key j of a thread
// is element warp * kRun + 32 j + lane.  Partners up to 16 apart are in another
// lane, 32 and 64 apart in the same thread, further in another warp and reached
// through shared memory (6 of the 55 stages; all of them through it took 13 us
// a tile).
constexpr int kPer = kRankTile / kThreads, kRun = 32 * kPer;
static_assert(kPer == 4, "partners within a thread");

__device__ __forceinline__ void sort_tile(unsigned long long (&k)[kPer], unsigned long long* sm) {
  const int e0 = (threadIdx.x >> 5) * kRun + (threadIdx.x & 31);
  for (int size = 2; size <= kRankTile; size <<= 1)
    for (int d = size >> 1; d > 0; d >>= 1) {
      unsigned long long o[kPer];
      if (d >= kRun) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j) sm[e0 + 32 * j] = k[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j) o[j] = sm[(e0 + 32 * j) ^ d];
      } else if (d >= 32) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) o[j] = d == 32 ? k[j ^ 1] : k[j ^ 2];
      } else {
#pragma unroll
        for (int j = 0; j < kPer; ++j) o[j] = __shfl_xor_sync(0xffffffffu, k[j], d);
      }
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int e = e0 + 32 * j;
        // the lower partner keeps the smaller key where the run ascends
        const bool smaller = ((e & d) == 0) == ((e & size) == 0);
        if ((o[j] < k[j]) == smaller) k[j] = o[j];
      }
    }
}

__device__ void rank_keys(const Layout& l, int n, int32_t* out0, int32_t* out1, int* d_count,
                          unsigned long long* sm) {
  const int tiles = (n + kRankTile - 1) / kRankTile;
  // warps of consecutive keys, dealt out over the blocks
  const int step = gridDim.x * kThreads;
  const int first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
  // a tile's keys in order, filled up with the largest value (no key: the two
  // labels of a pair differ)
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    unsigned long long k[kPer];
    const int e0 = (threadIdx.x >> 5) * kRun + (threadIdx.x & 31);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = t * kRankTile + e0 + 32 * j;
      k[j] = i < n ? l.keys[0][i] : ~0ull;
    }
    sort_tile(k, sm);
#pragma unroll
    for (int j = 0; j < kPer; ++j) l.keys[1][t * kRankTile + e0 + 32 * j] = k[j];
  }
  if (!grid_barrier(l.hdr)) return;
  // per tile, the keys that go out (1), then the number of those before each
  // and, past the last, of all
  int* const out = reinterpret_cast<int*>(l.keys[0]);   // [tiles][kRankTile + 1]
  const unsigned long long* const a = l.keys[1];
  for (int i = first; i < n; i += step) {
    const unsigned long long key = a[i];
    const int t = i / kRankTile;
    bool seen = i % kRankTile != 0 && a[i - 1] == key;
    for (int e = 0; e < t && !seen; e += kWide) {
      int at[kWide];
      lower_bounds(a, e, t, key, at);
#pragma unroll
      for (int g = 0; g < kWide; ++g)
        seen |= at[g] < kRankTile && a[min(e + g, t - 1) * kRankTile + at[g]] == key;
    }
    out[i + t] = !seen;
  }
  if (!grid_barrier(l.hdr)) return;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    int* const o = out + t * (kRankTile + 1);
    int v[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = threadIdx.x * kPer + k;
      v[k] = t * kRankTile + i < n ? o[i] : 0;
      sum += v[k];
    }
    int all;
    int at = scan_threads<kThreads>(sum, all);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      o[threadIdx.x * kPer + k] = at;
      at += v[k];
    }
    if (threadIdx.x == 0) o[kRankTile] = all;
  }
  if (!grid_barrier(l.hdr)) return;
  for (int i = first; i < n; i += step) {
    const int* const o = out + i + i / kRankTile;
    if (o[0] == o[1]) continue;
    const unsigned long long key = a[i];
    int pos = 0;
    for (int e = 0; e < tiles; e += kWide) {
      int at[kWide];
      lower_bounds(a, e, tiles, key, at);
#pragma unroll
      for (int g = 0; g < kWide; ++g)
        if (e + g < tiles) pos += out[(e + g) * (kRankTile + 1) + at[g]];
    }
    out0[pos] = (int)((unsigned)(key >> 32) ^ 0x80000000u);
    out1[pos] = (int)((unsigned)key ^ 0x80000000u);
  }
  if (blockIdx.x == 0) {
    int mine = 0, all;
    for (int t = threadIdx.x; t < tiles; t += kThreads) mine += out[t * (kRankTile + 1) + kRankTile];
    scan_threads<kThreads>(mine, all);
    if (threadIdx.x == 0) *d_count = all;
  }
}

// ---- distinct keys in order, by a stable LSD radix sort -----------------------
// Per digit: counts per tile, digit-major (hist[d * nb + b]); each digit's
// counts scanned by one block, its total behind them; then the stable scatter.
// A block moves a tile's items in index order, kThreads at a time; an item's
// place is its digit's offset for the tile, plus the items of that digit in
// earlier rounds, in earlier warps of this round, and in earlier lanes of its
// warp.  Last, the first key of every run goes out.
struct RadixSmem {
  unsigned off[256], wc[kWarps][256];
};

__device__ void radix_keys(const Layout& l, int n, int32_t* out0, int32_t* out1, int* d_count,
                           RadixSmem& sm) {
  const int nb = blocks_of(n), warp = threadIdx.x >> 5;
  unsigned* const totals = l.hist + (size_t)256 * nb;
  unsigned lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  for (int p = 0; p < 8; ++p) {
    if (!pass_runs(l.bits, p)) continue;
    const int q = pass_parity(l.bits, p);
    const unsigned long long* in = l.keys[q];
    unsigned long long* out = l.keys[q ^ 1];
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
      sm.off[threadIdx.x] = 0;
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < kItems; ++k) {
        const int i = (b * kItems + k) * kThreads + threadIdx.x;
        if (i < n) atomicAdd(&sm.off[(in[i] >> (8 * p)) & 0xff], 1u);
      }
      __syncthreads();
      l.hist[(size_t)threadIdx.x * nb + b] = sm.off[threadIdx.x];
      __syncthreads();
    }
    if (!grid_barrier(l.hdr)) return;
    for (int d = blockIdx.x; d < 256; d += gridDim.x) {
      const unsigned all = block_scan<kThreads>(l.hist + (size_t)d * nb, nb);
      if (threadIdx.x == 0) totals[d] = all;
    }
    if (!grid_barrier(l.hdr)) return;
    unsigned all;
    const unsigned below = scan_threads<kThreads>(totals[threadIdx.x], all);
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
      sm.off[threadIdx.x] = below + l.hist[(size_t)threadIdx.x * nb + b];
      for (int w = 0; w < kWarps; ++w) sm.wc[w][threadIdx.x] = 0;
      __syncthreads();
      for (int k = 0; k < kItems; ++k) {
        const int i = (b * kItems + k) * kThreads + threadIdx.x;
        if (i - (int)threadIdx.x >= n) break;   // the same in every thread
        const bool ok = i < n;
        const unsigned long long key = ok ? in[i] : 0ull;
        const int digit = ok ? (int)((key >> (8 * p)) & 0xff) : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, digit);
        const int rank = __popc(peers & lt);
        if (ok && rank == 0) sm.wc[warp][digit] = __popc(peers);
        __syncthreads();
        if (ok) {
          unsigned pos = sm.off[digit] + rank;
          for (int w = 0; w < warp; ++w) pos += sm.wc[w][digit];
          out[pos] = key;
        }
        __syncthreads();
        // the round's counts move into the digit offsets
        unsigned t = 0;
        for (int w = 0; w < kWarps; ++w) {
          t += sm.wc[w][threadIdx.x];
          sm.wc[w][threadIdx.x] = 0;
        }
        sm.off[threadIdx.x] += t;
        __syncthreads();
      }
    }
    if (!grid_barrier(l.hdr)) return;
  }
  const unsigned long long* const a = l.keys[pass_parity(l.bits, 8)];
  auto starts = [&](int i) { return i < n && (i == 0 || a[i] != a[i - 1]); };
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    int c = 0, all;
#pragma unroll 4
    for (int k = 0; k < kItems; ++k) c += starts((b * kItems + k) * kThreads + threadIdx.x);
    scan_threads<kThreads>(c, all);
    if (threadIdx.x == 0) l.block_sum[b] = all;
  }
  if (!grid_barrier(l.hdr)) return;
  if (blockIdx.x == 0) {
    const int all = block_scan<kThreads>(l.block_sum, nb);
    if (threadIdx.x == 0) *d_count = all;
  }
  if (!grid_barrier(l.hdr)) return;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    int base = l.block_sum[b];
    for (int k = 0; k < kItems; ++k) {
      const int i = (b * kItems + k) * kThreads + threadIdx.x;
      int all;
      const int at = base + scan_threads<kThreads>((int)starts(i), all);
      if (starts(i)) {
        out0[at] = (int)((unsigned)(a[i] >> 32) ^ 0x80000000u);
        out1[at] = (int)((unsigned)a[i] ^ 0x80000000u);
      }
      base += all;
    }
  }
}

// One cooperative launch: the number of keys is known on the device only, and
// launches for the path not taken would cost more than ranking does.
// Two blocks per SM: the searches' registers, and half the arrivals of four.
__global__ void __launch_bounds__(kThreads, 2) sort_kernel(const Layout l, int32_t* out0,
                                                         int32_t* out1, int* d_count) {
  __shared__ union {
    unsigned long long tile[kRankTile];
    RadixSmem radix;
  } sm;
  const int n = *l.total;
  if (n <= kFewKeys) rank_keys(l, n, out0, out1, d_count, sm.tile);
  else radix_keys(l, n, out0, out1, d_count, sm.radix);
}

}  // namespace adj
}  // namespace sg

using namespace sg;

extern "C" size_t split_segment_adjacency_edges_workspace_size(int width, int height) {
  if (width < 1 || height < 1) return 0;
  return adj::carve(nullptr, (int64_t)width * height, false).bytes;
}

extern "C" int split_segment_adjacency_edges(const int32_t* labels, int width, int height,
                                             int32_t* edges, int32_t* d_count, void* workspace,
                                             size_t workspace_bytes, void* stream) {
  if (!labels || !edges || !d_count || width < 1 || height < 1) return SPLIT_ERR_INVALID;
  const int64_t n = (int64_t)width * height;
  if (n > adj::kMaxPixels) return SPLIT_ERR_INVALID;
  adj::Layout l = adj::carve(nullptr, n, false);
  if (!workspace || workspace_bytes < l.bytes || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return SPLIT_ERR_WORKSPACE;
  l = adj::carve(workspace, n, false);
  cudaStream_t st = as_stream(stream);
  const int tiles = adj::blocks_of(n);
  launch_pdl(adj::count_kernel, dim3(tiles), dim3(adj::kThreads), 0, st, labels, width, height,
             l.block_sum);
  SG_TRY(launch_status());
  launch_pdl(adj::scan_blocks_kernel, dim3(1), dim3(adj::kScanThreads), 0, st, tiles, l.block_sum,
             d_count, l.hdr);
  SG_TRY(launch_status());
  launch_pdl(adj::write_kernel, dim3(tiles), dim3(adj::kThreads), 0, st, labels, width, height,
             (const int*)l.block_sum, (const int*)d_count, edges);
  return launch_status();
}

extern "C" size_t split_segment_adjacency_workspace_size(int width, int height) {
  if (width < 1 || height < 1) return 0;
  return adj::carve(nullptr, (int64_t)width * height, true).bytes;
}

extern "C" int split_segment_adjacency(const int32_t* labels, int width, int height,
                                       int32_t* keys, int32_t* adjacency, int32_t* d_count,
                                       void* workspace, size_t workspace_bytes, void* stream) {
  if (!labels || !keys || !adjacency || !d_count || width < 1 || height < 1)
    return SPLIT_ERR_INVALID;
  const int64_t n = (int64_t)width * height;
  if (n > adj::kMaxPixels) return SPLIT_ERR_INVALID;
  adj::Layout l = adj::carve(nullptr, n, true);
  if (!workspace || workspace_bytes < l.bytes || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return SPLIT_ERR_WORKSPACE;
  l = adj::carve(workspace, n, true);
  cudaStream_t st = as_stream(stream);
  // 1: the distinct pair keys of every tile, and the digits that vary
  launch_pdl(adj::reset_kernel, dim3(1), dim3(32), 0, st, l, (int*)d_count);
  SG_TRY(launch_status());
  const int tiles = ((width + adj::kPixW - 1) / adj::kPixW) * ((height + adj::kPixH - 1) / adj::kPixH);
  launch_pdl(adj::pair_kernel, dim3(tiles), dim3(adj::kThreads), 0, st, labels, width, height, l);
  SG_TRY(launch_status());
  // 2: sorted, one of each
  DeviceInfo di;
  SG_TRY(device_info(&di));
  int per_sm = 0;
  SG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, adj::sort_kernel,
                                                            adj::kThreads, 0));
  if (per_sm < 1) return SPLIT_ERR_UNSUPPORTED;
  int* count = d_count;
  void* args[] = {&l, &keys, &adjacency, &count};
  SG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)adj::sort_kernel,
                                          dim3(di.sm_count * std::min(per_sm, 2)),
                                          dim3(adj::kThreads), args, 0, st));
  return launch_status();
}
