// Small-segment merge: a boundary-histogram pass plus a relabel.
//
// Restates split/src/split/device/ccl/merge_small_segments.cu:92-196 with its
// helpers segment_adjacency.cu:112-142 (8-neighbour edge set),
// detail/fix_map_cycles.cuh:14-44 (mutual pairs keep the larger id) and
// detail/map_until_converged.cuh:14-31 (every label follows its map chain to
// the end).  Instead of materialising 16 ints per pixel of edges and radix
// sorting them, pixels of small segments insert their (segment, neighbour
// segment) pairs into a hash table with multiplicities; each pair then bids
// for its segment with one 64-bit atomicMax:
//   MOST_BOUNDARY: (edge count << 32) | ~neighbour      (most edges, lowest id)
//   REF_CHROMA   : ~((bits(d2) << 32) | neighbour)       (least d2, lowest id)
// and the winning pair writes the segment's map entry.  A small segment that
// lies wholly inside one tile has all its pairs in that tile's table: it is
// decided there and never enters the global table.
//
// Workspace state (kept clean between calls):
//   table keys / counts / slot list   zero outside a call
//   best[n]                            zero outside a call
// Per-call arrays: size[n] (unless the caller passes component sizes),
// map[n], fin[n] (final target of every small segment), sum[n] (chroma),
// dec[n] (the decided segments).
//
// The table holds at most half its capacity (2^ceil(log2 n) slots) of pairs.
// An image cut into very many small segments can have more distinct pairs
// than that (up to about 8 per pixel).  Then the pair pass stops inserting and
// flags the overflow, and the decision kernel takes the overflow path: the
// small segments are split into classes by the top bits of a hash of their
// id, and each class goes through its own round of pair pass, bids and
// decisions in the emptied table; a class whose pairs still do not fit is
// split in two again.  Bids only compare pairs of one segment, so rounds over
// disjoint classes decide exactly what one pass over a large enough table
// would.  The chains then resolve over the decided segments.
#include <algorithm>
#include <mutex>

#include "geom.cuh"
#include "merge_state.cuh"

namespace sg {
namespace mrg {

constexpr int kThreads = 256;
// the pair pass: six blocks of 256 threads per SM (three of 512 take 8% more
// on the maze's 32768 tiles, 5% less on a 512 x 512 frame of 128)
constexpr int kPairThreads = 256, kPairBlocks = 6;
constexpr int kListThreads = 512;   // the decision launch (1024: the 4K frame 4 us more)
constexpr int kProbeCap = 1 << 16;
constexpr int kNearProbes = 4;   // from one of eight starts: eleven slots of a segment
constexpr unsigned kChainCap = 1u << 24;
// overflow path: pending classes (level, class) on a stack, and a bound on rounds
constexpr int kStackCap = 64;
constexpr unsigned kRoundCap = 1u << 20;

struct Layout {
  WsHeader* hdr;
  State* state;
  int32_t* size;
  int32_t* map;
  int32_t* fin;
  unsigned long long* best;
  double* sum;
  unsigned long long* keys;
  unsigned* counts;
  int32_t* list;
  int32_t* dec;
  int* stack;   // [1 + 2 * kStackCap]: depth, then (level, class) pairs
  int cap_log2;
  size_t bytes;
};

inline int cap_log2_for(int64_t n) {
  int l = 12;
  while ((1ll << l) < n && l < 31) ++l;
  return l;
}

inline Layout carve(void* ws, int64_t n) {
  Carver c(ws);
  Layout l;
  l.hdr = c.take<WsHeader>(1);
  l.state = c.take<State>(1);
  l.size = c.take<int32_t>((size_t)n);
  l.map = c.take<int32_t>((size_t)n);
  l.fin = c.take<int32_t>((size_t)n);
  l.best = c.take<unsigned long long>((size_t)n);
  l.sum = c.take<double>((size_t)n);
  l.cap_log2 = cap_log2_for(n);
  const size_t cap = (size_t)1 << l.cap_log2;
  l.keys = c.take<unsigned long long>(cap);
  l.counts = c.take<unsigned>(cap);
  l.list = c.take<int32_t>(cap);
  l.dec = c.take<int32_t>((size_t)n);
  l.stack = c.take<int>(1 + 2 * kStackCap);
  l.bytes = c.size();
  return l;
}

__device__ __forceinline__ unsigned long long pair_key(int s, int t) {
  return (((unsigned long long)(unsigned)s << 32) | (unsigned)t) + 1ull;
}
__device__ __forceinline__ int key_s(unsigned long long k) { return (int)((k - 1ull) >> 32); }
__device__ __forceinline__ int key_t(unsigned long long k) { return (int)(unsigned)((k - 1ull) & 0xffffffffull); }

// Adds m edges to pair (s, t) of the global table.  Returns the slot of a
// pair not seen before (which the caller lists), -1 for one already there,
// -2 (and flags the overflow) when a probe sequence runs out.
__device__ __forceinline__ int claim(const Layout& L, int s, int t, unsigned m) {
  const unsigned long long key = pair_key(s, t);
  const unsigned mask = (1u << L.cap_log2) - 1u;
  // A segment's first pairs share eleven slots, so that its claims, counts and
  // bids meet in a cache line or two; a pair that finds no room there goes on at
  // a hash of both ids.  Without that a segment of d neighbours probes a run of
  // its own pairs d long.
  unsigned h = (((unsigned)s * 0x9E3779B9u) >> (32 - L.cap_log2)) +
               (((unsigned)t * 0x9E3779B9u) >> 29);
  h &= mask;
  for (int probe = 0; probe < kProbeCap; ++probe) {
    if (probe == kNearProbes)
      h = (unsigned)((key * 0x9E3779B97F4A7C15ull) >> (64 - L.cap_log2));
    else if (probe > 0)
      h = (h + 1) & mask;
    unsigned long long k = *(volatile unsigned long long*)(L.keys + h);
    if (k == 0ull) {
      k = atomicCAS(L.keys + h, 0ull, key);
      if (k == 0ull) {
        atomicAdd(L.counts + h, m);
        return (int)h;
      }
    }
    if (k == key) {
      atomicAdd(L.counts + h, m);
      return -1;
    }
  }
  *(volatile int*)&L.state->overflow = 1;
  return -2;
}

// Lists claimed slot h at place idx.  A pair past half the table's capacity
// flags the overflow and returns false: the caller then stops inserting (the
// pass decides class by class instead), and so does every tile that starts
// after the flag is set, so the table never grows past half by more than the
// lanes running at once.  Every claimed slot is listed (the list holds as
// many entries as the table), so the table can always be cleared through it.
__device__ __forceinline__ bool list_slot(const Layout& L, unsigned idx, int h) {
  L.list[idx] = h;
  if (idx < (((1u << L.cap_log2) - 1u) >> 1)) return true;
  *(volatile int*)&L.state->overflow = 1;
  return false;
}

// claim, listing a new pair with one atomic for the lanes that arrive
// together; returns whether to go on inserting
__device__ bool insert(const Layout& L, int s, int t, unsigned m) {
  const int h = claim(L, s, t, m);
  if (h < 0) return h == -1;
  const unsigned am = __activemask();
  const int lane = threadIdx.x & 31, leader = __ffs(am) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(&L.state->list_count, (unsigned)__popc(am));
  base = __shfl_sync(am, base, leader);
  return list_slot(L, base + __popc(am & ((1u << lane) - 1u)), h);
}

// Class of segment s at split level `lev`: the top lev bits of a hash of s
// (level 0: every segment in class 0).
__device__ __forceinline__ unsigned seg_class(int s, int lev) {
  return lev == 0 ? 0u : ((unsigned)s * 2654435761u) >> (32 - lev);
}

// Sum of x over the lanes of `peers` (the lanes that hold this lane's value),
// left in the lowest of them: pairs of peers add up in log2 steps (the peer
// reduction by rank parity of E. Westphal, "Voting and Shuffling to Optimize
// Atomic Operations", 2015).
__device__ __forceinline__ double sum_peers(unsigned peers, double x) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  unsigned rank = __popc(peers & ((1u << lane) - 1u));
  unsigned above = peers & (0xfffffffeu << lane);
  while (__any_sync(full, above != 0u)) {
    const int next = __ffs(above);
    const double y = __shfl_sync(full, x, next ? next - 1 : lane);
    if (next) x += y;
    above &= __ballot_sync(full, !(rank & 1u));
    rank >>= 1;
  }
  return x;
}

// Sizes (generic path) and chroma sums; REF_CHROMA also notes whether the
// labels were already sorted (merge_small_segments.cu:124-126, :192-195).
//
// What bounds it: atomics on the few words of the large segments, when every
// pixel issues its own.  A warp takes 256 consecutive pixels; while they carry
// one label its lanes add up in registers, and a step of several labels
// issues one atomic per label (1283 x 957 sample frame: 149 to 19 us).
constexpr int kSizeRounds = 8;
__global__ void __launch_bounds__(kThreads)
size_kernel(const int32_t* __restrict__ lab, int64_t n, Layout L, bool count_sizes,
            const float* __restrict__ chroma, int* status) {
  pdl_wait();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32 *
                      kSizeRounds;
       base < n; base += nwarps * 32 * kSizeRounds) {
    int s[kSizeRounds];
    float c[kSizeRounds];
#pragma unroll
    for (int j = 0; j < kSizeRounds; ++j) {
      const int64_t i = base + 32 * j + lane;
      s[j] = i < n ? __ldg(lab + i) : -1;
      c[j] = i < n && chroma ? __ldg(chroma + i) : 0.0f;
    }
    int cur = -1, cnt = 0;   // the running label and its pixels (warp-uniform)
    double acc = 0.0;
    auto flush = [&]() {
      if (cur < 0) return;
      if (chroma) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(full, acc, o);
        if (lane == 0) atomicAdd(L.sum + cur, acc);
        acc = 0.0;
      }
      if (count_sizes && lane == 0) atomicAdd(L.size + cur, cnt);
      cnt = 0;
    };
#pragma unroll
    for (int j = 0; j < kSizeRounds; ++j) {
      const int64_t i = base + 32 * j + lane;
      const bool bad = i < n && (s[j] < 0 || s[j] >= n);
      if (bad) set_status(status, SPLIT_ERR_INVALID);
      if (chroma) {
        int after = __shfl_down_sync(full, s[j], 1);
        if (lane == 31 && i + 1 < n) after = __ldg(lab + i + 1);
        if (!bad && i + 1 < n && after < s[j]) L.state->unsorted = 1;
      }
      const int v = bad ? -1 : s[j];
      const int v0 = __shfl_sync(full, v, 0);
      if (__all_sync(full, v == v0)) {
        if (v0 < 0) continue;
        if (v0 != cur) {
          flush();
          cur = v0;
        }
        cnt += 32;
        acc += (double)c[j];
        continue;
      }
      const unsigned peers = __match_any_sync(full, v);
      const bool leader = v >= 0 && lane == __ffs(peers) - 1;
      if (count_sizes && leader) atomicAdd(L.size + v, __popc(peers));
      if (chroma) {
        const double sum = sum_peers(peers, (double)c[j]);
        if (leader) atomicAdd(L.sum + v, sum);
      }
    }
    flush();
  }
}

__device__ __forceinline__ float seg_mean(const Layout& L, const int32_t* sizes, int s) {
  return (float)L.sum[s] / (float)__ldg(sizes + s);
}

// what pair (s, t) with `count` edges bids for its segment s
__device__ __forceinline__ unsigned long long bid_of(const Layout& L, const int32_t* sizes,
                                                     int policy, int s, int t, unsigned count) {
  if (policy == SPLIT_MERGE_MOST_BOUNDARY)
    return ((unsigned long long)count << 32) | (unsigned)(0xffffffffu - (unsigned)t);
  const float x = seg_mean(L, sizes, s) - seg_mean(L, sizes, t);
  const float d2 = __fadd_rn(__fmul_rn(x, x), __fmul_rn(x, x));
  return ~(((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)t);
}

__device__ __forceinline__ int bid_target(unsigned long long b, int policy) {
  if (policy == SPLIT_MERGE_MOST_BOUNDARY) return (int)(0xffffffffu - (unsigned)(b & 0xffffffffull));
  return (int)(unsigned)((~b) & 0xffffffffull);
}

// Appends s of the calling lanes to the decided list, one atomic per group of
// lanes that arrive together.
__device__ __forceinline__ void list_decided(const Layout& L, int s) {
  const unsigned am = __activemask();
  const int lane = threadIdx.x & 31, leader = __ffs(am) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(&L.state->dec_count, (unsigned)__popc(am));
  base = __shfl_sync(am, base, leader);
  L.dec[base + __popc(am & ((1u << lane) - 1u))] = s;
}

// The distinct neighbour segments of the pixel at `c` (row pitch `pitch`) of
// small segment s, each once with its number of edges: f(t, m) returns
// whether to go on.
template <class F>
__device__ __forceinline__ void for_neighbours(const int* c, int pitch, int s, long long n,
                                               int* status, F&& f) {
  int v[8] = {c[-pitch - 1], c[-pitch], c[-pitch + 1], c[-1],
              c[1],          c[pitch - 1], c[pitch],   c[pitch + 1]};
  bool any = false;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    if (v[a] >= n) {
      set_status(status, SPLIT_ERR_INVALID);
      v[a] = -1;
    }
    if (v[a] < 0) v[a] = s;
    any |= v[a] != s;
  }
  if (!any) return;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    bool first = v[a] != s;
    unsigned m = 1;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (b < a) first &= v[b] != v[a];
      if (b > a) m += v[b] == v[a];
    }
    if (first && !f(v[a], m)) return;
  }
}

// One tile's tables: its small segments of several pixels (pixels in the
// tile, best bid) and their pairs.
constexpr int kHaloW = kTileW + 2, kHaloH = kTileH + 2;
// a table this long into a probe sequence is called full: near capacity the
// sequences of every pixel grow long (a dense tile took 100 us to fill up)
constexpr int kTileProbes = 16;
template <int THREADS, int SEG_BITS, int PAIR_BITS>
struct TileTables {
  static constexpr int kThreads = THREADS, kSegBits = SEG_BITS, kPairBits = PAIR_BITS;
  static constexpr int kSegs = 1 << SEG_BITS, kPairs = 1 << PAIR_BITS;
  union {
    int lab[kHaloH * kHaloW];            // until the pairs are counted
    unsigned long long best[kSegs];      // after
  };
  unsigned long long pair[kPairs];       // (segment slot + 1, t); 0: free
  unsigned edges[kPairs];
  int seg[kSegs];                        // -1: free
  int pixels[kSegs];
  unsigned short out[kPairs];            // pairs for the global table
  int nout, nclaim, full;
  unsigned base;
  int scan[THREADS / 32];
};
// The pair pass: 28 KB, six blocks per SM.  Ordinary tiles hold up to a few
// hundred pairs (the maze's at most 250); a tile of dense speckle has
// thousands and is left to the decision launch's tables (146 KB, one block per
// SM), which hold any realistic tile; past that, pairs go into the global
// table pixel by pixel.
using PassTables = TileTables<kPairThreads, 9, 10>;
using DenseTables = TileTables<kListThreads, 11, 13>;

template <class T>
__device__ __forceinline__ int tile_seg_slot(T& tab, int s) {
  unsigned h = ((unsigned)s * 2654435761u) >> (32 - T::kSegBits);
  for (int probe = 0; probe < kTileProbes; ++probe, h = (h + 1) & (T::kSegs - 1)) {
    int k = *(volatile int*)&tab.seg[h];
    if (k == -1) k = atomicCAS(&tab.seg[h], -1, s);
    if (k == -1 || k == s) return (int)h;
  }
  return -1;
}

template <class T>
__device__ __forceinline__ bool tile_add_pair(T& tab, int slot, int t, unsigned m) {
  const unsigned long long key = ((unsigned long long)(slot + 1) << 32) | (unsigned)t;
  unsigned h = (unsigned)((key * 0x9E3779B97F4A7C15ull) >> (64 - T::kPairBits));
  for (int probe = 0; probe < kTileProbes; ++probe, h = (h + 1) & (T::kPairs - 1)) {
    unsigned long long k = *(volatile unsigned long long*)&tab.pair[h];
    if (k == 0ull) k = atomicCAS(&tab.pair[h], 0ull, key);
    if (k == 0ull || k == key) {
      atomicAdd(&tab.edges[h], m);
      return true;
    }
  }
  return false;
}

// Boundary histogram of the small segments (of class (lev, cls) when CLASSES)
// in one 32 x 64 tile, by the block.  DEFER: a tile that does not fit the
// tables is listed for the decision launch instead (at the end of dec, which
// never meets its front: every such tile has segments of several pixels, so
// more pixels than decided segments).
//
// What bounds it: the latency of global atomics where segments are small and
// many: an insert is a table probe, a compare-and-swap and two adds in turn.
// So the shared tables take one round of them per distinct pair and tile,
// segments inside the tile (most segments below a few dozen pixels) none at all,
// and segments of one pixel are decided from registers; list places are taken
// with one atomic per block.  8192 x 8192 maze, 1.4 M segments: 1.15 ms.
template <bool CLASSES, bool DEFER, class T>
__device__ __forceinline__ void pair_tile(const int32_t* __restrict__ lab, const Geoms& gs,
                                          const Layout& L, const int32_t* sizes, int P, int policy,
                                          T& tab, int tile, int lev, unsigned cls, int* status) {
  constexpr int NT = T::kThreads;
  constexpr int kPer = kTileH * kTileW / NT;
  static_assert(kTileH * kTileW % NT == 0, "whole pixels per thread in a tile");
  const long long n = gs.total_px;
  const TileRef tr = tile_ref(gs, tile);
  const int W = tr.W, H = tr.H;
  // every label load, then every size gather, before any pixel is examined
  int seg[kPer], sz[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int q = threadIdx.x + j * NT;
    const int x = tr.tx0 + q % kTileW, y = tr.ty0 + q / kTileW;
    seg[j] = (x < W && y < H) ? __ldg(lab + tr.off + (long long)y * W + x) : -1;
  }
  // an overflow flagged before the tile starts: nothing more to insert
  const bool stopped = *(volatile int*)&L.state->overflow != 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) sz[j] = (seg[j] >= 0 && seg[j] < n) ? __ldg(sizes + seg[j]) : P;
  // bit j: pixel j belongs to a small segment (of the class) of several
  // pixels / is one by itself
  unsigned small = 0, single = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (sz[j] >= P || (CLASSES && seg_class(seg[j], lev) != cls)) continue;
    if (!CLASSES && sz[j] == 1)
      single |= 1u << j;
    else
      small |= 1u << j;
  }
  if (!__syncthreads_or((small | single) != 0u)) return;
  for (int q = threadIdx.x; q < kHaloH * kHaloW; q += NT) {
    const int y = tr.ty0 - 1 + q / kHaloW, x = tr.tx0 - 1 + q % kHaloW;
    tab.lab[q] = (x >= 0 && y >= 0 && x < W && y < H)
                     ? __ldg(lab + tr.off + (long long)y * W + x)
                     : -1;
  }
  if (threadIdx.x == 0) {
    tab.nout = 0;
    tab.nclaim = 0;
    tab.full = 0;
  }
  // (one thread's view of the overflow flag decides for the block)
  if (__syncthreads_or(threadIdx.x == 0 && stopped)) return;
  auto at = [&](int j) {
    const int q = threadIdx.x + j * NT;
    return tab.lab + (q / kTileW + 1) * kHaloW + q % kTileW + 1;
  };
  unsigned decided = 0;   // bit j: the single pixel j has a target
  if (!CLASSES) {
    // a segment of one pixel: its eight neighbours are all there is to know
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (!((single >> j) & 1u)) continue;
      const int s = seg[j];
      unsigned long long best = 0ull;
      for_neighbours(at(j), kHaloW, s, n, status, [&](int t, unsigned m) {
        best = max(best, bid_of(L, sizes, policy, s, t, m));
        return true;
      });
      L.fin[s] = s;
      if (best == 0ull) continue;
      L.best[s] = best;
      L.map[s] = bid_target(best, policy);
      decided |= 1u << j;
    }
  }
  const bool tables = __syncthreads_or(small != 0u);
  if (tables) {
    for (int i = threadIdx.x; i < T::kSegs; i += NT) {
      tab.seg[i] = -1;
      tab.pixels[i] = 0;
    }
    for (int i = threadIdx.x; i < T::kPairs; i += NT) {
      tab.pair[i] = 0ull;
      tab.edges[i] = 0u;
    }
    __syncthreads();
    for (int j = 0; j < kPer; ++j) {
      if (!((small >> j) & 1u)) continue;
      if (*(volatile int*)&tab.full) break;
      const int* c = at(j);
      const int s = *c;
      const int slot = tile_seg_slot(tab, s);
      if (slot < 0) {
        *(volatile int*)&tab.full = 1;
        break;
      }
      atomicAdd(&tab.pixels[slot], 1);
      for_neighbours(c, kHaloW, s, n, status, [&](int t, unsigned m) {
        const bool ok = tile_add_pair(tab, slot, t, m);
        if (!ok) *(volatile int*)&tab.full = 1;
        return ok;
      });
    }
    __syncthreads();
  }
  const bool full = tables && tab.full;
  if (DEFER && full) {
    if (threadIdx.x == 0) L.dec[n - 1 - atomicAdd(&L.state->dense_count, 1u)] = tile;
    return;
  }
  if (full) {
    // more segments or pairs than the tables hold: straight into the global one
    for (int j = 0; j < kPer; ++j) {
      if (!((small >> j) & 1u)) continue;
      const int* c = at(j);
      const int s = *c;
      L.fin[s] = s;
      bool go = true;
      for_neighbours(c, kHaloW, s, n, status, [&](int t, unsigned m) {
        go = insert(L, s, t, m);
        return go;
      });
      if (!go) break;
    }
  } else if (tables) {
    for (int i = threadIdx.x; i < T::kSegs; i += NT) {
      tab.best[i] = 0ull;
      const int s = tab.seg[i];
      if (s < 0) continue;
      L.fin[s] = s;
      // only a segment wholly inside the tile keeps its count
      if (CLASSES || tab.pixels[i] != __ldg(sizes + s)) tab.pixels[i] = 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T::kPairs; i += NT) {
      const unsigned long long k = tab.pair[i];
      if (k == 0ull) continue;
      const int slot = (int)(k >> 32) - 1, t = (int)(unsigned)(k & 0xffffffffull);
      if (tab.pixels[slot])
        atomicMax(&tab.best[slot], bid_of(L, sizes, policy, tab.seg[slot], t, tab.edges[i]));
      else
        tab.out[atomicAdd(&tab.nout, 1)] = (unsigned short)i;
    }
    __syncthreads();
    const int nout = tab.nout;
    bool go = true;
    for (int o0 = 0; o0 < nout; o0 += NT) {
      const int o = o0 + threadIdx.x;
      int h = -1;
      if (o < nout && go) {
        const int i = tab.out[o];
        const unsigned long long k = tab.pair[i];
        h = claim(L, tab.seg[(int)(k >> 32) - 1], (int)(unsigned)(k & 0xffffffffull),
                  tab.edges[i]);
        go = h != -2;
      }
      const int place = h >= 0 ? atomicAdd(&tab.nclaim, 1) : 0;
      __syncthreads();
      if (threadIdx.x == 0) {
        tab.base = tab.nclaim ? atomicAdd(&L.state->list_count, (unsigned)tab.nclaim) : 0u;
        tab.nclaim = 0;
      }
      __syncthreads();
      if (h >= 0) go = list_slot(L, tab.base + (unsigned)place, h) && go;
    }
  }
  if (CLASSES) {
    __syncthreads();   // the tables are reused by the block's next tile
    return;
  }
  // the tile's decided segments, listed with one atomic
  int mine = __popc(decided);
  if (tables && !full)
    for (int i = threadIdx.x; i < T::kSegs; i += NT) mine += tab.best[i] != 0ull;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) tab.scan[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < NT / 32; ++w) {
      const int c = tab.scan[w];
      tab.scan[w] = sum;
      sum += c;
    }
    tab.base = sum ? atomicAdd(&L.state->dec_count, (unsigned)sum) : 0u;
  }
  __syncthreads();
  unsigned place = tab.base + (unsigned)(tab.scan[warp] + incl - mine);
#pragma unroll
  for (int j = 0; j < kPer; ++j)
    if ((decided >> j) & 1u) L.dec[place++] = seg[j];
  if (tables && !full)
    for (int i = threadIdx.x; i < T::kSegs; i += NT) {
      const unsigned long long b = tab.best[i];
      if (b == 0ull) continue;
      const int s = tab.seg[i];
      L.best[s] = b;
      L.map[s] = bid_target(b, policy);
      L.dec[place++] = s;
    }
  if (!DEFER) __syncthreads();   // the tables are reused by the block's next tile
}

// boundary histogram of small segments, one block per 32 x 64 tile
__global__ void __launch_bounds__(kPairThreads, kPairBlocks)
pair_kernel(const int32_t* __restrict__ lab, Geoms gs, Layout L, const int32_t* sizes, int P,
            int policy, int* status) {
  __shared__ PassTables tab;
  pdl_wait();
  // from here the table and the bids hold this call's words: the stamp comes
  // back only when the call has cleared them
  if (blockIdx.x == 0 && threadIdx.x == 0) L.hdr->stamp = kStampDirty;
  pair_tile<false, true>(lab, gs, L, sizes, P, policy, tab, blockIdx.x, 0, 0u, status);
}

__device__ void bid_phase(const Layout& L, const int32_t* sizes, int policy) {
  const unsigned cnt = *(volatile unsigned*)&L.state->list_count;
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const int h = L.list[j];
    const unsigned long long k = L.keys[h];
    const int s = key_s(k), t = key_t(k);
    const unsigned long long bid = bid_of(L, sizes, policy, s, t, L.counts[h]);
    atomicMax(L.best + s, bid);
  }
}

// next segment along the map: small segments with a winning neighbour move
__device__ __forceinline__ int next_of(const Layout& L, const int32_t* sizes, int P, int r) {
  if (__ldg(sizes + r) >= P) return r;
  if (*(volatile unsigned long long*)(L.best + r) == 0ull) return r;
  const int nx = *(volatile int*)(L.map + r);
  // map entries come from winning pairs, so they are segment ids; anything
  // else is a corrupted workspace: stop the chain here
  if (nx < 0 || nx >= L.state->n) {
    set_status(&L.hdr->status, SPLIT_ERR_INVALID);
    return r;
  }
  return nx;
}

// empties the table slots listed in the claimed-slot list
__device__ void clear_table(const Layout& L) {
  const unsigned cnt = *(volatile unsigned*)&L.state->list_count;
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const int h = L.list[j];
    L.keys[h] = 0ull;
    L.counts[h] = 0u;
  }
}

// the winning pairs of the global table: map entries and the decided list
__device__ void decide_phase(const Layout& L, int policy) {
  const unsigned cnt = *(volatile unsigned*)&L.state->list_count;
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const unsigned long long k = L.keys[L.list[j]];
    const int s = key_s(k), t = key_t(k);
    if (bid_target(L.best[s], policy) == t) {
      L.map[s] = t;
      list_decided(L, s);
    }
  }
}

// The end of every decided segment's chain.  Of a mutual pair the larger id
// keeps itself (fix_map_cycles.cuh:28-43): a chain that meets one ends at the
// larger id, so the map itself need not be changed first.
__device__ void resolve_phase(const Layout& L, const int32_t* sizes, int P, int* status) {
  const unsigned cnt = *(volatile unsigned*)&L.state->dec_count;
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const int s = L.dec[j];
    int r = s, nx = next_of(L, sizes, P, r);
    unsigned steps = 0;
    while (nx != r) {
      const int nn = next_of(L, sizes, P, nx);
      if (nn == r) {
        r = max(r, nx);
        break;
      }
      r = nx;
      nx = nn;
      if (++steps > kChainCap) {
        set_status(status, SPLIT_ERR_NOT_CONVERGED);
        break;
      }
    }
    L.fin[s] = r;
  }
}

// returns the bids of the decided segments to zero
__device__ void clear_bids(const Layout& L) {
  const unsigned cnt = *(volatile unsigned*)&L.state->dec_count;
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x)
    L.best[L.dec[j]] = 0ull;
}

// Records that the table and the bids are clean for the layout `stamp`, at the
// end of a call and behind its last barrier.  A call that gave up has bids of
// segments that no list names: its next call clears everything.
__device__ __forceinline__ void set_stamp(WsHeader* h, unsigned long long stamp) {
  if (*(volatile int*)&h->status == SPLIT_OK) h->stamp = stamp;
}

// ---- overflow path -----------------------------------------------------
// The pair pass overflowed: decide class by class (see the top of the file).
// Runs inside the cooperative decision launch; every phase sits behind a
// bounded grid barrier and the round count is bounded.  Segments the pair pass
// decided inside their tiles are decided again, to the same end.
__device__ void overflow_path(const Layout& L, const int32_t* lab, const Geoms& gs,
                              const int32_t* sizes, int P, int policy,
                              unsigned long long stamp, unsigned& nbar, DenseTables& tab) {
  WsHeader* h = L.hdr;
  State* st = L.state;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  clear_table(L);
  if (!grid_barrier_counted(h, ++nbar)) return;
  if (lead) {
    st->list_count = 0;
    st->overflow = 0;
    st->dec_count = 0;
    L.stack[0] = 2;            // the two halves of level 1
    L.stack[1] = 1, L.stack[2] = 1;
    L.stack[3] = 1, L.stack[4] = 0;
  }
  if (!grid_barrier_counted(h, ++nbar)) return;
  __shared__ int lev, cls;
  for (unsigned round = 0;; ++round) {
    if (threadIdx.x == 0) {
      const int depth = *(volatile int*)L.stack;
      lev = depth > 0 && round < kRoundCap ? *(volatile int*)(L.stack + 2 * depth - 1) : -1;
      cls = depth > 0 ? *(volatile int*)(L.stack + 2 * depth) : 0;
    }
    __syncthreads();
    if (lev < 0) break;   // the same decision in every block
    for (int t = blockIdx.x; t < gs.total_tiles; t += gridDim.x)
      pair_tile<true, false>(lab, gs, L, sizes, P, policy, tab, t, lev, (unsigned)cls,
                             &h->status);
    if (!grid_barrier_counted(h, ++nbar)) return;
    const bool split = *(volatile int*)&st->overflow != 0;
    if (!split) {
      bid_phase(L, sizes, policy);
      if (!grid_barrier_counted(h, ++nbar)) return;
      decide_phase(L, policy);
      if (!grid_barrier_counted(h, ++nbar)) return;
    }
    clear_table(L);
    if (!grid_barrier_counted(h, ++nbar)) return;
    if (lead) {
      int depth = L.stack[0] - 1;   // pop (lev, cls)
      if (split) {
        if (lev >= 31 || depth + 2 > kStackCap) {
          set_status(&h->status, SPLIT_ERR_OVERFLOW);
          depth = 0;
        } else {
          L.stack[1 + 2 * depth] = lev + 1, L.stack[2 + 2 * depth] = 2 * cls + 1;
          L.stack[3 + 2 * depth] = lev + 1, L.stack[4 + 2 * depth] = 2 * cls;
          depth += 2;
        }
      }
      L.stack[0] = depth;
      st->list_count = 0;
      st->overflow = 0;
      if (round + 1 >= kRoundCap) set_status(&h->status, SPLIT_ERR_NOT_CONVERGED);
    }
    if (!grid_barrier_counted(h, ++nbar)) return;
  }
  resolve_phase(L, sizes, P, &h->status);
  if (!grid_barrier_counted(h, ++nbar)) return;
  clear_bids(L);
  if (lead) set_stamp(h, stamp);
}

// The decision, one cooperative launch (at most one block per SM, see
// merge_run): the dense tiles the pair pass left, bids and decisions over the
// global pair list (each skipped when there is none), chains, cleanup, each
// phase behind a bounded grid barrier.  The last step records the layout the
// guard cleared for.  When the table overflowed, the overflow path decides
// instead.
__global__ void __launch_bounds__(kListThreads, 1)
list_kernel(Layout L, const int32_t* lab, Geoms gs, const int32_t* sizes, int P, int policy,
            unsigned long long stamp) {
  extern __shared__ __align__(16) unsigned char list_smem[];
  DenseTables& tab = *reinterpret_cast<DenseTables*>(list_smem);
  WsHeader* h = L.hdr;
  // grid barriers passed (the guard zeroed the counter they count on)
  unsigned nbar = 0;
  // written before this launch only: the same in every block, so all of them
  // pass the barrier or none
  const unsigned dense = *(volatile unsigned*)&L.state->dense_count;
  if (dense) {
    // (a tile that starts after an overflow was flagged returns at once)
    for (unsigned k = blockIdx.x; k < dense; k += gridDim.x) {
      const int tile = *(volatile int*)&L.dec[gs.total_px - 1 - k];
      if (tile >= 0 && tile < gs.total_tiles)
        pair_tile<false, false>(lab, gs, L, sizes, P, policy, tab, tile, 0, 0u, &h->status);
    }
    if (!grid_barrier_counted(h, ++nbar)) return;
  }
  // The dense tiles set the flag too, so it is read behind that barrier only:
  // every insert has come before, and the overflow path resets the flag behind
  // its next barrier.  A block that read it earlier could miss a faster
  // block's overflow, or see one and leave out a barrier that the others wait
  // at.
  const bool over = *(volatile int*)&L.state->overflow != 0;
  if (over) {
    overflow_path(L, lab, gs, sizes, P, policy, stamp, nbar, tab);
    return;
  }
  if (*(volatile unsigned*)&L.state->list_count) {
    bid_phase(L, sizes, policy);
    if (!grid_barrier_counted(h, ++nbar)) return;
    decide_phase(L, policy);
    if (!grid_barrier_counted(h, ++nbar)) return;
  }
  resolve_phase(L, sizes, P, &h->status);
  if (!grid_barrier_counted(h, ++nbar)) return;
  clear_table(L);
  clear_bids(L);
  if (blockIdx.x == 0 && threadIdx.x == 0) set_stamp(h, stamp);
}

// out = the final label of every pixel (out may be in), four pixels per
// thread where the addresses allow it; equal neighbours share one look-up.
template <bool VEC>
__global__ void relabel_kernel(const int32_t* in, int32_t* out, int64_t n, const State* stp,
                               const int32_t* fin) {
  pdl_wait();
  const State st = *stp;
  const int64_t step = gridDim.x * (int64_t)blockDim.x;
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (VEC) {
    for (; i < n / 4; i += step) {
      const int4 v = reinterpret_cast<const int4*>(in)[i];
      int4 r;
      r.x = relabel(st, fin, v.x);
      r.y = v.y == v.x ? r.x : relabel(st, fin, v.y);
      r.z = v.z == v.y ? r.y : relabel(st, fin, v.z);
      r.w = v.w == v.z ? r.z : relabel(st, fin, v.w);
      if (in != out || r.x != v.x || r.y != v.y || r.z != v.z || r.w != v.w)
        reinterpret_cast<int4*>(out)[i] = r;
    }
    i = n / 4 * 4 + (blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
  }
  for (; i < n; i += step) out[i] = relabel(st, fin, in[i]);
}

// Sets the run's parameters (block 0) and clears the state that every call
// leaves at zero (hash table, bids) when the workspace was last used with
// another layout (or never): reusing one workspace for images of different
// sizes moves these regions.  list_kernel records the new layout at its end,
// unless the call failed.
__global__ void guard_kernel(WsHeader* h, unsigned long long stamp, Layout L, long long n,
                             const int32_t* sizes, int P, int policy) {
  pdl_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    State* st = L.state;
    st->n = (int)n;
    st->sizes = sizes;
    st->P = P;
    st->policy = policy;
    st->unsorted = 0;
    st->list_count = 0;
    st->cap_log2 = L.cap_log2;
    st->overflow = 0;
    st->dec_count = 0;
    st->dense_count = 0;
    h->barrier_count = 0;
  }
  if (*(volatile const unsigned long long*)&h->stamp == stamp) return;
  const long long cap = 1ll << L.cap_log2;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cap; i += stride) {
    L.keys[i] = 0ull;
    L.counts[i] = 0u;
  }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
    L.best[i] = 0ull;
}

// The decision launch's shared memory is above the default limit: allowed once
// per device (no stream work, so a graph capture may be under way).
static int list_attributes() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  SG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return SPLIT_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return SPLIT_OK;
  SG_CUDA_TRY(cudaFuncSetAttribute((const void*)list_kernel,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(DenseTables)));
  done[dev] = true;
  return SPLIT_OK;
}

}  // namespace mrg

int merge_view_n(const void* ws, int64_t n, MergeView* out) {
  if (!ws || n < 1) return SPLIT_ERR_INVALID;
  mrg::Layout l = mrg::carve(const_cast<void*>(ws), n);
  out->state = l.state;
  out->fin = l.fin;
  return SPLIT_OK;
}

int merge_view(const void* ws, int width, int height, MergeView* out) {
  if (!ws || width < 1 || height < 1) return SPLIT_ERR_INVALID;
  mrg::Layout l = mrg::carve(const_cast<void*>(ws), (int64_t)width * height);
  out->state = l.state;
  out->fin = l.fin;
  return SPLIT_OK;
}

}  // namespace sg

using namespace sg;

extern "C" size_t split_merge_small_workspace_size(int width, int height) {
  if (width < 1 || height < 1) return 0;
  return mrg::carve(nullptr, (int64_t)width * height).bytes;
}

static int merge_relabel_run(const int32_t* in, int32_t* out, int64_t n, const mrg::State* state,
                             const int32_t* fin, cudaStream_t st) {
  DeviceInfo di;
  SG_TRY(device_info(&di));
  const bool vec =
      ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const int64_t items = vec ? (n + 3) / 4 : n;
  const int grid = (int)std::min<int64_t>((items + mrg::kThreads - 1) / mrg::kThreads,
                                          (int64_t)di.sm_count * 8);
  launch_pdl(vec ? mrg::relabel_kernel<true> : mrg::relabel_kernel<false>, dim3(grid),
             dim3(mrg::kThreads), 0, st, in, out, n, state, fin);
  return launch_status();
}

// Runs the decision passes over a geometry table (labels are arena-global
// segment ids); the labels are relabelled unless `relabel_labels` is false
// (the fused erosion relabels instead).
static int merge_run(int32_t* labels, const Geoms& gs, int P, int policy, const float* chroma,
                     const int32_t* d_sizes, void* workspace, size_t workspace_bytes,
                     cudaStream_t st, bool relabel_labels) {
  const int64_t n = gs.total_px;
  if (!labels || n < 1 || n > 0x7fffffffLL) return SPLIT_ERR_INVALID;
  if (policy != SPLIT_MERGE_MOST_BOUNDARY && policy != SPLIT_MERGE_REF_CHROMA)
    return SPLIT_ERR_INVALID;
  if (policy == SPLIT_MERGE_REF_CHROMA && !chroma) return SPLIT_ERR_INVALID;
  mrg::Layout l = mrg::carve(nullptr, n);
  if (!workspace || workspace_bytes < l.bytes || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return SPLIT_ERR_WORKSPACE;
  l = mrg::carve(workspace, n);
  DeviceInfo di;
  SG_TRY(device_info(&di));
  const int64_t size_px = (int64_t)mrg::kThreads * mrg::kSizeRounds;
  const int grid = (int)std::min<int64_t>((n + size_px - 1) / size_px, (int64_t)di.sm_count * 8);
  const int32_t* sizes = d_sizes ? d_sizes : l.size;
  const bool ref = policy == SPLIT_MERGE_REF_CHROMA;
  const unsigned long long stamp = ((unsigned long long)l.cap_log2 << 40) | (unsigned long long)n;
  // the guard usually finds the stamp unchanged and exits: one block per SM
  // is enough for the rare full clear
  launch_pdl(mrg::guard_kernel, dim3(di.sm_count), dim3(mrg::kThreads), 0, st, l.hdr, stamp, l,
             (long long)n, sizes, P, policy);
  SG_TRY(launch_status());
  if (!d_sizes) SG_CUDA_TRY(cudaMemsetAsync(l.size, 0, sizeof(int32_t) * (size_t)n, st));
  if (ref) SG_CUDA_TRY(cudaMemsetAsync(l.sum, 0, sizeof(double) * (size_t)n, st));
  if (!d_sizes || ref) {
    launch_pdl(mrg::size_kernel, dim3(grid), dim3(mrg::kThreads), 0, st, labels, n, l, !d_sizes,
               ref ? chroma : nullptr, &l.hdr->status);
    SG_TRY(launch_status());
  }
  launch_pdl(mrg::pair_kernel, dim3(gs.total_tiles), dim3(mrg::kPairThreads), 0, st, labels, gs, l,
             sizes, P, policy, &l.hdr->status);
  SG_TRY(launch_status());
  {
    // At most one co-resident block per SM and one per 8192
    // pixels: the lists of most images are short and the decision is bound by
    // its grid barriers, which slow with the block count.
    SG_TRY(mrg::list_attributes());
    const int list_blocks = (int)std::max<int64_t>(1, std::min<int64_t>(di.sm_count, n / 8192));
    unsigned long long stamp_arg = stamp;
    int P_arg = P, policy_arg = policy;
    const int32_t* sizes_arg = sizes;
    const int32_t* lab_arg = labels;
    Geoms gs_arg = gs;
    void* args[] = {&l, &lab_arg, &gs_arg, &sizes_arg, &P_arg, &policy_arg, &stamp_arg};
    SG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)mrg::list_kernel, dim3(list_blocks),
                                            dim3(mrg::kListThreads), args, sizeof(mrg::DenseTables),
                                            st));
  }
  SG_TRY(launch_status());
  if (relabel_labels)
    return merge_relabel_run(labels, labels, n, (const mrg::State*)l.state,
                             (const int32_t*)l.fin, st);
  return SPLIT_OK;
}

static int merge_decide(int32_t* labels, int width, int height, int P, int policy,
                        const float* chroma, const int32_t* d_sizes, void* workspace,
                        size_t workspace_bytes, cudaStream_t st, bool relabel_labels) {
  if (!labels || width < 1 || height < 1) return SPLIT_ERR_INVALID;
  if ((int64_t)width * height > 0x7fffffffLL) return SPLIT_ERR_INVALID;
  return merge_run(labels, single_geom(width, height), P, policy, chroma, d_sizes, workspace,
                   workspace_bytes, st, relabel_labels);
}

namespace sg {
int merge_geoms(const int32_t* labels, const Geoms& gs, int P, int policy, const int32_t* d_sizes,
                void* workspace, size_t workspace_bytes, cudaStream_t st) {
  return merge_run(const_cast<int32_t*>(labels), gs, P, policy, nullptr, d_sizes, workspace,
                   workspace_bytes, st, false);
}
size_t merge_workspace_bytes(int64_t n) { return mrg::carve(nullptr, n).bytes; }
}  // namespace sg

extern "C" int split_merge_small(int32_t* labels, int width, int height, int P, int policy,
                                 const float* chroma, const int32_t* d_sizes, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  return merge_decide(labels, width, height, P, policy, chroma, d_sizes, workspace,
                      workspace_bytes, as_stream(stream), true);
}

namespace sg {
int merge_decide_only(const int32_t* labels, int width, int height, int P, int policy,
                      const float* chroma, const int32_t* d_sizes, void* workspace,
                      size_t workspace_bytes, cudaStream_t st) {
  return merge_decide(const_cast<int32_t*>(labels), width, height, P, policy, chroma, d_sizes,
                      workspace, workspace_bytes, st, false);
}
int merge_relabel(const int32_t* in, int32_t* out, int width, int height, const void* workspace,
                  cudaStream_t st) {
  MergeView v;
  SG_TRY(merge_view(workspace, width, height, &v));
  return merge_relabel_run(in, out, (int64_t)width * height, v.state, v.fin, st);
}
}  // namespace sg
