// Smooth-boundary merge: segments join the adjacent segment across whose
// shared boundary the features change least.
//
// Restates the documented behaviour of split/src/split/device/ccl/
// merge_smooth_boundaries.cu:134-243:
//   * directed 8-neighbour edges (p, q) between pixels of different labels,
//     the image border excluded (segment_adjacency.cu:112-142, :170-254);
//   * per segment pair (s, t): the number of such edges and the mean over
//     them of |x_p - x_q| (Euclidean norm of feature rows 0..2, in FP32,
//     VecNorm :25-35), averaged per pair (:176-186);
//   * pairs with mean >= D or with 15 edges or fewer are dropped (:197-205),
//     D = threshold * max_i |x_i| (:193-195, max_colwise_norm :37-55);
//   * every segment with candidates maps to the one with the smallest
//     (mean, id) (:207-226: "if we are faced with multiple options, we take
//     the smallest scalar"); mutual pairs keep the larger id
//     (fix_map_cycles.cuh:14-44) and labels follow their map chains to the
//     end (map_until_converged.cuh:14-31).
// The reference file does not compile as written (its reduce_by_key is given
// thrust::less, a predicate, as the reduction), so the stated intent above
// is what this restates.
//
// An edge and its reverse have the same norm, so a pair's statistics are those
// of its reverse: the table holds unordered pairs (s < t), filled from four of
// the eight neighbours, and every entry bids for both segments.  The table is
// open-addressing (key, edge count, 96-bit fixed-point sum of the edge norms
// at scale 2^32), so the means do not depend on the order edges are added in.
// Bids are one 64-bit atomicMax per segment and pair on
// ~((bits(mean) << 32) | t).
#include "geom.cuh"

namespace sg {
namespace smooth {

constexpr int kThreads = 256;
constexpr int kProbeCap = 1 << 16;
constexpr unsigned kChainCap = 1u << 24;

// One pair of segments.
struct Slot {
  unsigned long long key;       // 0: free
  unsigned long long lo, hi;    // sums of the norms' low and high 32-bit words
  unsigned count;
  unsigned pad;
};

struct Layout {
  WsHeader* hdr;
  unsigned* maxsq;              // bits of the largest |x|^2 (non-negative float)
  unsigned* list_count;
  unsigned* call;               // the call's number: marks this call's entries of fin
  unsigned* full;               // a pair found no slot: the rest is not looked for
  unsigned long long* best;     // [n] winning bid per segment, 0 = none
  unsigned long long* fin;      // [n] (call number, final label)
  Slot* slots;                  // [cap]
  int32_t* list;                // [cap] claimed slots
  int cap_log2;
  size_t bytes;
};

inline int cap_log2_for(int64_t n) {
  int l = 11;
  while ((1ll << l) < n && l < 30) ++l;
  return l;
}

inline Layout carve(void* ws, int64_t n) {
  Carver c(ws);
  Layout l;
  l.hdr = c.take<WsHeader>(1);
  l.maxsq = l.hdr ? l.hdr->counter : nullptr;
  l.list_count = l.hdr ? l.hdr->counter + 1 : nullptr;
  l.call = l.hdr ? reinterpret_cast<unsigned*>(l.hdr->pad) : nullptr;
  l.full = l.hdr ? reinterpret_cast<unsigned*>(l.hdr->pad) + 1 : nullptr;
  l.best = c.take<unsigned long long>((size_t)n);
  l.fin = c.take<unsigned long long>((size_t)n);
  l.cap_log2 = cap_log2_for(n);
  const size_t cap = (size_t)1 << l.cap_log2;
  l.slots = c.take<Slot>(cap);
  l.list = c.take<int32_t>(cap);
  l.bytes = c.size();
  return l;
}

__device__ __forceinline__ unsigned long long pair_key(int s, int t) {
  return ((unsigned long long)(unsigned)min(s, t) << 32) | (unsigned)max(s, t);
}
__device__ __forceinline__ int key_s(unsigned long long k) { return (int)(k >> 32); }
__device__ __forceinline__ int key_t(unsigned long long k) { return (int)(unsigned)k; }
__device__ __forceinline__ unsigned key_hash(unsigned long long key, int bits) {
  return (unsigned)((key * 0x9E3779B97F4A7C15ull) >> (64 - bits));
}

// The call's words of the header to zero; and, unless the workspace was last
// used for this layout and left clean, or never used (another image size moves
// the pieces over each other, another entry point writes over them), the pieces
// that every call leaves clean.  relabel_kernel records the layout.  The call
// numbers start again when they run out: the entries of fin go with them.
__global__ void __launch_bounds__(kThreads)
guard_kernel(Layout L, unsigned long long stamp, long long n) {
  pdl_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0)
    L.hdr->barrier_count = *L.maxsq = *L.list_count = *L.full = 0u;
  const unsigned long long last = L.hdr->stamp;
  if ((last == stamp || last == 0ull) && *L.call != ~0u) return;
  const long long step = (long long)gridDim.x * blockDim.x;
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = first; i < n; i += step) L.best[i] = L.fin[i] = 0ull;
  for (long long i = first; i < 1ll << L.cap_log2; i += step) L.slots[i] = Slot{};
}

// |p - q| over feature rows 0..2, the sum of squares in row order
__device__ __forceinline__ float edge_norm(const float (&p)[3], const float (&q)[3]) {
  float s = 0.0f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float v = __fsub_rn(p[d], q[d]);
    s = __fadd_rn(s, __fmul_rn(v, v));
  }
  return __fsqrt_rn(s);
}

__device__ void insert(const Layout& L, unsigned long long key, unsigned m, unsigned long long lo,
                       unsigned long long hi, int* status) {
  const unsigned mask = (1u << L.cap_log2) - 1u;
  unsigned h = key_hash(key, L.cap_log2);
  for (int probe = 0; probe < kProbeCap; ++probe, h = (h + 1) & mask) {
    Slot* const e = L.slots + h;
    unsigned long long k = *(volatile unsigned long long*)&e->key;
    if (k == 0ull) {
      k = atomicCAS(&e->key, 0ull, key);
      if (k == 0ull) {
        const unsigned idx = atomicAdd(L.list_count, 1u);
        L.list[idx] = (int)h;
        k = key;
      }
    }
    if (k == key) {
      atomicAdd(&e->count, m);
      atomicAdd(&e->lo, lo);
      if (hi) atomicAdd(&e->hi, hi);
      return;
    }
  }
  set_status(status, SPLIT_ERR_OVERFLOW);
  *(volatile unsigned*)L.full = 1u;
}

// One block per 32 x 64 tile: the largest feature norm, and the statistics of
// the tile's boundary edges (to the east, south-west, south and south-east).
//
// Bound by the reads of the features when few pixels lie on a boundary and by
// the latency of the edges otherwise.  The features are read once for the
// norm; the pixels that have an edge go to a list, which the block then walks
// densely, so that a boundary's loads overlap instead of following each other
// down the columns of one warp; the edges of a pair meet in a shared-memory
// table and reach the global one as one entry per tile and pair.  The norms'
// 62-bit values are added as four 16-bit pieces: a tile has at most 2^13
// edges, so a piece's sum stays below 2^29.  Pairs that the tile's table has no
// room for within a short probe take another round in it: one by one into the
// global table they cost a 64 x 48 image of 3 x 3 pixel segments 150 us.  1080p, 400
// segments and 4000 single pixels: 81 us for a norm kernel and a kernel that
// pushed every directed edge into the global table, 24 us; seven blocks per SM
// hold the 1020 tiles at once (six: 33 us).
constexpr int kHaloW = kTileW + 2, kHaloH = kTileH + 1;
constexpr int kPairBits = 9, kPairs = 1 << kPairBits, kPairProbes = 16;
constexpr int kTilePx = kTileH * kTileW;
static_assert(kTilePx <= 1 << 11 && kThreads % kTileW == 0, "list entries; pixels per thread");

__global__ void __launch_bounds__(kThreads, 7)
edge_kernel(const int32_t* __restrict__ lab, const float* __restrict__ pts, Geoms gs, Layout L,
            int* status) {
  __shared__ int tile[kHaloH * kHaloW];
  __shared__ unsigned long long key[kPairs];
  __shared__ unsigned count[kPairs], piece[4][kPairs];
  __shared__ unsigned short todo[kTilePx];   // local pixel, then its edges in 4 bits
  __shared__ unsigned ntodo, maxsq, stopped;
  pdl_wait();
  const long long n = gs.total_px;
  const TileRef tr = tile_ref(gs, blockIdx.x);
  const int W = tr.W, H = tr.H;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned last = *L.call;
    *L.call = last == ~0u ? 1u : last + 1u;   // never 0, the mark of a cleared entry
    L.hdr->stamp = kStampDirty;               // until the call has cleared its words
  }
  if (threadIdx.x == 0) {
    ntodo = maxsq = 0u;
    stopped = *(volatile unsigned*)L.full;
  }
  // -1: outside the image, or no label
  bool bad = false;
  for (int q = threadIdx.x; q < kHaloH * kHaloW; q += kThreads) {
    const int x = tr.tx0 - 1 + q % kHaloW, y = tr.ty0 + q / kHaloW;
    int v = -1;
    if (x >= 0 && x < W && y < H) {
      v = __ldg(lab + tr.off + (long long)y * W + x);
      if (v < 0 || v >= n) {
        bad = true;
        v = -1;
      }
    }
    tile[q] = v;
  }
  if (bad) set_status(status, SPLIT_ERR_INVALID);
  for (int i = threadIdx.x; i < kPairs; i += kThreads) {
    key[i] = 0ull;
    count[i] = piece[0][i] = piece[1][i] = piece[2][i] = piece[3][i] = 0u;
  }
  __syncthreads();
  const int lx = threadIdx.x % kTileW, ly0 = threadIdx.x / kTileW;
  unsigned largest = 0u;
#pragma unroll
  for (int r = 0; r < kTileH; r += kThreads / kTileW) {
    const int ly = ly0 + r;
    const int* c = tile + ly * kHaloW + lx + 1;
    const int v = c[0];
    if (tr.tx0 + lx < W && tr.ty0 + ly < H) {
      const long long i = tr.off + (long long)(tr.ty0 + ly) * W + tr.tx0 + lx;
      float s = 0.0f;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float f = __ldg(pts + d * n + i);
        s = __fadd_rn(s, __fmul_rn(f, f));
      }
      // non-negative floats order like their bit patterns (NaN is skipped)
      if (s >= 0.0f) largest = max(largest, __float_as_uint(s));
    }
    const int e = c[1], sw = c[kHaloW - 1], so = c[kHaloW], se = c[kHaloW + 1];
    unsigned m = 0u;
    if (v >= 0)
      m = (e >= 0 && e != v ? 1u : 0u) | (sw >= 0 && sw != v ? 2u : 0u) |
          (so >= 0 && so != v ? 4u : 0u) | (se >= 0 && se != v ? 8u : 0u);
    const unsigned any = __ballot_sync(0xffffffffu, m != 0u);
    if (any) {
      const int lane = threadIdx.x & 31;
      unsigned at = lane == 0 ? atomicAdd(&ntodo, (unsigned)__popc(any)) : 0u;
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(any & ((1u << lane) - 1u));
      if (m) todo[at] = (unsigned short)((ly * kTileW + lx) << 4 | m);
    }
  }
  largest = __reduce_max_sync(0xffffffffu, largest);
  if ((threadIdx.x & 31) == 0) atomicMax(&maxsq, largest);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(L.maxsq, maxsq);
  const unsigned nt = ntodo;
  if (nt == 0u || stopped) return;
  // Edges whose pair finds no room stay in the list for another round with an
  // emptied table.
  for (bool again = true; again;) {
    unsigned left = 0u;
    for (unsigned q = threadIdx.x; q < nt; q += kThreads) {
      const unsigned item = todo[q], m = item & 15u, px = item >> 4;
      if (m == 0u) continue;
      const int* c = tile + (px / kTileW) * kHaloW + px % kTileW + 1;
      const int v = c[0];
      const long long i =
          tr.off + (long long)(tr.ty0 + (int)(px / kTileW)) * W + tr.tx0 + (int)(px % kTileW);
      const int t[4] = {c[1], c[kHaloW - 1], c[kHaloW], c[kHaloW + 1]};
      const long long j[4] = {i + 1, i + W - 1, i + W, i + W + 1};
      float f[3], g[4][3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        f[d] = __ldg(pts + d * n + i);
#pragma unroll
        for (int k = 0; k < 4; ++k) g[k][d] = m >> k & 1u ? __ldg(pts + d * n + j[k]) : 0.0f;
      }
      unsigned rest = 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!(m >> k & 1u)) continue;
        const float e = edge_norm(f, g[k]);
        const long long w = __float2ll_rn(__fmul_rn(e, 4294967296.0f));
        const unsigned long long kk = pair_key(v, t[k]);
        if (!(e < 1073741824.0f)) {   // 2^30, or NaN: too large for the pieces
          set_status(status, SPLIT_ERR_OVERFLOW);
          insert(L, kk, 1u, (unsigned long long)w & 0xffffffffull, (unsigned long long)(w >> 32),
                 status);
          continue;
        }
        unsigned h = key_hash(kk, kPairBits);
        bool in = false;
        for (int probe = 0; probe < kPairProbes; ++probe, h = (h + 1) & (kPairs - 1)) {
          unsigned long long o = *(volatile unsigned long long*)&key[h];
          if (o == 0ull) o = atomicCAS(&key[h], 0ull, kk);
          in = o == 0ull || o == kk;
          if (in) break;
        }
        if (!in) {
          rest |= 1u << k;
          continue;
        }
        atomicAdd(&count[h], 1u);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const unsigned p = (unsigned)(w >> (16 * a)) & 0xffffu;
          if (p) atomicAdd(&piece[a][h], p);
        }
      }
      if (rest != m) todo[q] = (unsigned short)(px << 4 | rest);
      left |= rest;
    }
    again = __syncthreads_or(left != 0u);
    for (int i = threadIdx.x; i < kPairs; i += kThreads) {
      if (!key[i]) continue;
      insert(L, key[i], count[i], piece[0][i] + ((unsigned long long)piece[1][i] << 16),
             piece[2][i] + ((unsigned long long)piece[3][i] << 16), status);
      if (again) {
        key[i] = 0ull;
        count[i] = piece[0][i] = piece[1][i] = piece[2][i] = piece[3][i] = 0u;
      }
    }
    // (a full global table: the call has failed, whatever else is tried)
    if (again && __syncthreads_or(*(volatile unsigned*)L.full != 0u)) return;
  }
}

// mean edge norm of a slot, rounded to FP32 (the reference keeps it as real);
// edge norms are below 2^30, so the high words sum to below 2^62
__device__ __forceinline__ float slot_mean(const Slot& e) {
  const double hi = (double)(long long)e.hi;
  const double lo = (double)e.lo;
  const double S = __dadd_rn(__dmul_rn(hi, 4294967296.0), lo);
  return __double2float_rn(__ddiv_rn(__dmul_rn(S, 1.0 / 4294967296.0), (double)e.count));
}

__device__ void bid_phase(const Layout& L, float threshold) {
  const unsigned cnt = *(volatile unsigned*)L.list_count;
  const float D = __fmul_rn(threshold, __fsqrt_rn(__uint_as_float(*(volatile unsigned*)L.maxsq)));
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const Slot e = L.slots[L.list[j]];
    const int s = key_s(e.key), t = key_t(e.key);
    if (e.count <= 15u) continue;
    const float d = slot_mean(e);
    if (!(d < D)) continue;
    const unsigned long long mean = (unsigned long long)__float_as_uint(d) << 32;
    atomicMax(L.best + s, ~(mean | (unsigned)t));
    atomicMax(L.best + t, ~(mean | (unsigned)s));
  }
}

// the winning bid of segment r after the bids are in
__device__ __forceinline__ unsigned long long bid_of(const Layout& L, int r) {
  return *(volatile unsigned long long*)(L.best + r);
}
__device__ __forceinline__ int bid_target(unsigned long long b) {
  return (int)(unsigned)((~b) & 0xffffffffull);
}

// The segment that r maps to: its bid's target; r itself without a bid, and
// the larger id of a pair that bid for each other.  A bid's target is a segment
// id; anything else is a corrupted workspace: the chain stops here.
__device__ __forceinline__ int next_of(const Layout& L, int n, int r) {
  const unsigned long long b = bid_of(L, r);
  if (b == 0ull) return r;
  const int t = bid_target(b);
  if (t < 0 || t >= n) {
    set_status(&L.hdr->status, SPLIT_ERR_INVALID);
    return r;
  }
  if (r > t) {
    const unsigned long long back = bid_of(L, t);
    if (back != 0ull && bid_target(back) == r) return r;
  }
  return t;
}

// The end of s's chain, for a segment that has a bid; one of its pairs, the
// one it bid for, does it.
__device__ __forceinline__ void resolve(const Layout& L, int n, int s, int t,
                                        unsigned long long call) {
  const unsigned long long b = bid_of(L, s);
  if (!b || bid_target(b) != t) return;
  int r = s;
  for (unsigned steps = 0;; ++steps) {
    const int nx = next_of(L, n, r);
    if (nx == r) break;
    r = nx;
    if (steps > kChainCap) {
      set_status(&L.hdr->status, SPLIT_ERR_NOT_CONVERGED);
      break;
    }
  }
  L.fin[s] = call << 32 | (unsigned)r;
}

// The decision over the pairs, one cooperative launch (one block per SM): the
// bids, a bounded grid barrier, then every segment's chain.  The fix of mutual
// pairs needs both bids and nothing else, so the chain reads it off the bids
// as it goes: no phase writes maps first, and two barriers of 1.5 us each are
// not needed.
__global__ void __launch_bounds__(kThreads) list_kernel(Layout L, float threshold, int n) {
  bid_phase(L, threshold);
  if (!grid_barrier(L.hdr)) return;
  const unsigned cnt = *(volatile unsigned*)L.list_count;
  const unsigned long long call = *L.call;
  for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x) {
    const unsigned long long k = L.slots[L.list[j]].key;
    resolve(L, n, key_s(k), key_t(k), call);
    resolve(L, n, key_t(k), key_s(k), call);
  }
}

__device__ __forceinline__ int final_of(const Layout& L, unsigned n, unsigned call, int v) {
  if ((unsigned)v >= n) return v;
  const unsigned long long f = __ldg(L.fin + v);
  return (unsigned)(f >> 32) == call ? (int)(unsigned)f : v;
}

// Final labels, four pixels per thread where the address allows it (equal
// neighbours share one look-up), and the slots and bids of the call back to
// zero for the next.  The look-up needs one word: an entry of fin counts when
// it carries the call's number, so fin is never cleared.
template <bool VEC>
__global__ void __launch_bounds__(kThreads)
relabel_kernel(int32_t* __restrict__ lab, long long n, Layout L, unsigned long long stamp) {
  pdl_wait();
  // (a call that failed may have left anything: the next one clears)
  if (blockIdx.x == 0 && threadIdx.x == 0 && L.hdr->status == SPLIT_OK) L.hdr->stamp = stamp;
  const unsigned call = *L.call, cnt = *L.list_count;
  const long long step = (long long)gridDim.x * blockDim.x;
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned un = (unsigned)n;
  long long i = first;
  if (VEC) {
    for (; i < n / 4; i += step) {
      const int4 v = reinterpret_cast<const int4*>(lab)[i];
      int4 r;
      r.x = final_of(L, un, call, v.x);
      r.y = v.y == v.x ? r.x : final_of(L, un, call, v.y);
      r.z = v.z == v.y ? r.y : final_of(L, un, call, v.z);
      r.w = v.w == v.z ? r.z : final_of(L, un, call, v.w);
      if (r.x != v.x || r.y != v.y || r.z != v.z || r.w != v.w)
        reinterpret_cast<int4*>(lab)[i] = r;
    }
    i = n / 4 * 4 + first;
  }
  for (; i < n; i += step) lab[i] = final_of(L, un, call, lab[i]);
  for (long long j = first; j < cnt; j += step) {
    Slot* const e = L.slots + L.list[j];
    L.best[key_s(e->key)] = 0ull;
    L.best[key_t(e->key)] = 0ull;
    *e = Slot{};
  }
}

}  // namespace smooth
}  // namespace sg

using namespace sg;

extern "C" size_t split_merge_smooth_workspace_size(int width, int height) {
  if (width < 1 || height < 1) return 0;
  return smooth::carve(nullptr, (int64_t)width * height).bytes;
}

extern "C" int split_merge_smooth(int32_t* labels, int width, int height, const float* points,
                                  float threshold, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  using namespace sg::smooth;
  if (!labels || !points || width < 1 || height < 1) return SPLIT_ERR_INVALID;
  const int64_t n = (int64_t)width * height;
  if (n > 0x7fffffffLL || !(threshold >= 0.0f)) return SPLIT_ERR_INVALID;
  Layout l = carve(nullptr, n);
  if (!workspace || workspace_bytes < l.bytes || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return SPLIT_ERR_WORKSPACE;
  l = carve(workspace, n);
  cudaStream_t st = as_stream(stream);
  DeviceInfo di;
  SG_TRY(device_info(&di));
  const Geoms gs = single_geom(width, height);
  // the high bit: another workspace layout than the small-segment merge's
  const unsigned long long stamp =
      1ull << 63 | (unsigned long long)l.cap_log2 << 40 | (unsigned long long)n;
  launch_pdl(guard_kernel, dim3(di.sm_count), dim3(kThreads), 0, st, l, stamp, (long long)n);
  SG_TRY(launch_status());
  launch_pdl(edge_kernel, dim3(gs.total_tiles), dim3(kThreads), 0, st, (const int32_t*)labels,
             points, gs, l, &l.hdr->status);
  SG_TRY(launch_status());
  {
    // one co-resident block per SM; the header clear above zeroed the barrier
    int per_sm = 0;
    SG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, list_kernel, kThreads, 0));
    if (per_sm < 1) return SPLIT_ERR_UNSUPPORTED;
    float thr = threshold;
    int n32 = (int)n;
    void* args[] = {&l, &thr, &n32};
    SG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)list_kernel, dim3(di.sm_count),
                                            dim3(kThreads), args, 0, st));
  }
  SG_TRY(launch_status());
  const bool vec = (reinterpret_cast<uintptr_t>(labels) & 15) == 0;
  const int64_t items = vec ? (n + 3) / 4 : n;
  int64_t blocks = (items + kThreads - 1) / kThreads;
  const int64_t cap = (int64_t)di.sm_count * 8;
  if (blocks > cap) blocks = cap;
  launch_pdl(vec ? relabel_kernel<true> : relabel_kernel<false>, dim3((unsigned)blocks),
             dim3(kThreads), 0, st, labels, (long long)n, l, stamp);
  return launch_status();
}
