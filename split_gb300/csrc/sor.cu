// Shape-from-shading normals from a shading image and a light direction.
//
// Restates split/src/split/device/sfs/estimate_normals.cu:251-308: the
// normals x (planar 3 x N) solve A x = b with
//   A = (L L^T) (x) I_N + 2 lambda B (x) I_3        (:260-278, build_M :85-121)
//   B = 5-point Poisson matrix of the H x W grid, off-diagonals -1 for the
//       in-grid 4-neighbours, diagonal 4 - [row on the border] - [column on
//       the border] (build_B :124-171, the reference's valence rule)
//   b = intensity * L  (build_L :232-248),  L normalised (:258-265)
// from x0 = (0, 0, 1) (:283-287) by relaxation until |b - A x| <=
// tol |b| or max_iter sweeps (apply_sor.cu:9-38: omega 1, tol 1e-5, 1500
// iterations), then normalised with z >= 0 (normalize_vectors.cu:15-41).
//
// The reference assembles A with cuSPARSE calls CUDA 12 no longer has
// (:174-230); here A is never stored.  Each sweep is a red-black block
// Gauss-Seidel pass: a pixel's three unknowns are solved together, the 3 x 3
// block c I + L L^T (c = 2 lambda * valence) inverted in closed form,
//   x_i = (r - L (L . r) / (c + L . L)) / c,  r = s_i L + 2 lambda * sum_j x_j,
// with pixels of one colour independent of each other.  B as the reference
// builds it is the grid's graph Laplacian (every row sums to zero), so A is
// only positive semi-definite: a constant field perpendicular to L is in its
// null space, and the relaxation order decides that component of the
// converged normals.  The order here (red, then black, within a sweep) is the
// one the FP64 restatement in the oracle follows.  The residual test runs
// before every sweep as in the reference's monitor; its sums are per-block
// partials added in one fixed order by every block, so every block takes the
// same decision and the result does not depend on timing.  The decision is the
// one of FP64 sums: the sums in two floats decide only where they are clear of
// the limit, anywhere near it (or not finite) the residual is summed again in
// FP64.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace sg {
namespace sor {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxBlocks = 1024;   // a thread holds one block's partial

// The unknowns are kept per colour (red: row + column even), one float4 per
// pixel (x0, x1, x2, shading intensity), row r of a colour holding its pixels
// in column order at [r * wh, r * wh + wh), wh = (W + 1) / 2: pixel k of row r
// and colour p is column 2 k + ((r + p) & 1).  A pixel's four neighbours are
// all of the other colour: k in the rows above and below, k and one of k - 1,
// k + 1 in its own row.
struct Args {
  const float* s;      // shading intensity, H x W
  float* normals;      // planar 3 x N
  float4 *red, *red_next, *black, *black_next;   // two iterates of each colour
  int W, H, wh;
  float L0, L1, L2;    // normalised light direction
  float lam2;          // 2 * smoothness weight
  int max_iter;
  float tol;
  double* partial;     // [2][kMaxBlocks]
  int32_t* d_iters;
  WsHeader* hdr;
};

__device__ __forceinline__ int valence(int r, int c, int H, int W) {
  return 4 - ((r == 0 || r == H - 1) ? 1 : 0) - ((c == 0 || c == W - 1) ? 1 : 0);
}

// A sum of squares in two floats (relative error below 2^-40): each square's
// product is exact as p + pe (the fma's rest), and so is each sum's rounding
// error (Knuth's two-sum), so only the small word rounds.  FP64 on this part
// runs at two lanes per clock and SM: summing the three squares of a pixel and
// the warp trees in FP64 takes 5.6 us of a VGA sweep, more than everything else
// in it.
struct Sum2 {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float v, float small) {
    const float s = __fadd_rn(hi, v);
    const float b = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(v, b));
    lo = __fadd_rn(lo, __fadd_rn(e, small));
    hi = s;
  }
  __device__ __forceinline__ void add_square(float e) {
    const float p = __fmul_rn(e, e);
    add(p, __fmaf_rn(e, e, -p));
  }
};

struct Problem {
  float L[3], LL, lam2;
  int W, H, wh;
};

// sum of the in-grid 4-neighbours' unknowns of pixel k of row r, column c:
// `y` holds the other colour
__device__ __forceinline__ void neighbour_sum(const Problem& P, const float4* y, int r, int k,
                                              int c, float (&S)[3]) {
  const long long i = (long long)r * P.wh + k;
  const int odd = c & 1;
  // up, left, right, down
  const long long at[4] = {i - P.wh, odd ? i : i - 1, odd ? i + 1 : i, i + P.wh};
  const bool in[4] = {r > 0, c > 0, c + 1 < P.W, r + 1 < P.H};
  float4 v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = in[q] ? y[at[q]] : make_float4(0.f, 0.f, 0.f, 0.f);
  S[0] = S[1] = S[2] = 0.0f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (!in[q]) continue;
    S[0] = __fadd_rn(S[0], v[q].x);
    S[1] = __fadd_rn(S[1], v[q].y);
    S[2] = __fadd_rn(S[2], v[q].z);
  }
}

// the residual of a pixel whose unknowns are x and whose neighbours sum to S:
// f(e) for each component
template <class F>
__device__ __forceinline__ void residual(const Problem& P, const float (&x)[3], float si, float v,
                                         const float (&S)[3], F&& f) {
  const float lx = __fadd_rn(__fadd_rn(__fmul_rn(P.L[0], x[0]), __fmul_rn(P.L[1], x[1])),
                             __fmul_rn(P.L[2], x[2]));
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float lap = __fsub_rn(__fmul_rn(v, x[d]), S[d]);
    const float ax = __fadd_rn(__fmul_rn(P.L[d], lx), __fmul_rn(P.lam2, lap));
    f(__fsub_rn(__fmul_rn(si, P.L[d]), ax));
  }
}

// the block solve of a pixel from its neighbours' sum
__device__ __forceinline__ void solve(const Problem& P, float si, float v, const float (&S)[3],
                                      float (&x)[3]) {
  float rv[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) rv[d] = __fadd_rn(__fmul_rn(si, P.L[d]), __fmul_rn(P.lam2, S[d]));
  const float cc = __fmul_rn(P.lam2, v);
  const float lr = __fadd_rn(__fadd_rn(__fmul_rn(P.L[0], rv[0]), __fmul_rn(P.L[1], rv[1])),
                             __fmul_rn(P.L[2], rv[2]));
  const float q = __fdiv_rn(lr, __fadd_rn(cc, P.LL));
#pragma unroll
  for (int d = 0; d < 3; ++d) x[d] = __fdiv_rn(__fsub_rn(rv[d], __fmul_rn(P.L[d], q)), cc);
}

// FP64 sum of the block's lanes in a fixed order: two-float warp trees, then
// the warps' values in FP64 by the first warp (valid in thread 0)
__device__ double block_sum(Sum2 v) {
  __shared__ double w[kWarps];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float h = __shfl_down_sync(0xffffffffu, v.hi, o);
    const float l = __shfl_down_sync(0xffffffffu, v.lo, o);
    v.add(h, l);
  }
  __syncthreads();   // the last call's words have been read
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = (double)v.hi + (double)v.lo;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = w[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  return t;
}

// What `of` makes of the FP64 sum of one value per thread, the same in every
// thread: warps whose lanes hold no value skip their tree, and one thread calls
// `of` (an FP64 operation of every warp takes the block's unit 16 clocks each).
template <class F>
__device__ __forceinline__ auto block_reduce(double v, int nvalues, F&& of) {
  __shared__ double w[kWarps];
  __shared__ decltype(of(0.0)) result;
  const int warp = threadIdx.x >> 5;
  __syncthreads();
  if (warp * 32 < nvalues) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) w[warp] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i * 32 < nvalues; ++i) t += w[i];
    result = of(t);
  }
  __syncthreads();
  return result;
}
__device__ double block_total(double v, int nvalues) {
  return block_reduce(v, nvalues, [](double t) { return t; });
}

// a sum in two floats against the limit -/+ what it may be off
enum Test { kBelow, kNear, kAbove };

// The pixels of one colour that a thread owns: packed indices first + j *
// kThreads below `end`, row and place stepped without divisions.
struct Walk {
  int i, r, k, dr, dk, end, wh;
  __device__ __forceinline__ Walk(const Problem& P, int chunk) : wh(P.wh) {
    const int n = P.H * P.wh;
    const int b = (int)blockIdx.x * chunk;
    end = min(n, b + chunk);
    i = b + (int)threadIdx.x;
    r = i / wh;
    k = i - r * wh;
    dr = kThreads / wh;
    dk = kThreads - dr * wh;
  }
  __device__ __forceinline__ bool more() const { return i < end; }
  __device__ __forceinline__ void next() {
    i += kThreads;
    r += dr;
    k += dk;
    if (k >= wh) {
      k -= wh;
      ++r;
    }
  }
};

// unit normal with z >= 0 of pixel i
__device__ __forceinline__ void store_normal(float* normals, long long n, long long i, float x,
                                             float y, float z) {
  const float m = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
  const float rmag = __fdiv_rn(1.0f, __fsqrt_rn(m));
  normals[i] = __fmul_rn(x, rmag);
  normals[n + i] = __fmul_rn(y, rmag);
  normals[2 * n + i] = __fmul_rn(fabsf(z), rmag);
}

__device__ __forceinline__ Problem problem_of(const Args& a) {
  Problem P;
  P.L[0] = a.L0;
  P.L[1] = a.L1;
  P.L[2] = a.L2;
  P.LL = __fadd_rn(__fadd_rn(__fmul_rn(P.L[0], P.L[0]), __fmul_rn(P.L[1], P.L[1])),
                   __fmul_rn(P.L[2], P.L[2]));
  P.lam2 = a.lam2;
  P.W = a.W;
  P.H = a.H;
  P.wh = a.wh;
  return P;
}

// The sweeps from iterate `it` on with the residual summed in FP64 before each,
// where sums in two floats do not tell it from the limit (or are not finite).
struct Iterate {
  int it;   // below 0: a barrier wait gave up
  float4 *red, *blk;
};
__device__ __noinline__ Iterate sweeps_fp64(Args a, int chunk, double limit2, Iterate x,
                                            float4* red_next, float4* blk_next, unsigned nbar) {
  const Problem P = problem_of(a);
  for (;; ++x.it) {
    double sum = 0.0;
    for (int colour = 0; colour < 2; ++colour)
      for (Walk w(P, chunk); w.more(); w.next()) {
        const int c = 2 * w.k + ((w.r + colour) & 1);
        if (c >= P.W) continue;
        const float4 o = (colour ? x.blk : x.red)[w.i];
        const float v[3] = {o.x, o.y, o.z};
        float S[3];
        neighbour_sum(P, colour ? x.red : x.blk, w.r, w.k, c, S);
        residual(P, v, o.w, (float)valence(w.r, c, P.H, P.W), S,
                 [&](float e) { sum += (double)e * (double)e; });
      }
    // (the partials of the other parity were read before the last barrier)
    double* part = a.partial + (size_t)(~x.it & 1) * kMaxBlocks;
    sum = block_total(sum, kThreads);
    if (threadIdx.x == 0) __stcg(part + blockIdx.x, sum);
    if (!grid_barrier_counted(a.hdr, ++nbar)) return Iterate{-1, nullptr, nullptr};
    const double e2 = block_total(threadIdx.x < gridDim.x ? __ldcg(part + threadIdx.x) : 0.0,
                                  (int)gridDim.x);
    if (e2 <= limit2 || x.it >= a.max_iter) return x;
    for (int colour = 0; colour < 2; ++colour) {
      for (Walk w(P, chunk); w.more(); w.next()) {
        const int c = 2 * w.k + ((w.r + colour) & 1);
        if (c >= P.W) continue;
        const float si = (colour ? x.blk : x.red)[w.i].w;
        float S[3], v[3];
        neighbour_sum(P, colour ? red_next : x.blk, w.r, w.k, c, S);
        solve(P, si, (float)valence(w.r, c, P.H, P.W), S, v);
        (colour ? blk_next : red_next)[w.i] = make_float4(v[0], v[1], v[2], si);
      }
      if (!grid_barrier_counted(a.hdr, ++nbar)) return Iterate{-1, nullptr, nullptr};
    }
    float4* r = x.red;
    x.red = red_next;
    red_next = r;
    r = x.blk;
    x.blk = blk_next;
    blk_next = r;
  }
}

// One persistent cooperative launch, one block per SM at most, every block
// owning the same contiguous packed pixels of both colours.
//
// What bounds it: at VGA a thread holds one pixel per colour, so a pass is
// the latency of one round of L2 loads and of a grid barrier; larger images
// are bound by L2 bandwidth.  So a sweep is two passes and two barriers, with
// no residual pass: the red pass reads the neighbours that the residual of
// the iterate before it needs as well, and a black pixel's neighbours do not
// change after its update, so the black pass adds the residuals of the next
// iterate.  The test's total is known after the barrier that ends the red
// pass and is added up beside the black pass, so both passes write a second
// buffer and the iterate before them is the result when the test holds.
// VGA: 8.2 us a sweep.
__global__ void __launch_bounds__(kThreads) sor_kernel(Args a, int chunk) {
  const Problem P = problem_of(a);
  if (blockIdx.x == 0 && threadIdx.x == 0) a.hdr->stamp = kStampDirty;
  unsigned nbar = 0;
  float4 *red = a.red, *red_next = a.red_next, *blk = a.black, *blk_next = a.black_next;
  // x0 = (0, 0, 1) and |b|^2 = sum s_i^2 |L|^2
  double acc = 0.0;
  for (int colour = 0; colour < 2; ++colour)
    for (Walk w(P, chunk); w.more(); w.next()) {
      const int c = 2 * w.k + ((w.r + colour) & 1);
      if (c >= P.W) continue;
      const float si = __ldg(a.s + (long long)w.r * P.W + c);
      (colour ? blk : red)[w.i] = make_float4(0.0f, 0.0f, 1.0f, si);
      acc += (double)si * (double)si;
    }
  acc = block_total(acc, kThreads);
  if (threadIdx.x == 0) __stcg(a.partial + kMaxBlocks + blockIdx.x, acc);
  if (!grid_barrier_counted(a.hdr, ++nbar)) return;
  const bool has = threadIdx.x < gridDim.x;
  const double bnorm2 =
      block_total(has ? __ldcg(a.partial + kMaxBlocks + threadIdx.x) : 0.0, (int)gridDim.x) *
      (double)P.LL;
  // the residual is summed scaled by a power of two near 1 / |b|, so that its
  // squares neither overflow nor vanish in FP32 at ordinary intensities
  int ex = 0;
  if (bnorm2 > 0.0 && bnorm2 < INFINITY) ex = -(ilogb(bnorm2) / 2);
  ex = max(-120, min(120, ex));
  const float scale = ldexpf(1.0f, ex);
  const double limit2 = (double)a.tol * (double)a.tol * bnorm2 * ldexp(1.0, 2 * ex);
  // The scaled sum's error: below 2^-40 of it, and what its squares lose below
  // FP32's range, under 2^-110 in all.  Within 2^-20 and 2^-90 FP64 decides.
  const double band = limit2 * 0x1p-20 + 0x1p-90;
  const double below = limit2 - band, above = limit2 + band;
  // the black pixels' residual at x0
  Sum2 black;
  for (Walk w(P, chunk); w.more(); w.next()) {
    const int c = 2 * w.k + ((w.r + 1) & 1);
    if (c >= P.W) continue;
    const float4 o = blk[w.i];
    const float x[3] = {o.x, o.y, o.z};
    float S[3];
    neighbour_sum(P, red, w.r, w.k, c, S);
    residual(P, x, o.w, (float)valence(w.r, c, P.H, P.W), S,
             [&](float e) { black.add_square(__fmul_rn(e, scale)); });
  }
  int it = 0;
  bool near = false;
  for (; it < a.max_iter; ++it) {
    double* part = a.partial + (size_t)(it & 1) * kMaxBlocks;
    // red: the residual of the current iterate and the next one's values
    Sum2 sum = black;
    for (Walk w(P, chunk); w.more(); w.next()) {
      const int c = 2 * w.k + (w.r & 1);
      if (c >= P.W) continue;
      const float4 o = red[w.i];
      float x[3] = {o.x, o.y, o.z}, S[3];
      const float v = (float)valence(w.r, c, P.H, P.W);
      neighbour_sum(P, blk, w.r, w.k, c, S);
      residual(P, x, o.w, v, S, [&](float e) { sum.add_square(__fmul_rn(e, scale)); });
      solve(P, o.w, v, S, x);
      red_next[w.i] = make_float4(x[0], x[1], x[2], o.w);
    }
    const double r2 = block_sum(sum);
    if (threadIdx.x == 0) __stcg(part + blockIdx.x, r2);
    if (!grid_barrier_counted(a.hdr, ++nbar)) return;
    const double mine = has ? __ldcg(part + threadIdx.x) : 0.0;
    // black: the next iterate's values and their residual
    black = Sum2();
    for (Walk w(P, chunk); w.more(); w.next()) {
      const int c = 2 * w.k + ((w.r + 1) & 1);
      if (c >= P.W) continue;
      const float si = blk[w.i].w;
      float x[3], S[3];
      const float v = (float)valence(w.r, c, P.H, P.W);
      neighbour_sum(P, red_next, w.r, w.k, c, S);
      solve(P, si, v, S, x);
      residual(P, x, si, v, S, [&](float e) { black.add_square(__fmul_rn(e, scale)); });
      blk_next[w.i] = make_float4(x[0], x[1], x[2], si);
    }
    const Test test = block_reduce(mine, (int)gridDim.x, [&](double t) {
      return t < below ? kBelow : t > above && t < INFINITY ? kAbove : kNear;
    });
    if (test == kBelow) break;   // iterate `it` is the result
    if (test == kNear) {
      near = true;               // (the same in every block)
      break;
    }
    if (!grid_barrier_counted(a.hdr, ++nbar)) return;
    float4* r = red;
    red = red_next;
    red_next = r;
    r = blk;
    blk = blk_next;
    blk_next = r;
  }
  if (near) {
    const Iterate x = sweeps_fp64(a, chunk, (double)a.tol * (double)a.tol * bnorm2,
                                  Iterate{it, red, blk}, red_next, blk_next, nbar);
    if (x.it < 0) return;
    it = x.it;
    red = x.red;
    blk = x.blk;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.d_iters) *a.d_iters = it;
  // unit normals with z >= 0, each thread from the pixels it wrote itself
  const long long n = (long long)P.W * P.H;
  for (int colour = 0; colour < 2; ++colour)
    for (Walk w(P, chunk); w.more(); w.next()) {
      const int c = 2 * w.k + ((w.r + colour) & 1);
      if (c >= P.W) continue;
      const long long i = (long long)w.r * P.W + c;
      const float4 x = (colour ? blk : red)[w.i];
      store_normal(a.normals, n, i, x.x, x.y, x.z);
    }
}

// The same relaxation with the unknowns in `normals`, for a workspace that holds
// the sums alone.  A sweep is a residual pass in FP64, a red and a black pass,
// each behind a barrier: the packed form above is several times faster and is
// taken wherever the workspace has room for it.
__global__ void __launch_bounds__(kThreads) sor_in_place_kernel(Args a) {
  const Problem P = problem_of(a);
  const long long n = (long long)P.W * P.H;
  const long long first = (long long)blockIdx.x * kThreads + threadIdx.x;
  const long long step = (long long)gridDim.x * kThreads;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.hdr->stamp = kStampDirty;
  float* const x = a.normals;   // (written and read by every block: no read-only loads)
  const bool has = threadIdx.x < gridDim.x;
  unsigned nbar = 0;
  // FP64 sum over the grid, every block's result the same (slot: two in turn)
  auto grid_sum = [&](double v, int slot, double* total) {
    double* part = a.partial + (size_t)slot * kMaxBlocks;
    v = block_total(v, kThreads);
    if (threadIdx.x == 0) __stcg(part + blockIdx.x, v);
    if (!grid_barrier_counted(a.hdr, ++nbar)) return false;
    *total = block_total(has ? __ldcg(part + threadIdx.x) : 0.0, (int)gridDim.x);
    return true;
  };
  auto sums = [&](int r, int c, float (&S)[3]) {
    const long long i = (long long)r * P.W + c;
    const long long at[4] = {i - P.W, i - 1, i + 1, i + P.W};
    const bool in[4] = {r > 0, c > 0, c + 1 < P.W, r + 1 < P.H};
    S[0] = S[1] = S[2] = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!in[q]) continue;
#pragma unroll
      for (int d = 0; d < 3; ++d) S[d] = __fadd_rn(S[d], __ldcg(x + d * n + at[q]));
    }
  };
  // x0 = (0, 0, 1) and |b|^2 = sum s_i^2 |L|^2
  double acc = 0.0, total = 0.0;
  for (long long i = first; i < n; i += step) {
    __stcg(x + i, 0.0f);
    __stcg(x + n + i, 0.0f);
    __stcg(x + 2 * n + i, 1.0f);
    const double si = (double)__ldg(a.s + i);
    acc += si * si;
  }
  if (!grid_sum(acc, 1, &total)) return;
  const double limit2 = (double)a.tol * (double)a.tol * (total * (double)P.LL);
  int it = 0;
  for (;; ++it) {
    acc = 0.0;
    for (long long i = first; i < n; i += step) {
      const int r = (int)(i / P.W), c = (int)(i - (long long)r * P.W);
      const float xi[3] = {__ldcg(x + i), __ldcg(x + n + i), __ldcg(x + 2 * n + i)};
      float S[3];
      sums(r, c, S);
      residual(P, xi, __ldg(a.s + i), (float)valence(r, c, P.H, P.W), S,
               [&](float e) { acc += (double)e * (double)e; });
    }
    if (!grid_sum(acc, it & 1, &total)) return;
    if (total <= limit2 || it >= a.max_iter) break;
    for (int colour = 0; colour < 2; ++colour) {
      for (long long k = first; k < (long long)P.H * P.wh; k += step) {
        const int r = (int)(k / P.wh);
        const int c = 2 * (int)(k - (long long)r * P.wh) + ((r + colour) & 1);
        if (c >= P.W) continue;
        const long long i = (long long)r * P.W + c;
        float S[3], v[3];
        sums(r, c, S);
        solve(P, __ldg(a.s + i), (float)valence(r, c, P.H, P.W), S, v);
#pragma unroll
        for (int d = 0; d < 3; ++d) __stcg(x + d * n + i, v[d]);
      }
      if (!grid_barrier_counted(a.hdr, ++nbar)) return;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.d_iters) *a.d_iters = it;
  for (long long i = first; i < n; i += step)
    store_normal(x, n, i, __ldcg(x + i), __ldcg(x + n + i), __ldcg(x + 2 * n + i));
}

struct Layout {
  WsHeader* hdr;
  double* partial;
  float4* x[2][2];     // the packed unknowns (null: they stay in the normals)
  size_t bytes;
};

constexpr int kPartials = 4096;   // words of a slot: 65 792 bytes without the unknowns
static_assert(kMaxBlocks <= kPartials, "a word per block");

inline Layout carve(void* ws, int W, int H, bool packed) {
  Carver c(ws);
  Layout l{};
  l.hdr = c.take<WsHeader>(1);
  l.partial = c.take<double>((size_t)2 * kPartials);
  for (int colour = 0; colour < 2 && packed; ++colour)
    for (int i = 0; i < 2; ++i) l.x[colour][i] = c.take<float4>((size_t)H * ((W + 1) / 2));
  l.bytes = c.size();
  return l;
}

}  // namespace sor
}  // namespace sg

using namespace sg;

extern "C" size_t split_estimate_normals_workspace_size(int width, int height) {
  if (width < 1 || height < 1) return 0;
  return sor::carve(nullptr, width, height, true).bytes;
}

extern "C" int split_estimate_normals(const float* intensity, int width, int height, float lx,
                                      float ly, float lz, float smoothness, int max_iter,
                                      float tol, float* normals, int32_t* d_iterations,
                                      void* workspace, size_t workspace_bytes, void* stream) {
  using namespace sg::sor;
  if (!intensity || !normals || width < 1 || height < 1 || max_iter < 0 || !(tol >= 0.0f) ||
      !(smoothness > 0.0f))
    return SPLIT_ERR_INVALID;
  if ((int64_t)width * height > 0x7fffffffLL / 3) return SPLIT_ERR_INVALID;
  const float mag2 = lx * lx + ly * ly + lz * lz;
  if (!(mag2 > 0.0f)) return SPLIT_ERR_INVALID;
  if (!workspace || workspace_bytes < carve(nullptr, width, height, false).bytes ||
      (reinterpret_cast<uintptr_t>(workspace) & 255))
    return SPLIT_ERR_WORKSPACE;
  const bool packed_x = workspace_bytes >= carve(nullptr, width, height, true).bytes;
  const Layout l = carve(workspace, width, height, packed_x);
  cudaStream_t st = as_stream(stream);
  SG_CUDA_TRY(cudaMemsetAsync(l.hdr, 0, offsetof(WsHeader, stamp), st));
  DeviceInfo di;
  SG_TRY(device_info(&di));
  // One block per SM at most, and one pixel of a colour per thread at least:
  // the barriers slow with the block count.
  const int wh = (width + 1) / 2;
  const int64_t packed = (int64_t)height * wh;
  int grid = std::min(di.sm_count, kMaxBlocks);
  grid = (int)std::min<int64_t>(grid, (packed + kThreads - 1) / kThreads);
  const int64_t chunk64 = (packed + grid - 1) / grid;
  int chunk = (int)chunk64;
  // the light direction normalised as the reference does (estimate_normals.cu:258-265)
  const float rmag = 1.0f / std::sqrt(mag2);
  Args a{intensity, normals, l.x[0][0], l.x[0][1], l.x[1][0], l.x[1][1], width, height, wh,
         lx * rmag, ly * rmag, lz * rmag, 2.0f * smoothness, max_iter, tol, l.partial,
         d_iterations, l.hdr};
  void* args[] = {&a, &chunk};   // (the in-place kernel takes the first)
  SG_CUDA_TRY(cudaLaunchCooperativeKernel(
      packed_x ? (const void*)sor_kernel : (const void*)sor_in_place_kernel, dim3(grid),
      dim3(kThreads), args, 0, st));
  return launch_status();
}
