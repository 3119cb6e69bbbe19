// Loads of a lane's consecutive pixels and their features, shared by the
// k-means kernels.
#pragma once

#include "common.cuh"
#include "f32x2.cuh"

namespace sg {

constexpr int kPx = 4;   // consecutive pixels per lane

// byte / 255 of a pair of values, correctly rounded like the division: with r
// = 1 / 255 rounded and e the rest, fma(b, r, b * e) gives it for every byte
// (no table look-ups and no bank conflicts).
__device__ __forceinline__ float2 unit_pair(float2 b) {
  constexpr float r = 1.0f / 255.0f;
  constexpr float e = (float)(1.0 / 255.0 - (double)r);
  return ffma2(b, make_float2(r, r), fmul2(b, make_float2(e, e)));
}

// The lane's kPx consecutive pixels of a row as loaded (RGB8: the words that
// hold their bytes), so that a batch's loads are under way before the one
// before it is examined.
template <int LAYOUT, int DIM>
struct RawPx {
  float v[LAYOUT == SPLIT_LAYOUT_RGB8 ? 1 : kPx][LAYOUT == SPLIT_LAYOUT_PLANAR ? DIM : 3];
  uint32_t w[LAYOUT == SPLIT_LAYOUT_RGB8 ? 4 : 1];
  int shift;   // RGB8: bits before the first byte

  // pixels px0 .. px0 + valid - 1 (valid <= kPx; 0: nothing is read).  Every
  // word that is read holds a byte of them.
  __device__ __forceinline__ void load(const void* points, int64_t n, int64_t px0, int valid) {
    if (LAYOUT == SPLIT_LAYOUT_FLOAT4) {
      const float4* p = static_cast<const float4*>(points) + px0;
#pragma unroll
      for (int j = 0; j < kPx; ++j) {
        const float4 x = j < valid ? __ldg(p + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[j][0] = x.x;
        v[j][1] = x.y;
        v[j][2] = x.z;
      }
    } else if (LAYOUT == SPLIT_LAYOUT_RGB8) {
      const uintptr_t at = reinterpret_cast<uintptr_t>(points) + 3 * px0;
      const uint32_t* p = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
      const int skip = (int)(at & 3);
      shift = 8 * skip;
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = valid > 0 && 4 * i < 3 * valid + skip ? __ldg(p + i) : 0u;
    } else {
      const float* p = static_cast<const float*>(points) + px0;
#pragma unroll
      for (int d = 0; d < DIM; ++d)
#pragma unroll
        for (int j = 0; j < kPx; ++j) v[j][d] = j < valid ? __ldg(p + (int64_t)d * n + j) : 0.0f;
    }
  }
  __device__ __forceinline__ void features(float xy_scale, int row, int col,
                                           float (&f)[kPx][DIM]) const {
    if (LAYOUT == SPLIT_LAYOUT_RGB8) {
      uint32_t x[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) x[i] = __funnelshift_r(w[i], w[i + 1], shift);
#pragma unroll
      for (int q = 0; q < kPx / 2; ++q)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int a = 6 * q + c, b = a + 3;
          // 2^23 + byte, minus 2^23
          const float2 m = make_float2(
              __uint_as_float(__byte_perm(x[a >> 2], 0x4b000000u, 0x7540u | (a & 3))),
              __uint_as_float(__byte_perm(x[b >> 2], 0x4b000000u, 0x7540u | (b & 3))));
          const float2 u = unit_pair(fadd2(m, make_float2(-8388608.0f, -8388608.0f)));
          f[2 * q][c] = u.x;
          f[2 * q + 1][c] = u.y;
        }
    } else {
#pragma unroll
      for (int j = 0; j < kPx; ++j)
#pragma unroll
        for (int d = 0; d < (LAYOUT == SPLIT_LAYOUT_PLANAR ? DIM : 3); ++d) f[j][d] = v[j][d];
    }
    if (DIM == 5 && LAYOUT != SPLIT_LAYOUT_PLANAR) {
      const float fy = __fmul_rn(xy_scale, (float)row);
#pragma unroll
      for (int j = 0; j < kPx; ++j) {
        f[j][3] = __fmul_rn(xy_scale, (float)(col + j));
        f[j][4] = fy;
      }
    }
  }
};

}  // namespace sg
