// Detector-ray rotation, square Lambert map and bilinear master-pattern
// sampling shared by the projector (K1) and the grid refinement (K9):
// qu_apply quaternions.py:186-213, rosca_lambert_side_by_side
// sphere.py:145-185, grid_sample master_pattern.py:197-206.
#pragma once

#include "common.cuh"

namespace ebsd {

__device__ __forceinline__ float2 lambert_side_by_side(float x, float y, float z) {
  const float fac = sqrtf(fmaxf(2.0f * (1.0f - fabsf(z)), 0.0f));
  const bool cond = fabsf(y) <= fabsf(x);
  const float big = cond ? x : y;
  const float sml = cond ? y : x;
  const float sgn = big < 0.0f ? -1.0f : 1.0f;
  const float simple = sgn * fac * 0.70710678118654752f;  // 2 / sqrt(8)
  const float arct = sgn * fac * atan2f(sml * sgn, fabsf(big)) * 0.90031631615710607f;  // 2 sqrt2/pi
  float u = cond ? simple : arct;
  const float v = cond ? arct : simple;
  u = u / 2.0f - 0.5f + (z < 0.0f ? 1.0f : 0.0f);
  return make_float2(u, v);
}

// grid_sample(bilinear, padding_mode="border") of one point (u, v) in
// [-1, 1]^2 on an (h, w) image; AC = align_corners (False for dictionary
// indexing, master_pattern.py:197-206; True for grid refinement,
// refining.py:206).
template <bool AC = false>
__device__ __forceinline__ float sample_border(const float* __restrict__ img, int h, int w, float u,
                                               float v) {
  float ix, iy;
  if constexpr (AC) {
    ix = (u + 1.0f) / 2.0f * (float)(w - 1);
    iy = (v + 1.0f) / 2.0f * (float)(h - 1);
  } else {
    ix = ((u + 1.0f) * (float)w - 1.0f) / 2.0f;
    iy = ((v + 1.0f) * (float)h - 1.0f) / 2.0f;
  }
  ix = fminf(fmaxf(ix, 0.0f), (float)(w - 1));
  iy = fminf(fmaxf(iy, 0.0f), (float)(h - 1));
  const float fx0 = floorf(ix), fy0 = floorf(iy);
  const int x0 = (int)fx0, y0 = (int)fy0;
  const int x1 = min(x0 + 1, w - 1), y1 = min(y0 + 1, h - 1);
  const float wnw = (fx0 + 1.0f - ix) * (fy0 + 1.0f - iy);
  const float wne = (ix - fx0) * (fy0 + 1.0f - iy);
  const float wsw = (fx0 + 1.0f - ix) * (iy - fy0);
  const float wse = (ix - fx0) * (iy - fy0);
  const float* r0 = img + (int64_t)y0 * w;
  const float* r1 = img + (int64_t)y1 * w;
  return __ldg(r0 + x0) * wnw + __ldg(r0 + x1) * wne + __ldg(r1 + x0) * wsw + __ldg(r1 + x1) * wse;
}

// The four taps of sample_border<AC> (same arithmetic), split from their
// loads so that a caller can issue the gathers of several samples together.
struct BorderTaps {
  int i00, i01, i10, i11;
  float w00, w01, w10, w11;
};

template <bool AC = false>
__device__ __forceinline__ BorderTaps border_taps(int h, int w, float u, float v) {
  float ix, iy;
  if constexpr (AC) {
    ix = (u + 1.0f) / 2.0f * (float)(w - 1);
    iy = (v + 1.0f) / 2.0f * (float)(h - 1);
  } else {
    ix = ((u + 1.0f) * (float)w - 1.0f) / 2.0f;
    iy = ((v + 1.0f) * (float)h - 1.0f) / 2.0f;
  }
  ix = fminf(fmaxf(ix, 0.0f), (float)(w - 1));
  iy = fminf(fmaxf(iy, 0.0f), (float)(h - 1));
  const float fx0 = floorf(ix), fy0 = floorf(iy);
  const int x0 = (int)fx0, y0 = (int)fy0;
  const int x1 = min(x0 + 1, w - 1), y1 = min(y0 + 1, h - 1);
  BorderTaps t;
  t.w00 = (fx0 + 1.0f - ix) * (fy0 + 1.0f - iy);
  t.w01 = (ix - fx0) * (fy0 + 1.0f - iy);
  t.w10 = (fx0 + 1.0f - ix) * (iy - fy0);
  t.w11 = (ix - fx0) * (iy - fy0);
  t.i00 = y0 * w + x0;
  t.i01 = y0 * w + x1;
  t.i10 = y1 * w + x0;
  t.i11 = y1 * w + x1;
  return t;
}

// Rotate v by unit quaternion q = (w, x, y, z): v + w t + q_vec x t,
// t = 2 q_vec x v (equal to q (0, v) q* for unit q).
__device__ __forceinline__ float3 rotate(float4 q, float vx, float vy, float vz) {
  const float tx = 2.0f * (q.z * vz - q.w * vy);
  const float ty = 2.0f * (q.w * vx - q.y * vz);
  const float tz = 2.0f * (q.y * vy - q.z * vx);
  return make_float3(vx + q.x * tx + (q.z * tz - q.w * ty), vy + q.x * ty + (q.w * tx - q.y * tz),
                     vz + q.x * tz + (q.y * ty - q.z * tx));
}

// ---- the projector's form of the chain above --------------------------------
// rotate -> lambert_side_by_side -> sample_border with the same roundings in
// fewer instructions. The roundings are written out (which product of a sum is
// fused), so that every route of the projector gives the same bits and a
// dictionary does not change with the compiler's choice of contractions: the
// scores of neighbouring orientations agree to about 1e-2, rounding moves them
// by 1e-6, and an index should not depend on that.
//  * exact scalings (2 q, w / 2) are folded into constants;
//  * signs are moved by copysign instead of multiplications by +-1;
//  * the lower tap is floor(i), read from the low mantissa bits after adding
//    1.5 * 2^23 rounding down (one addition instead of a floor and a
//    conversion);
//  * 1 - (i - i0) equals (i0 + 1) - i, both being exact.
constexpr float kTapBias = 12582912.0f;
constexpr unsigned kTapBiasBits = 0x4B400000u;

struct LambertGrid {
  float half_w, half_h, x_max, y_max;
  unsigned w, bias;  // bias: of y0 * w + x0 formed from biased bits, modulo 2^32
};

__host__ __device__ inline LambertGrid lambert_grid(int h, int w) {
  return {0.5f * (float)w, 0.5f * (float)h, (float)(w - 1), (float)(h - 1), (unsigned)w,
          kTapBiasBits * (unsigned)(w + 1)};
}

// Offset of the lower tap (x0, y0) and the weights of the upper taps.
struct LambertTap {
  int i;
  float fx, fy;
};

// a b - c d with the second product rounded first
__device__ __forceinline__ float diff_of_products(float a, float b, float c, float d) {
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}

// q2 = 2 (x, y, z) of the quaternion q = (w, x, y, z)
__device__ __forceinline__ LambertTap lambert_tap(const LambertGrid& g, float4 q, float3 q2, float vx, float vy,
                                                  float vz) {
  const float tx = diff_of_products(q2.y, vz, q2.z, vy);
  const float ty = diff_of_products(q2.z, vx, q2.x, vz);
  const float tz = diff_of_products(q2.x, vy, q2.y, vx);
  const float x = __fadd_rn(__fmaf_rn(q.x, tx, vx), diff_of_products(q.z, tz, q.w, ty));
  const float y = __fadd_rn(__fmaf_rn(q.x, ty, vy), diff_of_products(q.w, tx, q.y, tz));
  const float z = __fadd_rn(__fmaf_rn(q.x, tz, vz), diff_of_products(q.y, ty, q.z, tx));
  const float ax = fabsf(x), ay = fabsf(y);
  const bool cond = ay <= ax;
  const float fac = sqrtf(fmaxf(__fmaf_rn(-2.0f, fabsf(z), 2.0f), 0.0f));
  const float simple = __fmul_rn(fac, 0.70710678118654752f);  // 2 / sqrt(8)
  const float arct = __fmul_rn(__fmul_rn(fac, atan2f(cond ? ay : ax, cond ? ax : ay)), 0.90031631615710607f);
  const float u = copysignf(cond ? simple : arct, x), v = copysignf(cond ? arct : simple, y);
  const float us = __fadd_rn(__fmaf_rn(u, 0.5f, -0.5f), z < 0.0f ? 1.0f : 0.0f);
  float ix = __fmaf_rn(__fadd_rn(us, 1.0f), g.half_w, -0.5f);
  float iy = __fmaf_rn(__fadd_rn(v, 1.0f), g.half_h, -0.5f);
  ix = fminf(fmaxf(ix, 0.0f), g.x_max);
  iy = fminf(fmaxf(iy, 0.0f), g.y_max);
  const float bx = __fadd_rd(ix, kTapBias), by = __fadd_rd(iy, kTapBias);
  LambertTap t;
  t.i = (int)(__float_as_uint(by) * g.w + __float_as_uint(bx) - g.bias);
  t.fx = __fadd_rn(ix, -__fadd_rn(bx, -kTapBias));
  t.fy = __fadd_rn(iy, -__fadd_rn(by, -kTapBias));
  return t;
}

__device__ __forceinline__ float blend(const LambertTap& t, float v00, float v01, float v10, float v11) {
  const float gx = __fadd_rn(1.0f, -t.fx), gy = __fadd_rn(1.0f, -t.fy);
  return __fmaf_rn(v11, __fmul_rn(t.fx, t.fy),
                   __fmaf_rn(v10, __fmul_rn(gx, t.fy),
                             __fmaf_rn(v00, __fmul_rn(gx, gy), __fmul_rn(v01, __fmul_rn(t.fx, gy)))));
}

}  // namespace ebsd
