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

// ---- the form that the projector and the refinement run -----------------------
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
  float half_w, half_h;  // of the extents, or of extents - 1 (align_corners)
  float x_max, y_max;
  unsigned w, bias;  // bias: of y0 * w + x0 formed from biased bits, modulo 2^32
};

template <bool AC = false>
__host__ __device__ inline LambertGrid lambert_grid(int h, int w) {
  return {0.5f * (float)(AC ? w - 1 : w), 0.5f * (float)(AC ? h - 1 : h), (float)(w - 1), (float)(h - 1), (unsigned)w,
          kTapBiasBits * (unsigned)(w + 1)};
}

// A sample's lower tap and the weights of the upper ones: the entry i of a
// gather table, or the pixel (x0, y0) of an image.
template <bool QUADS>
struct LambertTap {
  float fx, fy;
  int i;
};
template <>
struct LambertTap<false> {
  float fx, fy;
  int x0, y0;
};

// Sizes that the biased floor and a 32-bit index reach; a table is not made for
// an image beyond them, and the route without one has neither.
inline bool quads_fit(int h, int w) {
  return h <= 65535 && w <= (1 << 22) && (int64_t)h * w <= INT32_MAX;
}

// a b - c d with the second product rounded first
__device__ __forceinline__ float diff_of_products(float a, float b, float c, float d) {
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}

// q2 = 2 (x, y, z) of the quaternion q = (w, x, y, z); AC = align_corners, as the
// grid was made
template <bool AC, bool QUADS>
__device__ __forceinline__ LambertTap<QUADS> lambert_tap(const LambertGrid& g, float4 q, float3 q2, float vx,
                                                         float vy, float vz) {
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
  float ix, iy;
  if constexpr (AC) {
    ix = __fmul_rn(__fadd_rn(us, 1.0f), g.half_w);
    iy = __fmul_rn(__fadd_rn(v, 1.0f), g.half_h);
  } else {
    ix = __fmaf_rn(__fadd_rn(us, 1.0f), g.half_w, -0.5f);
    iy = __fmaf_rn(__fadd_rn(v, 1.0f), g.half_h, -0.5f);
  }
  ix = fminf(fmaxf(ix, 0.0f), g.x_max);
  iy = fminf(fmaxf(iy, 0.0f), g.y_max);
  LambertTap<QUADS> t;
  if constexpr (QUADS) {
    const float bx = __fadd_rd(ix, kTapBias), by = __fadd_rd(iy, kTapBias);
    t.i = (int)(__float_as_uint(by) * g.w + __float_as_uint(bx) - g.bias);
    t.fx = __fadd_rn(ix, -__fadd_rn(bx, -kTapBias));
    t.fy = __fadd_rn(iy, -__fadd_rn(by, -kTapBias));
  } else {
    const float x0 = floorf(ix), y0 = floorf(iy);
    t.x0 = (int)x0;
    t.y0 = (int)y0;
    t.fx = __fadd_rn(ix, -x0);
    t.fy = __fadd_rn(iy, -y0);
  }
  return t;
}

// The four taps of a sample: one float4 of a gather table, or four values of
// the image (upper taps clamped to the border).
template <bool QUADS>
__device__ __forceinline__ float4 load_taps(const float* __restrict__ img, int h, const LambertGrid& g,
                                            const LambertTap<QUADS>& t) {
  if constexpr (QUADS) {
    return __ldg(reinterpret_cast<const float4*>(img) + t.i);
  } else {
    const float* lo = img + (int64_t)t.y0 * g.w + t.x0;
    const float* hi = t.y0 < h - 1 ? lo + g.w : lo;
    const int dx = t.x0 < (int)g.w - 1 ? 1 : 0;
    return make_float4(__ldg(lo), __ldg(lo + dx), __ldg(hi), __ldg(hi + dx));
  }
}

template <bool QUADS>
__device__ __forceinline__ float blend(const LambertTap<QUADS>& t, const float4& v) {
  const float gx = __fadd_rn(1.0f, -t.fx), gy = __fadd_rn(1.0f, -t.fy);
  return __fmaf_rn(v.w, __fmul_rn(t.fx, t.fy),
                   __fmaf_rn(v.z, __fmul_rn(gx, t.fy),
                             __fmaf_rn(v.x, __fmul_rn(gx, gy), __fmul_rn(v.y, __fmul_rn(t.fx, gy)))));
}

}  // namespace ebsd
