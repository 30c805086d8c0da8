// Lens distortion / TCA gather (crates/optics/src/{plan,resample}.rs) and
// exact separable area reduction (crates/core/src/resample.rs) on sm_103a.
//
// Optics: the per-column and per-row halves of the pre-transform
// (plan.rs:448-455 and correction.rs input_coordinate_x/y) are resolved on the
// host in f64 and uploaded as f32 tables, so a pixel starts from two loads.
// The inverse distortion has the values of the lensfun Newton iteration in f64
// from the f32 coordinates (radius sqrt(f64(x*x + y*y)), <= 7 steps, |F| < 1e-5,
// input kept on non-convergence; Poly3 returns NaN), computed in pairs of f32
// wherever those decide the result (see below), TCA is applied in f32 and the
// post-transform back to pixels is f64 narrowed once, as in
// plan.rs:466-483. Each channel is a 4x4 Catmull-Rom gather with the
// reference's tap order (resample.rs:21-33); a footprint outside [1, W-2]
// sets the error word, which the host turns into RD_INVALID_INPUT.
//
// Area reduction: the host builds the overlap tables exactly as
// AreaReductionAxis::new (f64 overlaps narrowed to f32); the horizontal and
// vertical passes accumulate taps in table order from 0, as the reference.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "lens_model.cuh"
#include "rd_internal.cuh"

namespace rd {
namespace {

struct FastOptics {
  float uh, ul;   // f64 unscale split into an FP32 pair
  float2 oh, ol;  // centre * unscale (x, y) split alike
  float2 err;     // what x and y may be off by before they are rounded
  float neg_zero;
};

struct OpticsParams {
  const float* in;   // planar RGB
  const float* mult; // vignetting multipliers, or null
  float* out;
  int W, H;
  const float* ix;   // per-column input x (f32, lens units)
  const float* iy;   // per-row input y
  double cx, cy, unscale;
  int dist_model;
  float d0, d1, d2;
  float inv_k1;      // Poly3: 1 / d0
  int tca_model;
  float tr[3], tb[3];
  unsigned* error;
  FastOptics fast;
};

__device__ __forceinline__ void undistort(const OpticsParams& p, float x, float y, float& ox, float& oy) {
  lens_undistort(p.dist_model, p.d0, p.d1, p.d2, x, y, ox, oy);
}

__device__ __forceinline__ void tca_poly3(const float* ch, float x, float y, float& ox, float& oy) {
  lens_tca_poly3(ch, x, y, ox, oy);
}

// ---- exact FP32 fast path -------------------------------------------------
// GB300 runs FP64 at a small fraction of its FP32 rate, so the per-pixel f64
// arithmetic of the reference (lensfun's Newton inversion, the f64 pixel
// transform) is evaluated in double-float FP32 arithmetic (~44-bit accuracy).
// The f64 result is then rounded to f32 exactly as the reference does; when
// the double-float value lies so close to an f32 rounding midpoint (or to the
// Newton break threshold) that the two could disagree, the pixel takes the
// f64 path instead. The output is therefore the f64 path's, bit for bit.
struct df {
  float h, l;
};
__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ df fast_two_sum(float a, float b) {
  const float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ df two_prod(float a, float b) {
  const float p = a * b;
  return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ df df_add(df x, df y) {
  const df s = two_sum(x.h, y.h);
  return fast_two_sum(s.h, s.l + x.l + y.l);
}
__device__ __forceinline__ df df_mul(df x, df y) {
  df p = two_prod(x.h, y.h);
  p.l = p.l + (x.h * y.l + x.l * y.h);
  return fast_two_sum(p.h, p.l);
}
__device__ __forceinline__ df df_mul_f(df x, float b) {
  df p = two_prod(x.h, b);
  p.l = p.l + x.l * b;
  return fast_two_sum(p.h, p.l);
}
__device__ __forceinline__ df df_div(df x, df y) {
  const float q1 = x.h / y.h;
  const df r = df_add(x, df_mul_f({-y.h, -y.l}, q1));
  const float q2 = r.h / y.h;
  return fast_two_sum(q1, q2);
}
// Nearest f32 of a normalised double-float value (|l| <= ulp(h)/2). The
// rounding midpoints next to h sit at h +- ulp(h)/2, so `amb` is set when |l|
// lies within a relative 2^-40 of ulp(h)/2, and also whenever the gaps around
// h are uneven or tiny (h a power of two, zero, subnormal-adjacent or not
// finite); the caller then takes the f64 path.
__device__ __forceinline__ float df_round(df v, bool& amb) {
  const float r = v.h + v.l;
  const unsigned bits = __float_as_uint(v.h) & 0x7fffffffu;
  const unsigned expo = bits >> 23;
  if (expo <= 25u || expo == 255u || (bits & 0x7fffffu) == 0u) {
    amb = true;
    return r;
  }
  const float half_ulp = __uint_as_float((expo - 24u) << 23);
  if (!(fabsf(fabsf(v.l) - half_ulp) > fabsf(v.h) * 9.094947e-13f)) amb = true;  // 2^-40
  return r;
}

// ---- packed FP32: x and y of a coordinate, or two taps, in one instruction ----
// Products are fused multiply-adds with -0.0 (`z`, from a launch argument):
// the exact product rounded once, and nothing for the compiler to contract.
__device__ __forceinline__ float2 pmul(float2 a, float2 b, float2 z) { return __ffma2_rn(a, b, z); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pneg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 pair(float v) { return make_float2(v, v); }

// (n + c) * unscale in f64, narrowed to f32 (plan.rs:476-478), of x and y, as
// n * unscale + (c * unscale) in double-float: the two differ by a few 2^-53 of
// the coordinate, the double-float sum by a few 2^-46. The sum is rounded with
// the error bound `err` (2^-40 of the largest coordinate) added and taken away
// (Ziv's test): when both give the same f32, so does the f64 value; otherwise
// `sure` is cleared and the caller takes the f64 form. 15 packed instructions
// against about 90 of the double-float form of the expression as it stands
// (two normalised double-float operations and an exponent test, for x and y).
__device__ __forceinline__ float2 post_transform(float2 n, const FastOptics& f, float2 z, bool& sure) {
  const float2 uh = pair(f.uh);
  const float2 ph = pmul(n, uh, z);
  const float2 pl = __ffma2_rn(n, uh, pneg(ph));
  const float2 sum = padd(ph, f.oh);
  const float2 bb = padd(sum, pneg(ph));
  const float2 sl = padd(padd(ph, pneg(padd(sum, pneg(bb)))), padd(f.oh, pneg(bb)));
  const float2 low = padd(sl, padd(pl, __ffma2_rn(n, pair(f.ul), f.ol)));
  const float2 r = padd(sum, padd(low, f.err)), r2 = padd(sum, padd(low, pneg(f.err)));
  sure = sure && r.x == r2.x && r.y == r2.y;
  return r;
}
__device__ __forceinline__ float post_transform_f64(float n, double c, double unscale) {
  return (float)(((double)n + c) * unscale);
}

// Poly5 inverse from f32 (x, y): the f64 Newton result, computed through the
// one-step closed form when that is what the iteration does (break at step 0:
// ratio 1; break at step 1: ratio = 1 - g/d with g = k1 u + k2 u^2 and
// d = 1 + 3 k1 u + 5 k2 u^2 for u = x^2 + y^2), else through f64.
__device__ __forceinline__ void undistort_poly5_fast(float x, float y, float a, float b, float& ox, float& oy,
                                                     bool& need_f64) {
  ox = x;
  oy = y;
  const float s = x * x + y * y;
  if (s == 0.0f) return;
  const float as32 = a * s, bss32 = b * (s * s);
  const float g32 = as32 + bss32;
  const float sq = sqrtf(s);
  const float f0 = sq * g32;
  const float thr = 1.0e-5f;
  // f0 is good to a few 2^-24 of itself and of the two terms, which cancel where the distortion crosses zero.
  const float off = thr * 1.0e-5f + sq * (fabsf(as32) + fabsf(bss32)) * 4.7683716e-7f;  // 2^-21
  if (fabsf(f0) < thr - off) return;  // |F(rd)| < 1e-5: frozen at the input
  if (fabsf(f0) <= thr + off) {
    need_f64 = true;
    return;
  }
  const float d32 = 1.0f + 3.0f * a * s + 5.0f * b * (s * s);
  const float q32 = f0 / d32;
  // F(ru1) for ru1 = rd - q, all of its terms: the second-order one vanishes at 3 k1 + 10 k2 u = 0. Their sum is good
  // to 2^-21 of the largest, 5e-8 while that is below 0.1.
  const float t2 = 3.0f * a * sq + 10.0f * b * sq * s, t3 = a + 10.0f * b * s, t4 = 5.0f * b * sq, q2 = q32 * q32;
  const float f1 = (t2 - q32 * (t3 - q32 * (t4 - q32 * b))) * q2;
  const float size = (fabsf(t2) + fabsf(q32) * (fabsf(t3) + fabsf(q32) * (fabsf(t4) + fabsf(q32 * b)))) * q2;
  if (!(fabsf(f1) < 1.0e-6f) || !(size < 0.1f) || !(d32 > 0.0f)) {
    need_f64 = true;
    return;
  }
  const df as = two_prod(a, s);
  const df ss = two_prod(s, s);
  const df bss = df_mul_f(ss, b);
  const df g = df_add(as, bss);
  const df d = df_add(df_add({1.0f, 0.0f}, df_mul_f(as, 3.0f)), df_mul_f(bss, 5.0f));
  const df q = df_div(g, d);
  const df ratio = fast_two_sum(1.0f, -q.h);
  const df rr = {ratio.h, ratio.l - q.l};
  if (!(rr.h > 0.0f)) {
    need_f64 = true;
    return;
  }
  bool amb = false;
  const float rx = df_round(df_mul_f(rr, x), amb);
  const float ry = df_round(df_mul_f(rr, y), amb);
  if (amb) {
    need_f64 = true;
    return;
  }
  ox = rx;
  oy = ry;
}

// Poly3 inverse from f32 (x, y), as above: with R = f32(rd / k1) and e =
// rd / k1 - R, F(rd) = rd^3 + e, so a break at step 0 gives ratio 1 and one at
// step 1 gives ratio = 1 - (u + e / rd) / (3 u + 1 / k1) for u = rd^2. In
// double-float R and e are the two halves of the product rd / k1. A Poly3 lens
// has no radial table (its freeze is ambiguous), so every pixel comes here; the
// f64 iteration took 4.32 ms per 8256x5504 frame at the FP64 rate.
__device__ __forceinline__ void undistort_poly3_fast(float x, float y, float inv_k1, float& ox, float& oy,
                                                     bool& need_more) {
  ox = x;
  oy = y;
  const float s = x * x + y * y;
  if (s == 0.0f) return;
  const float rh = sqrtf(s);
  const float rl = __fmaf_rn(-rh, rh, s) * __fdividef(0.5f, rh);  // sqrt(s) = rh + rl
  df p = two_prod(rh, inv_k1);
  p = fast_two_sum(p.h, p.l + rl * inv_k1);
  const float thr = 1.0e-5f;
  const float f0 = s * rh + p.l;
  const float d0 = 3.0f * s + inv_k1;
  const float step = __fdividef(f0, d0);
  const float f1 = 3.0f * rh * step * step;  // F(ru1) = 3 rd step^2 - step^3
  // p.h is R unless p.l is within 2^-18 of half its ulp. 1 / k1 below 3e4 keeps e below 1e-3, so that f0 is good to
  // 1e-10 (and to 2^-23 of itself) and the f64 iteration's own rounding is far below the margins of the tests.
  const bool plain = s > 1.0e-12f && s < 1.0e2f && fabsf(inv_k1) > 1.0e-2f && fabsf(inv_k1) < 3.0e4f &&
                     fabsf(d0) > 0.25f * fabsf(inv_k1) && p.h + p.l * 1.0000038f == p.h;
  if (!plain) {
    need_more = true;
    return;
  }
  if (fabsf(f0) < thr * (1.0f - 1.0e-4f)) return;  // frozen at the input
  if (fabsf(f0) <= thr * (1.0f + 1.0e-4f) || !(fabsf(f1) < thr * 0.9f)) {
    need_more = true;
    return;
  }
  const df d = df_add(two_prod(s, 3.0f), {inv_k1, 0.0f});
  const df q = df_div(two_sum(s, __fdividef(p.l, rh)), d);
  const df ratio = fast_two_sum(1.0f, -q.h);
  const df rr = {ratio.h, ratio.l - q.l};
  bool amb = !(rr.h > 0.0f);
  const float rx = df_round(df_mul_f(rr, x), amb);
  const float ry = df_round(df_mul_f(rr, y), amb);
  if (amb) {
    need_more = true;
    return;
  }
  ox = rx;
  oy = ry;
}

// The Newton inversion of lens_undistort and lens_tca_poly3 step by step in
// double-float, for what the closed forms do not cover: each iterate is within
// a few 2^-45 of the f64 one. False where a break test or a rounding is too
// close to call; the caller then takes the f64 iteration. `model` as
// lens_undistort's, 4 for the TCA polynomial (k0, k1, k2 = v, c, b).
__device__ __forceinline__ df df_sub(df x, df y) { return df_add(x, {-y.h, -y.l}); }
__device__ bool newton_df(int model, float k0, float k1, float k2, float x, float y, float& ox, float& oy) {
  const float s = x * x + y * y;
  if (!(s > 1.0e-12f && s < 1.0e4f)) return false;
  const float rh = sqrtf(s);
  const df rd = fast_two_sum(rh, __fdividef(__fmaf_rn(-rh, rh, s), 2.0f * rh));
  df target = rd;
  float inv_k1 = 0.0f;
  if (model == 1) {
    inv_k1 = 1.0f / k0;
    if (!(fabsf(inv_k1) > 1.0e-4f && fabsf(inv_k1) < 1.0e8f)) return false;
    const df p = df_mul_f(rd, inv_k1);
    bool amb = false;
    target = {df_round(p, amb), 0.0f};
    if (amb) return false;
  }
  df ru = rd;
  for (int k = 0; k < 7; ++k) {
    const df r2 = df_mul(ru, ru);
    df f, d;
    float size;  // the magnitude that the rounding errors of f go with
    if (model == 1) {
      f = df_sub(df_add(df_mul(r2, ru), df_mul_f(ru, inv_k1)), target);
      d = df_add(df_mul_f(r2, 3.0f), {inv_k1, 0.0f});
      size = fabsf(r2.h * ru.h) + fabsf(target.h);
    } else if (model == 2) {
      const df r4 = df_mul(r2, r2), ar = df_mul_f(r2, k0), br = df_mul_f(r4, k1);
      f = df_sub(df_mul(ru, df_add({1.0f, 0.0f}, df_add(ar, br))), target);
      d = df_add({1.0f, 0.0f}, df_add(df_mul_f(ar, 3.0f), df_mul_f(br, 5.0f)));
      size = fabsf(ru.h) * (1.0f + fabsf(ar.h) + fabsf(br.h)) + rh;
    } else if (model == 3) {
      const df ar = df_mul_f(df_mul(r2, ru), k0), br = df_mul_f(r2, k1), cr = df_mul_f(ru, k2);
      f = df_sub(df_mul(ru, df_add(df_add(df_add(ar, br), cr), {1.0f, 0.0f})), target);
      d = df_add(df_add(df_add(df_mul_f(ar, 4.0f), df_mul_f(br, 3.0f)), df_mul_f(cr, 2.0f)), {1.0f, 0.0f});
      size = fabsf(ru.h) * (1.0f + fabsf(ar.h) + fabsf(br.h) + fabsf(cr.h)) + rh;
    } else {
      const df br = df_mul_f(r2, k2), cr = df_mul_f(ru, k1);
      f = df_sub(df_mul(ru, df_add(df_add(br, cr), {k0, 0.0f})), target);
      d = df_add(df_add(df_mul_f(br, 3.0f), df_mul_f(cr, 2.0f)), {k0, 0.0f});
      size = fabsf(ru.h) * (fabsf(k0) + fabsf(br.h) + fabsf(cr.h)) + rh;
    }
    const float margin = 1.0e-5f * 1.0e-6f + size * 1.8189894e-12f;  // 2^-39 of the terms
    if (!(fabsf(f.h) < 1.0e30f) || !(fabsf(d.h) > 1.0e-3f * (model == 1 ? fabsf(inv_k1) : 1.0f))) return false;
    if (fabsf(fabsf(f.h) - 1.0e-5f) <= margin) return false;
    if (fabsf(f.h) < 1.0e-5f) {
      if (!(ru.h > 0.0f)) return false;
      if (k == 0) {  // ru / rd is 1 exactly
        ox = x;
        oy = y;
        return true;
      }
      const df ratio = df_div(ru, rd);
      bool amb = false;
      ox = df_round(df_mul_f(ratio, x), amb);
      oy = df_round(df_mul_f(ratio, y), amb);
      return !amb;
    }
    ru = df_sub(ru, df_div(f, d));
    if (!(ru.h > 1.0e-3f * rh && ru.h < 1.0e3f * rh)) return false;
  }
  return false;
}

// cubic_weight (resample.rs) at the four distances x - (fx - 1) .. x - (fx + 2)
// of a footprint with fx = floor(x) >= 1, from d = x - fx. Those differences
// are exact and lie in [1, 2), [0, 1), [-1, 0) and [-2, -1), so they are d + 1,
// d, d - 1 and d - 2, and each weight takes one fixed branch: |d| <= 1 for the
// middle two, 1 < |d| < 2 for the outer two. The outer distances reach 1 or 2
// only when x is an integer, where the reference's branch and this one both
// give +0.0.
// Of x and y at once. A product with a power of two is exact, so fusing it with
// the addition that follows changes nothing (0.5 a a a = 0.5 (a a a), 4 a).
__device__ __forceinline__ void cubic_weights(float2 d, float2 (&w)[4], float2 z) {
  const float2 one = pair(1.0f), two = pair(2.0f);
  const float2 a0 = padd(d, one), a2 = padd(one, pneg(d)), a3 = padd(two, pneg(d));
  auto outer = [&](float2 a) {
    const float2 cube = pmul(pmul(a, a, z), a, z), square = pmul(pmul(pair(2.5f), a, z), a, z);
    return padd(__ffma2_rn(pair(-4.0f), a, __ffma2_rn(pair(-0.5f), cube, square)), two);
  };
  auto inner = [&](float2 a) {
    const float2 cube = pmul(pmul(pmul(pair(1.5f), a, z), a, z), a, z), square = pmul(pmul(pair(-2.5f), a, z), a, z);
    return padd(padd(cube, square), one);
  };
  w[0] = outer(a0);
  w[1] = inner(d);
  w[2] = inner(a2);
  w[3] = outer(a3);
}

// Four samples of a row (the vignetted source values).
template <bool VIG>
__device__ __forceinline__ void load_taps(const float* __restrict__ plane, const float* __restrict__ mult, long long at,
                                          float2 (&s)[2], float2 z) {
  const float* row = plane + at;
  s[0] = make_float2(__ldg(row), __ldg(row + 1));
  s[1] = make_float2(__ldg(row + 2), __ldg(row + 3));
  if (VIG) {
    const float* mrow = mult + at;
    s[0] = pmul(s[0], make_float2(__ldg(mrow), __ldg(mrow + 1)), z);
    s[1] = pmul(s[1], make_float2(__ldg(mrow + 2), __ldg(mrow + 3)), z);
  }
}
// The sum over a footprint (resample.rs:3-41) whose rows are s[0] .. s[3].
__device__ __forceinline__ float sum_taps(const float2 (*s)[2], float2 d, float2 z) {
  float2 w[4];
  cubic_weights(d, w, z);
  const float2 wx01 = make_float2(w[0].x, w[1].x), wx23 = make_float2(w[2].x, w[3].x);
  float value = 0.0f;
#pragma unroll
  for (int oy = 0; oy < 4; ++oy) {
    const float2 wy = pair(w[oy].y);
    const float2 t01 = pmul(s[oy][0], pmul(wy, wx01, z), z), t23 = pmul(s[oy][1], pmul(wy, wx23, z), z);
    value += t01.x;
    value += t01.y;
    value += t23.x;
    value += t23.y;
  }
  return value;
}

// Output pixels (x, y) and (x, y + 1) from the positions n of their channels
// (lens units): post-transform, then the Catmull-Rom gather. The footprints of
// two pixels one above the other mostly lie one row apart, so the second takes
// three of its rows from the first (62 % of the loads and vignetting products)
// and loads them again only where the distortion moves it by another column or
// row. What bounds the gather is the FP32 pipe (about 540 of 640 issue slots a
// pixel) and the latency of its loads: 0.54 ms per 24 MP frame with the radial
// table (0.71 with a pixel per thread, scalar weights and the coordinates'
// double-float form), 1.21 ms per 45 MP frame through a Poly3 lens (4.32 with
// its Newton steps in f64). A non-finite coordinate or a footprint that leaves the image is an error.
template <bool VIG>
__device__ __forceinline__ void gather_pair(const OpticsParams& p, const float (&n0)[6], const float (&n1)[6],
                                            bool bad0, bool bad1, int x, int y) {
  const long long plane = (long long)p.W * p.H;
  const long long o = (long long)y * p.W + x;
  const bool two = y + 1 < p.H;
  const float2 z = pair(p.fast.neg_zero);
  float2 c[6];
  bool sure = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    c[k] = post_transform(make_float2(n0[2 * k], n0[2 * k + 1]), p.fast, z, sure);
    c[3 + k] = post_transform(make_float2(n1[2 * k], n1[2 * k + 1]), p.fast, z, sure);
  }
  if (!sure) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      c[k].x = post_transform_f64(n0[2 * k], p.cx, p.unscale);
      c[k].y = post_transform_f64(n0[2 * k + 1], p.cy, p.unscale);
      c[3 + k].x = post_transform_f64(n1[2 * k], p.cx, p.unscale);
      c[3 + k].y = post_transform_f64(n1[2 * k + 1], p.cy, p.unscale);
    }
  }
  bool bad = bad0 || (two && bad1);
  const int W = p.W;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float* src = p.in + k * plane;
    // The conversion saturates and takes NaN to 0, which is outside.
    const int fx = __float2int_rd(c[k].x), fy = __float2int_rd(c[k].y);
    const int gx = __float2int_rd(c[3 + k].x), gy = __float2int_rd(c[3 + k].y);
    const bool in0 = !bad0 && fx >= 1 && fy >= 1 && fx < W - 2 && fy < p.H - 2;
    const bool in1 = !bad1 && gx >= 1 && gy >= 1 && gx < W - 2 && gy < p.H - 2;
    float2 s[5][2];
    float v0 = 0.0f, v1 = 0.0f;
    if (in0) {
      const long long at = (long long)(fy - 1) * W + (fx - 1);
#pragma unroll
      for (int r = 0; r < 4; ++r) load_taps<VIG>(src, p.mult, at + (long long)r * W, s[r], z);
      v0 = sum_taps(s, padd(c[k], make_float2(-(float)fx, -(float)fy)), z);
    }
    if (two && in1) {
      const long long at = (long long)(gy - 1) * W + (gx - 1);
      if (!(in0 && gx == fx && gy == fy + 1)) {
#pragma unroll
        for (int r = 0; r < 3; ++r) load_taps<VIG>(src, p.mult, at + (long long)r * W, s[1 + r], z);
      }
      load_taps<VIG>(src, p.mult, at + 3ll * W, s[4], z);
      v1 = sum_taps(s + 1, padd(c[3 + k], make_float2(-(float)gx, -(float)gy)), z);
    }
    bad = bad || !in0 || (two && !in1) || !isfinite(v0) || !isfinite(v1);
    p.out[k * plane + o] = isfinite(v0) ? v0 : 0.0f;
    if (two) p.out[k * plane + o + W] = isfinite(v1) ? v1 : 0.0f;
  }
  if (bad) atomicOr(p.error, 8u);
}

// The position of each channel before the post-transform by the Newton path;
// false when it is not finite. One copy for a thread's two pixels (inlined
// twice, the code of all models measured 1 % slower).
__device__ __noinline__ bool newton_positions(const OpticsParams& p, float ix, float iy, float (&n)[6]) {
  float gx, gy;
  if (p.dist_model == RD_DISTORTION_NONE) {
    gx = ix;
    gy = iy;
  } else {
    bool need_more = true;
    if (p.dist_model == RD_DISTORTION_POLY5) {
      need_more = false;
      undistort_poly5_fast(ix, iy, p.d0, p.d1, gx, gy, need_more);
    } else if (p.dist_model == RD_DISTORTION_POLY3) {
      need_more = false;
      undistort_poly3_fast(ix, iy, p.inv_k1, gx, gy, need_more);
    }
    if (need_more && !newton_df(p.dist_model, p.d0, p.d1, p.d2, ix, iy, gx, gy)) undistort(p, ix, iy, gx, gy);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    n[2 * k] = gx;
    n[2 * k + 1] = gy;
  }
  if (p.tca_model == RD_TCA_LINEAR) {
    n[0] = gx * p.tr[0];
    n[1] = gy * p.tr[0];
    n[4] = gx * p.tb[0];
    n[5] = gy * p.tb[0];
  } else if (p.tca_model == RD_TCA_POLY3) {
    if (!newton_df(4, p.tr[0], p.tr[1], p.tr[2], gx, gy, n[0], n[1])) tca_poly3(p.tr, gx, gy, n[0], n[1]);
    if (!newton_df(4, p.tb[0], p.tb[1], p.tb[2], gx, gy, n[4], n[5])) tca_poly3(p.tb, gx, gy, n[4], n[5]);
  }
  return isfinite(gx) && isfinite(gy);
}

template <bool VIG>
__global__ void __launch_bounds__(256, 4) optics_kernel(const OpticsParams p) {
  const int x = blockIdx.x * 32 + (threadIdx.x & 31);
  const int y = 2 * (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5));
  if (x >= p.W || y >= p.H) return;
  const float ix = p.ix[x];
  float n0[6], n1[6];
  const bool bad0 = !newton_positions(p, ix, p.iy[y], n0);
  const bool bad1 = !newton_positions(p, ix, p.iy[min(y + 1, p.H - 1)], n1);
  gather_pair<VIG>(p, n0, n1, bad0, bad1, x, y);
}

// f32 hypot as the reference gets it (f32::hypot, glibc hypotf): the double
// sum of the two exact double squares, its double square root, narrowed once.
// Here the square root is taken in double-float from the FP32-pair sum of
// squares (one Newton correction of an approximate root) and rounded by Ziv's
// test as in post_transform (the root is within a few 2^-45 of the f64 one);
// the rare result too close to an f32 rounding boundary, and sums outside the
// plain range, are computed in f64.
__device__ __forceinline__ float hypot_f32(float x, float y) {
  const df xx = two_prod(x, x), yy = two_prod(y, y);
  const df s = two_sum(xx.h, yy.h);
  const float low = s.l + (xx.l + yy.l);
  const float inv = rsqrtf(s.h);
  const float r0 = s.h * inv;
  const float correction = (__fmaf_rn(-r0, r0, s.h) + low) * (0.5f * inv);
  const float err = r0 * 9.094947e-13f;  // 2^-40
  const float r = r0 + (correction + err);
  if (r == r0 + (correction - err) && s.h > 1.0e-20f && s.h < 1.0e20f) return r;
  return (float)sqrt((double)x * (double)x + (double)y * (double)y);
}

// Self-check of hypot_f32: x runs over every f32 in [first, last), y is a
// hashed f32 of either sign with |y| < 2; counts results that differ from the
// double computation.
__global__ void hypot_check_kernel(unsigned first, unsigned last, unsigned long long* mismatches) {
  unsigned long long bad = 0;
  for (unsigned b = first + blockIdx.x * blockDim.x + threadIdx.x; b < last; b += gridDim.x * blockDim.x) {
    unsigned h = b * 2654435761u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    const float x = __uint_as_float(b);
    const float y = __uint_as_float((h & 0x807fffffu) | ((109u + (h >> 23) % 19u) << 23));  // 2^-18 <= |y| < 2
    const float want = (float)sqrt((double)x * (double)x + (double)y * (double)y);
    if (__float_as_uint(hypot_f32(x, y)) != __float_as_uint(want)) ++bad;
    if (__float_as_uint(hypot_f32(x, 0.0f)) != __float_as_uint(x)) ++bad;
  }
  if (bad) atomicAdd(mismatches, bad);
}

// The radial-table branch of the remap (correction.rs:122-151): the three
// channel multipliers come from one lookup at the pixel's input radius
// (RadialMultipliers::lookup, radial.rs:212-229: nearest knot on the pixel's
// side of a pinned freeze boundary, else the linear blend of the two knots),
// then plan.rs:136-141's post-transform and the Catmull-Rom gather per
// channel. `knots` holds [m_r, m_g, m_b, pin] per knot; it is 16 KB and stays
// in L1.
__device__ __forceinline__ void table_positions(const float4* __restrict__ knots, float step, float ix, float iy,
                                                float (&n)[6]) {
  const float radius = hypot_f32(ix, iy);
  const float position = radius / step;
  const int index = position < (float)(RADIAL_KNOTS - 2) ? (int)position : RADIAL_KNOTS - 2;
  const float4 lo = __ldg(knots + index), hi = __ldg(knots + index + 1);
  float m[3];
  if (lo.w == lo.w) {  // pinned segment
    const float4 k = radius >= lo.w ? hi : lo;
    m[0] = k.x;
    m[1] = k.y;
    m[2] = k.z;
  } else {
    float blend = position - (float)index;
    if (blend > 1.0f) blend = 1.0f;
    m[0] = lo.x * (1.0f - blend) + hi.x * blend;
    m[1] = lo.y * (1.0f - blend) + hi.y * blend;
    m[2] = lo.z * (1.0f - blend) + hi.z * blend;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    n[2 * k] = ix * m[k];
    n[2 * k + 1] = iy * m[k];
  }
}

template <bool VIG>
__global__ void __launch_bounds__(256, 4) optics_lut_kernel(const OpticsParams p, const float4* __restrict__ knots,
                                                         float step) {
  const int x = blockIdx.x * 32 + (threadIdx.x & 31);
  const int y = 2 * (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5));
  if (x >= p.W || y >= p.H) return;
  const float ix = p.ix[x];
  float n0[6], n1[6];
  table_positions(knots, step, ix, p.iy[y], n0);
  table_positions(knots, step, ix, p.iy[min(y + 1, p.H - 1)], n1);
  gather_pair<VIG>(p, n0, n1, false, false, x, y);
}

// Horizontal area pass: one thread per (row, target column, channel-plane).
template <bool VIG>
__device__ __forceinline__ float area_row(const float* __restrict__ row, const float* __restrict__ mrow,
                                          const float* __restrict__ hw, int hn) {
  float mid = 0.0f;
  for (int j = 0; j < hn; ++j) {
    float sample = __ldg(row + j);
    if (VIG) sample = sample * __ldg(mrow + j);
    mid += sample * __ldg(hw + j);
  }
  return mid;
}

// Exact separable area reduction in one pass: a thread owns one output
// column and channel of a tile of AREA_ROWS output rows and streams the
// tile's input rows in order. Each input row's horizontal sum is computed
// once and added to the vertical sum of every output row it belongs to (the
// row where two output rows meet goes to both), so neither pass stores the
// intermediate rows. Both sums accumulate their taps in table order from 0,
// as the two-pass form (and resample.rs) does, so the outputs are the same
// bit for bit.
constexpr int AREA_ROWS = 16;

template <bool VIG, int TAPS>
__global__ void __launch_bounds__(128) area_kernel(const float* __restrict__ in, const float* __restrict__ mult,
                                                   int W, int H, int tw, int th, const int* __restrict__ hfirst,
                                                   const int* __restrict__ hoffset, const int* __restrict__ hcount,
                                                   const float* __restrict__ hweights,
                                                   const int* __restrict__ vfirst, const int* __restrict__ voffset,
                                                   const int* __restrict__ vcount, const float* __restrict__ vweights,
                                                   float* __restrict__ out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.z;
  if (s >= tw) return;
  const int t0 = blockIdx.y * AREA_ROWS, t1 = min(t0 + AREA_ROWS, th);
  const float* plane = in + (long long)c * W * H + hfirst[s];
  const float* mplane = VIG ? mult + hfirst[s] : nullptr;
  const float* hw = hweights + hoffset[s];
  const int hn = hcount[s];
  float* o = out + (long long)c * tw * th + s;
  int t = t0;
  int first = vfirst[t], end = first + vcount[t];
  const float* vw = vweights + voffset[t];
  float acc = 0.0f;
  const int r_end = vfirst[t1 - 1] + vcount[t1 - 1];
  // Adds one input row's horizontal sum to the vertical sum(s) it belongs to;
  // false once the tile's last output row is written.
  auto take = [&](int r, float mid) {
    acc += mid * __ldg(vw + (r - first));
    if (r == end - 1) {
      o[(long long)t * tw] = acc;
      if (++t == t1) return false;
      const int nf = vfirst[t];
      vw = vweights + voffset[t];
      // The next output row starts at or before this input row (they share
      // at most this one).
      acc = 0.0f;
      if (nf <= r) acc += mid * __ldg(vw + (r - nf));
      first = nf;
      end = nf + vcount[t];
    }
    return true;
  };
  if constexpr (TAPS > 0) {
    // No column has more than TAPS taps: the samples of four rows are loaded
    // together before any of their sums, so their latencies overlap; each sum
    // still adds its taps in order from 0. With four as the only such form, a
    // reduction by 3.2 (45 MP to 2560 pixels) had columns of four and of five
    // taps in every warp and took both ways: 0.31 ms, 0.12 with six.
    float w[TAPS];
#pragma unroll
    for (int j = 0; j < TAPS; ++j) w[j] = j < hn ? __ldg(hw + j) : 0.0f;
    for (int r0 = first; r0 < r_end; r0 += 4) {
      float smp[4][TAPS];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float* row = plane + (long long)(r0 + q) * W;
        const float* mrow = VIG ? mplane + (long long)(r0 + q) * W : nullptr;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
          float v = 0.0f;
          if (r0 + q < r_end && j < hn) {
            v = __ldg(row + j);
            if (VIG) v = v * __ldg(mrow + j);
          }
          smp[q][j] = v;
        }
      }
      bool more = true;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (!more || r0 + q >= r_end) break;
        float mid = 0.0f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
          if (j < hn) mid += smp[q][j] * w[j];
        more = take(r0 + q, mid);
      }
      if (!more) break;
    }
    return;
  }
  for (int r = first; r < r_end; ++r)
    if (!take(r, area_row<VIG>(plane + (long long)r * W, VIG ? mplane + (long long)r * W : nullptr, hw, hn))) break;
}

struct AxisTable {
  std::vector<int> first, offset, count;
  std::vector<float> weights;
};

// AreaReductionAxis::new (resample.rs:45-113).
AxisTable build_axis(int source, int target) {
  AxisTable a;
  const double scale = (double)source / (double)target;
  for (int t = 0; t < target; ++t) {
    const double left = (double)t * scale, right = (double)(t + 1) * scale;
    const int first = (int)std::floor(left);
    const int end = std::min((int)std::ceil(right), source);
    a.first.push_back(first);
    a.offset.push_back((int)a.weights.size());
    a.count.push_back(end - first);
    for (int s = first; s < end; ++s) {
      const double overlap = std::min(right, (double)(s + 1)) - std::max(left, (double)s);
      a.weights.push_back((float)(overlap / scale));
    }
  }
  return a;
}

}  // namespace

// Per-axis pre-transform, plan.rs:448-455 / correction.rs input_coordinate_x,y.
std::vector<float> optics_input_coordinates(const rd_optics_desc& o) {
  const int W = (int)o.width, H = (int)o.height;
  std::vector<float> tab((size_t)W + H);
  const double cpx = o.center_x * o.norm_unscale, cpy = o.center_y * o.norm_unscale;
  for (int x = 0; x < W; ++x) {
    const double mapped = cpx + ((double)x - cpx) / (double)o.scale;
    tab[x] = (float)(mapped * o.norm_scale - o.center_x);
  }
  for (int y = 0; y < H; ++y) {
    const double mapped = cpy + ((double)y - cpy) / (double)o.scale;
    tab[W + y] = (float)(mapped * o.norm_scale - o.center_y);
  }
  return tab;
}

Status run_optics_gather(Context& ctx, const rd_optics_desc& o, const float* rgb_in, const float* mult,
                         float* rgb_out) {
  const int W = (int)o.width, H = (int)o.height;
  const std::vector<float> tab = optics_input_coordinates(o);
  // The remap's branch is decided once per apply (correction.rs:110-121).
  const RadialTable radial = build_radial_table(o, tab.data(), tab.data() + W);
  const bool lut = radial.guard == RD_RADIAL_ACCEPTED;
  std::vector<float> staged = lut ? radial.knots : std::vector<float>();
  const size_t knot_floats = staged.size();  // a multiple of 4: the coordinate tables stay 16-byte aligned
  staged.insert(staged.end(), tab.begin(), tab.end());
  const size_t bytes = sizeof(float) * staged.size();
  void* d = nullptr;
  RD_TRY(device_alloc(ctx, bytes, &d));
  float* dbuf = static_cast<float*>(d);
  RD_TRY(upload(ctx, dbuf, staged.data(), bytes));
  const float* dtab = dbuf + knot_floats;
  OpticsParams p{};
  p.in = rgb_in;
  p.mult = mult;
  p.out = rgb_out;
  p.W = W;
  p.H = H;
  p.ix = dtab;
  p.iy = dtab + W;
  p.cx = o.center_x;
  p.cy = o.center_y;
  p.unscale = o.norm_unscale;
  p.dist_model = o.distortion_model;
  p.d0 = o.distortion[0];
  p.d1 = o.distortion[1];
  p.d2 = o.distortion[2];
  p.tca_model = o.tca_model;
  for (int c = 0; c < 3; ++c) {
    p.tr[c] = o.tca_red[c];
    p.tb[c] = o.tca_blue[c];
  }
  p.error = ctx.d_error;
  auto split = [](double v, float& h, float& l) {
    h = (float)v;
    l = (float)(v - (double)h);
  };
  split(o.norm_unscale, p.fast.uh, p.fast.ul);
  split(o.center_x * o.norm_unscale, p.fast.oh.x, p.fast.ol.x);
  split(o.center_y * o.norm_unscale, p.fast.oh.y, p.fast.ol.y);
  // Coordinates that matter lie within twice the image and the centre; one further out fails its footprint test
  // in either form.
  p.fast.err.x = (float)((2.0 * W + std::fabs(o.center_x * o.norm_unscale)) * 0x1p-40);
  p.fast.err.y = (float)((2.0 * H + std::fabs(o.center_y * o.norm_unscale)) * 0x1p-40);
  p.fast.neg_zero = -0.0f;
  p.inv_k1 = 1.0f / o.distortion[0];
  // Tiles of 32 columns and `rows` rows (one warp per two rows), tuned across
  // calls per image shape: the tile only decides which CTA takes which pixels.
  // 32 rows, a CTA of 16 warps, would not hold four CTAs' worth of warps at 64
  // registers; with fewer registers (54, 48, 40) the gather is 5 to 8 % slower.
  const ShapeKey key{TUNE_OPTICS, W, H, 0};
  const ShapePick pick = shape_begin(ctx, key, 16, {8});
  const int rows = pick.value;
  const dim3 grid((W + 31) / 32, (H + rows - 1) / rows);
  const unsigned block = 16u * (unsigned)rows;
  const float4* knots = reinterpret_cast<const float4*>(dbuf);
  if (lut && p.mult) {
    RD_LAUNCH(ctx, K_OPTICS, optics_lut_kernel<true><<<grid, block, 0, ctx.stream>>>(p, knots, radial.step));
  } else if (lut) {
    RD_LAUNCH(ctx, K_OPTICS, optics_lut_kernel<false><<<grid, block, 0, ctx.stream>>>(p, knots, radial.step));
  } else if (p.mult) {
    RD_LAUNCH(ctx, K_OPTICS, optics_kernel<true><<<grid, block, 0, ctx.stream>>>(p));
  } else {
    RD_LAUNCH(ctx, K_OPTICS, optics_kernel<false><<<grid, block, 0, ctx.stream>>>(p));
  }
  shape_end(ctx, key, pick);
  const cudaError_t launch = cudaGetLastError();
  device_free(ctx, dbuf, bytes);
  if (launch != cudaSuccess) return Status{RD_SYNCHRONIZATION, cudaGetErrorString(launch)};
  return Status{};
}


Status run_hypot_check(Context& ctx, uint64_t* result) {
  void* p = nullptr;
  RD_TRY(device_alloc(ctx, 16, &p));
  RD_CUDA_TRY(cudaMemsetAsync(p, 0, 16, ctx.stream));
  const float lo = 0x1p-12f, hi = 2.0f;
  unsigned first = 0, last = 0;
  std::memcpy(&first, &lo, 4);
  std::memcpy(&last, &hi, 4);
  const int grid = (ctx.sm_count > 0 ? ctx.sm_count : 152) * 8;
  RD_LAUNCH(ctx, K_OPTICS, (hypot_check_kernel<<<grid, 256, 0, ctx.stream>>>(
                               first, last, static_cast<unsigned long long*>(p))));
  Status st;
  uint64_t v = 0;
  if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(&v, p, 8, cudaMemcpyDeviceToHost, ctx.stream) != cudaSuccess ||
      cudaStreamSynchronize(ctx.stream) != cudaSuccess)
    st = Status{RD_SYNCHRONIZATION, "hypot check failed"};
  device_free(ctx, p, 16);
  if (st.ok()) *result = v;
  return st;
}

Status run_area_reduce(Context& ctx, const float* rgb, const float* mult, int W, int H, int tw, int th, float* out) {
  const AxisTable ha = build_axis(W, tw), va = build_axis(H, th);
  const size_t ints = ha.first.size() * 3 + va.first.size() * 3;
  const size_t bytes = ints * sizeof(int) + (ha.weights.size() + va.weights.size()) * sizeof(float);
  std::vector<unsigned char> host(bytes);
  unsigned char* q = host.data();
  auto put = [&](const void* src, size_t n) {
    std::memcpy(q, src, n);
    q += n;
  };
  put(ha.first.data(), tw * sizeof(int));
  put(ha.offset.data(), tw * sizeof(int));
  put(ha.count.data(), tw * sizeof(int));
  put(va.first.data(), th * sizeof(int));
  put(va.offset.data(), th * sizeof(int));
  put(va.count.data(), th * sizeof(int));
  put(ha.weights.data(), ha.weights.size() * sizeof(float));
  put(va.weights.data(), va.weights.size() * sizeof(float));
  void* d = nullptr;
  RD_TRY(device_alloc(ctx, bytes, &d));
  unsigned char* b = static_cast<unsigned char*>(d);
  RD_TRY(upload(ctx, b, host.data(), bytes));
  const int* hf = reinterpret_cast<const int*>(b);
  const int* ho = hf + tw;
  const int* hc = ho + tw;
  const int* vf = hc + tw;
  const int* vo = vf + th;
  const int* vc = vo + th;
  const float* hw = reinterpret_cast<const float*>(vc + th);
  const float* vw = hw + ha.weights.size();
  const dim3 grid((tw + 127) / 128, (th + AREA_ROWS - 1) / AREA_ROWS, 3);
  const int taps = *std::max_element(ha.count.begin(), ha.count.end());
#define RD_AREA_LAUNCH(V, T)                                                                                          \
  RD_LAUNCH(ctx, K_AREA, (area_kernel<V, T><<<grid, 128, 0, ctx.stream>>>(rgb, mult, W, H, tw, th, hf, ho, hc, hw, vf, \
                                                                        vo, vc, vw, out)))
#define RD_AREA_TAPS(V)                        \
  if (taps <= 4) RD_AREA_LAUNCH(V, 4);         \
  else if (taps <= 6) RD_AREA_LAUNCH(V, 6);    \
  else if (taps <= 8) RD_AREA_LAUNCH(V, 8);    \
  else RD_AREA_LAUNCH(V, 0)
  if (mult) {
    RD_AREA_TAPS(true);
  } else {
    RD_AREA_TAPS(false);
  }
#undef RD_AREA_TAPS
#undef RD_AREA_LAUNCH
  const cudaError_t launch = cudaGetLastError();
  device_free(ctx, b, bytes);
  if (launch != cudaSuccess) return Status{RD_SYNCHRONIZATION, cudaGetErrorString(launch)};
  return Status{};
}

}  // namespace rd
