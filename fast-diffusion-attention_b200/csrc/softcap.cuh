// Capped scores: tanh(x), x = score * scale / cap, without the special-function unit where the scores allow it.
//
// That unit gives 16 results per clock and SM, and a capped score needs two of them (tanh and exp2): at head dimension 64
// twice the time of the tensor products. Scores mostly stay well inside the cap, where an odd polynomial of degree 7 does:
// packed multiply-adds for two columns, which run on the FMA pipe beside the exponentials. A warp whose scores of a step
// all satisfy |x| <= 0.5 takes it, any other one (NaN included) the unit's tanh. The polynomial is a least-maximum fit of
// tanh(x) / x in x^2: relative error at most 5.5e-7 there. tanh.approx is as good for small arguments only (its bound is
// 2^-11). The same four coefficients fitted up to |x| = 1 would be 8.2e-5 off, and the log-sum-exp of scores of unit variance
// under a cap of 30 by 1.1e-5 instead of 1e-7; a fifth one up to 0.75 takes registers that cost the 128-wide forward what the
// polynomial gains it.
//
// Used in the forward up to head dimension 128 (with one query tile an item, where it hardly matters, too: both give the same
// bits) and in the single-pass backward at head dimension 64. With 32 heads of 64 on 4 x 8192 tokens (cap
// 30) the forward went from 1325 to 1257 us and the backward kernel from 2763 to 2615, with 16 heads of 128 on 4 x 4096 tokens
// the forward from 242 to 220.
// Elsewhere the unit's tanh is as fast or faster (forward of 256-wide heads 98.2 against 101.2 us on 2 x 4096 tokens, 8 heads;
// single-pass backward of 128-wide heads 629 against 658 us on 4 x 4096 tokens, 16 heads; split backward 396 against 418).
#pragma once

#include "ptx.cuh"

namespace fda {

// Part of the kernels' parameters. The order and the alignment count: the packed multiply-adds read their constants from there.
// With k0 on an odd multiple of 8 bytes the forward takes 1158 us (4 x 8192 tokens, 32 heads of 64), at the other offsets 1172
// to 1180; the single-pass kernel 2643 against 2688 to 2749.
struct alignas(16) CapPoly {
  float limit;            // |score| up to which the polynomial holds; negative: never (a scale that is not positive, or whose
                          // powers leave the fp32 range)
  float pre;              // x = score * pre
  float k0, k1, k2, k3;   // tanh(x) = score * (k0 + y (k1 + y (k2 + y k3))), y = score^2
};

__host__ __device__ __forceinline__ CapPoly make_cap_poly(float pre) {
  CapPoly c;
  const float p2 = pre * pre;
  c.pre = pre;
  c.k0 = 0.999999463558197f * pre;
  c.k1 = -0.3332631587982178f * pre * p2;
  c.k2 = 0.13190287351608276f * pre * p2 * p2;
  c.k3 = -0.04440191388130188f * pre * p2 * p2 * p2;
  c.limit = (pre > 1e-4f && pre < 1e4f) ? 0.5f / pre : -1.f;
  return c;
}

// Whether a warp's scores v[0 .. kN) all lie where the polynomial holds. Whole warps; the answer is the same in all lanes.
template <int kN>
__device__ __forceinline__ bool cap_poly_holds(const float* v, const CapPoly& c) {
  static_assert(kN % 8 == 0, "four running maxima of two columns each");
  float mx[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) mx[i] = ptx::max_nan(fabsf(v[2 * i]), fabsf(v[2 * i + 1]));
#pragma unroll
  for (int j = 8; j < kN; j += 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) mx[i] = ptx::max3_nan(mx[i], fabsf(v[j + 2 * i]), fabsf(v[j + 2 * i + 1]));
  }
  return __all_sync(0xffffffffu, ptx::max_nan(ptx::max3_nan(mx[0], mx[1], mx[2]), mx[3]) <= c.limit);
}

// tanh(x) / score of two columns, for scores inside the limit
__device__ __forceinline__ void cap_poly2(float& t0, float& t1, float s0, float s1, const CapPoly& c) {
  float y0, y1;
  ptx::mul2(y0, y1, s0, s1, s0, s1);
  ptx::fma2(t0, t1, y0, y1, c.k3, c.k3, c.k2, c.k2);
  ptx::fma2(t0, t1, y0, y1, t0, t1, c.k1, c.k1);
  ptx::fma2(t0, t1, y0, y1, t0, t1, c.k0, c.k0);
}

// Two scores become their tanh.
template <bool kPoly>
__device__ __forceinline__ void cap2(float& s0, float& s1, const CapPoly& c) {
  if (kPoly) {
    float t0, t1;
    cap_poly2(t0, t1, s0, s1, c);
    ptx::mul2(s0, s1, s0, s1, t0, t1);
  } else {
    s0 = ptx::tanh_fast(s0 * c.pre);
    s1 = ptx::tanh_fast(s1 * c.pre);
  }
}

template <int kN>
__device__ __forceinline__ void cap_scores(float* v, const CapPoly& c, bool poly) {
  if (poly) {
#pragma unroll
    for (int j = 0; j < kN; j += 2) cap2<true>(v[j], v[j + 1], c);
  } else {
#pragma unroll
    for (int j = 0; j < kN; j += 2) cap2<false>(v[j], v[j + 1], c);
  }
}

}  // namespace fda
