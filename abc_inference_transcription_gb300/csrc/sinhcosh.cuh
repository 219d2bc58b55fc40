// sinhcosh.cuh — sinh and cosh as unevaluated sums of two floats, for results
// that are rounded to float: the FP64 pipe needs some 3,500 issue slots of a
// scheduler for a warp's sinh and cosh, these about 300.
//
// Sums and products of two floats with their errors: T. J. Dekker, "A
// floating-point technique for extending the available precision", Numer. Math.
// 18 (1971); the exponential by a table of 2^(j/32) and a short polynomial:
// P. T. P. Tang, "Table-driven implementation of the exponential function in
// IEEE floating-point arithmetic", ACM TOMS 15 (1989).  Relative errors below
// kSinhCoshErr over the range that sinh_cosh accepts (measured: 2^-42), so
// that a caller can tell when the rounding to float is beyond doubt
// (rounds_to) and compute in FP64 where it is not.
//
// Every operation is rounded by itself: no contraction on the device
// (__fmul_rn and the like); a host build needs -ffp-contract=off.
#pragma once
#include "common.cuh"

namespace abc {

constexpr float kSinhCoshErr = 1.8189894e-12f;  // 2^-39

struct FF {
  float h, l;  // h = RN(h + l)
};

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ float f_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float f_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float f_mul(float a, float b) { return __fmul_rn(a, b); }
#else
ABC_HD float f_add(float a, float b) { return a + b; }
ABC_HD float f_sub(float a, float b) { return a - b; }
ABC_HD float f_mul(float a, float b) { return a * b; }
#endif

ABC_HD FF two_sum(float a, float b) {
  const float s = f_add(a, b), v = f_sub(s, a);
  return {s, f_add(f_sub(a, f_sub(s, v)), f_sub(b, v))};
}
ABC_HD FF quick_sum(float a, float b) {  // |a| >= |b| or a = 0
  const float s = f_add(a, b);
  return {s, f_sub(b, f_sub(s, a))};
}
ABC_HD FF two_prod(float a, float b) {
  const float p = f_mul(a, b);
  return {p, fmaf(a, b, -p)};
}
ABC_HD FF ff_add(FF a, FF b) {
  const FF s = two_sum(a.h, b.h);
  return quick_sum(s.h, f_add(s.l, f_add(a.l, b.l)));
}
ABC_HD FF ff_mul(FF a, FF b) {
  const FF p = two_prod(a.h, b.h);
  return quick_sum(p.h, f_add(p.l, fmaf(a.h, b.l, f_mul(a.l, b.h))));
}
ABC_HD FF ff_mul1(FF a, float b) {
  const FF p = two_prod(a.h, b);
  return quick_sum(p.h, fmaf(a.l, b, p.l));
}
// a b + c, rounded nowhere but in the low part
ABC_HD FF ff_muladd(float a, float b, float c) {
  const FF p = two_prod(a, b), s = two_sum(p.h, c), t = two_sum(s.l, p.l), u = two_sum(s.h, t.h);
  return {u.h, f_add(u.l, t.l)};
}

// x to the float nearest to x.h + x.l, true if every value within a relative
// err of it rounds there too
ABC_HD bool rounds_to(FF x, float err, float& out) {
  const float e = f_mul(fabsf(x.h), err);
  out = f_add(x.h, f_add(x.l, e));
  return out == f_add(x.h, f_sub(x.l, e));
}

// 2^(j/32)
#define ABC_POW32 \
  {               \
    {1.0f, 0.0f}, {1.0218972f, -4.81156e-08f}, {1.0442737f, 4.83347e-08f}, {1.0671405f, -5.933752e-08f},  \
    {1.0905077f, -1.307754e-08f}, {1.1143868f, -5.43554e-08f}, {1.1387886f, 5.3862223e-08f}, {1.1637249f, -4.0514415e-08f},  \
    {1.1892071f, 3.7976353e-08f}, {1.2152474f, -3.267395e-08f}, {1.2418578f, 4.496838e-08f}, {1.269051f, 1.4193333e-09f},  \
    {1.2968396f, -4.0189995e-08f}, {1.3252367f, -3.4963733e-08f}, {1.3542556f, -1.0123349e-08f}, {1.38391f, -5.8755774e-08f},  \
    {1.4142135f, 2.4203235e-08f}, {1.4451808f, 3.3242e-08f}, {1.4768262f, -4.500899e-08f}, {1.5091645f, -2.4959373e-08f},  \
    {1.5422108f, 8.070905e-09f}, {1.5759809f, -5.6610254e-08f}, {1.6104903f, 9.836217e-09f}, {1.6457555f, -5.124972e-08f},  \
    {1.6817929f, -2.4755327e-08f}, {1.7186193f, -4.8496176e-08f}, {1.7562522f, -9.23577e-09f}, {1.7947091f, -1.1415045e-08f},  \
    {1.8340081f, -1.1239278e-08f}, {1.8741677f, -4.6630056e-08f}, {1.9152066f, 9.845328e-09f}, {1.9571441f, -1.7021804e-08f}  \
  }
#if defined(__CUDACC__)
static __device__ const float2 kPow32Dev[32] = ABC_POW32;
#endif
ABC_HD FF pow32(int j) {
#if defined(__CUDA_ARCH__)
  const float2 t = __ldg(kPow32Dev + j);
  return {t.x, t.y};
#else
  static const FF t[32] = ABC_POW32;
  return t[j];
#endif
}

ABC_HD float bits_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

// 2^k (t (1 + r + r^2 / 2 + tail)) for t = 2^(j/32), scaled by sc = 2^k
ABC_HD FF scaled_exp(FF t, float rh, float rl, float tail, FF r2, float sc) {
  const FF p = quick_sum(rh, f_mul(r2.h, 0.5f));
  const float pl = f_add(p.l, f_add(rl, fmaf(r2.l, 0.5f, tail)));
  const FF m = two_prod(t.h, p.h), s = quick_sum(t.h, m.h);
  const float lo = f_add(s.l, f_add(m.l, fmaf(t.h, pl, fmaf(t.l, p.h, t.l))));
  return {f_mul(s.h, sc), f_mul(lo, sc)};
}

// sinh(u) and cosh(u); false outside 2^-30 <= |u| <= 30
ABC_HD bool sinh_cosh(FF u, FF& sh, FF& ch) {
  const bool neg = u.h < 0.0f;
  const float a = neg ? -u.h : u.h, al = neg ? -u.l : u.l;
  if (!(a >= 9.3132257e-10f && a <= 30.0f)) return false;
  if (a < 0.35f) {
    // Taylor sums, the leading terms in two floats: the last one left out is below 2^-47
    FF z = two_prod(a, a);
    z = quick_sum(z.h, fmaf(2.0f * a, al, z.l));
    const float s3 = fmaf(z.h, fmaf(z.h, 2.5052108e-8f, 2.7557319e-6f), 1.9841270e-4f);
    // z / 6 + z^2 / 120 + z^3 (1 / 5040 + ...)
    FF q = ff_add({8.3333338e-3f, -4.346172e-10f}, two_prod(z.h, s3));
    q = ff_add({0.16666667f, -4.967054e-9f}, ff_mul(z, q));
    q = ff_mul(z, q);
    sh = ff_add({a, al}, ff_mul({a, al}, q));
    // z / 2 + z^2 / 24 + z^3 (1 / 720 + ...)
    const float c3 = fmaf(z.h, fmaf(z.h, fmaf(z.h, 2.0876757e-9f, 2.7557319e-7f), 2.4801587e-5f), 1.3888889e-3f);
    q = ff_add({4.1666668e-2f, -1.2417635e-9f}, two_prod(z.h, c3));
    q = ff_add({0.5f, 0.0f}, ff_mul(z, q));
    ch = ff_add({1.0f, 0.0f}, ff_mul(z, q));
  } else {
    // a = n ln 2 / 32 + r, n = 32 k + j; ln 2 / 32 in parts of 13, 13 and 24 bits,
    // so that n times the first two is exact
    const float n = rintf(f_mul(a, 46.166241f));
    const int ni = (int)n, j = ni & 31, k = ni >> 5;
    FF r = two_sum(fmaf(-n, 0.021659851f, a), f_mul(-n, 9.98145e-07f));
    r = two_sum(r.h, f_add(r.l, fmaf(-n, 1.733102e-10f, al)));
    const FF r2 = {f_mul(r.h, r.h), 0.0f};
    const FF rr = {r2.h, f_add(fmaf(r.h, r.h, -r2.h), f_mul(2.0f * r.h, r.l))};
    // r^3 / 6 + r^5 / 120 and r^4 / 24
    const float odd = f_mul(f_mul(rr.h, r.h), fmaf(rr.h, 8.3333333e-3f, 0.16666667f));
    const float even = f_mul(f_mul(rr.h, rr.h), 4.1666668e-2f);
    // e^a / 2^k and e^-a / 2^k
    const FF ep = scaled_exp(pow32(j), r.h, r.l, f_add(even, odd), rr, 1.0f);
    const FF en = scaled_exp(pow32((32 - j) & 31), -r.h, -r.l, f_sub(even, odd), rr,
                             bits_float((uint32_t)(127 - 2 * k - (j ? 1 : 0)) << 23));
    const float half = bits_float((uint32_t)(126 + k) << 23);
    const FF d = two_sum(ep.h, -en.h), s = two_sum(ep.h, en.h);
    sh = quick_sum(f_mul(d.h, half), f_mul(f_add(d.l, f_sub(ep.l, en.l)), half));
    ch = quick_sum(f_mul(s.h, half), f_mul(f_add(s.l, f_add(ep.l, en.l)), half));
  }
  if (neg) sh = {-sh.h, -sh.l};
  return true;
}

ABC_HD bool within(float x, float lo, float hi) { return fabsf(x) > lo && fabsf(x) < hi; }

// The mean and variance of y = c sinh(u), u = mu sd + mean with variance var sd^2
// (delta method), or of u itself where c is not positive: what FP64 gives, rounded to float.
// False where that takes FP64: next to a rounding boundary, or outside the range in which
// the errors of the products are representable.
ABC_HD bool unscale32(float mu, float var, float sd, float mean, float c, float& m, float& v) {
  const FF u = ff_muladd(mu, sd, mean);
  const FF vu = ff_mul1(two_prod(var, sd), sd);
  if (!within(vu.h, 1e-9f, 1e9f)) return false;
  if (!(c > 0.0f)) return within(u.h, 1e-9f, 1e9f) && rounds_to(u, kSinhCoshErr, m) && rounds_to(vu, kSinhCoshErr, v);
  FF sh, ch;
  if (!sinh_cosh(u, sh, ch)) return false;
  sh = ff_mul1(sh, c);
  ch = ff_mul1(ch, c);
  if (!within(sh.h, 1e-15f, 1e15f) || !within(ch.h, 1e-6f, 1e14f)) return false;
  return rounds_to(sh, kSinhCoshErr, m) && rounds_to(ff_mul(ff_mul(ch, ch), vu), 2.0f * kSinhCoshErr, v);
}

}  // namespace abc
