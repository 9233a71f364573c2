// Elementary functions rounded once from more than float precision, without the FP64 pipe (its rate on
// sm_103a is far below the FP32 one): a value is evaluated as an unevaluated sum of two floats, to within
// 2^-40.5 of its magnitude (measured against extended precision over the floats of the ranges below),
// and rounded when every value within PAIR_ERR of it rounds to the same float; otherwise (about one
// call in 10,000) FP64 decides.  The results are those of the FP64 function rounded to float.
// Operations are the error-free transformations of Dekker (1971) and Knuth; the functions are their
// Taylor series after a reduction of the argument by split constants (Cody and Waite).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace fg {

#ifdef __CUDA_ARCH__
#define PAIR_ADD(a, b) __fadd_rn(a, b)
#define PAIR_SUB(a, b) __fsub_rn(a, b)
#define PAIR_MUL(a, b) __fmul_rn(a, b)
#define PAIR_FMA(a, b, c) __fmaf_rn(a, b, c)
#else  // compiled without contraction on the host
#define PAIR_ADD(a, b) ((a) + (b))
#define PAIR_SUB(a, b) ((a) - (b))
#define PAIR_MUL(a, b) ((a) * (b))
#define PAIR_FMA(a, b, c) fmaf(a, b, c)
#endif
#define PAIR_FN __host__ __device__ __forceinline__

struct Pair {
  float h, l;  // |l| <= ulp(h) / 2
};

PAIR_FN uint32_t pair_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t b;
  std::memcpy(&b, &f, sizeof(b));
  return b;
#endif
}
PAIR_FN float pair_float(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  std::memcpy(&f, &b, sizeof(f));
  return f;
#endif
}
PAIR_FN uint64_t pair_bits64(double v) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(v));
#else
  uint64_t b;
  std::memcpy(&b, &v, sizeof(b));
  return b;
#endif
}

constexpr float PAIR_ERR = 3.637978807091713e-12f;  // 2^-38, relative

// a + b for |a| >= |b| (or a = 0).
PAIR_FN Pair pair_fast(float a, float b) {
  const float s = PAIR_ADD(a, b);
  return Pair{s, PAIR_SUB(b, PAIR_SUB(s, a))};
}
PAIR_FN Pair pair_sum(float a, float b) {
  const float s = PAIR_ADD(a, b), t = PAIR_SUB(s, a);
  return Pair{s, PAIR_ADD(PAIR_SUB(a, PAIR_SUB(s, t)), PAIR_SUB(b, t))};
}
PAIR_FN Pair pair_prod(float a, float b) {
  const float p = PAIR_MUL(a, b);
  return Pair{p, PAIR_FMA(a, b, -p)};
}
PAIR_FN Pair pair_add(Pair a, Pair b) {
  const Pair s = pair_sum(a.h, b.h);
  return pair_fast(s.h, PAIR_ADD(s.l, PAIR_ADD(a.l, b.l)));
}
// c + a for |c| >= |a|.
PAIR_FN Pair pair_add(Pair c, float a) {
  const Pair s = pair_fast(c.h, a);
  return pair_fast(s.h, PAIR_ADD(s.l, c.l));
}
PAIR_FN Pair pair_mul(Pair a, Pair b) {
  const Pair p = pair_prod(a.h, b.h);
  return pair_fast(p.h, PAIR_FMA(a.h, b.l, PAIR_FMA(a.l, b.h, p.l)));
}
PAIR_FN Pair pair_mul(Pair a, float b) {
  const Pair p = pair_prod(a.h, b);
  return pair_fast(p.h, PAIR_FMA(a.l, b, p.l));
}

// A quotient and its remainder's.
PAIR_FN Pair pair_div(Pair n, Pair d) {
  const float inv = 1.0f / d.h;
  const float q = PAIR_MUL(n.h, inv);
  const float rem = PAIR_ADD(PAIR_FMA(-q, d.h, n.h), PAIR_FMA(-q, d.l, n.l));
  return pair_fast(q, PAIR_MUL(rem, inv));
}

// Whether the value's rounding to float is settled; r receives it.
PAIR_FN bool pair_round(Pair a, float& r) {
  const float e = PAIR_MUL(fabsf(a.h), PAIR_ERR);
  r = PAIR_ADD(a.h, PAIR_ADD(a.l, e));
  return r == PAIR_ADD(a.h, PAIR_SUB(a.l, e));
}

// log of a positive normal float plus a low part: x = 2^k m, m in [sqrt(1/2), sqrt(2));
// log m = 2 atanh(s), s = (m - 1) / (m + 1), |s| < .1716.  (From 2^127.5 on, k is 128 and the low part's
// scale overflows: the result is a NaN, which pair_round does not settle.)
PAIR_FN Pair pair_log(float x, float xl = 0.0f) {
  const int b = static_cast<int>(pair_bits(x));
  const int k = (b - 0x3f3504f3) >> 23;  // 0x3f3504f3: sqrt(1/2)
  const float m = pair_float(static_cast<uint32_t>(b - (k << 23)));
  const float up = pair_float(static_cast<uint32_t>(127 - k) << 23);
  const float f = PAIR_SUB(m, 1.0f), fl = PAIR_MUL(xl, up);  // f is exact
  const Pair n = pair_fast(f, fl);
  Pair d = pair_sum(2.0f, f);
  d = pair_fast(d.h, PAIR_ADD(d.l, fl));
  const Pair s = pair_div(n, d);
  const Pair z = pair_mul(s, s);
  // 2 s (1 + z / 3 + z^2 / 5 + ...), z < .0295: the first two terms as pairs.
  float p = 0.13333334f;  // 2 / 15
  p = PAIR_FMA(p, z.h, 0.15384616f);
  p = PAIR_FMA(p, z.h, 0.18181819f);
  p = PAIR_FMA(p, z.h, 0.22222222f);
  p = PAIR_FMA(p, z.h, 0.2857143f);
  Pair t = pair_add(Pair{0.400000006f, -5.96046457e-09f}, PAIR_MUL(p, z.h));
  t = pair_mul(t, z);
  t = pair_add(Pair{0.666666687f, -1.98682155e-08f}, t);
  t = pair_mul(pair_mul(t, z), s);
  const Pair lm = pair_add(Pair{2.0f * s.h, 2.0f * s.l}, t);
  // k log 2: the first part has 16 bits, its product is exact.
  const float kf = static_cast<float>(k);
  const Pair lk = pair_mul(Pair{1.42860677e-06f, 5.49792315e-14f}, kf);
  return pair_add(pair_add(Pair{PAIR_MUL(kf, 0.693145751953125f), 0.0f}, lk), lm);
}

// exp for |x| <= 70 (the low part stays a normal float): x = k log 2 + r, |r| < .347, by the series of r / 8 and three squarings.
PAIR_FN Pair pair_exp(float x) {
  const float kf = rintf(PAIR_MUL(x, 1.4426950f));
  const Pair c = pair_prod(-kf, 1.42860677e-06f);
  Pair r = pair_sum(PAIR_FMA(-kf, 0.693145751953125f, x), c.h);
  r = pair_fast(r.h, PAIR_ADD(r.l, PAIR_FMA(-kf, 5.49792315e-14f, c.l)));
  r = Pair{PAIR_MUL(0.125f, r.h), PAIR_MUL(0.125f, r.l)};
  // 1 + r + r^2 / 2 + r^3 / 6 + r^4 (1 / 24 + ...), |r| < .0434.
  float p = 0.0013888889f;
  p = PAIR_FMA(p, r.h, 0.008333334f);
  p = PAIR_FMA(p, r.h, 0.041666668f);
  Pair t = pair_add(Pair{0.166666672f, -4.96705388e-09f}, PAIR_MUL(p, r.h));
  t = pair_add(Pair{0.5f, 0.0f}, pair_mul(t, r));
  t = pair_add(Pair{1.0f, 0.0f}, pair_mul(t, r));
  t = pair_add(Pair{1.0f, 0.0f}, pair_mul(t, r));
  t = pair_mul(t, t);
  t = pair_mul(t, t);
  t = pair_mul(t, t);
  const float up = pair_float(static_cast<uint32_t>(127 + static_cast<int>(kf)) << 23);
  return Pair{PAIR_MUL(t.h, up), PAIR_MUL(t.l, up)};
}

// sin and cos for |x| <= 8: x = k pi / 2 + r, |r| <= pi / 4; the first part of pi / 2 has 20 bits, so
// its product and the difference are exact.
PAIR_FN void pair_sincos(float x, Pair& sn, Pair& cs) {
  const float kf = rintf(PAIR_MUL(x, 0.63661975f));
  const Pair c = pair_prod(-kf, 1.26759085e-06f);
  Pair r = pair_sum(PAIR_FMA(-kf, 1.5707950592041016f, x), c.h);
  r = pair_fast(r.h, PAIR_ADD(r.l, PAIR_FMA(-kf, -5.14531146e-14f, c.l)));
  const Pair z = pair_mul(r, r);
  // sin r = r + r z (S1 + z (S2 + z (S3 + ...))), cos r = 1 + z (-1/2 + z (C2 + z (C3 + ...))),
  // z < .617: three coefficients each as pairs.
  float p = 1.6059044e-10f;
  p = PAIR_FMA(p, z.h, -2.5052108e-08f);
  p = PAIR_FMA(p, z.h, 2.7557319e-06f);
  Pair t = pair_add(Pair{-0.000198412701f, 2.72559687e-12f}, PAIR_MUL(p, z.h));
  t = pair_add(Pair{0.00833333377f, -4.34617203e-10f}, pair_mul(t, z));
  t = pair_add(Pair{-0.166666672f, 4.96705388e-09f}, pair_mul(t, z));
  t = pair_mul(pair_mul(t, z), r);
  const Pair s = pair_add(r, t);
  p = -1.1470746e-11f;
  p = PAIR_FMA(p, z.h, 2.0876757e-09f);
  p = PAIR_FMA(p, z.h, -2.7557319e-07f);
  p = PAIR_FMA(p, z.h, 2.4801588e-05f);
  t = pair_add(Pair{-0.00138888892f, 3.36310944e-11f}, PAIR_MUL(p, z.h));
  t = pair_add(Pair{0.0416666679f, -1.24176347e-09f}, pair_mul(t, z));
  t = pair_add(Pair{-0.5f, 0.0f}, pair_mul(t, z));
  const Pair q = pair_add(Pair{1.0f, 0.0f}, pair_mul(t, z));
  const int k = static_cast<int>(kf) & 3;
  const Pair a = k & 1 ? q : s, b = k & 1 ? s : q;
  sn = k & 2 ? Pair{-a.h, -a.l} : a;
  cs = (k + 1) & 2 ? Pair{-b.h, -b.l} : b;
}

// hi = v rounded to float, lo = v - hi (exact) rounded to float.  In integer arithmetic: hi takes the
// upper 24 bits of v's 53, lo is the signed rest of at most 2^28.  Zero and magnitudes outside 2^-60 ..
// 2^120 are converted.
PAIR_FN void split64(double v, float& hi, float& lo) {
  const uint64_t b = pair_bits64(v);
  const uint32_t h = static_cast<uint32_t>(b >> 32), l = static_cast<uint32_t>(b);
  const uint32_t e = (h >> 20) & 0x7ffu;
  if (e - 963u > 180u) {
    hi = static_cast<float>(v);
    lo = static_cast<float>(v - static_cast<double>(hi));
    return;
  }
  const uint32_t q = ((h & 0xfffffu) << 3) | (l >> 29), r = l & 0x1fffffffu;  // q: 23 bits below the leading one
  const bool up = r > 0x10000000u || (r == 0x10000000u && (q & 1u));           // to nearest, ties to even
  const int d = static_cast<int>(r) - (up ? 0x20000000 : 0);
  hi = pair_float((h & 0x80000000u) | (((e - 896u) << 23) + q + (up ? 1u : 0u)));
  // d in units of 2^(e - 1075); a rest of zero is +0 whatever the sign.
  lo = PAIR_MUL(static_cast<float>(static_cast<int>(h) < 0 ? -d : d), pair_float((e - 948u) << 23));
}

// n / d of FP64 values, given also as pairs (to 2^-48), rounded to float.
PAIR_FN float pair_quotf(double n, double d, Pair np, Pair dp) {
  float r;
  // About 2^-50, 2^50: quotients from 2^-100 on, whose low parts a float's smallest step (2^-149) holds to
  // 2^-49 of the quotient.  (With 2^-60 and 2^60, quotients below 2^-115 could round the wrong way.)
  const float lo = 8.9e-16f, hi = 1.1e15f;
  if (fabsf(np.h) > lo && fabsf(np.h) < hi && fabsf(dp.h) > lo && fabsf(dp.h) < hi && pair_round(pair_div(np, dp), r)) return r;
  return static_cast<float>(n / d);
}

// The FP64 functions rounded to float.
PAIR_FN float pair_expf(float x) {
  float r;
  if (fabsf(x) <= 70.0f && pair_round(pair_exp(x), r)) return r;
  return static_cast<float>(exp(static_cast<double>(x)));
}
PAIR_FN float pair_logf(float x) {
  float r;
  if (x >= 1.17549435e-38f && x <= 3.4028235e38f && pair_round(pair_log(x), r)) return r;
  return static_cast<float>(log(static_cast<double>(x)));
}
PAIR_FN void pair_sincosf(float x, float& sn, float& cs) {
  Pair s, c;
  pair_sincos(x, s, c);
  const bool in = fabsf(x) <= 8.0f;
  if (!(in && pair_round(s, sn))) sn = static_cast<float>(sin(static_cast<double>(x)));
  if (!(in && pair_round(c, cs))) cs = static_cast<float>(cos(static_cast<double>(x)));
}

// The density -log10(clamp(T, 1e-4, 1)) + 0.05 of a transmittance.
PAIR_FN float pair_densityf(float T) {
  float r;
  const bool in = T > 1.0001e-4f && T <= 1.0f;
  const Pair v = pair_add(pair_mul(pair_log(in ? T : 1.0f), Pair{-0.434294492f, 1.010305e-08f}),
                          Pair{0.0500000007f, -7.45058071e-10f});
  if (in && pair_round(v, r)) return r;
  const double tc = fmin(fmax(static_cast<double>(T), 1e-4), 1.0);
  return tc == 1e-4 ? 4.05f : (tc == 1.0 ? 0.05f : static_cast<float>(-log10(tc) + 0.05));
}

}  // namespace fg
