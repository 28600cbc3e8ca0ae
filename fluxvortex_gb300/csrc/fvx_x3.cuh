// fvx_x3.cuh -- the regularising cores f and f'(r)/r of the FP64 particle sweeps
// in three-float arithmetic, off the FP64 pipe.
//
// This GPU issues 1.7 FP64 operations per clock and SM against 123 FP32 ones,
// so one FP64 operation costs as much as 70 FP32 operations.  A pair's scalar
// chain -- r^2 + sigma^2, its root, powers, or the Gaussian core's erf and exp
// -- is 20 to 130 FP64 operations; as unevaluated sums of three floats (72
// bits) it is 400 to 800 FP32 operations, which run beside the FP64 vector part
// (9 to 21 operations).  The operations are built from the error-free
// transformations of Knuth (two_sum), Dekker (fast_two_sum) and an FMA
// (two_prod); f and f'/r carry a relative error below 2^-60 (Winckelmans) and
// 2^-56 (Gaussian) against 40-digit arithmetic over r / sigma from 1e-9 to 1e3
// (tests/test_x3_host.py), the FP64 forms they replace about 2^-51.
//
// Ranges: coordinates up to 2^13, cores of 2^-22 .. 2^13, so that every
// product and error term is a normal float; the caller keeps pairs outside of
// them on the FP64 forms.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define FVX_X3 __device__ __forceinline__
#else
#define FVX_X3 static inline
#endif

namespace fvx {
namespace x3 {

struct F3 {
  float h, m, l;  // h + m + l; |m| below 2^-21 |h| ("loose"), or ulp(h) / 2 after renorm
};

#if defined(__CUDA_ARCH__)
FVX_X3 float rcp_seed(float x) { return __frcp_rn(x); }
FVX_X3 uint64_t words(double x) { return (uint64_t)__double_as_longlong(x); }
FVX_X3 float add(float a, float b) { return __fadd_rn(a, b); }
FVX_X3 float sub(float a, float b) { return __fsub_rn(a, b); }
FVX_X3 float mul(float a, float b) { return __fmul_rn(a, b); }
FVX_X3 float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
FVX_X3 float rsqrt_seed(float x) { return rsqrtf(x); }
FVX_X3 uint32_t bits(float x) { return __float_as_uint(x); }
FVX_X3 float from_bits(uint32_t b) { return __uint_as_float(b); }
FVX_X3 double from_words(uint32_t hi, uint32_t lo) { return __hiloint2double(hi, lo); }
FVX_X3 int to_int(float x) { return __float2int_rn(x); }
FVX_X3 int to_int_down(float x) { return __float2int_rd(x); }
FVX_X3 float round_int(float x) { return rintf(x); }
#else
// the host's forms (compiled without contraction): the tests run them
FVX_X3 float rcp_seed(float x) { return 1.0f / x; }
FVX_X3 uint64_t words(double x) { uint64_t w; memcpy(&w, &x, 8); return w; }
FVX_X3 float add(float a, float b) { return a + b; }
FVX_X3 float sub(float a, float b) { return a - b; }
FVX_X3 float mul(float a, float b) { return a * b; }
FVX_X3 float fma_(float a, float b, float c) { return fmaf(a, b, c); }
FVX_X3 float rsqrt_seed(float x) { return (float)(1.0 / sqrt((double)x)) * (1.0f + 1.5e-7f); }
FVX_X3 uint32_t bits(float x) { uint32_t b; memcpy(&b, &x, 4); return b; }
FVX_X3 float from_bits(uint32_t b) { float x; memcpy(&x, &b, 4); return x; }
FVX_X3 double from_words(uint32_t hi, uint32_t lo) {
  uint64_t w = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &w, 8);
  return x;
}
FVX_X3 int to_int(float x) { return (int)lrintf(x); }
FVX_X3 int to_int_down(float x) { return (int)floorf(x); }
FVX_X3 float round_int(float x) { return rintf(x); }
#endif

// The ranges of coordinates (or offsets) and cores: magnitudes below 2^13, cores of
// 2^-22 .. 2^13; not NaN.
FVX_X3 bool coord_in_range(double x) {
  return ((uint32_t)(words(x) >> 32) & 0x7fffffffu) < (uint32_t)((1023 + 13) << 20);
}
FVX_X3 bool core_in_range(double s) {
  const uint32_t h = (uint32_t)(words(s) >> 32);
  return h >= (uint32_t)((1023 - 22) << 20) && h < (uint32_t)((1023 + 13) << 20);
}

// s + e = a + b exactly
FVX_X3 float two_sum(float a, float b, float& e) {
  const float s = add(a, b);
  const float v = sub(s, a);
  e = add(sub(a, sub(s, v)), sub(b, v));
  return s;
}
// the same for |a| >= |b| (or a = 0)
FVX_X3 float fast_two_sum(float a, float b, float& e) {
  const float s = add(a, b);
  e = sub(b, sub(s, a));
  return s;
}
// p + e = a b exactly
FVX_X3 float two_prod(float a, float b, float& e) {
  const float p = mul(a, b);
  e = fma_(a, b, -p);
  return p;
}

// FP64 -> three floats (exact within the ranges above)
FVX_X3 F3 split(double x) {
  F3 r;
  r.h = (float)x;
  const double y = x - (double)r.h;
  r.m = (float)y;
  r.l = (float)(y - (double)r.m);
  return r;
}

// The same for a positive FP64 number of 2^-60 .. 2^60 by integer operations: the
// leading 24 bits, the next 15 and the last 14.
FVX_X3 F3 split_positive(double x) {
  const uint64_t w = words(x);
  const uint32_t hi = (uint32_t)(w >> 32), lo = (uint32_t)w;
  const uint32_t b = ((hi << 3) | (lo >> 29)) - ((uint32_t)(1023 - 127) << 23);
  const uint32_t e = b & 0x7f800000u;  // 2^exponent
  F3 r;
  r.h = from_bits(b);
  r.m = mul((float)(int)((lo >> 14) & 0x7fffu), from_bits(e - (38u << 23)));
  r.l = mul((float)(int)(lo & 0x3fffu), from_bits(e - (52u << 23)));
  return r;
}

// h >= m >= l (in magnitude, loosely) -> without overlap
FVX_X3 F3 renorm(float h, float m, float l) {
  F3 r;
  float e;
  r.h = fast_two_sum(h, m, e);
  r.m = fast_two_sum(e, l, r.l);
  return r;
}

// split() of any FP64 number, off the FP64 pipe where its magnitude allows
FVX_X3 F3 split_fast(double x) {
  const uint64_t w = words(x);
  const uint32_t e = (uint32_t)(w >> 52) & 2047u;
  if (e - (1023u - 60u) < 120u) {
    F3 r = split_positive(from_words((uint32_t)(w >> 32) & 0x7fffffffu, (uint32_t)w));
    const uint32_t sign = (uint32_t)(w >> 32) & 0x80000000u;
    r.h = from_bits(bits(r.h) ^ sign);
    r.m = from_bits(bits(r.m) ^ sign);
    r.l = from_bits(bits(r.l) ^ sign);
    return renorm(r.h, r.m, r.l);
  }
  if ((w << 1) == 0) return F3{0.0f, 0.0f, 0.0f};
  return split(x);
}

// Three floats -> the FP64 number nearest to their sum, by integer operations:
// normalised, so that |m| <= ulp(h) / 2; then h's bits widened, and m + l in units
// of h's last FP64 place.  Only a power of two h can step down a binade, where
// a place is half.
FVX_X3 double to_double(const F3& loose) {
  F3 a = loose;
  float e;
  a.h = fast_two_sum(loose.h, loose.m, e);
  a.m = fast_two_sum(e, loose.l, a.l);
  const uint32_t b = bits(a.h);
  // 2^(52 - exponent of h), in two factors (it may exceed a float)
  const int ex = (int)((b >> 23) & 255u) - 127;
  const float s = from_bits((uint32_t)(127 + 26 - (ex >> 1)) << 23);
  const float s2 = from_bits((uint32_t)(127 + 26 - (ex - (ex >> 1))) << 23);
  const float m = mul(mul(a.m, s), s2), mi = round_int(m);
  int d = to_int(mi) + to_int(add(sub(m, mi), mul(mul(a.l, s), s2)));
  if ((int)b < 0) d = -d;  // places count magnitudes
  if ((b & 0x7fffffu) == 0 && d < 0) d += d;
  if ((b << 1) == 0) return 0.0;
  const uint32_t hi = ((b & 0x7fffffffu) >> 3) + ((uint32_t)(1023 - 127) << 20);
  const uint64_t w = (((uint64_t)hi << 32) | (b << 29)) + (uint64_t)(int64_t)d;
  return from_words((uint32_t)(w >> 32) | (b & 0x80000000u), (uint32_t)w);
}

// a - b with full relative accuracy of the difference
FVX_X3 F3 diff(const F3& a, const F3& b) {
  float e0, e1, e2, r;
  const float h = two_sum(a.h, -b.h, e0);
  const float m = two_sum(a.m, -b.m, e1);
  float l = add(e1, sub(a.l, b.l));
  const float v = two_sum(e0, m, e2);
  l = add(l, e2);
  F3 d;
  d.h = two_sum(h, v, r);
  d.m = two_sum(r, l, d.l);
  return d;
}

// a + b of numbers whose sum does not cancel
FVX_X3 F3 sum(const F3& a, const F3& b) {
  float e0, e1, e2;
  const float h = two_sum(a.h, b.h, e0);
  const float m = two_sum(a.m, b.m, e1);
  const float v = two_sum(m, e0, e2);
  return F3{h, v, add(add(a.l, b.l), add(e1, e2))};
}

// a b; a and b may be loose, and the result is
FVX_X3 F3 prod(const F3& a, const F3& b) {
  float e0, e1, e2, e3, e4;
  const float h = two_prod(a.h, b.h, e0);
  const float x = two_prod(a.h, b.m, e1);
  const float y = two_prod(a.m, b.h, e2);
  const float s = two_sum(x, y, e3);
  const float v = two_sum(e0, s, e4);
  float l = fma_(a.h, b.l, add(e1, e2));
  l = fma_(a.m, b.m, l);
  l = fma_(a.l, b.h, l);
  return F3{h, v, add(l, add(e3, e4))};
}

// a (1 + c), c = ch + cl small (below 2^-18); loose
FVX_X3 F3 scale1p(const F3& a, float ch, float cl) {
  float e0, e1;
  const float p = two_prod(a.h, ch, e0);
  const float v = two_sum(a.m, p, e1);
  const float l = add(fma_(a.m, ch, fma_(a.h, cl, a.l)), add(e0, e1));
  return F3{a.h, v, l};
}

// dx^2 + dy^2 + dz^2 (+ s)
template <bool ADD>
FVX_X3 F3 norm2(const F3& x, const F3& y, const F3& z, const F3& s) {
  float ex, ey, ez, fx, fy, fz, ea, eb = 0.0f, ec, r[8];
  const float px = two_prod(x.h, x.h, ex), py = two_prod(y.h, y.h, ey),
              pz = two_prod(z.h, z.h, ez);
  const float dx = add(x.h, x.h), dy = add(y.h, y.h), dz = add(z.h, z.h);
  const float mx = two_prod(dx, x.m, fx), my = two_prod(dy, y.m, fy), mz = two_prod(dz, z.m, fz);
  float l = add(fma_(x.m, x.m, fma_(dx, x.l, fx)), fma_(y.m, y.m, fma_(dy, y.l, fy)));
  l = add(l, fma_(z.m, z.m, fma_(dz, z.l, fz)));
  if (ADD) l = add(l, s.l);
  const float a = two_sum(px, py, ea), b = ADD ? two_sum(pz, s.h, eb) : pz,
              h = two_sum(a, b, ec);
  const float u0 = two_sum(ex, mx, r[0]), u1 = two_sum(ey, my, r[1]), u2 = two_sum(ez, mz, r[2]);
  const float u3 = two_sum(ea, ec, r[3]);
  const float v0 = two_sum(u0, u1, r[4]), v1 = two_sum(u2, u3, r[5]);
  float m = two_sum(v0, v1, r[6]);
  l = add(l, add(add(add(r[0], r[1]), add(r[2], r[3])), add(add(r[4], r[5]), r[6])));
  if (ADD) {
    float c;
    const float w = two_sum(eb, s.m, r[7]);
    m = two_sum(m, w, c);
    l = add(l, add(r[7], c));
  }
  return renorm(h, m, l);
}

// The reciprocal root's seed t and its defect E = 1 - q t^2 (|E| < 2^-20), with
// t^2 = p + pe exactly: 1/sqrt(q) = t (1 - E)^-1/2, and a power is t^k times the
// binomial series in E.
struct Root {
  float t, p, pe, eh, el;
};
FVX_X3 Root root(const F3& q) {
  Root R;
  R.t = rsqrt_seed(q.h);
  R.p = two_prod(R.t, R.t, R.pe);
  float re, we, ve, ea, eb, ec;
  const float r = two_prod(q.h, R.p, re);
  const float w = two_prod(q.h, R.pe, we);
  const float v = two_prod(q.m, R.p, ve);
  const float a = two_sum(sub(1.0f, r), -re, ea);
  const float b = two_sum(w, v, eb);
  const float e = two_sum(a, -b, ec);
  const float l = sub(add(sub(ea, eb), ec), add(add(we, ve), fma_(q.m, R.pe, mul(q.l, R.p))));
  R.eh = fast_two_sum(e, l, R.el);
  return R;
}

// a (1 - E)^-k: (1 - E)^-k - 1 = k E + k (k + 1) / 2 E^2 + k (k + 1)(k + 2) / 6 E^3
FVX_X3 F3 power_series(const F3& a, const Root& R, float k, float k2, float k3) {
  float e, cl;
  const float c = two_prod(k, R.eh, e);
  const float l = fma_(mul(R.eh, fma_(k3, R.eh, k2)), R.eh, fma_(k, R.el, e));
  const float ch = fast_two_sum(c, l, cl);
  return scale1p(a, ch, cl);
}
FVX_X3 F3 scale_float(const F3& a, float t) {
  float e0, e1, e2;
  const float h = two_prod(a.h, t, e0);
  const float m = two_prod(a.m, t, e1);
  const float v = two_sum(e0, m, e2);
  return F3{h, v, add(fma_(a.l, t, e1), e2)};
}
// q^-1/2, q^-1 and q^-5/2
FVX_X3 F3 power_m1_2(const Root& R) {
  return power_series(F3{R.t, 0.0f, 0.0f}, R, 0.5f, 0.375f, 0.3125f);
}
FVX_X3 F3 power_m1(const Root& R) { return power_series(F3{R.p, R.pe, 0.0f}, R, 1.0f, 1.0f, 1.0f); }
FVX_X3 F3 power_m5_2(const Root& R) {
  float e0, e1, e2;
  const float h = two_prod(R.p, R.p, e0);
  const float m = two_prod(add(R.p, R.p), R.pe, e1);
  const float v = two_sum(e0, m, e2);
  const F3 t4{h, v, add(fma_(R.pe, R.pe, e1), e2)};
  return power_series(scale_float(t4, R.t), R, 2.5f, 4.375f, 6.5625f);
}

// a / d for an FP64 d of 2^-60 .. 2^60: with y = 1/d's float and E = 1 - d y, a / d =
// a y (1 + E + E^2 + ..), |E| < 2^-23
FVX_X3 F3 quotient(const F3& a, double d) {
  const F3 q = split_positive(d);
  const float y = rcp_seed(q.h);
  float re, ve, ea, cl;
  const float r = two_prod(q.h, y, re);
  const float v = two_prod(q.m, y, ve);
  const float e = two_sum(sub(1.0f, r), -add(re, v), ea);
  // re + v rounds: what it loses (below 2^-24 of 2^-24) joins the low part
  const float s = add(re, v), back = sub(v, sub(s, re));
  const float l = sub(ea, add(add(back, ve), mul(q.l, y)));
  const float ch = fast_two_sum(e, fma_(e, e, l), cl);
  return scale1p(scale_float(a, y), ch, cl);
}

// Staged constants of a source: Winckelmans s2 = sigma^2, k = 1.5 sigma^2;
// Gaussian s2 = 1 / sigma^2, k = 1 / sigma^3, k5 = 1 / sigma^5.
struct Core {
  F3 s2, k, k5;
};

// 2 f + f'/r r^2, the vorticity's isotropic term
FVX_X3 F3 twice_f_plus(const F3& f, const F3& fpr, const F3& r2) {
  const F3 p = prod(fpr, r2);
  return diff(F3{add(f.h, f.h), add(f.m, f.m), add(f.l, f.l)}, F3{-p.h, -p.m, -p.l});
}

FVX_X3 Core winckelmans_core(const F3& s) {
  const F3 p = prod(s, s);
  Core c = {};
  c.s2 = renorm(p.h, p.m, p.l);
  c.k = scale_float(c.s2, 1.5f);
  return c;
}
FVX_X3 Core winckelmans_core(double sigma) { return winckelmans_core(split(sigma)); }
// (to three floats, so that sigma cancels where the core is the singular one)
FVX_X3 Core gaussian_core(double sigma) {
  const double r = 1.0 / sigma;
  F3 s = split(r);
  s.l = add(s.l, (float)(fma(-sigma, r, 1.0) * r));
  Core c;
  const F3 p = prod(s, s);
  c.s2 = renorm(p.h, p.m, p.l);
  c.k = prod(c.s2, s);
  c.k5 = prod(c.k, c.s2);
  return c;
}

// Winckelmans: f = (q + 1.5 s^2) q^-5/2 and, with FPR, f'/r =
// -3 (q + 2.5 s^2) q^-1 q^-5/2, q = r^2 + s^2; with SUM also f'/r r^2 + 2 f.
template <bool FPR, bool SUM>
FVX_X3 void winckelmans(const F3& x, const F3& y, const F3& z, const Core& c, F3& f, F3& fpr,
                        F3& s) {
  const F3 q = norm2<true>(x, y, z, c.s2);
  const Root R = root(q);
  const F3 g = power_m5_2(R);
  const F3 qk = sum(q, c.k);
  f = prod(qk, g);
  if (FPR) fpr = scale_float(prod(prod(sum(qk, c.s2), power_m1(R)), g), -3.0f);
  if (SUM) {
    s = twice_f_plus(f, fpr, norm2<false>(x, y, z, F3{}));
  }
}

// ---- the Gaussian core's polynomials (fvx_core_table.cuh) --------------------------
// F(x) = g(rho) / rho^3 and G(x) = 2 F'(x), x = rho^2 < kCoreEnd, by one degree-9
// polynomial per interval of a quarter about its middle: c0 and c1 as three
// floats, c2 .. c5 as two, c6 .. c9 as one (their terms are below 2^-35 of the
// value).  Horner in one, two and three floats to match.
constexpr int kRowFloats = 20;

FVX_X3 void step2(float ch, float cm, const F3& t, float& h, float& l) {
  float e, r;
  const float p = two_prod(t.h, h, e);
  e = fma_(t.h, l, fma_(t.m, h, e));
  h = fast_two_sum(ch, p, r);
  l = add(r, add(cm, e));
}

struct Row {
  float c[kRowFloats];
};

FVX_X3 F3 polynomial(const Row& r, const F3& t) {
  const float* c = r.c;
  float e;
  const float s = fma_(t.h, fma_(t.h, fma_(t.h, c[17], c[16]), c[15]), c[14]);
  float h = fast_two_sum(c[12], mul(t.h, s), e);
  float l = add(e, c[13]);
  step2(c[10], c[11], t, h, l);
  step2(c[8], c[9], t, h, l);
  step2(c[6], c[7], t, h, l);
  h = fast_two_sum(h, l, l);
  const F3 v = sum(F3{c[3], c[4], c[5]}, prod(t, F3{h, l, 0.0f}));
  return sum(F3{c[0], c[1], c[2]}, prod(t, v));
}

// Interval i of x, t = x - its middle; beyond `end` the core is the singular one
// (to 1e-18), F = x^-3/2 and G = -3 x^-5/2, homogeneous in x: x is brought to
// [64, 256) by a power of four, 4^-k, where intervals of one follow the others,
// and F and G come back by s3 = 8^-k and s3 s2 = 32^-k.  (A second branch for the
// singular core, which most warps then run beside the first, took 200
// operations.)
FVX_X3 int interval(const F3& x, float end, int rows, F3& t, float& s2, float& s3) {
  F3 v = x;
  const bool far = x.h >= end;
  s2 = s3 = 1.0f;
  int i;
  float mid;
  if (far) {
    // x.h = 2^ex (1 + ..): k = (ex - 6) / 2 rounded down
    const int k = ((int)(bits(x.h) >> 23) - 127 - 6) >> 1;
    s2 = from_bits((uint32_t)(127 - 2 * k) << 23);
    s3 = from_bits((uint32_t)(127 - 3 * k) << 23);
    v = F3{mul(x.h, s2), mul(x.m, s2), mul(x.l, s2)};
    const int j = to_int_down(v.h);
    mid = add((float)j, 0.5f);
    i = rows + j - 64;
  } else {
    i = to_int_down(mul(x.h, 4.0f));
    mid = fma_((float)i, 0.25f, 0.125f);
  }
  float e, u;
  const float h = two_sum(v.h, -mid, e);
  const float m = two_sum(e, v.m, u);
  t = renorm(h, m, add(u, v.l));
  return i;
}

// Gaussian-erf: f = F(x) / sigma^3, f'/r = G(x) / sigma^5, x = r^2 / sigma^2;
// rows(i, k) gives interval i's polynomial of F (k = 0) or G (k = 1).
template <bool FPR, bool SUM, typename Rows>
FVX_X3 void gaussian(const F3& x, const F3& y, const F3& z, const Core& c, float end, int n_rows,
                     Rows rows, F3& f, F3& fpr, F3& s) {
  const F3 r2 = norm2<false>(x, y, z, F3{});
  const F3 u = prod(r2, c.s2);
  F3 t;
  float s2, s3;
  const int i = interval(renorm(u.h, u.m, u.l), end, n_rows, t, s2, s3);
  auto scaled = [](const F3& a, float k) { return F3{mul(a.h, k), mul(a.m, k), mul(a.l, k)}; };
  f = prod(polynomial(rows(i, 0), t), scaled(c.k, s3));
  if (FPR) fpr = prod(polynomial(rows(i, 1), t), scaled(scaled(c.k5, s3), s2));
  if (SUM) s = twice_f_plus(f, fpr, r2);
}

}  // namespace x3
}  // namespace fvx
