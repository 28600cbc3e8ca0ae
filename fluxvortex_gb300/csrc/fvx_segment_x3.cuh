// fvx_segment_x3.cuh -- the line vortex of fvx_segment_math.cuh with its scalar
// parts in three-float arithmetic (fvx_x3.cuh), for the Biot-Savart sweeps.
//
// Per corner the offset, its length and reciprocal length, and per leg
//   c4 = Gamma / 8pi (1/la + 1/lb) (r0^2 - (la - lb)^2) / (|r3|^2 + r0^2 rc^2)
// are formed on the FP32 pipe; FP64 keeps r3 = d_a x d_b, its square and the
// sums: 55 operations per ring against about 140, beside some 2,700 FP32 ones.
// The 72 bits also carry the law of cosines' form of la lb - c3 to within a
// thousandth of a leg's length of a corner.  Points nearer than that, and all
// pairs outside the arithmetic's range, keep the FP64 forms.
#pragma once

#include "fvx_segment_math.cuh"
#include "fvx_x3.cuh"

namespace fvx {
namespace seg {

// Corners and leg constants of one vortex.
struct RingX3 {
  x3::F3 c[4][3];   // corners BR, FR, FL, BL
  x3::F3 r0sq[4];   // |end - start|^2 per leg
  double c2[4];     // |end - start|^2 r_c^2 per leg
  double half_c1;   // Gamma / (8 pi)
  float near;       // |d|^2 below this at a corner: general path, unless zero (all: > kNoX3)
  int pad;
};

// Legs of 2^-20 .. 2^15 (high words of their squares) and core terms to 2^50:
// with corners and points within 2^13 every product is a normal float, and a
// corner whose |d|^2 is zero in floats (|d| < 2^-74) is within every tolerance
// (1e-10 of 2^-20).
constexpr int kX3LegMin = (1023 - 40) << 20, kX3LegMax = (1023 + 30) << 20;
constexpr int kX3CoreMax = (1023 + 50) << 20;

constexpr float kNoX3 = 1e30f;

__device__ __forceinline__ bool x3_range(double x) {
  return (__double2hiint(x) & 0x7fffffff) < ((1023 + 13) << 20);
}

template <int LEGS>
__device__ __forceinline__ void prep_x3(RingX3& X, const VortexRec& R) {
  bool ok = R.lo < kHiMax;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      X.c[c][k] = x3::split_fast(R.c[c][k]);
      ok = ok && x3_range(R.c[c][k]);
    }
  float far = 0.0f;
#pragma unroll
  for (int l = Legs<LEGS>::n; l < 4; ++l) {
    X.r0sq[l] = x3::F3{};
    X.c2[l] = 0.0;
  }
#pragma unroll
  for (int l = 0; l < Legs<LEGS>::n; ++l) {
    const x3::F3* s = X.c[Legs<LEGS>::s(l)];
    const x3::F3* e = X.c[Legs<LEGS>::e(l)];
    X.r0sq[l] = x3::norm2<false>(x3::diff(e[0], s[0]), x3::diff(e[1], s[1]),
                                 x3::diff(e[2], s[2]), x3::F3{});
    X.c2[l] = R.c2[l];
    const int h = __double2hiint(R.r0sq[l]);
    ok = ok && h >= kX3LegMin && h < kX3LegMax && __double2hiint(R.c2[l]) < kX3CoreMax;
    far = fmaxf(far, X.r0sq[l].h);
  }
  X.half_c1 = 0.5 * R.c1;
  X.near = ok ? far * 2.168404344971009e-19f : __int_as_float(0x7f800000);  // 2^-62 far
}

// Reads a RingX3 (shared memory, by broadcast).
struct RingView {
  const RingX3& X;
  __device__ __forceinline__ x3::F3 corner(int c, int k) const { return X.c[c][k]; }
  __device__ __forceinline__ x3::F3 r0sq(int l) const { return X.r0sq[l]; }
  __device__ __forceinline__ double c2(int l) const { return X.c2[l]; }
  __device__ __forceinline__ float near() const { return X.near; }
  __device__ __forceinline__ double half_c1() const { return X.half_c1; }
};

// A corner as a point sees it: offset, |d|^2 and, in three floats, |d| and 1/|d|.
// on: the point is the corner itself.
struct CornerX3 {
  double d[3];
  x3::F3 inv, len;
  float sq;
  bool on;
};
template <typename View>
__device__ __forceinline__ CornerX3 see_corner(const View& V, int c, const x3::F3* p,
                                               bool& general) {
  CornerX3 C;
  x3::F3 o[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    o[k] = x3::diff(V.corner(c, k), p[k]);
    C.d[k] = x3::to_double(o[k]);
  }
  x3::F3 q = x3::norm2<false>(o[0], o[1], o[2], x3::F3{});
  C.sq = q.h;
  C.on = !(q.h > V.near());
  if (C.on) {
    general = general || q.h != 0.0f;
    q.h = 1.0f;
  }
  const x3::Root R = x3::root(q);
  C.inv = x3::power_m1_2(R);
  C.len = x3::prod(q, C.inv);
  return C;
}

// Velocity of one vortex (all legs), its `near` at most kNoX3, at the point p, within
// 2^13; rare(v, cnt): the general path's velocity and skips.  The legs are a loop, not
// unrolled: 3,000 instructions in a row run from the instruction cache's next
// level (14.6 ms for 10,000 x 10,000 rings, against 12.5 ms so).
template <int LEGS, typename View, typename Rare>
__device__ __forceinline__ void vortex_velocity_x3(const View& V, const x3::F3* p, double& vx,
                                                   double& vy, double& vz, int cnt[4],
                                                   Rare rare) {
  constexpr bool kChain = LEGS != FVX_LEGS_CHORDWISE;  // a leg starts where the last one ended
  bool general = false;
  double ux = 0.0, uy = 0.0, uz = 0.0;
  int on_start = 0, on_end = 0, on_line = 0;
  CornerX3 a, first;
  if (kChain) {
    a = see_corner(V, 0, p, general);
    if (LEGS == FVX_LEGS_RING) first = a;
  }
#pragma unroll 1
  for (int l = 0; l < Legs<LEGS>::n; ++l) {
    CornerX3 b;
    if (!kChain) a = see_corner(V, 2 * l, p, general);
    if (LEGS == FVX_LEGS_RING && l == 3)
      b = first;
    else
      b = see_corner(V, kChain ? l + 1 : 2 * l + 1, p, general);
    const double r3x = fma(a.d[1], b.d[2], -(a.d[2] * b.d[1]));
    const double r3y = fma(a.d[2], b.d[0], -(a.d[0] * b.d[2]));
    const double r3z = fma(a.d[0], b.d[1], -(a.d[1] * b.d[0]));
    const double r3_sq = fma(r3z, r3z, fma(r3y, r3y, r3x * r3x));
    // high words of |d_a|^2 and |d_b|^2 from their floats'
    const int ha = static_cast<int>(x3::bits(a.sq) >> 3) + ((1023 - 127) << 20);
    const int hb = static_cast<int>(x3::bits(b.sq) >> 3) + ((1023 - 127) << 20);
    if (a.on || b.on) {
      if (a.on)
        on_start++;
      else
        on_end++;
    } else if (__double2hiint(r3_sq) < ha + (hb + kHiLine) &&
               on_leg_line(r3_sq, a.d[0] * a.d[0] + a.d[1] * a.d[1] + a.d[2] * a.d[2],
                           b.d[0] * b.d[0] + b.d[1] * b.d[1] + b.d[2] * b.d[2])) {
      on_line++;
    } else {
      const x3::F3 r0sq = V.r0sq(l);
      const x3::F3 gap = x3::diff(a.len, b.len);
      x3::F3 num = x3::diff(r0sq, x3::prod(gap, gap));  // 2 (la lb - c3)
      const bool near = fminf(a.sq, b.sq) < 9.5367431640625e-7f * r0sq.h;  // 2^-20
      if (__any_sync(__activemask(), near)) {
        const double c3 = a.d[0] * b.d[0] + a.d[1] * b.d[1] + a.d[2] * b.d[2];
        if (near) num = x3::split(2.0 * fma(x3::to_double(a.len), x3::to_double(b.len), -c3));
      }
      const x3::F3 t = x3::prod(x3::sum(a.inv, b.inv), num);
      const double den = r3_sq + V.c2(l);
      const int hd = __double2hiint(den);
      double c4;
      if (hd >= ((1023 - 59) << 20) && hd < ((1023 + 59) << 20))
        c4 = x3::to_double(x3::quotient(t, den));
      else
        c4 = x3::to_double(t) * rcp_newton(den);
      ux = fma(c4, r3x, ux);
      uy = fma(c4, r3y, uy);
      uz = fma(c4, r3z, uz);
    }
    if (kChain) a = b;
  }
  if (general) {
    double g[3] = {0.0, 0.0, 0.0};
    int gc[4] = {0, 0, 0, 0};
    rare(g, gc);
    vx += g[0];
    vy += g[1];
    vz += g[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) cnt[k] += gc[k];
    return;
  }
  cnt[1] += on_start;
  cnt[2] += on_end;
  cnt[3] += on_line;
  const double half = V.half_c1();
  vx = fma(half, ux, vx);
  vy = fma(half, uy, vy);
  vz = fma(half, uz, vz);
}

}  // namespace seg
}  // namespace fvx
