// fvx_segment_math.cuh -- per-pair arithmetic of the PteraSoftware line
// vortex (Lamb-Oseen + Squire core), shared by the Biot-Savart sweeps
// (fvx_segments.cu) and the panel-method kernels (fvx_uvlm.cu).
//
// The quantities of src/fluxvortex/warp_kernels.py:46-96 with the legs of one
// vortex fused: corner offsets and their lengths are computed once and shared
// by the two legs meeting at a corner, and the per-leg constants are hoisted
// into a VortexRec.
//
// FP64 issue bounds these sweeps: this GPU's FP64 pipe takes 1.7 operations
// per clock and SM, and a square root, a division and a comparison cost it 7.4,
// 7.4 and 1.  The common path therefore avoids all three:
//   * one reciprocal square root per corner (seed instruction plus one cubic
//     Newton step) gives the length |d| = d^2 / |d| and its reciprocal;
//   * c4 = Gamma/4pi (la + lb)(la lb - c3) / (la lb D), D = |r3|^2 + r0^2 rc^2,
//     is (1/la + 1/lb) times la lb - c3 times 1/D (seed plus the Newton
//     step's quadratic form).  Where both ends are at least a leg length away
//     la lb - c3 is (r0^2 - (la - lb)^2) / 2 by the law of cosines: two
//     operations instead of four, and it loses r0 / la digits less to
//     cancellation; nearer, where it would lose more, it is as it stands;
//   * every skip test is first a comparison of the high words, as integers,
//     with a threshold on the safe side; only a pair inside that margin takes
//     the tests themselves.
// About 140 FP64 operations per ring and point against about 300: the AIC of 192
// panels 20.6 us (26.7 with the reference's sequence), of 64 systems 955 us
// (1,370).  The sweeps (fvx_segments.cu) go further and form the scalar parts in
// three floats (fvx_segment_x3.cuh), which pays where a vortex's record serves
// many points.
// Against 113-bit arithmetic (max |error| / max |velocity|) the AIC of 120 panels
// is off by 3.1e-16 (1.8e-15 by the reference's sequence), 400 points of a wake of
// 1,000 rings by 2.4e-16 in three floats (9.4e-15): it was la lb - c3's
// cancellation (tests/test_gpu_ring_precision.py).
#pragma once

#include "fvx_common.cuh"

namespace fvx {
namespace seg {

constexpr double kEps0 = 2.22e-16;           // warp_kernels.py:52
constexpr double kTol = 1.0e-10;             // warp_kernels.py:70,81
constexpr double kFourLamb = 5.02572;        // 4 * 1.25643, warp_kernels.py:88
constexpr double kSquire = 1.0e-4;           // warp_kernels.py:88
constexpr double kInv4Pi = 0.07957747154594767;  // warp_kernels.py:89

template <int LEGS>
struct Legs;
template <>
struct Legs<FVX_LEGS_RING> {
  static constexpr int n = 4;
  __device__ static constexpr int s(int l) { return l; }
  __device__ static constexpr int e(int l) { return (l + 1) & 3; }
};
template <>
struct Legs<FVX_LEGS_CHORDWISE> {
  static constexpr int n = 2;
  __device__ static constexpr int s(int l) { return l == 0 ? 0 : 2; }
  __device__ static constexpr int e(int l) { return l == 0 ? 1 : 3; }
};
template <>
struct Legs<FVX_LEGS_HORSESHOE> {
  static constexpr int n = 3;
  __device__ static constexpr int s(int l) { return l; }
  __device__ static constexpr int e(int l) { return l + 1; }
};

// Hoisted per-vortex record (shared memory, read by broadcast).
struct VortexRec {
  double c[4][3];   // corners BR, FR, FL, BL
  double r0sq[4];   // |end - start|^2 per leg
  double tol[4];    // 1e-10 |end - start| per leg
  double c2[4];     // |end - start|^2 * r_c^2 per leg
  double c1;        // Gamma / (4 pi)
  int valid;        // bit l: leg l passes the zero-length test
  int lo;           // corners this near or nearer (high word of d^2): general path
};

__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// 1/sqrt(x) of a normal x: with e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^-1/2, and
// the binomial series to e^2; the seed's |e| < 2^-18 leaves 5/16 e^3 < 2^-55.
__device__ __forceinline__ double rsqrt_newton(double x) {
  const double y = rsqrt_seed(x);
  const double e = fma(-x, y * y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1/x of a normal x: with e = 1 - x y, 1/x = y (1 + e + e^2 + ...); as above.
__device__ __forceinline__ double rcp_newton(double x) {
  const double y = rcp_seed(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// High words of the squared corner distances that the fast path takes: within
// 2^-240 .. 2^240 all of its products are normal numbers.
constexpr int kHiMin = (1023 - 240) << 20, kHiMax = (1023 + 240) << 20, kHiOne = 1023 << 20;
// |r3|^2 < 2^-62 la^2 lb^2 in high words (each within 0.09 of a binary
// logarithm): covers the margin |r3|^2 < 2e-20 la^2 lb^2 = 2^-65.4 la^2 lb^2.
constexpr int kHiLine = -(62 << 20) - kHiOne;
// |d|^2 < 2^-62 r0^2 covers the corner tests' |d|^2 < 1e-20 r0^2 = 2^-66.4 r0^2
constexpr int kHiNear = 62 << 20;
constexpr int kHiC2 = (1023 + 400) << 20;  // core terms beyond 2^400: general path

// TOL: keep the legs' tolerances in the record (for a caller that takes the
// general path throughout); else that path forms them when it needs them.
template <int LEGS, bool TOL = false>
__device__ __forceinline__ void prep_vortex(VortexRec& R, const double* br, const double* fr,
                                            const double* fl, const double* bl, double strength,
                                            double rc0, double age, double nu) {
  const double* cs[4] = {br, fr, fl, bl};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    R.c[c][0] = cs[c][0];
    R.c[c][1] = cs[c][1];
    R.c[c][2] = cs[c][2];
  }
  double rc_sq = rc0 * rc0 + kFourLamb * (nu + kSquire * fabs(strength)) * age;
  R.c1 = strength * kInv4Pi;
  int valid = 0, far = 0;
  bool fast = true;
#pragma unroll
  for (int l = 0; l < Legs<LEGS>::n; ++l) {
    const double* s = cs[Legs<LEGS>::s(l)];
    const double* e = cs[Legs<LEGS>::e(l)];
    double r0x = e[0] - s[0], r0y = e[1] - s[1], r0z = e[2] - s[2];
    double r0_sq = r0x * r0x + r0y * r0y + r0z * r0z;
    R.r0sq[l] = r0_sq;
    R.c2[l] = r0_sq * rc_sq;
    // the zero-length test needs the root itself only near its threshold
    const int h0 = __double2hiint(r0_sq), h2 = __double2hiint(R.c2[l]);
    bool ok = h0 >= kHiMin && h0 < kHiMax;
    if (TOL || !ok || h0 < ((1023 - 100) << 20)) {
      const double r0_len = sqrt(r0_sq);
      if (TOL) R.tol[l] = r0_len * kTol;
      if (!(r0_len < kEps0)) valid |= 1 << l;
    } else {
      valid |= 1 << l;
    }
    fast = fast && ok && h2 >= 0 && h2 < kHiC2;
    far = max(far, h0);
  }
  R.valid = valid;
  // points within a margin of a leg's tolerance of a corner are left to the
  // general path, and so are all points where a leg is degenerate or a
  // constant leaves the fast path's range
  fast = fast && valid == (1 << Legs<LEGS>::n) - 1;
  R.lo = fast ? max(kHiMin, far - kHiNear) : kHiMax;
}

// The legs of one vortex at point p, in order, by the reference's own sequence
// of operations: take(l, c4, r3) for a leg that contributes c4 r3, skip(l, k)
// for one that skip test k leaves out.  The pairs that the fast path leaves
// out take it, and callers that keep the reference's rounding.  The skip tests
// are the reference's; where all distances are within the fast path's range
// (no NaN among them) integer comparisons decide them as far as they can:
// lengths and tolerances are not negative, so their words order them.
template <int LEGS, bool TOL, typename Take, typename Skip>
__device__ __forceinline__ void vortex_legs(const VortexRec& R, double px, double py, double pz,
                                            Take take, Skip skip) {
  double dx[4], dy[4], dz[4], sq[4], len[4];
  int lo = 0x7fffffff, hi = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    dx[c] = R.c[c][0] - px;
    dy[c] = R.c[c][1] - py;
    dz[c] = R.c[c][2] - pz;
    sq[c] = dx[c] * dx[c] + dy[c] * dy[c] + dz[c] * dz[c];
    len[c] = sqrt(sq[c]);
    lo = min(lo, __double2hiint(sq[c]));
    hi = max(hi, __double2hiint(sq[c]));
  }
  const bool in_range = lo >= kHiMin && hi < kHiMax;
  const int valid = R.valid;
#pragma unroll
  for (int l = 0; l < Legs<LEGS>::n; ++l) {
    const int a = Legs<LEGS>::s(l), b = Legs<LEGS>::e(l);
    if (!((valid >> l) & 1)) {
      skip(l, 0);
      continue;
    }
    // without a kept tolerance its root is taken only where a corner may be
    // within it
    const int near = __double2hiint(R.r0sq[l]) - kHiNear;
    if (TOL || !in_range || min(__double2hiint(sq[a]), __double2hiint(sq[b])) <= near) {
      const double tol = TOL ? R.tol[l] : sqrt(R.r0sq[l]) * kTol;
      if (in_range ? __double_as_longlong(len[a]) < __double_as_longlong(tol) : len[a] < tol) {
        skip(l, 1);
        continue;
      }
      if (in_range ? __double_as_longlong(len[b]) < __double_as_longlong(tol) : len[b] < tol) {
        skip(l, 2);
        continue;
      }
    }
    double r3x = dy[a] * dz[b] - dz[a] * dy[b];
    double r3y = dz[a] * dx[b] - dx[a] * dz[b];
    double r3z = dx[a] * dy[b] - dy[a] * dx[b];
    double r3_sq = r3x * r3x + r3y * r3y + r3z * r3z;
    double r1r2 = len[a] * len[b];
    if (!in_range ||
        __double2hiint(r3_sq) < __double2hiint(sq[a]) + (__double2hiint(sq[b]) + kHiLine)) {
      const double thr = kTol * r1r2;
      if (r3_sq < 2.0 * thr * thr && sqrt(r3_sq) < thr) {
        skip(l, 3);
        continue;
      }
    }
    double c3 = dx[a] * dx[b] + dy[a] * dy[b] + dz[a] * dz[b];
    double c4 = R.c1 * (len[a] + len[b]) * (r1r2 - c3) / (r1r2 * (r3_sq + R.c2[l]));
    take(l, c4, r3x, r3y, r3z);
  }
}

// Velocity of one vortex (all legs) at point p; cnt[k] counts skips.
template <int LEGS, bool TOL>
__device__ __forceinline__ void vortex_velocity_general(const VortexRec& R, double px, double py,
                                                        double pz, double& vx, double& vy,
                                                        double& vz, int cnt[4]) {
  vortex_legs<LEGS, TOL>(
      R, px, py, pz,
      [&](int, double c4, double r3x, double r3y, double r3z) {
        vx += c4 * r3x;
        vy += c4 * r3y;
        vz += c4 * r3z;
      },
      [&](int, int k) { cnt[k]++; });
}

template <int LEGS>
__device__ __noinline__ void vortex_velocity_rare(const VortexRec& R, double px, double py,
                                                  double pz, double* v, int* cnt) {
  vortex_velocity_general<LEGS, false>(R, px, py, pz, v[0], v[1], v[2], cnt);
}

// Skip test of a leg whose line the point may lie on (warp_kernels.py:81).
static __device__ __noinline__ bool on_leg_line(double r3_sq, double la_sq, double lb_sq) {
  const double thr = kTol * (sqrt(la_sq) * sqrt(lb_sq));
  return r3_sq < 2.0 * thr * thr && sqrt(r3_sq) < thr;
}

// Skip tests of a point that may lie on corner c (warp_kernels.py:70-74): bit l
// for a leg that starts there, bit 4 + l for one that ends there; -1 where the
// tests of the corner's legs, whose lengths differ, do not agree.
template <int LEGS>
__device__ __noinline__ int on_corner(const VortexRec& R, int c, double sq) {
  int skip = 0, legs = 0;
  for (int l = 0; l < Legs<LEGS>::n; ++l) {
    const int bit = Legs<LEGS>::s(l) == c ? 1 << l : (Legs<LEGS>::e(l) == c ? 16 << l : 0);
    if (bit == 0) continue;
    legs |= bit;
    // below 2^-68 r0^2 < 1e-20 r0^2 (the corner itself, as a rule) no root is needed
    if (__double2hiint(sq) < __double2hiint(R.r0sq[l]) - (68 << 20) ||
        sqrt(sq) < sqrt(R.r0sq[l]) * kTol)
      skip |= bit;
  }
  return skip == 0 || skip == legs ? skip : -1;
}

// As vortex_velocity_general, on the fast path wherever the pair is clear of
// the ends of FP64's range (see above).  Points on a corner stay on it, as a
// free wake's own vertices are targets: all legs that meet there are skipped,
// and the corner's distance, which only they use, is replaced by one.
template <int LEGS>
__device__ __forceinline__ void vortex_velocity(const VortexRec& R, double px, double py,
                                                double pz, double& vx, double& vy, double& vz,
                                                int cnt[4]) {
  double dx[4], dy[4], dz[4], sq[4];
  int lo = 0x7fffffff, hi = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    dx[c] = R.c[c][0] - px;
    dy[c] = R.c[c][1] - py;
    dz[c] = R.c[c][2] - pz;
    sq[c] = dx[c] * dx[c] + dy[c] * dy[c] + dz[c] * dz[c];
    // (a NaN may carry a sign, inf - inf on x86 does: it is above kHiMax either way)
    const int h = __double2hiint(sq[c]) & 0x7fffffff;
    lo = min(lo, h);
    hi = max(hi, h);
  }
  int skip = 0;
  if (lo <= R.lo || hi >= kHiMax) {
    bool general = hi >= kHiMax || R.lo == kHiMax;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (!general && __double2hiint(sq[c]) <= R.lo) {
        const int m = on_corner<LEGS>(R, c, sq[c]);
        general = m < 0 || (m == 0 && __double2hiint(sq[c]) < kHiMin);
        if (m > 0) {
          skip |= m;
          sq[c] = 1.0;
        }
      }
    if (general) {
      double g[3] = {0.0, 0.0, 0.0};
      int gc[4] = {0, 0, 0, 0};
      vortex_velocity_rare<LEGS>(R, px, py, pz, g, gc);
      vx += g[0];
      vy += g[1];
      vz += g[2];
#pragma unroll
      for (int k = 0; k < 4; ++k) cnt[k] += gc[k];
      return;
    }
  }
  double len[4], inv[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    inv[c] = rsqrt_newton(sq[c]);
    len[c] = sq[c] * inv[c];
  }
  double ux = 0.0, uy = 0.0, uz = 0.0;
#pragma unroll
  for (int l = 0; l < Legs<LEGS>::n; ++l) {
    const int a = Legs<LEGS>::s(l), b = Legs<LEGS>::e(l);
    if (skip & (17 << l)) {
      cnt[skip & (1 << l) ? 1 : 2]++;
      continue;
    }
    const double r3x = dy[a] * dz[b] - dz[a] * dy[b];
    const double r3y = dz[a] * dx[b] - dx[a] * dz[b];
    const double r3z = dx[a] * dy[b] - dy[a] * dx[b];
    const double r3_sq = r3x * r3x + r3y * r3y + r3z * r3z;
    if (__double2hiint(r3_sq) < __double2hiint(sq[a]) + (__double2hiint(sq[b]) + kHiLine) &&
        on_leg_line(r3_sq, sq[a], sq[b])) {
      cnt[3]++;
      continue;
    }
    const double gap = len[a] - len[b];
    double num = fma(-gap, gap, R.r0sq[l]);  // 2 (la lb - c3)
    const bool near = min(__double2hiint(sq[a]), __double2hiint(sq[b])) <
                      __double2hiint(R.r0sq[l]);
    // a vote, so that the compiler keeps this a branch: far warps skip it
    if (__any_sync(__activemask(), near)) {
      const double c3 = dx[a] * dx[b] + dy[a] * dy[b] + dz[a] * dz[b];
      if (near) {
        num = fma(len[a], len[b], -c3);
        num = __hiloint2double(__double2hiint(num) + (1 << 20), __double2loint(num));  // doubled
      }
    }
    const double c4 = (inv[a] + inv[b]) * num * rcp_newton(r3_sq + R.c2[l]);
    ux = fma(c4, r3x, ux);
    uy = fma(c4, r3y, uy);
    uz = fma(c4, r3z, uz);
  }
  const double half = 0.5 * R.c1;
  vx = fma(half, ux, vx);
  vy = fma(half, uy, vy);
  vz = fma(half, uz, vz);
}

}  // namespace seg
}  // namespace fvx
