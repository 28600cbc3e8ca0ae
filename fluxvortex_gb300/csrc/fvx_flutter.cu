// fvx_flutter.cu -- batched aeroelastic flutter sweep: one persistent CTA per
// environment (airspeed) runs the coupled UVLM + beam time history.
//
// Per step, all in the CTA (FP64 unless noted):
//   deform the base vertex grid by the beam's heave/twist (linear span
//   interpolation, rotation about the elastic axis) and take the vertex
//   velocities from the beam velocities; build the ring lattice (quarter-
//   chord rings, 3/4-chord collocation points, normals, areas, bound legs);
//   AIC[i][j] = (unit ring j at collocation i) . n_i; wake ring rows and the
//   particle wake induced at the 2P points (collocation + bound-leg centres),
//   in FP64 or -- mixed precision -- in FP32 on FP64 offsets with compensated
//   particle sums (particles staged through shared memory, split over thread
//   slices, slices reduced in fixed order); the
//   right-hand side; an LU solve with partial pivoting (first largest
//   pivot, as LAPACK's getrf); Kutta-Joukowski forces on the bound
//   legs with the full induced velocity and the unsteady term; station lift
//   and torque about the elastic axis distributed to the beam nodes; the
//   Newmark average-acceleration step with the precomputed inverse of the
//   effective stiffness; the tip history; the wake update (convect with the
//   freestream, shed the trailing-edge row at the new geometry, convert the
//   row past n_keep into 4 particles per ring, FIFO-capped particle store).
// The FP64 pipe bounds a step (1.7 operations per clock and SM), so the step's
// serial parts are spread over the warps and the mixed-precision sums keep off
// it (diff_f32) -- all bit for bit the sums they were, since the FP32 ring law
// amplifies a rounding difference anywhere upstream.  64 airspeeds, 20 chords,
// mixed precision: 104.3 ms with the loads' bound rings on one warp, both CTAs
// forming the whole AIC, one thread searching the pivots and converting rows,
// and eleven FP64 operations and conversions per particle; 31.1 ms so.
// Reference: src/fluxvortex/aeroelastic_solver.py:68-221 and beam_fe.py:231-351
// around PteraSoftware's ring-vortex UVLM; the PteraSoftware-free model is
// described in fluxvortex_gb300/flutter.py.
#include <cooperative_groups.h>

#include "fvx_common.cuh"
#include "fvx_pair_math.cuh"
#include "fvx_parts.cuh"
#include "fvx_segment_math.cuh"

namespace fvx {
namespace flutter {

constexpr int kMaxP = 64;       // panels per environment
constexpr int kMaxNV = 128;     // vertices
constexpr int kMaxRows = 16;    // n_keep + 1 wake ring rows
constexpr int kMaxNS = 16;      // spanwise panels
constexpr int kMaxDof = 48;     // beam DOF (all nodes)
constexpr int kTile = 128;      // particles staged per tile
constexpr double kC = -0.07957747154594767;  // -1/(4 pi): particle strength scaling

constexpr int kLegItems = 256;  // (point, ring) pairs per pass of the loads' leg terms
constexpr int kLegStride = 17;  // doubles per pair: 4 legs of (c4, r3), one of padding

// A wake ring for the mixed-precision sweep: corners in FP64 and in parts
// (split_f32), and the leg constants rounded once here instead of per point.
struct RingF32 {
  double c[4][3];
  Parts p[4][3];
  float c2[4], tol[4];
  float c1;
  int valid;
};

struct Smem {
  double verts[kMaxNV][3], vvel[kMaxNV][3];
  double colloc[kMaxP][3], normal[kMaxP][3], legc[kMaxP][3], legv[kMaxP][3];
  double vcol[kMaxP][3], vleg[kMaxP][3], area[kMaxP];
  seg::VortexRec bound[kMaxP];
  union {  // the wake's rings, FP64 or mixed precision
    seg::VortexRec wake[kMaxRows * kMaxNS];
    RingF32 wakef[kMaxRows * kMaxNS];
  };
  double A[kMaxP][kMaxP + 1];  // AIC; the right-hand side is column P of the LU
  double rhs[kMaxP], gam[kMaxP], gprev[kMaxP];
  double Vind[2 * kMaxP][3];
  double Vsum[2 * kMaxP][3];  // cluster form: both CTAs' partial inductions summed
  double Vbound[kMaxP][3];    // bound rings at the bound-leg centres
  double W[kMaxRows + 1][kMaxNS + 1][3];
  double wgam[kMaxRows][kMaxNS], wage[kMaxRows];
  double d[kMaxDof], v[kMaxDof], a[kMaxDof], F[kMaxDof], feff[kMaxDof], gd[kMaxDof];
  // two tiles of staged particles: x y z | a' (C-scaled) | sigma^2, 2.5 sigma^2
  double tile[2 * kTile][8];
  // mixed precision: the parts of x y z with sigma^2 and 2.5 sigma^2, and a'
  __align__(16) float tile_h[2 * kTile][4], tile_l[2 * kTile][4], tile_r[2 * kTile][4],
      tile_a[2 * kTile][4];
  double newmark[6];  // a0 .. a5 of the Newmark step
  double legs[kLegItems * kLegStride];
  double udiag_inv[kMaxP];  // reciprocals of U's diagonal
  int perm[kMaxP];
  int lu_ok;
  double red[8];
};

static_assert(sizeof(Smem) <= 227 * 1024, "the environment's state must fit shared memory");

// Deformed vertices and their velocities from the beam state in S.d / S.v.
__device__ void deform(Smem& S, const FlutterParams& p) {
  const int nv = (p.nc + 1) * (p.ns + 1);
  for (int k = threadIdx.x; k < nv; k += blockDim.x) {
    const int n = p.vert_node[k];
    const double xi = p.vert_xi[k];
    const double w = S.d[3 * n] * (1.0 - xi) + S.d[3 * (n + 1)] * xi;
    const double th = S.d[3 * n + 2] * (1.0 - xi) + S.d[3 * (n + 1) + 2] * xi;
    const double wd = S.v[3 * n] * (1.0 - xi) + S.v[3 * (n + 1)] * xi;
    const double thd = S.v[3 * n + 2] * (1.0 - xi) + S.v[3 * (n + 1) + 2] * xi;
    const double* b = p.base_verts + 3 * k;
    const double xr = b[0] - p.x_ea;
    const double s = sin(th), c = cos(th);
    S.verts[k][0] = p.x_ea + xr * c;
    S.verts[k][1] = b[1];
    S.verts[k][2] = b[2] + w - xr * s;
    S.vvel[k][0] = -xr * s * thd;
    S.vvel[k][1] = 0.0;
    S.vvel[k][2] = wd - xr * c * thd;
  }
}

// quarter-chord point of vertex column j at chordwise station i (0..nc)
__device__ __forceinline__ void quarter(const double (*V)[3], int nc, int ns, int i, int j,
                                        double* q) {
  const int s1 = ns + 1;
  const double* a = V[i * s1 + j];
  if (i < nc) {
    const double* b = V[(i + 1) * s1 + j];
    for (int c = 0; c < 3; ++c) q[c] = a[c] + 0.25 * (b[c] - a[c]);
  } else {
    const double* b = V[(i - 1) * s1 + j];
    for (int c = 0; c < 3; ++c) q[c] = a[c] + 0.25 * (a[c] - b[c]);
  }
}

// (geometry on the first warps, ring records on the next)
__device__ void build_lattice(Smem& S, const FlutterParams& p) {
  const int P = p.nc * p.ns, s1 = p.ns + 1, w = (P + 31) & ~31;
  for (int t = threadIdx.x; t < 2 * w; t += blockDim.x) {
    const int k = t < w ? t : t - w;
    if (k >= P) continue;
    const int i = k / p.ns, j = k % p.ns;
    double fl[3], fr[3];
    quarter(S.verts, p.nc, p.ns, i, j, fl);
    quarter(S.verts, p.nc, p.ns, i, j + 1, fr);
    if (t >= w) {
      double br[3], bl[3];
      quarter(S.verts, p.nc, p.ns, i + 1, j + 1, br);
      quarter(S.verts, p.nc, p.ns, i + 1, j, bl);
      seg::prep_vortex<FVX_LEGS_RING, true>(S.bound[k], br, fr, fl, bl, 1.0, p.rc0, 0.0, p.nu);
      continue;
    }
    double vfl[3], vfr[3];
    quarter(S.vvel, p.nc, p.ns, i, j, vfl);
    quarter(S.vvel, p.nc, p.ns, i, j + 1, vfr);
    const double* v00 = S.verts[i * s1 + j];
    const double* v01 = S.verts[i * s1 + j + 1];
    const double* v10 = S.verts[(i + 1) * s1 + j];
    const double* v11 = S.verts[(i + 1) * s1 + j + 1];
    const double* u00 = S.vvel[i * s1 + j];
    const double* u01 = S.vvel[i * s1 + j + 1];
    const double* u10 = S.vvel[(i + 1) * s1 + j];
    const double* u11 = S.vvel[(i + 1) * s1 + j + 1];
    double d1[3], d2[3];
    for (int c = 0; c < 3; ++c) {
      const double c0 = v00[c] + 0.75 * (v10[c] - v00[c]);
      const double c1 = v01[c] + 0.75 * (v11[c] - v01[c]);
      S.colloc[k][c] = 0.5 * (c0 + c1);
      const double e0 = u00[c] + 0.75 * (u10[c] - u00[c]);
      const double e1 = u01[c] + 0.75 * (u11[c] - u01[c]);
      S.vcol[k][c] = 0.5 * (e0 + e1);
      S.legc[k][c] = 0.5 * (fr[c] + fl[c]);
      S.legv[k][c] = fl[c] - fr[c];
      S.vleg[k][c] = 0.5 * (vfr[c] + vfl[c]);
      d1[c] = v11[c] - v00[c];
      d2[c] = v01[c] - v10[c];
    }
    const double cx = d1[1] * d2[2] - d1[2] * d2[1];
    const double cy = d1[2] * d2[0] - d1[0] * d2[2];
    const double cz = d1[0] * d2[1] - d1[1] * d2[0];
    const double nrm = sqrt(cx * cx + cy * cy + cz * cz);
    S.normal[k][0] = cx / nrm;
    S.normal[k][1] = cy / nrm;
    S.normal[k][2] = cz / nrm;
    S.area[k] = 0.5 * nrm;
  }
}

// The reference's panel deformation (coupling 1; aeroelastic_solver.py:150-221):
// panel k of strip j moves with the heave w and twist th (nose-up) of the
// displacements S.gd interpolated at the strip's collocation span station; its
// corners and ring vertices by dz = w - (x - x_ea) sin th, dx = (x - x_ea)
// (cos th - 1), its collocation point by dz only.  Normal and area from the
// moved corners; no motion velocity.
__device__ __forceinline__ void ref_motion(const FlutterParams& p, const Smem& S, int j,
                                           double& w, double& s, double& c1) {
  const int n = p.station_node[j];
  const double xi = p.station_xi[j];
  w = S.gd[3 * n] * (1.0 - xi) + S.gd[3 * (n + 1)] * xi;
  const double th = S.gd[3 * n + 2] * (1.0 - xi) + S.gd[3 * (n + 1) + 2] * xi;
  s = sin(th);
  c1 = cos(th) - 1.0;
}
__device__ __forceinline__ void ref_move(const FlutterParams& p, double w, double s, double c1,
                                         double* q) {
  const double xr = q[0] - p.x_ea;
  q[0] += xr * c1;
  q[2] += w - xr * s;
}
__device__ void build_lattice_reference(Smem& S, const FlutterParams& p) {
  const int P = p.nc * p.ns, s1 = p.ns + 1;
  const double(*B)[3] = reinterpret_cast<const double(*)[3]>(p.base_verts);
  for (int k = threadIdx.x; k < P; k += blockDim.x) {
    const int i = k / p.ns, j = k % p.ns;
    double w, sn, c1;
    ref_motion(p, S, j, w, sn, c1);
    double fl[3], fr[3], br[3], bl[3], v00[3], v01[3], v10[3], v11[3];
    quarter(B, p.nc, p.ns, i, j, fl);
    quarter(B, p.nc, p.ns, i, j + 1, fr);
    quarter(B, p.nc, p.ns, i + 1, j + 1, br);
    quarter(B, p.nc, p.ns, i + 1, j, bl);
    for (int c = 0; c < 3; ++c) {
      v00[c] = B[i * s1 + j][c];
      v01[c] = B[i * s1 + j + 1][c];
      v10[c] = B[(i + 1) * s1 + j][c];
      v11[c] = B[(i + 1) * s1 + j + 1][c];
      const double c0 = v00[c] + 0.75 * (v10[c] - v00[c]);
      const double c1b = v01[c] + 0.75 * (v11[c] - v01[c]);
      S.colloc[k][c] = 0.5 * (c0 + c1b);
    }
    S.colloc[k][2] += w - (S.colloc[k][0] - p.x_ea) * sn;
    ref_move(p, w, sn, c1, fl);
    ref_move(p, w, sn, c1, fr);
    ref_move(p, w, sn, c1, br);
    ref_move(p, w, sn, c1, bl);
    ref_move(p, w, sn, c1, v00);
    ref_move(p, w, sn, c1, v01);
    ref_move(p, w, sn, c1, v10);
    ref_move(p, w, sn, c1, v11);
    double d1[3], d2[3];
    for (int c = 0; c < 3; ++c) {
      S.vcol[k][c] = 0.0;
      S.vleg[k][c] = 0.0;
      S.legc[k][c] = 0.5 * (fr[c] + fl[c]);
      S.legv[k][c] = fl[c] - fr[c];
      d1[c] = v11[c] - v00[c];
      d2[c] = v01[c] - v10[c];
    }
    const double cx = d1[1] * d2[2] - d1[2] * d2[1];
    const double cy = d1[2] * d2[0] - d1[0] * d2[2];
    const double cz = d1[0] * d2[1] - d1[1] * d2[0];
    const double nrm = sqrt(cx * cx + cy * cy + cz * cz);
    S.normal[k][0] = cx / nrm;
    S.normal[k][1] = cy / nrm;
    S.normal[k][2] = cz / nrm;
    S.area[k] = 0.5 * nrm;
    seg::prep_vortex<FVX_LEGS_RING, true>(S.bound[k], br, fr, fl, bl, 1.0, p.rc0, 0.0, p.nu);
  }
}

// The reference's trailing edge for the wake's new row (coupling 1): the back
// vertices of the last chordwise rings, strip k's back-left one and the last
// strip's back-right one, each moved with its strip's deformation.
__device__ void trailing_edge_reference(const Smem& S, const FlutterParams& p, double* out,
                                        int k) {
  const double(*B)[3] = reinterpret_cast<const double(*)[3]>(p.base_verts);
  const int j = k < p.ns ? k : p.ns - 1;
  double w, sn, c1;
  ref_motion(p, S, j, w, sn, c1);
  quarter(B, p.nc, p.ns, p.nc, k, out);
  ref_move(p, w, sn, c1, out);
}

// The mixed-precision record of a wake ring (prep_vortex's constants, rounded).
__device__ __forceinline__ void prep_ring_f32(RingF32& Q, const double* br, const double* fr,
                                              const double* fl, const double* bl, double strength,
                                              double rc0, double age, double nu) {
  seg::VortexRec R;
  seg::prep_vortex<FVX_LEGS_RING, true>(R, br, fr, fl, bl, strength, rc0, age, nu);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      Q.c[c][k] = R.c[c][k];
      Q.p[c][k] = split_f32(R.c[c][k]);
    }
    Q.c2[c] = static_cast<float>(R.c2[c]);
    Q.tol[c] = static_cast<float>(R.tol[c]);
  }
  Q.c1 = static_cast<float>(R.c1);
  Q.valid = R.valid;
}

// A target point of the wake induction, in FP64 and in parts.
struct Point {
  double p[3];
  Parts s[3];
};

// One wake ring at a point in FP32 on the FP64 offsets' floats (the
// ring-vortex formula and skip tests of seg::vortex_legs, ring leg set).
__device__ __forceinline__ void ring_velocity_f32(const RingF32& R, const Point& P, float& vx,
                                                  float& vy, float& vz) {
  float d[4][3], len[4];
  bool same = true;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      d[c][k] = diff_f32(R.p[c][k], P.s[k], same);
  if (!same) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int k = 0; k < 3; ++k) d[c][k] = static_cast<float>(R.c[c][k] - P.p[k]);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
    len[c] = sqrtf(d[c][0] * d[c][0] + d[c][1] * d[c][1] + d[c][2] * d[c][2]);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int a = l, b = (l + 1) & 3;
    if (!((R.valid >> l) & 1)) continue;
    const float tol = R.tol[l];
    if (len[a] < tol || len[b] < tol) continue;
    const float r3x = d[a][1] * d[b][2] - d[a][2] * d[b][1];
    const float r3y = d[a][2] * d[b][0] - d[a][0] * d[b][2];
    const float r3z = d[a][0] * d[b][1] - d[a][1] * d[b][0];
    const float r3_sq = r3x * r3x + r3y * r3y + r3z * r3z;
    const float r1r2 = len[a] * len[b];
    const float thr = 1.0e-10f * r1r2;
    if (r3_sq < 2.f * thr * thr && sqrtf(r3_sq) < thr) continue;
    const float c3 = d[a][0] * d[b][0] + d[a][1] * d[b][1] + d[a][2] * d[b][2];
    const float c4 = R.c1 * (len[a] + len[b]) * (r1r2 - c3) / (r1r2 * (r3_sq + R.c2[l]));
    vx += c4 * r3x;
    vy += c4 * r3y;
    vz += c4 * r3z;
  }
}

// Induced velocity of the wake rings and particles at the 2P points
// (collocation points, then bound-leg centres) into S.Vind.
// CL > 1: the environment runs on a cluster of CL CTAs; CTA `crank` takes
// every CL-th ring (by slice) and every CL-th particle tile, and the partial
// inductions are summed in rank order through distributed shared memory, so
// both CTAs hold the same total.
template <bool F32, int CL>
__device__ void wake_induction(Smem& S, const FlutterParams& p, const FlutterState& st, int env,
                               int R, int head, int count, int crank) {
  const int P = p.nc * p.ns, T2 = 2 * P;
  const int slices = blockDim.x / T2;
  const int tgt = threadIdx.x % T2, sl = threadIdx.x / T2;
  const bool active = sl < slices;
  double px = 0.0, py = 0.0, pz = 0.0;
  Point pt = {};
  if (active) {
    const double* q = tgt < P ? S.colloc[tgt] : S.legc[tgt - P];
    px = q[0];
    py = q[1];
    pz = q[2];
    if constexpr (F32) {
      for (int k = 0; k < 3; ++k) {
        pt.p[k] = q[k];
        pt.s[k] = split_f32(q[k]);
      }
    }
  }
  // wake rings: slice sl takes rings sl, sl + slices, ...
  double vx = 0.0, vy = 0.0, vz = 0.0;
  int cnt[4] = {0, 0, 0, 0};
  if (active) {
    if constexpr (F32) {
      float fx = 0.f, fy = 0.f, fz = 0.f;
      for (int r = sl + crank * slices; r < R * p.ns; r += slices * CL)
        ring_velocity_f32(S.wakef[r], pt, fx, fy, fz);
      vx = fx;
      vy = fy;
      vz = fz;
    } else {
      for (int r = sl + crank * slices; r < R * p.ns; r += slices * CL)
        seg::vortex_velocity_general<FVX_LEGS_RING, true>(S.wake[r], px, py, pz, vx, vy, vz, cnt);
    }
  }
  // particles, staged in tiles, oldest first
  const int Pm = p.max_particles;
  const double* pp = st.ppos + static_cast<int64_t>(env) * Pm * 3;
  const double* pa = st.palp + static_cast<int64_t>(env) * Pm * 3;
  const double* ps = st.psig + static_cast<int64_t>(env) * Pm;
  float hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  // this CTA's tiles, two at a time: a thread per particle stages them
  for (int t0 = crank * kTile; t0 < count; t0 += 2 * kTile * CL) {
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * kTile; e += blockDim.x) {
      const int at = t0 + (e / kTile) * kTile * CL + e % kTile;
      if (at >= count) continue;
      const int q = (head + at) % Pm;
      const double s = ps[q];
      S.tile[e][0] = pp[3 * q];
      S.tile[e][1] = pp[3 * q + 1];
      S.tile[e][2] = pp[3 * q + 2];
      if constexpr (F32) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const Parts w = split_f32(S.tile[e][k]);
          S.tile_h[e][k] = w.h;
          S.tile_l[e][k] = w.l;
          S.tile_r[e][k] = w.r;
          S.tile_a[e][k] = static_cast<float>(kC * pa[3 * q + k]);
        }
        S.tile_h[e][3] = static_cast<float>(s * s);
        S.tile_l[e][3] = static_cast<float>(2.5 * s * s);
      } else {
        S.tile[e][3] = kC * pa[3 * q];
        S.tile[e][4] = kC * pa[3 * q + 1];
        S.tile[e][5] = kC * pa[3 * q + 2];
        S.tile[e][6] = s * s;
        S.tile[e][7] = 2.5 * s * s;
      }
    }
    __syncthreads();
    if (!active) continue;
    for (int h = 0; h < 2; ++h) {
      const int nt = min(kTile, count - t0 - h * kTile * CL);
      const int e1 = h * kTile + nt;
      if constexpr (F32) {
        // FP32 pair arithmetic on the FP64 offset's float, compensated sums;
        // two particles side by side (two warps per quarter leave a single
        // particle's chain exposed), added in order
        for (int e = h * kTile + sl; e < e1; e += 2 * slices) {
          const int pair_n = e + slices < e1 ? 2 : 1;
          float d[2][3], s2[2], k2[2], al[2][3], u[2][3];
          bool same = true;
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const int em = m < pair_n ? e + m * slices : e;
            const float4 sh = *reinterpret_cast<const float4*>(S.tile_h[em]);
            const float4 so = *reinterpret_cast<const float4*>(S.tile_l[em]);
            const float4 sr = *reinterpret_cast<const float4*>(S.tile_r[em]);
            const float4 av = *reinterpret_cast<const float4*>(S.tile_a[em]);
            d[m][0] = diff_f32(pt.s[0], Parts{sh.x, so.x, sr.x}, same);
            d[m][1] = diff_f32(pt.s[1], Parts{sh.y, so.y, sr.y}, same);
            d[m][2] = diff_f32(pt.s[2], Parts{sh.z, so.z, sr.z}, same);
            s2[m] = sh.w;
            k2[m] = so.w;
            al[m][0] = av.x;
            al[m][1] = av.y;
            al[m][2] = av.z;
          }
          if (!same) {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              const double* s = S.tile[m < pair_n ? e + m * slices : e];
#pragma unroll
              for (int c = 0; c < 3; ++c) d[m][c] = static_cast<float>(pt.p[c] - s[c]);
            }
          }
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const float r2 = d[m][0] * d[m][0] + d[m][1] * d[m][1] + d[m][2] * d[m][2];
            float f, fpr;
            pair::core_f32<FVX_KERNEL_WINCKELMANS, false>(r2, s2[m], k2[m], f, fpr);
            const float ex = f * d[m][0], ey = f * d[m][1], ez = f * d[m][2];
            u[m][0] = ey * al[m][2] - ez * al[m][1];
            u[m][1] = ez * al[m][0] - ex * al[m][2];
            u[m][2] = ex * al[m][1] - ey * al[m][0];
          }
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            if (m >= pair_n) break;
            float t = hx + u[m][0];
            lx += (hx - t) + u[m][0];
            hx = t;
            t = hy + u[m][1];
            ly += (hy - t) + u[m][1];
            hy = t;
            t = hz + u[m][2];
            lz += (hz - t) + u[m][2];
            hz = t;
          }
        }
      } else {
        for (int e = h * kTile + sl; e < e1; e += slices) {
          const double* s = S.tile[e];
          const double dx = px - s[0], dy = py - s[1], dz = pz - s[2];
          const double r2 = dx * dx + dy * dy + dz * dz;
          double f, fpr;
          pair::core_f64<FVX_KERNEL_WINCKELMANS, false>(r2, s[6], s[7], f, fpr);
          const double ex = f * dx, ey = f * dy, ez = f * dz;
          vx += ey * s[5] - ez * s[4];
          vy += ez * s[3] - ex * s[5];
          vz += ex * s[4] - ey * s[3];
        }
      }
    }
  }
  if constexpr (F32) {
    vx += static_cast<double>(hx) + static_cast<double>(lx);
    vy += static_cast<double>(hy) + static_cast<double>(ly);
    vz += static_cast<double>(hz) + static_cast<double>(lz);
  }
  // slice partials -> fixed-order sum: reuse A's storage as scratch
  __syncthreads();
  double* part = &S.A[0][0];  // needs slices * 2P * 3 <= kMaxP * (kMaxP + 1)
  if (active) {
    part[(sl * T2 + tgt) * 3 + 0] = vx;
    part[(sl * T2 + tgt) * 3 + 1] = vy;
    part[(sl * T2 + tgt) * 3 + 2] = vz;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < T2; k += blockDim.x) {
    double x = 0.0, y = 0.0, z = 0.0;
    for (int s2 = 0; s2 < slices; ++s2) {
      x += part[(s2 * T2 + k) * 3 + 0];
      y += part[(s2 * T2 + k) * 3 + 1];
      z += part[(s2 * T2 + k) * 3 + 2];
    }
    S.Vind[k][0] = x;
    S.Vind[k][1] = y;
    S.Vind[k][2] = z;
  }
  __syncthreads();
  if constexpr (CL > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();  // every CTA's partial is complete
    for (int k = threadIdx.x; k < T2; k += blockDim.x) {
      double x = 0.0, y = 0.0, z = 0.0;
      for (int r = 0; r < CL; ++r) {
        const double(*V)[3] = r == crank ? S.Vind : cl.map_shared_rank(S.Vind, r);
        x += V[k][0];
        y += V[k][1];
        z += V[k][2];
      }
      S.Vsum[k][0] = x;
      S.Vsum[k][1] = y;
      S.Vsum[k][2] = z;
    }
    cl.sync();  // every CTA has read the others' partials
    for (int k = threadIdx.x; k < T2; k += blockDim.x)
      for (int c = 0; c < 3; ++c) S.Vind[k][c] = S.Vsum[k][c];
    __syncthreads();
  }
}

// LU solve of S.A x = S.rhs into S.gam (partial pivoting, first largest
// |pivot|).  Four warps (one per SM quarter's FP64 pipe) eliminate the rows
// under each pivot, the right-hand side being column P; every warp finds the
// pivot itself, by integer comparisons of the magnitudes' words, and rows are
// permuted by index, so a step costs one barrier.  The chain of a step is
// pivot search, reciprocal, one multiplier per row, one FMA per element.
constexpr int kLuWarps = 4;

__device__ bool lu_solve(Smem& S, int P) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < P; i += blockDim.x) S.A[i][P] = S.rhs[i];
  __syncthreads();
  const int nw = min(kLuWarps, static_cast<int>(blockDim.x) >> 5);
  if (warp < nw) {
    int p0 = lane, p1 = lane + 32;  // physical rows of logical rows lane, lane + 32
    bool ok = true;
    for (int k = 0; k < P; ++k) {
      // |A[i][k]| as (hi, lo) words; rows above k and NaNs count as zero
      unsigned h0 = 0, l0 = 0, h1 = 0, l1 = 0;
      bool nan_diag = false;
      if (lane >= k && lane < P) {
        const double v = S.A[p0][k];
        h0 = __double2hiint(v) & 0x7fffffff;
        l0 = __double2loint(v);
        if (v != v) {
          nan_diag = lane == k;
          h0 = l0 = 0;
        }
      }
      if (lane + 32 >= k && lane + 32 < P) {
        const double v = S.A[p1][k];
        h1 = __double2hiint(v) & 0x7fffffff;
        l1 = __double2loint(v);
        if (v != v) {
          nan_diag = nan_diag || lane + 32 == k;
          h1 = l1 = 0;
        }
      }
      const unsigned hm = __reduce_max_sync(0xffffffffu, max(h0, h1));
      const unsigned c0 = h0 == hm ? l0 : 0u, c1 = h1 == hm ? l1 : 0u;
      const unsigned lm = __reduce_max_sync(0xffffffffu, max(c0, c1));
      if (__any_sync(0xffffffffu, nan_diag) || (hm | lm) == 0) {
        ok = false;
        break;
      }
      const unsigned b0 =
          __ballot_sync(0xffffffffu, lane >= k && lane < P && h0 == hm && l0 == lm);
      const unsigned b1 =
          __ballot_sync(0xffffffffu, lane + 32 >= k && lane + 32 < P && h1 == hm && l1 == lm);
      const int piv = b0 ? __ffs(b0) - 1 : 31 + __ffs(b1);
      // swap logical rows k and piv
      const int pk = __shfl_sync(0xffffffffu, k < 32 ? p0 : p1, k & 31);
      const int pp = __shfl_sync(0xffffffffu, piv < 32 ? p0 : p1, piv & 31);
      if (lane == k) p0 = pp;
      if (lane + 32 == k) p1 = pp;
      if (piv != k) {
        if (lane == piv) p0 = pk;
        if (lane + 32 == piv) p1 = pk;
      }
      const double inv = 1.0 / S.A[pp][k];
      // this lane's rows' multipliers; the warp's rows take them by shuffles
      double m0 = 0.0, m1 = 0.0;
      if (lane > k && lane < P) m0 = S.A[p0][k] * inv;
      if (lane + 32 > k && lane + 32 < P) m1 = S.A[p1][k] * inv;
      // columns k + 1 .. P (P: the right-hand side)
      const int j0 = k + 1 + lane, j1 = j0 + 32, j2 = j1 + 32;
      const double u0 = j0 <= P ? S.A[pp][j0] : 0.0;
      const double u1 = j1 <= P ? S.A[pp][j1] : 0.0;
      const double u2 = j2 <= P ? S.A[pp][j2] : 0.0;
      // four rows at a time, loads first: a row's store would hold up the next
      // row's loads
      for (int i0 = k + 1 + warp; i0 < P; i0 += 4 * nw) {
        double l[4], a0[4], a1[4], a2[4];
        double* row[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const int i = min(i0 + m * nw, P - 1);
          l[m] = __shfl_sync(0xffffffffu, i < 32 ? m0 : m1, i & 31);
          row[m] = S.A[__shfl_sync(0xffffffffu, i < 32 ? p0 : p1, i & 31)];
          a0[m] = j0 <= P ? row[m][j0] : 0.0;
          a1[m] = j1 <= P ? row[m][j1] : 0.0;
          a2[m] = j2 <= P ? row[m][j2] : 0.0;
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (i0 + m * nw >= P) break;
          if (j0 <= P) row[m][j0] = a0[m] - l[m] * u0;
          if (j1 <= P) row[m][j1] = a1[m] - l[m] * u1;
          if (j2 <= P) row[m][j2] = a2[m] - l[m] * u2;
        }
      }
      asm volatile("bar.sync 1, %0;" ::"r"(32 * nw) : "memory");
    }
    if (warp == 0) {
      if (lane < P) S.perm[lane] = p0;
      if (lane + 32 < P) S.perm[lane + 32] = p1;
      if (lane == 0) S.lu_ok = ok;
      __syncwarp();
      // back substitution, each row's terms in order: one thread's chain.  The
      // diagonals' correctly rounded reciprocals are formed side by side first;
      // q = s r and one step q + (s - q d) r is then the correctly rounded s / d
      // (Markstein, 1990), at a third of a division's latency.
      if (lane < P) S.udiag_inv[lane] = 1.0 / S.A[p0][lane];
      if (lane + 32 < P) S.udiag_inv[lane + 32] = 1.0 / S.A[p1][lane + 32];
      __syncwarp();
      if (ok && lane == 0) {
        for (int i = P - 1; i >= 0; --i) {
          const double* row = S.A[S.perm[i]];
          double s = row[P];
          const double diag = row[i], r = S.udiag_inv[i];
#pragma unroll 4
          for (int j = i + 1; j < P; ++j) s -= row[j] * S.gam[j];
          const double q = s * r;
          const double rem = fma(-q, diag, s);
          // (a quotient or remainder at the ends of the range: the division)
          const int h = __double2hiint(q) & 0x7ff00000;
          S.gam[i] = h > (200 << 20) && h < (1800 << 20) && fabs(diag) < 1e200 && fabs(diag) > 1e-200
                         ? fma(rem, r, q)
                         : s / diag;
        }
      }
    }
  }
  __syncthreads();
  return S.lu_ok != 0;
}

// CL CTAs per environment (a cluster, launched with that cluster size): they
// share the wake induction (wake_induction), the AIC's rows and the loads'
// points, through distributed shared memory, and run the rest of the step
// redundantly; rank 0 alone writes the environment's global state, and a
// cluster barrier at the start of every step makes its particle writes of
// the last step visible to the others.
template <bool F32, int CL>
__global__ void __launch_bounds__(512) sweep_kernel(FlutterParams p, FlutterState st, int step_end) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  int crank = 0;
  if constexpr (CL > 1) crank = static_cast<int>(cooperative_groups::this_cluster().block_rank());
  const bool writer = crank == 0;
  const int env = blockIdx.x / CL;
  const int P = p.nc * p.ns, s1 = p.ns + 1, ndof = 3 * p.nnodes, nf = ndof - 3;
  const int last = min(step_end, p.n_steps[env]);
  int step = st.step[env];
  if (step >= last) return;
  const double ux = p.u_inf[3 * env], uy = p.u_inf[3 * env + 1], uz = p.u_inf[3 * env + 2];
  const double dt = p.dt;
  // load state
  const bool ref = p.coupling == 1;
  for (int k = threadIdx.x; k < ndof; k += blockDim.x) {
    S.d[k] = st.d[env * ndof + k];
    S.v[k] = st.v[env * ndof + k];
    S.a[k] = st.a[env * ndof + k];
    S.gd[k] = ref ? st.gd[env * ndof + k] : 0.0;
  }
  int R = st.nrows[env];
  for (int k = threadIdx.x; k < (R + 1) * s1 * 3; k += blockDim.x)
    (&S.W[0][0][0])[(k / (s1 * 3)) * (kMaxNS + 1) * 3 + k % (s1 * 3)] =
        st.W[(static_cast<int64_t>(env) * (p.n_keep + 2)) * s1 * 3 + k];
  for (int k = threadIdx.x; k < R * p.ns; k += blockDim.x)
    S.wgam[k / p.ns][k % p.ns] = st.wgam[env * (p.n_keep + 1) * p.ns + k];
  for (int k = threadIdx.x; k < R; k += blockDim.x) S.wage[k] = st.wage[env * (p.n_keep + 1) + k];
  for (int k = threadIdx.x; k < P; k += blockDim.x) S.gprev[k] = st.gprev[env * P + k];
  if (threadIdx.x == 0) {
    const double b = p.beta, g = p.gamma;
    S.newmark[0] = 1.0 / (b * dt * dt);
    S.newmark[1] = 1.0 / (b * dt);
    S.newmark[2] = 1.0 / (2.0 * b) - 1.0;
    S.newmark[3] = g / (b * dt);
    S.newmark[4] = g / b - 1.0;
    S.newmark[5] = dt * (g / (2.0 * b) - 1.0);
  }
  int has_prev = st.has_prev[env];
  int head = st.phead[env], count = st.pcount[env];
  __syncthreads();
  bool ok = true, first = true;
  for (; step < last && ok; ++step) {
    if constexpr (CL > 1) {
      __threadfence();
      cooperative_groups::this_cluster().sync();  // rank 0's particle writes visible
    }
    // 1. geometry and lattice
    if (ref) {
      build_lattice_reference(S, p);
    } else {
      // the last step's deform already holds this step's vertices
      if (first) deform(S, p);
      first = false;
      __syncthreads();
      build_lattice(S, p);
    }
    // the wake's rings on the threads after the lattice's warps
    const int t0 = (2 * ((P + 31) & ~31)) % blockDim.x;
    for (int k = threadIdx.x >= t0 ? threadIdx.x - t0 : threadIdx.x + blockDim.x - t0;
         k < R * p.ns; k += blockDim.x) {
      const int r = k / p.ns, j = k % p.ns;
      if constexpr (F32)
        prep_ring_f32(S.wakef[k], S.W[r + 1][j + 1], S.W[r][j + 1], S.W[r][j], S.W[r + 1][j],
                      S.wgam[r][j], p.rc0, S.wage[r], p.nu);
      else
        seg::prep_vortex<FVX_LEGS_RING, true>(S.wake[k], S.W[r + 1][j + 1], S.W[r][j + 1],
                                              S.W[r][j], S.W[r + 1][j], S.wgam[r][j], p.rc0,
                                              S.wage[r], p.nu);
    }
    __syncthreads();
    // 2. wake + particles at collocation points and bound-leg centres
    wake_induction<F32, CL>(S, p, st, env, R, head, count, crank);
    // 3. AIC (written after the induction, whose scratch overlaps it) and rhs;
    // each CTA of a cluster takes a share of the rows and stores them in all
    const int rows = (P + CL - 1) / CL, row0 = crank * rows, row1 = min(P, row0 + rows);
    for (int e = threadIdx.x; e < (row1 - row0) * P; e += blockDim.x) {
      const int i = row0 + e / P, j = e % P;
      double vx = 0.0, vy = 0.0, vz = 0.0;
      int cnt[4] = {0, 0, 0, 0};
      seg::vortex_velocity_general<FVX_LEGS_RING, true>(S.bound[j], S.colloc[i][0],
                                                        S.colloc[i][1], S.colloc[i][2], vx, vy,
                                                        vz, cnt);
      const double w = vx * S.normal[i][0] + vy * S.normal[i][1] + vz * S.normal[i][2];
      S.A[i][j] = w;
      if constexpr (CL > 1) {
        for (int r = 0; r < CL; ++r)
          if (r != crank) *cooperative_groups::this_cluster().map_shared_rank(&S.A[i][j], r) = w;
      }
    }
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      const double wx = (ux - S.vcol[i][0]) + S.Vind[i][0];
      const double wy = (uy - S.vcol[i][1]) + S.Vind[i][1];
      const double wz = (uz - S.vcol[i][2]) + S.Vind[i][2];
      S.rhs[i] = -(wx * S.normal[i][0] + wy * S.normal[i][1] + wz * S.normal[i][2]);
    }
    if constexpr (CL > 1)
      cooperative_groups::this_cluster().sync();  // all rows are in place
    else
      __syncthreads();
    // 4. strengths
    if (!lu_solve(S, P)) {
      ok = false;
      break;
    }
    // 5. loads: bound rings with strengths gamma at the bound-leg centres
    for (int k = threadIdx.x; k < P; k += blockDim.x) S.bound[k].c1 = S.gam[k] * seg::kInv4Pi;
    __syncthreads();
    double* Fz = &S.A[0][0];     // P station-force z components (A is free now)
    double* arm = Fz + kMaxP;
    // A pass forms the leg terms of up to kLegItems (point, ring) pairs side by
    // side, then a thread per point and component adds them in ring and leg
    // order; each CTA of a cluster takes the points of its AIC rows.
    {
      const int np = row1 - row0;
      const int per = max(1, kLegItems / max(np, 1));  // rings per pass
      double acc[2] = {0.0, 0.0};  // values 3 point + component: this thread's (at most two)
      for (int jb = 0; jb < P; jb += per) {
        const int nj = min(per, P - jb);
        for (int e = threadIdx.x; e < np * nj; e += blockDim.x) {
          const int k = row0 + e / nj, j = jb + e % nj;
          double* o = S.legs + e * kLegStride;
          seg::vortex_legs<FVX_LEGS_RING, true>(
              S.bound[j], S.legc[k][0], S.legc[k][1], S.legc[k][2],
              [&](int l, double c4, double r3x, double r3y, double r3z) {
                o[4 * l] = c4;
                o[4 * l + 1] = r3x;
                o[4 * l + 2] = r3y;
                o[4 * l + 3] = r3z;
              },
              [&](int l, int) { o[4 * l] = o[4 * l + 1] = o[4 * l + 2] = o[4 * l + 3] = 0.0; });
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int v = threadIdx.x + m * blockDim.x;
          if (v >= 3 * np) continue;
          const double* o = S.legs + (v / 3) * nj * kLegStride;
          for (int j = 0; j < nj; ++j, o += kLegStride)
#pragma unroll
            for (int l = 0; l < 4; ++l) acc[m] = fma(o[4 * l], o[4 * l + 1 + v % 3], acc[m]);
        }
        __syncthreads();
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int v = threadIdx.x + m * blockDim.x;
        if (v >= 3 * np) continue;
        double* o = &S.Vbound[row0][0] + v;
        *o = acc[m];
        if constexpr (CL > 1) {
          for (int r = 0; r < CL; ++r)
            if (r != crank) *cooperative_groups::this_cluster().map_shared_rank(o, r) = acc[m];
        }
      }
      if constexpr (CL > 1)
        cooperative_groups::this_cluster().sync();
      else
        __syncthreads();
    }
    for (int k = threadIdx.x; k < P; k += blockDim.x) {
      const double vx = S.Vbound[k][0], vy = S.Vbound[k][1], vz = S.Vbound[k][2];
      const double Vx = (ux - S.vleg[k][0]) + (S.Vind[P + k][0] + vx);
      const double Vy = (uy - S.vleg[k][1]) + (S.Vind[P + k][1] + vy);
      const double Vz = (uz - S.vleg[k][2]) + (S.Vind[P + k][2] + vz);
      const int i = k / p.ns;
      const double geff = i > 0 ? S.gam[k] - S.gam[k - p.ns] : S.gam[k];
      const double dg = has_prev ? (S.gam[k] - S.gprev[k]) / dt : 0.0;
      const double* l = S.legv[k];
      const double cz = Vx * l[1] - Vy * l[0];
      const double fz = p.rho * geff * cz - p.rho * dg * S.area[k] * S.normal[k][2];
      // physical: torque about the elastic axis with the bound leg's arm;
      // reference: the lift's moment about x = 0 with the collocation
      // point's arm (nose-up: -x_c F_z)
      Fz[k] = fz;
      arm[k] = ref ? -S.colloc[k][0] : p.x_ea - S.legc[k][0];
    }
    __syncthreads();
    // the reference couples from step 1 to the step before the last
    const bool couple = !ref || (step >= 1 && step < p.n_steps[env] - 1);
    // 6. station loads -> nodal forces: lift and torque per station, then each
    // degree of freedom adds its stations' shares in station order
    double* lift = arm + kMaxP;
    double* torque = lift + kMaxNS;
    if (couple && threadIdx.x < p.ns) {
      const int j = threadIdx.x;
      double lf = 0.0, tq = 0.0;
      for (int i = 0; i < p.nc; ++i) lf += Fz[i * p.ns + j];
      for (int i = 0; i < p.nc; ++i) tq += Fz[i * p.ns + j] * arm[i * p.ns + j];
      lift[j] = lf;
      torque[j] = tq;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < ndof && couple; k += blockDim.x) {
      const int n = k / 3, c = k % 3;
      double f = 0.0;
      for (int j = 0; j < p.ns && c != 1; ++j) {
        const double q = c == 0 ? lift[j] : torque[j], xi = p.station_xi[j];
        if (p.station_node[j] == n) f += q * (1.0 - xi);
        if (p.station_node[j] + 1 == n) f += q * xi;
      }
      S.F[k] = f;
    }
    // 7. Newmark: F_eff = F + M (a0 d + a1 v + a2 a) + C (a3 d + a4 v + a5 a)
    const double g = p.gamma;
    const double a0 = S.newmark[0], a1 = S.newmark[1], a2 = S.newmark[2], a3 = S.newmark[3],
                 a4 = S.newmark[4], a5 = S.newmark[5];
    double* xm = torque + kMaxNS;
    double* xc = xm + kMaxDof;
    for (int c = threadIdx.x; c < nf && couple; c += blockDim.x) {
      const double dc = S.d[3 + c], vc = S.v[3 + c], ac = S.a[3 + c];
      xm[c] = a0 * dc + a1 * vc + a2 * ac;
      xc[c] = a3 * dc + a4 * vc + a5 * ac;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nf && couple; r += blockDim.x) {
      double fm = 0.0, fc = 0.0;
      for (int c = 0; c < nf; ++c) {
        fm += p.mr[r * nf + c] * xm[c];
        fc += p.cr[r * nf + c] * xc[c];
      }
      S.feff[r] = S.F[3 + r] + fm + fc;
    }
    __syncthreads();
    double dn = 0.0, an = 0.0, vn = 0.0;
    for (int r = threadIdx.x; r < nf && couple; r += blockDim.x) {
      for (int c = 0; c < nf; ++c) dn += p.kinv[r * nf + c] * S.feff[c];
      const double d0 = S.d[3 + r], v0 = S.v[3 + r], acc0 = S.a[3 + r];
      an = a0 * (dn - d0) - a1 * v0 - a2 * acc0;
      vn = v0 + dt * ((1.0 - g) * acc0 + g * an);
    }
    __syncthreads();
    if (couple && threadIdx.x < nf) {
      S.d[3 + threadIdx.x] = dn;
      S.v[3 + threadIdx.x] = vn;
      S.a[3 + threadIdx.x] = an;
    }
    __syncthreads();
    if (couple && writer && threadIdx.x == 0) {
      const int h = ref ? step - 1 : step;
      st.hist_w[static_cast<int64_t>(env) * p.max_steps + h] = S.d[ndof - 3];
      st.hist_th[static_cast<int64_t>(env) * p.max_steps + h] = S.d[ndof - 1];
    }
    if (couple && writer && st.hist_nodes != nullptr) {
      const int h = ref ? step - 1 : step;
      double* hn = st.hist_nodes + (static_cast<int64_t>(env) * p.max_steps + h) * p.nnodes * 2;
      for (int n = threadIdx.x; n < p.nnodes; n += blockDim.x) {
        hn[2 * n] = S.d[3 * n];
        hn[2 * n + 1] = S.d[3 * n + 2];
      }
    }
    // the coupling's displacements shape the next step (reference)
    if (ref && couple)
      for (int k = threadIdx.x; k < ndof; k += blockDim.x) S.gd[k] = S.d[k];
    // 8. wake: next geometry's trailing edge, convect rows and particles
    if (!ref) deform(S, p);
    __syncthreads();
    const int Pm = p.max_particles;
    double* pp = st.ppos + static_cast<int64_t>(env) * Pm * 3;
    double* pa = st.palp + static_cast<int64_t>(env) * Pm * 3;
    double* ps = st.psig + static_cast<int64_t>(env) * Pm;
    for (int e = threadIdx.x; e < (writer ? count : 0); e += blockDim.x) {
      const int q = (head + e) % Pm;
      pp[3 * q] += ux * dt;
      pp[3 * q + 1] += uy * dt;
      pp[3 * q + 2] += uz * dt;
    }
    // shift rows down by one (new row 0), from the back so nothing is overwritten
    // early: a thread per coordinate of a column, strip or age
    for (int k = threadIdx.x; k < 3 * s1 + p.ns + 1; k += blockDim.x) {
      if (k < 3 * s1) {
        const int j = k / 3, c = k % 3;
        const double step_c = (c == 0 ? ux : (c == 1 ? uy : uz)) * dt;
        for (int r = R; r >= 0; --r) S.W[r + 1][j][c] = S.W[r][j][c] + step_c;
      } else if (k < 3 * s1 + p.ns) {
        const int j = k - 3 * s1;
        for (int r = R - 1; r >= 0; --r) S.wgam[r + 1][j] = S.wgam[r][j];
      } else {
        for (int r = R - 1; r >= 0; --r) S.wage[r + 1] = S.wage[r] + dt;
      }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < s1; k += blockDim.x) {
      if (ref)
        trailing_edge_reference(S, p, S.W[0][k], k);
      else
        quarter(S.verts, p.nc, p.ns, p.nc, k, S.W[0][k]);
    }
    for (int k = threadIdx.x; k < p.ns; k += blockDim.x) S.wgam[0][k] = S.gam[(p.nc - 1) * p.ns + k];
    if (threadIdx.x == 0) S.wage[0] = 0.0;
    ++R;
    __syncthreads();
    // 9. rows >= n_keep -> particles, appended in the reference's order (row,
    // strip, edge): a lane per edge, its place by a count of the edges before
    // it that convert.  Place t of this step goes to slot head + count + t of
    // the ring buffer, full or not: when it is full that slot holds the oldest.
    if (R > p.n_keep) {
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const int edges = (R - p.n_keep) * p.ns * 4;
        int added = 0;
        for (int e0 = 0; e0 < edges; e0 += 32) {
          const int e = e0 + lane;
          const int r = p.n_keep + e / (4 * p.ns), j = (e / 4) % p.ns;
          double a[3] = {}, bb[3] = {}, al[3] = {}, sg = 0.0;
          bool take = false;
          if (e < edges) {
            const double gr = S.wgam[r][j];
            const double* fl = S.W[r][j];
            const double* fr = S.W[r][j + 1];
            const double* bl = S.W[r + 1][j];
            const double* br = S.W[r + 1][j + 1];
            const double* from = (e & 3) == 0 ? fr : ((e & 3) == 1 ? fl : ((e & 3) == 2 ? bl : br));
            const double* to = (e & 3) == 0 ? fl : ((e & 3) == 1 ? bl : ((e & 3) == 2 ? br : fr));
            for (int c = 0; c < 3; ++c) {
              a[c] = from[c];
              bb[c] = to[c];
              al[c] = gr * (bb[c] - a[c]);
            }
            take = !(fabs(gr) < 1e-15) && al[0] * al[0] + al[1] * al[1] + al[2] * al[2] > 1e-30;
            auto dist = [](const double* x, const double* y) {
              const double u = x[0] - y[0], v = x[1] - y[1], w = x[2] - y[2];
              return sqrt(u * u + v * v + w * w);
            };
            sg = 1.3 * 0.25 * (dist(fl, fr) + dist(bl, fl) + dist(br, bl) + dist(fr, br));
          }
          const unsigned m = __ballot_sync(0xffffffffu, take);
          const int place = __popc(m & ((1u << lane) - 1u));
          // (of two places in one slot, Pm apart, the later one stays)
          if (take && writer && place + Pm >= __popc(m)) {
            const int q = (head + (count + added + place) % Pm) % Pm;
            for (int c = 0; c < 3; ++c) {
              pp[3 * q + c] = 0.5 * (a[c] + bb[c]);
              pa[3 * q + c] = al[c];
            }
            ps[q] = sg;
          }
          added += __popc(m);
          __syncwarp();
        }
        if (lane == 0) {
          const int over = max(0, count + added - Pm);
          S.red[0] = static_cast<double>((head + over) % Pm);
          S.red[1] = static_cast<double>(count + added - over);
        }
      }
      R = p.n_keep;
      __syncthreads();
      head = static_cast<int>(S.red[0]);
      count = static_cast<int>(S.red[1]);
    }
    for (int k = threadIdx.x; k < P; k += blockDim.x) S.gprev[k] = S.gam[k];
    has_prev = 1;
    __syncthreads();
  }
  if (!ok) {
    if (threadIdx.x == 0) flag_status(kStatusNonFinite);
  }
  // store state (rank 0)
  if (!writer) return;
  for (int k = threadIdx.x; k < ndof; k += blockDim.x) {
    st.d[env * ndof + k] = S.d[k];
    st.v[env * ndof + k] = S.v[k];
    st.a[env * ndof + k] = S.a[k];
    if (ref) st.gd[env * ndof + k] = S.gd[k];
  }
  for (int k = threadIdx.x; k < (R + 1) * s1 * 3; k += blockDim.x)
    st.W[(static_cast<int64_t>(env) * (p.n_keep + 2)) * s1 * 3 + k] =
        (&S.W[0][0][0])[(k / (s1 * 3)) * (kMaxNS + 1) * 3 + k % (s1 * 3)];
  for (int k = threadIdx.x; k < R * p.ns; k += blockDim.x)
    st.wgam[env * (p.n_keep + 1) * p.ns + k] = S.wgam[k / p.ns][k % p.ns];
  for (int k = threadIdx.x; k < R; k += blockDim.x) st.wage[env * (p.n_keep + 1) + k] = S.wage[k];
  for (int k = threadIdx.x; k < P; k += blockDim.x) st.gprev[env * P + k] = S.gprev[k];
  if (threadIdx.x == 0) {
    st.nrows[env] = R;
    st.has_prev[env] = has_prev;
    st.phead[env] = head;
    st.pcount[env] = count;
    st.step[env] = step;
  }
}

}  // namespace flutter
}  // namespace fvx

extern "C" int fvx_flutter_sweep(const FlutterParams* params, const FlutterState* state,
                                 int step_end, int precision, int threads, void* stream) {
  using namespace fvx::flutter;
  FVX_ARG_CHECK(params && state, "null argument");
  const FlutterParams& p = *params;
  const int P = p.nc * p.ns;
  FVX_ARG_CHECK(p.n_env > 0 && p.nc >= 2 && p.ns >= 1 && P <= kMaxP && p.ns <= kMaxNS &&
                    (p.nc + 1) * (p.ns + 1) <= kMaxNV,
                "lattice %d x %d outside the kernel's limits", p.nc, p.ns);
  FVX_ARG_CHECK(p.n_keep >= 1 && p.n_keep + 1 <= kMaxRows, "n_keep %d out of range", p.n_keep);
  FVX_ARG_CHECK(3 * p.nnodes <= kMaxDof && p.nnodes >= 2, "beam too large");
  FVX_ARG_CHECK(p.max_particles >= 1 && p.max_steps >= 1, "bad capacities");
  FVX_ARG_CHECK(precision == FVX_PREC_F64 || precision == FVX_PREC_F32C, "bad precision");
  FVX_ARG_CHECK(p.coupling == 0 || (p.coupling == 1 && state->gd != nullptr),
                "coupling %d unknown (or its displacement array missing)", p.coupling);
  FVX_ARG_CHECK(threads >= 2 * P && threads <= 512 && threads % (2 * P) == 0 && threads % 32 == 0,
                "threads must be a multiple of 2 x panels (and of 32), at most 512");
  FVX_ARG_CHECK((threads / (2 * P)) * 2 * P * 3 <= kMaxP * (kMaxP + 1),
                "too many slices for the reduction scratch");
  const size_t smem = sizeof(Smem);
  // two CTAs per environment (a cluster sharing its wake induction) when the
  // sweep leaves half of the SMs idle with one
  const int cl = 2 * p.n_env <= fvx::device_sm_count() ? 2 : 1;
  static bool attr_done[4] = {false, false, false, false};
  auto launch = [&](auto kernel, int idx) -> int {
    if (!attr_done[idx]) {
      FVX_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(smem)));
      attr_done[idx] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(p.n_env * cl));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cl);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FVX_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, *state, step_end));
    fvx::note_launch();
    return FVX_OK;
  };
  if (cl == 2) {
    if (precision == FVX_PREC_F32C) return launch(sweep_kernel<true, 2>, 3);
    return launch(sweep_kernel<false, 2>, 2);
  }
  if (precision == FVX_PREC_F32C) return launch(sweep_kernel<true, 1>, 1);
  return launch(sweep_kernel<false, 1>, 0);
}
