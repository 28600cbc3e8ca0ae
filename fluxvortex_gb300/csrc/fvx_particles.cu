// fvx_particles.cu -- all-pairs vortex-particle sweeps (velocity, stretching,
// velocity gradient, vorticity) with the Winckelmans or Gaussian-erf core.
//
// Replaces src/fluxvortex/kernel.py:69-190 (NumPy, 512 x 512 chunks) and its
// unused Warp ports src/fluxvortex/warp_vpm.py:20-141 (one thread per pair,
// one atomic per pair and component).
//
// Closed forms used (C = -1/(4 pi) folded into alpha on staging; d = x_t - x_s;
// f(r) = g(r/sigma)/r^3 and fpr = f'(r)/r, both finite at r = 0):
//   u      += f (d x a)                                      kernel.py:103-114
//   J_ij   += fpr (d x a)_i d_j + f eps_ijl a_l              kernel.py:156-188
//   S       = J . G_t = f (G_t x a) + fpr (d . G_t)(d x a)   particles.py:148-151
//   omega_i = eps_ijk J_kj = fpr (d (d . a) - a r^2) - 2 f a particles.py:219-225
// Winckelmans: f = (r^2 + 2.5 s^2) q^-5/2, fpr = -(3 r^2 + 10.5 s^2) q^-7/2,
//   q = r^2 + s^2 (kernel.py:42-55 rewritten without r_bar = r/sigma).
// Gaussian-erf: for r/sigma >= 0.5 the kernel.py:16-31 formula; below it the
//   Taylor series of g(r)/r^3 (the reference's erf - c r exp form cancels
//   there and is pure rounding noise at its r = 1e-12 self-pair clamp).
//
// FP64 sweeps (pairs_f64_kernel): the FP64 pipe bounds them, so the scalar core
// of a pair (f, f'/r) is formed in three-float arithmetic on the FP32 pipe
// (fvx_x3.cuh) and only the vector part stays in FP64; tiles with values outside
// that arithmetic's range take the FP64 core (core_f64).
//
// Layout and tiling: a CTA owns 128 (FP64) or 256 (FP32, two per thread) targets
// held in registers.  Source tiles of 128 particles (AoS pos, alpha,
// sigma exactly as the caller stores them) are staged by 1-D TMA bulk copies
// (cp.async.bulk) into a double-buffered raw area, then converted by all
// threads into a compute tile (alpha pre-scaled by C, sigma^2 and the core's
// second constant precomputed; FP32 positions re-centred in FP64 on the first
// of the target's block of 256 or 512 before rounding).  Every thread then sweeps the tile reading
// shared memory by broadcast.  FP32 sums are kept per tile and folded into a
// two-sum (hi, lo) pair per component.  When targets alone cannot fill the
// SMs the source range is split over gridDim.y; partial sums go to scratch
// and a second kernel adds them in fixed order.
#include <cfloat>

#include "fvx_common.cuh"
#include "fvx_core_table.cuh"
#include "fvx_pair_math.cuh"
#include "fvx_x2.cuh"
#include "fvx_x3.cuh"

namespace fvx {
namespace {

using namespace pair;

constexpr int kThreads = 128;
constexpr int kSrcTile = 128;
constexpr double kC = -0.07957747154594767;  // -1/(4 pi)

template <int TILE>
struct RawSrc {
  double pos[TILE * 3];
  double alpha[TILE * 3];
  double sigma[TILE];
};

// Compute tile of the FP32 sweeps: two 4-vectors per source so that a thread
// fetches a source with two 128-bit shared loads and reuses it for all its
// targets.
struct SrcTile {
  float4 p[kSrcTile];  // x, y, z, sigma^2
  float4 a[kSrcTile];  // C*alpha_x, C*alpha_y, C*alpha_z, k2
};

// FP32 sweeps: two targets per thread, the halves of f32x2 registers.  (Four took
// half the shared-memory loads but 96-106 registers and half as many CTAs:
// 32,768 particles 918 us against 841 for the velocity, 1,340 against 1,222 for the
// stretching.)  Blocks of `origin` targets share a re-centring origin.
constexpr int kTargetsF32 = 2 * kThreads;
template <int MODE>
constexpr int kOrigin = kThreads * (ModeInfo<MODE>::ncomp <= 3 ? 4 : 2);

struct PairArgs {
  const double* tgt;
  const double* tgt_gamma;
  int64_t n_tgt;
  const double* pos;
  const double* alpha;
  const double* sigma;
  int64_t n_src;
  int64_t chunk;  // sources per split (even)
  double* out_a;
  double* out_b;
  double* partial;  // (S, M, ncomp) when gridDim.y > 1
  int use_tma;
};

template <int TILE>
__device__ void issue_src(const PairArgs& A, RawSrc<TILE>& raw, int64_t j0, int cnt, uint64_t* bar) {
  BulkPlan pp = plan_bulk(A.pos, j0, cnt, 24, A.use_tma);
  BulkPlan pa = plan_bulk(A.alpha, j0, cnt, 24, A.use_tma);
  BulkPlan ps = plan_bulk(A.sigma, j0, cnt, 8, A.use_tma);
  mbar_arrive_expect_tx(bar, pp.bulk_bytes + pa.bulk_bytes + ps.bulk_bytes);
  if (pp.bulk_bytes) bulk_g2s(raw.pos, A.pos + 3 * j0, pp.bulk_bytes, bar);
  if (pa.bulk_bytes) bulk_g2s(raw.alpha, A.alpha + 3 * j0, pa.bulk_bytes, bar);
  if (ps.bulk_bytes) bulk_g2s(raw.sigma, A.sigma + j0, ps.bulk_bytes, bar);
}

template <int TILE>
__device__ void tail_src(const PairArgs& A, RawSrc<TILE>& raw, int64_t j0, int cnt) {
  BulkPlan p = plan_bulk(A.pos, j0, cnt, 24, A.use_tma);
  if (p.tail_bytes) plain_copy8(raw.pos, A.pos + 3 * j0, p.bulk_bytes, p.tail_bytes);
  p = plan_bulk(A.alpha, j0, cnt, 24, A.use_tma);
  if (p.tail_bytes) plain_copy8(raw.alpha, A.alpha + 3 * j0, p.bulk_bytes, p.tail_bytes);
  p = plan_bulk(A.sigma, j0, cnt, 8, A.use_tma);
  if (p.tail_bytes) plain_copy8(raw.sigma, A.sigma + j0, p.bulk_bytes, p.tail_bytes);
}

template <typename T>
__device__ __forceinline__ void two_sum_fold(T& hi, T& lo, T p) {
  T s = hi + p;
  T bp = s - hi;
  T err = (hi - (s - bp)) + (p - bp);
  hi = s;
  lo += err;
}

// One source against a thread's pair of targets (Winckelmans): core_f32 and
// accumulate in paired arithmetic, each product and sum with the scalar form's
// roundings, so the sums are the scalar loop's bit for bit.  The FP32 pipe bounds
// the loop (25 operations a pair for the velocity, 36 for the stretching); scalar
// instructions fill the issue slots before the pipe (79 % issue, 72 % of the
// pipe), paired ones take half of them.  32,768 particles: velocity
// 1,184 -> 839 us, stretching 1,538 -> 1,197 us (85 % of the pipe).
// NORMAL: q = r^2 + s^2 is a normal number whatever r (core_f32's rsqrtf scales
// its argument in case it is not: three of a pair's forty instructions).
template <int MODE, bool NORMAL>
__device__ __forceinline__ void pair_x2(const float4 pv, const float4 av, const uint64_t (&t)[3],
                                        const uint64_t (&g)[3],
                                        uint64_t (&acc)[ModeInfo<MODE>::ncomp]) {
  const uint64_t a[3] = {x2::dup(av.x), x2::dup(av.y), x2::dup(av.z)};
  const uint64_t na[3] = {x2::dup(-av.x), x2::dup(-av.y), x2::dup(-av.z)};
  const uint64_t s2 = x2::dup(pv.w);
  const uint64_t d[3] = {x2::sub(t[0], x2::dup(pv.x)), x2::sub(t[1], x2::dup(pv.y)),
                         x2::sub(t[2], x2::dup(pv.z))};
  const uint64_t r2 = x2::fma(d[2], d[2], x2::fma(d[0], d[0], x2::mul(d[1], d[1])));
  float qa, qb;
  x2::unpack(x2::add(r2, s2), qa, qb);
  const uint64_t T = NORMAL ? x2::pack(rsqrt_ftz(qa), rsqrt_ftz(qb))
                            : x2::pack(rsqrtf(qa), rsqrtf(qb));
  const uint64_t T2 = x2::mul(T, T);
  const uint64_t T5 = x2::mul(x2::mul(T2, T2), T);
  const uint64_t f = x2::mul(x2::add(r2, x2::dup(av.w)), T5);
  uint64_t fpr = 0;
  if constexpr (ModeInfo<MODE>::need_fpr)
    fpr = x2::mul(
        x2::mul(x2::fma(x2::dup(-10.5f), s2, x2::mul(x2::dup(-3.0f), r2)), T2), T5);
  // (v x a)_c = v_i a_j - v_j a_i, (c, i, j) cyclic
  auto cross = [&](const uint64_t (&v)[3], int c) {
    const int i = (c + 1) % 3, j = (c + 2) % 3;
    return x2::fma(v[i], a[j], x2::mul(v[j], na[i]));
  };
  auto dot = [&](const uint64_t (&v)[3]) {
    return x2::fma(d[2], v[2], x2::fma(d[0], v[0], x2::mul(d[1], v[1])));
  };
  if constexpr (MODE == FVX_PAIR_VELOCITY || MODE == FVX_PAIR_VELOCITY_STRETCH) {
    const uint64_t e[3] = {x2::mul(f, d[0]), x2::mul(f, d[1]), x2::mul(f, d[2])};
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] = x2::add(acc[c], cross(e, c));
  }
  if constexpr (MODE == FVX_PAIR_STRETCH || MODE == FVX_PAIR_VELOCITY_STRETCH) {
    constexpr int o = MODE == FVX_PAIR_STRETCH ? 0 : 3;
    const uint64_t w = x2::mul(fpr, dot(g));
    uint64_t v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = x2::fma(f, g[c], x2::mul(w, d[c]));
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[o + c] = x2::add(acc[o + c], cross(v, c));
  }
  if constexpr (MODE == FVX_PAIR_JACOBIAN) {
    const uint64_t q[3] = {x2::mul(fpr, cross(d, 0)), x2::mul(fpr, cross(d, 1)),
                           x2::mul(fpr, cross(d, 2))};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        uint64_t& o = acc[3 * i + j];
        if (i == j) {
          o = x2::fma(q[i], d[i], o);
        } else {  // + f a_l where (i, j, l) is cyclic, - f a_l otherwise
          const int l = 3 - i - j;
          o = x2::add(o, x2::fma(q[i], d[j], x2::mul(f, (j - i + 3) % 3 == 1 ? a[l] : na[l])));
        }
      }
  }
  if constexpr (MODE == FVX_PAIR_VORTICITY) {
    const uint64_t u = x2::mul(fpr, dot(a));
    const uint64_t v = x2::fma(fpr, r2, x2::add(f, f));
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] = x2::add(acc[c], x2::fma(d[c], u, x2::mul(na[c], v)));
  }
}

// (the stated minimum of one CTA per SM leaves ptxas its registers: 839 and 1,197 us
// at 32,768 particles; 873 and 1,207 with the default's 64)
template <int MODE, int KERNEL>
__global__ void __launch_bounds__(kThreads, 1) pairs_f32_kernel(PairArgs A) {
  using T = float;
  constexpr int TPT = kTargetsF32 / kThreads;  // targets per thread
  constexpr bool PAIRED = KERNEL == FVX_KERNEL_WINCKELMANS;
  constexpr int NC = ModeInfo<MODE>::ncomp;
  constexpr bool NEED_FPR = ModeInfo<MODE>::need_fpr;
  constexpr bool NEED_TG = ModeInfo<MODE>::need_tg;

  __shared__ __align__(128) RawSrc<kSrcTile> raw[2];
  __shared__ __align__(16) SrcTile tile;
  __shared__ __align__(8) uint64_t bar[2];

  const int64_t base = static_cast<int64_t>(blockIdx.x) * kTargetsF32;
  const int64_t ob = base / kOrigin<MODE> * kOrigin<MODE>;
  const double ox = A.tgt[3 * ob + 0], oy = A.tgt[3 * ob + 1], oz = A.tgt[3 * ob + 2];
  T tx[TPT], ty[TPT], tz[TPT], gx[TPT], gy[TPT], gz[TPT];
  bool act[TPT];
#pragma unroll
  for (int j = 0; j < TPT; ++j) {
    const int64_t i = base + threadIdx.x + j * kThreads;
    act[j] = i < A.n_tgt;
    double px = 0, py = 0, pz = 0, qx = 0, qy = 0, qz = 0;
    if (act[j]) {
      px = A.tgt[3 * i + 0] - ox;
      py = A.tgt[3 * i + 1] - oy;
      pz = A.tgt[3 * i + 2] - oz;
      if (NEED_TG) {
        qx = A.tgt_gamma[3 * i + 0];
        qy = A.tgt_gamma[3 * i + 1];
        qz = A.tgt_gamma[3 * i + 2];
      }
    }
    tx[j] = static_cast<T>(px);
    ty[j] = static_cast<T>(py);
    tz[j] = static_cast<T>(pz);
    gx[j] = static_cast<T>(qx);
    gy[j] = static_cast<T>(qy);
    gz[j] = static_cast<T>(qz);
  }

  const int64_t jb = static_cast<int64_t>(blockIdx.y) * A.chunk;
  const int64_t je = min(jb + A.chunk, A.n_src);
  const int ntiles = jb < je ? static_cast<int>((je - jb + kSrcTile - 1) / kSrcTile) : 0;

  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  T hi[TPT][NC], lo[TPT][NC];
#pragma unroll
  for (int j = 0; j < TPT; ++j)
#pragma unroll
    for (int c = 0; c < NC; ++c) hi[j][c] = lo[j][c] = T(0);
  const uint64_t t2[3] = {x2::pack(tx[0], tx[1]), x2::pack(ty[0], ty[1]), x2::pack(tz[0], tz[1])};
  const uint64_t g2[3] = {x2::pack(gx[0], gx[1]), x2::pack(gy[0], gy[1]), x2::pack(gz[0], gz[1])};

  uint32_t phase[2] = {0u, 0u};
  bool ok = true;
  if (ntiles > 0 && threadIdx.x == 0)
    issue_src(A, raw[0], jb, static_cast<int>(min64(kSrcTile, je - jb)), &bar[0]);
  int t = 0;
  for (; t < ntiles; ++t) {
    const int buf = t & 1;
    const int64_t j0 = jb + static_cast<int64_t>(t) * kSrcTile;
    const int n = static_cast<int>(min64(kSrcTile, je - j0));
    if (t + 1 < ntiles && threadIdx.x == 0) {
      const int64_t j1 = j0 + kSrcTile;
      issue_src(A, raw[buf ^ 1], j1, static_cast<int>(min64(kSrcTile, je - j1)),
                &bar[buf ^ 1]);
    }
    const bool got = mbar_wait(&bar[buf], phase[buf]);
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    phase[buf] ^= 1u;
    tail_src(A, raw[buf], j0, n);
    __syncthreads();
    bool subnormal = false;
    for (int k = threadIdx.x; k < n; k += kThreads) {
      const double sg = raw[buf].sigma[k];
      float4 pv, av;
      pv.x = static_cast<T>(raw[buf].pos[3 * k + 0] - ox);
      pv.y = static_cast<T>(raw[buf].pos[3 * k + 1] - oy);
      pv.z = static_cast<T>(raw[buf].pos[3 * k + 2] - oz);
      pv.w = static_cast<T>(sg * sg);
      av.x = static_cast<T>(kC * raw[buf].alpha[3 * k + 0]);
      av.y = static_cast<T>(kC * raw[buf].alpha[3 * k + 1]);
      av.z = static_cast<T>(kC * raw[buf].alpha[3 * k + 2]);
      av.w = static_cast<T>(KERNEL == FVX_KERNEL_WINCKELMANS ? 2.5 * sg * sg : 1.0 / sg);
      tile.p[k] = pv;
      tile.a[k] = av;
      if (PAIRED) subnormal |= !(pv.w >= FLT_MIN);  // (or NaN)
    }
    bool normal = false;
    if constexpr (PAIRED)
      normal = !__syncthreads_or(subnormal);
    else
      __syncthreads();
    T part[TPT][NC];
    if constexpr (PAIRED) {
      uint64_t part2[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) part2[c] = 0ull;
      if (normal) {
#pragma unroll 4
        for (int k = 0; k < n; ++k) pair_x2<MODE, true>(tile.p[k], tile.a[k], t2, g2, part2);
      } else {
#pragma unroll 1
        for (int k = 0; k < n; ++k) pair_x2<MODE, false>(tile.p[k], tile.a[k], t2, g2, part2);
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) x2::unpack(part2[c], part[0][c], part[1][c]);
    } else {
#pragma unroll
      for (int j = 0; j < TPT; ++j)
#pragma unroll
        for (int c = 0; c < NC; ++c) part[j][c] = T(0);
#pragma unroll 2
      for (int k = 0; k < n; ++k) {
        const float4 pv = tile.p[k], av = tile.a[k];
#pragma unroll
        for (int j = 0; j < TPT; ++j) {
          const T dx = tx[j] - pv.x, dy = ty[j] - pv.y, dz = tz[j] - pv.z;
          const T r2 = dx * dx + dy * dy + dz * dz;
          T f, fpr = T(0);
          core_f32<KERNEL, NEED_FPR>(r2, pv.w, av.w, f, fpr);
          accumulate<MODE, T>(part[j], dx, dy, dz, r2, av.x, av.y, av.z, f, fpr, gx[j], gy[j],
                              gz[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < TPT; ++j)
#pragma unroll
      for (int c = 0; c < NC; ++c) two_sum_fold(hi[j][c], lo[j][c], part[j][c]);
    __syncthreads();
  }
  if (!ok) {
    flag_status(kStatusTimeout);
    if (threadIdx.x == 0 && t + 1 < ntiles) mbar_wait(&bar[(t + 1) & 1], phase[(t + 1) & 1]);
    return;
  }
#pragma unroll
  for (int j = 0; j < TPT; ++j) {
    if (!act[j]) continue;
    const int64_t i = base + threadIdx.x + j * kThreads;
    double v[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c)
      v[c] = static_cast<double>(hi[j][c]) + static_cast<double>(lo[j][c]);
    if (gridDim.y > 1) {
      double* o = A.partial + (static_cast<int64_t>(blockIdx.y) * A.n_tgt + i) * NC;
#pragma unroll
      for (int c = 0; c < NC; ++c) o[c] = v[c];
    } else {
      constexpr int NA = ModeInfo<MODE>::na;
#pragma unroll
      for (int c = 0; c < NA; ++c) A.out_a[i * NA + c] = v[c];
#pragma unroll
      for (int c = NA; c < NC; ++c) A.out_b[i * (NC - NA) + (c - NA)] = v[c];
    }
  }
}

// ---- FP64 sweeps ------------------------------------------------------------------
// A staged source: scaled strength in FP64, position and core constants as three
// floats each (96 bytes: six 16-byte broadcast loads).
struct alignas(16) SrcX3 {
  double a[3];
  x3::F3 x[3];
  x3::F3 s2, k, k5;  // x3::Core
};
static_assert(sizeof(SrcX3) == 96, "a source is six 16-byte words");

// Sources per tile: short, so that two CTAs and their copies of the Gaussian
// core's table (88 KB) fit an SM.
constexpr int kSrc64 = 64;

// Dynamic shared memory: raw tiles, compute tile, barriers, and for the
// Gaussian core its polynomials ([interval][F, G or F alone][20]).
struct F64Smem {
  RawSrc<kSrc64> raw[2];
  SrcX3 tile[kSrc64];
  uint64_t bar[2];
  alignas(16) float table[];
};

__device__ const __align__(16) float g_core_table[] = {FVX_CORE_TABLE};
constexpr int kTableRows = x3::kCoreRows + x3::kFarRows;
constexpr int kTableFloats = kTableRows * x3::kRowFloats;  // of F, and of G

// Sums of one pair in FP64 given f and f'/r (and, for the vorticity, iso = f'/r
// r^2 + 2 f): accumulate() with every product fused into its sum.  The
// Jacobian's antisymmetric part goes to acc[9..11] = sum of f a and is put in
// place per tile (fold_tile).
template <int MODE>
struct F64Acc {
  static constexpr int n = MODE == FVX_PAIR_JACOBIAN ? 12 : ModeInfo<MODE>::ncomp;
};
template <int MODE>
__device__ __forceinline__ void accumulate_f64(double* acc, double dx, double dy, double dz,
                                               double ax, double ay, double az, double f,
                                               double fpr, double iso, double gx, double gy,
                                               double gz) {
  auto cross = [&](double* o, double vx, double vy, double vz) {
    o[0] = fma(-vz, ay, fma(vy, az, o[0]));
    o[1] = fma(-vx, az, fma(vz, ax, o[1]));
    o[2] = fma(-vy, ax, fma(vx, ay, o[2]));
  };
  if (MODE == FVX_PAIR_VELOCITY || MODE == FVX_PAIR_VELOCITY_STRETCH)
    cross(acc, f * dx, f * dy, f * dz);
  if (MODE == FVX_PAIR_STRETCH || MODE == FVX_PAIR_VELOCITY_STRETCH) {
    const double w = fpr * fma(dz, gz, fma(dy, gy, dx * gx));
    cross(acc + (MODE == FVX_PAIR_STRETCH ? 0 : 3), fma(w, dx, f * gx), fma(w, dy, f * gy),
          fma(w, dz, f * gz));
  }
  if (MODE == FVX_PAIR_JACOBIAN) {
    const double px = fpr * fma(dy, az, -(dz * ay));
    const double py = fpr * fma(dz, ax, -(dx * az));
    const double pz = fpr * fma(dx, ay, -(dy * ax));
    acc[0] = fma(px, dx, acc[0]);
    acc[1] = fma(px, dy, acc[1]);
    acc[2] = fma(px, dz, acc[2]);
    acc[3] = fma(py, dx, acc[3]);
    acc[4] = fma(py, dy, acc[4]);
    acc[5] = fma(py, dz, acc[5]);
    acc[6] = fma(pz, dx, acc[6]);
    acc[7] = fma(pz, dy, acc[7]);
    acc[8] = fma(pz, dz, acc[8]);
    acc[9] = fma(f, ax, acc[9]);
    acc[10] = fma(f, ay, acc[10]);
    acc[11] = fma(f, az, acc[11]);
  }
  if (MODE == FVX_PAIR_VORTICITY) {
    const double s = fpr * fma(dz, az, fma(dy, ay, dx * ax));
    acc[0] = fma(-ax, iso, fma(dx, s, acc[0]));
    acc[1] = fma(-ay, iso, fma(dy, s, acc[1]));
    acc[2] = fma(-az, iso, fma(dz, s, acc[2]));
  }
}
template <int MODE>
__device__ __forceinline__ void fold_tile(double* sum, double* part) {
  if (MODE == FVX_PAIR_JACOBIAN) {
    part[1] += part[11];
    part[2] -= part[10];
    part[3] -= part[11];
    part[5] += part[9];
    part[6] += part[10];
    part[7] -= part[9];
  }
#pragma unroll
  for (int c = 0; c < ModeInfo<MODE>::ncomp; ++c) sum[c] += part[c];
}

// One target per thread and slice.  The FP64 pipe and the FP32 issue bound it
// about alike: 9 (velocity), 16 (stretching), 21 (gradient), 10 (vorticity) FP64
// operations per pair, the offset being converted from its three floats, against
// 31, 40, 55 and 43 with the Winckelmans core in FP64 and 100 more with the
// Gaussian one; and the 450 to 850 FP32 operations of the scalar core beside
// them.  Velocity at 384 points of 131,071 particles 2.70 -> 0.94 ms (54e9
// pairs/s); gradient of 7,001 particles at themselves, Gaussian core, 13.9 ->
// 2.15 ms; the field step of 3,001 (three velocity, three stretching and a
// vorticity sweep, Gaussian) 15.5 -> 2.3 ms.
// Two slices of 128 threads share a CTA's targets, one taking the even sources,
// the other the odd ones, and its table.  (One: 1,392 us for 384 targets x 131,071
// sources with a CTA per SM, two: 1,017; four leave 64 registers a thread, and
// the stretching sums then spill: 336 us against 150 for 2,049 particles.)
constexpr int kSlices = 2;

template <int MODE, int KERNEL>
size_t f64_smem_bytes() {
  const size_t table = KERNEL == FVX_KERNEL_GAUSSIANERF
                           ? sizeof(float) * kTableFloats * (ModeInfo<MODE>::need_fpr ? 2 : 1)
                           : 0;
  const size_t tiles = sizeof(F64Smem) + table;
  const size_t sums = sizeof(double) * (kSlices - 1) * kThreads * ModeInfo<MODE>::ncomp;
  return tiles > sums ? tiles : sums;
}

template <int MODE, int KERNEL>
__global__ void __launch_bounds__(kSlices* kThreads) pairs_f64_kernel(PairArgs A) {
  constexpr int NC = ModeInfo<MODE>::ncomp;
  constexpr bool FPR = ModeInfo<MODE>::need_fpr;
  constexpr bool ISO = MODE == FVX_PAIR_VORTICITY;
  constexpr bool GAUSS = KERNEL == FVX_KERNEL_GAUSSIANERF;
  constexpr int kParts = FPR ? 2 : 1;  // polynomials staged per interval

  extern __shared__ __align__(128) unsigned char f64_smem[];
  F64Smem& S = *reinterpret_cast<F64Smem*>(f64_smem);

  constexpr int kRun = 32;
  constexpr int kAll = kSlices * kThreads;
  const int slice = threadIdx.x / kThreads, lt = threadIdx.x % kThreads;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + lt;
  const bool act = i < A.n_tgt;
  double tx = 0, ty = 0, tz = 0, gx = 0, gy = 0, gz = 0;
  if (act) {
    tx = A.tgt[3 * i + 0];
    ty = A.tgt[3 * i + 1];
    tz = A.tgt[3 * i + 2];
    if (ModeInfo<MODE>::need_tg) {
      gx = A.tgt_gamma[3 * i + 0];
      gy = A.tgt_gamma[3 * i + 1];
      gz = A.tgt_gamma[3 * i + 2];
    }
  }
  const bool tgt_ok = x3::coord_in_range(tx) && x3::coord_in_range(ty) && x3::coord_in_range(tz);
  const x3::F3 px = x3::split_fast(tx), py = x3::split_fast(ty), pz = x3::split_fast(tz);

  const int64_t jb = static_cast<int64_t>(blockIdx.y) * A.chunk;
  const int64_t je = min(jb + A.chunk, A.n_src);
  const int ntiles = jb < je ? static_cast<int>((je - jb + kSrc64 - 1) / kSrc64) : 0;

  if (threadIdx.x == 0) {
    mbar_init(&S.bar[0], 1);
    mbar_init(&S.bar[1], 1);
    fence_mbar_init();
  }
  if constexpr (GAUSS) {
    for (int e = threadIdx.x; e < kTableRows * kParts * (x3::kRowFloats / 4); e += kAll) {
      const int row = e / (x3::kRowFloats / 4), q = e % (x3::kRowFloats / 4);
      reinterpret_cast<float4*>(S.table)[e] = *reinterpret_cast<const float4*>(
          g_core_table + (row * 2 / kParts) * x3::kRowFloats + 4 * q);
    }
  }
  __syncthreads();

  double sum[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) sum[c] = 0.0;

  uint32_t phase[2] = {0u, 0u};
  bool ok = true;
  if (ntiles > 0 && threadIdx.x == 0)
    issue_src(A, S.raw[0], jb, static_cast<int>(min64(kSrc64, je - jb)), &S.bar[0]);
  int t = 0;
  for (; t < ntiles; ++t) {
    const int buf = t & 1;
    const int64_t j0 = jb + static_cast<int64_t>(t) * kSrc64;
    const int n = static_cast<int>(min64(kSrc64, je - j0));
    if (t + 1 < ntiles && threadIdx.x == 0) {
      const int64_t j1 = j0 + kSrc64;
      issue_src(A, S.raw[buf ^ 1], j1, static_cast<int>(min64(kSrc64, je - j1)),
                &S.bar[buf ^ 1]);
    }
    const bool got = mbar_wait(&S.bar[buf], phase[buf]);
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    phase[buf] ^= 1u;
    RawSrc<kSrc64>& raw = S.raw[buf];
    tail_src(A, raw, j0, n);
    __syncthreads();
    bool in_range = tgt_ok;
    for (int k = threadIdx.x; k < n; k += kAll) {
      const double sg = raw.sigma[k];
      SrcX3 v = {};
      in_range = in_range && x3::core_in_range(sg);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double p = raw.pos[3 * k + c];
        v.a[c] = kC * raw.alpha[3 * k + c];
        v.x[c] = x3::split_fast(p);
        in_range = in_range && x3::coord_in_range(p);
      }
      const x3::Core core = GAUSS ? x3::gaussian_core(sg) : x3::winckelmans_core(sg);
      v.s2 = core.s2;
      v.k = core.k;
      v.k5 = core.k5;
      S.tile[k] = v;
    }
    // sums of kRun sources at a time join the thread's: short partial sums
    // round less than the whole tile's did
    if (__syncthreads_and(in_range)) {
#pragma unroll 1
      for (int k0 = slice; k0 < n; k0 += kRun * kSlices) {
        double part[F64Acc<MODE>::n] = {};
        const int k1 = min(n, k0 + kRun * kSlices);
#pragma unroll 1
        for (int k = k0; k < k1; k += kSlices) {
          const SrcX3& s = S.tile[k];
          const x3::F3 x = x3::diff(px, s.x[0]), y = x3::diff(py, s.x[1]), z = x3::diff(pz, s.x[2]);
          const x3::Core core{s.s2, s.k, s.k5};
          x3::F3 f, fpr = {}, iso = {};
          if constexpr (GAUSS)
            x3::gaussian<FPR, ISO>(x, y, z, core, x3::kCoreEnd, x3::kCoreRows,
                                   [&](int row, int part_) {
                                     x3::Row r;
                                     const float4* q = reinterpret_cast<const float4*>(
                                         S.table + (row * kParts + part_) * x3::kRowFloats);
  #pragma unroll
                                     for (int w = 0; w < x3::kRowFloats / 4; ++w) {
                                       const float4 v4 = q[w];
                                       r.c[4 * w] = v4.x;
                                       r.c[4 * w + 1] = v4.y;
                                       r.c[4 * w + 2] = v4.z;
                                       r.c[4 * w + 3] = v4.w;
                                     }
                                     return r;
                                   },
                                   f, fpr, iso);
          else
            x3::winckelmans<FPR, ISO>(x, y, z, core, f, fpr, iso);
          accumulate_f64<MODE>(part, x3::to_double(x), x3::to_double(y), x3::to_double(z), s.a[0],
                               s.a[1], s.a[2], x3::to_double(f), FPR ? x3::to_double(fpr) : 0.0,
                               ISO ? x3::to_double(iso) : 0.0, gx, gy, gz);
        }
        fold_tile<MODE>(sum, part);
      }
    } else {
      // the same sums with the core in FP64
#pragma unroll 1
      for (int k0 = slice; k0 < n; k0 += kRun * kSlices) {
        double part[F64Acc<MODE>::n] = {};
        const int k1 = min(n, k0 + kRun * kSlices);
#pragma unroll 1
        for (int k = k0; k < k1; k += kSlices) {
          const double sg = raw.sigma[k];
          const double dx = tx - raw.pos[3 * k], dy = ty - raw.pos[3 * k + 1],
                       dz = tz - raw.pos[3 * k + 2];
          const double r2 = dx * dx + dy * dy + dz * dz;
          double f, fpr = 0.0;
          core_f64<KERNEL, FPR>(r2, sg * sg, GAUSS ? 1.0 / sg : 2.5 * sg * sg, f, fpr);
          accumulate_f64<MODE>(part, dx, dy, dz, kC * raw.alpha[3 * k], kC * raw.alpha[3 * k + 1],
                               kC * raw.alpha[3 * k + 2], f, fpr, fpr * r2 + (f + f), gx, gy, gz);
        }
        fold_tile<MODE>(sum, part);
      }
    }
    __syncthreads();
  }
  if (!ok) {
    flag_status(kStatusTimeout);
    if (threadIdx.x == 0 && t + 1 < ntiles) mbar_wait(&S.bar[(t + 1) & 1], phase[(t + 1) & 1]);
    return;
  }
  {
    // the slices' sums, in slice order (tiles, barriers and table are done with)
    double* q = reinterpret_cast<double*>(f64_smem);
    if (slice > 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c) q[((slice - 1) * NC + c) * kThreads + lt] = sum[c];
    }
    __syncthreads();
    if (slice > 0) return;
#pragma unroll
    for (int s = 0; s < kSlices - 1; ++s)
#pragma unroll
      for (int c = 0; c < NC; ++c) sum[c] += q[(s * NC + c) * kThreads + lt];
  }
  if (!act) return;
  if (gridDim.y > 1) {
    double* o = A.partial + (static_cast<int64_t>(blockIdx.y) * A.n_tgt + i) * NC;
#pragma unroll
    for (int c = 0; c < NC; ++c) o[c] = sum[c];
  } else {
    constexpr int NA = ModeInfo<MODE>::na;
#pragma unroll
    for (int c = 0; c < NA; ++c) A.out_a[i * NA + c] = sum[c];
#pragma unroll
    for (int c = NA; c < NC; ++c) A.out_b[i * (NC - NA) + (c - NA)] = sum[c];
  }
}

// The split partial sums of every output value, in a fixed order: a warp per
// value, lane l adding splits l, l + 32, ... in turn, then a fixed shuffle
// tree over the lanes.  (A thread per value would leave a few hundred values
// to a handful of CTAs, each thread waiting on one dependent load per split.)
__global__ void reduce_pairs_kernel(const double* __restrict__ partial, int64_t n_tgt, int nc,
                                    int na, int splits, double* __restrict__ out_a,
                                    double* __restrict__ out_b) {
  const int64_t idx = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t n_vals = n_tgt * nc;
  if (idx >= n_vals) return;  // the whole warp: idx is the warp's
  double s = 0.0;
  for (int k = lane; k < splits; k += 32) s += partial[static_cast<int64_t>(k) * n_vals + idx];
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (lane != 0) return;
  const int64_t i = idx / nc;
  const int c = static_cast<int>(idx - i * nc);
  if (c < na)
    out_a[i * na + c] = s;
  else
    out_b[i * (nc - na) + (c - na)] = s;
}

int mode_ncomp(int mode) {
  switch (mode) {
    case FVX_PAIR_VELOCITY:
    case FVX_PAIR_STRETCH:
    case FVX_PAIR_VORTICITY:
      return 3;
    case FVX_PAIR_VELOCITY_STRETCH:
      return 6;
    case FVX_PAIR_JACOBIAN:
      return 9;
    default:
      return -1;
  }
}

int mode_na(int mode) { return mode == FVX_PAIR_VELOCITY_STRETCH ? 3 : mode_ncomp(mode); }

// Targets of one row of the split rule's grid.
int targets_per_cta(int mode, int precision) {
  if (precision != FVX_PREC_F32C) return kThreads;
  return kThreads * (mode_ncomp(mode) <= 3 ? 4 : 2);
}

// Splits of the source range for six CTAs of a row's targets per SM, of at least
// two source tiles: few targets (the panel points against every particle) split
// the sources that far.
int splits_f32(int64_t gx, int64_t n_src, int64_t* chunk) {
  const int64_t want = 6LL * device_sm_count();
  int64_t s = gx >= want ? 1 : (want + gx - 1) / gx;
  const int64_t maxs = (n_src + 2 * kSrcTile - 1) / (2 * kSrcTile);
  if (s > maxs) s = maxs;
  if (s < 1) s = 1;
  int64_t c = (n_src + s - 1) / s;
  c = (c + 1) & ~int64_t(1);
  s = (n_src + c - 1) / c;
  *chunk = c;
  return static_cast<int>(s);
}

// An FP64 sweep takes as long as the SM with the most CTAs: `rounds` CTAs of
// `chunk` sources each and a prologue that costs as much as kPrologue of them (the
// first tile's latency, the Gaussian core's table), and an eighth longer where
// the SM has only one CTA's warps to overlap (less with more: 1,017, 955 and 916 us
// with 1, 4 .. 8 and 8 .. 16 rounds for 384 targets x 131,071 sources).  The
// number of rounds, up to 24, that makes the least of that: one for 240 targets
// x 2,001 sources (24 us; 28 with 4, 35 with 8), 3 for 2,049 x 2,049.
int splits_f64(int64_t gx, int64_t n_src, int64_t* chunk) {
  constexpr int64_t kPrologue = 4;
  const int64_t sms = device_sm_count();
  int64_t best = -1, best_c = n_src;
  for (int64_t rounds = 1; rounds <= 24; ++rounds) {
    int64_t s = rounds * sms / gx;
    if (s < 1) continue;
    if (s > n_src) s = n_src;
    int64_t c = (n_src + s - 1) / s;
    c = (c + 1) & ~int64_t(1);
    const int64_t per_sm = (gx * ((n_src + c - 1) / c) + sms - 1) / sms;
    const int64_t cost = (per_sm * 8 + 1) * (c + kPrologue);
    if (best < 0 || cost < best) {
      best = cost;
      best_c = c;
    }
  }
  *chunk = best_c;
  return static_cast<int>((n_src + best_c - 1) / best_c);
}

// coarse: the FP32 rule for FP64 too, for a caller whose scratch holds no more
int pair_splits(int mode, int precision, int64_t n_tgt, int64_t n_src, int64_t* chunk,
                bool coarse = false) {
  const int per_cta = targets_per_cta(mode, precision);
  const int64_t gx = (n_tgt + per_cta - 1) / per_cta;
  return precision == FVX_PREC_F32C || coarse ? splits_f32(gx, n_src, chunk)
                                              : splits_f64(gx, n_src, chunk);
}

template <int MODE, int KERNEL>
void launch_mode(int precision, dim3 grid, cudaStream_t stream, const PairArgs& A) {
  if (precision == FVX_PREC_F32C) {
    grid.x = static_cast<unsigned>((A.n_tgt + kTargetsF32 - 1) / kTargetsF32);
    pairs_f32_kernel<MODE, KERNEL><<<grid, kThreads, 0, stream>>>(A);
    return;
  }
  const size_t smem = f64_smem_bytes<MODE, KERNEL>();
  // (each call: the attribute is the current device's; a failure shows at the launch)
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(pairs_f64_kernel<MODE, KERNEL>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  pairs_f64_kernel<MODE, KERNEL><<<grid, kSlices * kThreads, smem, stream>>>(A);
}

template <int KERNEL>
void launch_kernel(int mode, int precision, dim3 grid, cudaStream_t stream, const PairArgs& A) {
  switch (mode) {
    case FVX_PAIR_VELOCITY:
      launch_mode<FVX_PAIR_VELOCITY, KERNEL>(precision, grid, stream, A);
      break;
    case FVX_PAIR_STRETCH:
      launch_mode<FVX_PAIR_STRETCH, KERNEL>(precision, grid, stream, A);
      break;
    case FVX_PAIR_VELOCITY_STRETCH:
      launch_mode<FVX_PAIR_VELOCITY_STRETCH, KERNEL>(precision, grid, stream, A);
      break;
    case FVX_PAIR_JACOBIAN:
      launch_mode<FVX_PAIR_JACOBIAN, KERNEL>(precision, grid, stream, A);
      break;
    default:
      launch_mode<FVX_PAIR_VORTICITY, KERNEL>(precision, grid, stream, A);
      break;
  }
}

}  // namespace

size_t particle_pairs_scratch(int mode, int precision, int64_t n_tgt, int64_t n_src) {
  const int nc = mode_ncomp(mode);
  if (nc < 0 || n_tgt <= 0 || n_src <= 0) return 0;
  int64_t chunk = 0;
  const int s = pair_splits(mode, precision, n_tgt, n_src, &chunk);
  return s > 1 ? sizeof(double) * static_cast<size_t>(nc) * n_tgt * s : 0;
}

int particle_pairs_launch(int mode, int kernel, int precision, const double* tgt,
                          const double* tgt_gamma, int64_t n_tgt, const double* pos,
                          const double* alpha, const double* sigma, int64_t n_src,
                          double* out_a, double* out_b, void* scratch, size_t scratch_bytes,
                          cudaStream_t stream) {
  const int nc = mode_ncomp(mode);
  FVX_ARG_CHECK(nc > 0, "unknown pair mode %d", mode);
  FVX_ARG_CHECK(kernel == FVX_KERNEL_GAUSSIANERF || kernel == FVX_KERNEL_WINCKELMANS,
                "unknown kernel %d", kernel);
  FVX_ARG_CHECK(precision == FVX_PREC_F64 || precision == FVX_PREC_F32C,
                "unknown precision %d", precision);
  FVX_ARG_CHECK(n_tgt >= 0 && n_src >= 0, "negative size");
  if (n_tgt == 0) return FVX_OK;
  const int na = mode_na(mode);
  FVX_ARG_CHECK(tgt && out_a, "null targets/output");
  FVX_ARG_CHECK(na == nc || out_b, "mode needs out_b");
  const bool need_tg = mode == FVX_PAIR_STRETCH || mode == FVX_PAIR_VELOCITY_STRETCH;
  FVX_ARG_CHECK(!need_tg || tgt_gamma, "mode needs target strengths");
  if (n_src == 0) {
    FVX_CUDA_TRY(cudaMemsetAsync(out_a, 0, sizeof(double) * na * n_tgt, stream));
    if (nc > na) FVX_CUDA_TRY(cudaMemsetAsync(out_b, 0, sizeof(double) * (nc - na) * n_tgt, stream));
    return FVX_OK;
  }
  FVX_ARG_CHECK(pos && alpha && sigma, "null source array");
  int64_t chunk = 0;
  int splits = pair_splits(mode, precision, n_tgt, n_src, &chunk);
  const size_t row = sizeof(double) * static_cast<size_t>(nc) * n_tgt;
  if (splits > 1 && (scratch == nullptr || scratch_bytes < row * splits)) {
    const size_t need = row * splits;
    splits = pair_splits(mode, precision, n_tgt, n_src, &chunk, true);
    if (splits > 1 && (scratch == nullptr || scratch_bytes < row * splits)) {
      set_last_error("particle_pairs needs %zu scratch bytes, got %zu", need, scratch_bytes);
      return FVX_ERR_SCRATCH;
    }
  }
  PairArgs A;
  A.tgt = tgt;
  A.tgt_gamma = tgt_gamma;
  A.n_tgt = n_tgt;
  A.pos = pos;
  A.alpha = alpha;
  A.sigma = sigma;
  A.n_src = n_src;
  A.chunk = chunk;
  A.out_a = out_a;
  A.out_b = out_b;
  A.partial = static_cast<double*>(scratch);
  A.use_tma = aligned16(pos) && aligned16(alpha) && aligned16(sigma);
  const int per_cta = targets_per_cta(mode, precision);
  const int64_t gx = (n_tgt + per_cta - 1) / per_cta;
  FVX_ARG_CHECK(gx < (1LL << 31), "too many targets");
  dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(splits));
  if (kernel == FVX_KERNEL_WINCKELMANS)
    launch_kernel<FVX_KERNEL_WINCKELMANS>(mode, precision, grid, stream, A);
  else
    launch_kernel<FVX_KERNEL_GAUSSIANERF>(mode, precision, grid, stream, A);
  FVX_LAUNCH_CHECK();
  if (splits > 1) {
    const int64_t nv = n_tgt * nc;  // a warp per value
    FVX_ARG_CHECK((nv * 32 + 255) / 256 < (1LL << 31), "too many output values");
    reduce_pairs_kernel<<<static_cast<unsigned>((nv * 32 + 255) / 256), 256, 0, stream>>>(
        static_cast<const double*>(scratch), n_tgt, nc, na, splits, out_a, out_b);
    FVX_LAUNCH_CHECK();
  }
  return FVX_OK;
}

}  // namespace fvx

extern "C" {

size_t fvx_particle_pairs_scratch_bytes(int mode, int precision, int64_t n_targets,
                                        int64_t n_sources) {
  return fvx::particle_pairs_scratch(mode, precision, n_targets, n_sources);
}

int fvx_particle_pairs(int mode, int kernel, int precision, const double* tgt_pos,
                       const double* tgt_gamma, int64_t n_targets, const double* src_pos,
                       const double* src_gamma, const double* src_sigma, int64_t n_sources,
                       double* out_a, double* out_b, void* scratch, size_t scratch_bytes,
                       void* stream) {
  return fvx::particle_pairs_launch(mode, kernel, precision, tgt_pos, tgt_gamma, n_targets,
                                    src_pos, src_gamma, src_sigma, n_sources, out_a, out_b,
                                    scratch, scratch_bytes, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
