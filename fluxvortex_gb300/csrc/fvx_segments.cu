// fvx_segments.cu -- line-vortex Biot-Savart for ring, chordwise-ring and
// horseshoe vortices with the PteraSoftware Lamb-Oseen + Squire core, FP64.
//
// Replaces the five functions of src/fluxvortex/warp_kernels.py:251-382 (one
// launch per leg with an atomic add per (point, vortex) pair, :188-246).
// Here all legs of a vortex are fused: corner offsets and their lengths are
// shared between the two legs that meet at a corner (the reference computes
// the same values twice, so sharing changes no bit), per-leg constants
// (|r0|^2, the 1e-10 |r0| tolerance, |r0|^2 r_c^2, Gamma/4pi) are hoisted
// into shared memory once per tile, and sums are reduced without atomics:
//
//   collapsed  CTA = 128 target points x a run of vortices.  Vortex tiles
//              (corners + strengths + core radii + ages) are staged into
//              shared memory by 1-D TMA bulk copies (cp.async.bulk), double
//              buffered on two mbarriers.  When the target blocks alone cannot
//              fill the SMs, all (block, vortex) work is laid end to end and
//              cut into equal runs, two CTAs per SM; the first run of a block
//              writes the result, the others' partial sums go to scratch and a
//              second kernel adds them in run order (deterministic).  Equal
//              runs matter because the FP64 pipe is the limit and has no
//              slack to hide a last wave: splitting each block alike left
//              10,000 points x 10,000 rings with 316 CTAs on 152 SMs, three
//              on some and two on the others.
//   expanded   one thread per vortex, looping over a few target points, so
//              that a warp writes 32 consecutive (point, vortex, 3) records.
//
// Arithmetic per (point, leg): fvx_segment_x3.cuh.  The four skip tests take
// the reference's decisions (warp_kernels.py:46-96).  10,000 points x 10,000
// rings: 61.4 ms with the reference's sequence in FP64, 25.4 ms with its roots,
// divisions and tests replaced (fvx_segment_math.cuh), 12.6 ms so; 501 points x
// 1,003 horseshoes expanded 213, 145 and 73 us; 200 points x 100 rings 30, 27
// and 18 us on the device.
#include "fvx_common.cuh"
#include "fvx_segment_math.cuh"
#include "fvx_segment_x3.cuh"

namespace fvx {
namespace {

using namespace seg;

constexpr int kCollThreads = 128;  // target points per collapsed CTA
constexpr int kCollSlices = 2;     // threads per point, each with every other vortex:
                                   // 16 warps per SM from the two CTAs' worth of runs
constexpr int kTile = 64;          // vortices per shared-memory tile
constexpr int kExpThreads = 64;    // vortices per expanded CTA
__device__ __forceinline__ void flush_counts(int cnt[4], int64_t* counts) {
  if (counts == nullptr) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    unsigned v = __reduce_add_sync(0xffffffffu, static_cast<unsigned>(cnt[k]));
    if ((threadIdx.x & 31) == 0 && v != 0)
      atomicAdd(reinterpret_cast<unsigned long long*>(counts + k),
                static_cast<unsigned long long>(v));
  }
}

struct RawTile {
  double c[4][kTile * 3];
  double strength[kTile];
  double rc0[kTile];
  double age[kTile];
};

// The runs of a collapsed call: CTA c takes (block, vortex) work c share ..
// (c + 1) share.  Partial sums: a slot of 128 rows of three values per CTA that
// starts inside a block (CTA 0 does not), in CTA order, and of the last block's
// rows for the CTAs from c_last on, which start inside that one.  With share >=
// the split's chunk, floor((blocks - 1) M / share) slots of 128 rows and
// ceil(M / share) at most of the last block's are within splits x points rows.
struct Runs {
  int64_t share, n_vort;
  int c_last, last_rows;
  __host__ __device__ int64_t row(int64_t c) const {
    return c < c_last ? (c - 1) * kCollThreads
                      : static_cast<int64_t>(c_last - 1) * kCollThreads + (c - c_last) * last_rows;
  }
};

struct SegArgs {
  const double* points;
  const double* corner[4];
  const double* strengths;
  const double* rc0s;
  const double* ages;  // may be null
  double nu;
  int64_t n_points;
  int64_t n_vort;
  Runs runs;        // collapsed: the CTAs' runs
  double* out;
  double* partial;  // collapsed: (rows, 3) per CTA that starts inside a block
  int64_t* counts;
  int use_tma;
};

// Issues the stage-in of vortices [v0, v0+cnt) into `raw`; thread 0 only.
__device__ void issue_tile(const SegArgs& A, RawTile& raw, int64_t v0, int cnt, uint64_t* bar) {
  uint32_t total = 0;
  BulkPlan pc[4], ps, pr, pa;
  for (int c = 0; c < 4; ++c) {
    pc[c] = plan_bulk(A.corner[c], v0, cnt, 24, A.use_tma);
    total += pc[c].bulk_bytes;
  }
  ps = plan_bulk(A.strengths, v0, cnt, 8, A.use_tma);
  pr = plan_bulk(A.rc0s, v0, cnt, 8, A.use_tma);
  pa = A.ages ? plan_bulk(A.ages, v0, cnt, 8, A.use_tma) : BulkPlan{0u, 0u};
  total += ps.bulk_bytes + pr.bulk_bytes + pa.bulk_bytes;
  mbar_arrive_expect_tx(bar, total);
  for (int c = 0; c < 4; ++c)
    if (pc[c].bulk_bytes) bulk_g2s(raw.c[c], A.corner[c] + 3 * v0, pc[c].bulk_bytes, bar);
  if (ps.bulk_bytes) bulk_g2s(raw.strength, A.strengths + v0, ps.bulk_bytes, bar);
  if (pr.bulk_bytes) bulk_g2s(raw.rc0, A.rc0s + v0, pr.bulk_bytes, bar);
  if (pa.bulk_bytes) bulk_g2s(raw.age, A.ages + v0, pa.bulk_bytes, bar);
}

// Plain copies of whatever the bulk copies of the tile did not cover.
__device__ void tail_tile(const SegArgs& A, RawTile& raw, int64_t v0, int cnt) {
  for (int c = 0; c < 4; ++c) {
    BulkPlan p = plan_bulk(A.corner[c], v0, cnt, 24, A.use_tma);
    if (p.tail_bytes) plain_copy8(raw.c[c], A.corner[c] + 3 * v0, p.bulk_bytes, p.tail_bytes);
  }
  BulkPlan p = plan_bulk(A.strengths, v0, cnt, 8, A.use_tma);
  if (p.tail_bytes) plain_copy8(raw.strength, A.strengths + v0, p.bulk_bytes, p.tail_bytes);
  p = plan_bulk(A.rc0s, v0, cnt, 8, A.use_tma);
  if (p.tail_bytes) plain_copy8(raw.rc0, A.rc0s + v0, p.bulk_bytes, p.tail_bytes);
  if (A.ages) {
    p = plan_bulk(A.ages, v0, cnt, 8, A.use_tma);
    if (p.tail_bytes) plain_copy8(raw.age, A.ages + v0, p.bulk_bytes, p.tail_bytes);
  }
}

// a / b, in 32 bits where both fit (a third of the instructions)
__device__ __forceinline__ int64_t div_small(int64_t a, int64_t b) {
  return ((a | b) >> 32) == 0 ? static_cast<uint32_t>(a) / static_cast<uint32_t>(b) : a / b;
}

// The whole tile by plain loads, every element in flight at once (array after
// array, the copies above wait for seven loads in a row; over the link to host
// memory that is 10 us).
__device__ void load_tile(const SegArgs& A, RawTile& raw, int64_t v0, int n) {
  const int words = (A.ages ? 15 : 14) * n;
  for (int e = threadIdx.x; e < words; e += blockDim.x) {
    if (e < 12 * n) {
      const int c = e / (3 * n), k = e - 3 * n * c;
      raw.c[c][k] = A.corner[c][3 * v0 + k];
    } else {
      const int f = e / n - 12, k = e - n * (f + 12);
      (f == 0 ? raw.strength : (f == 1 ? raw.rc0 : raw.age))[k] =
          (f == 0 ? A.strengths : (f == 1 ? A.rc0s : A.ages))[v0 + k];
    }
  }
}

template <int LEGS>
__device__ __forceinline__ void add_general(const VortexRec& R, double px, double py, double pz,
                                            double& vx, double& vy, double& vz, int* cnt) {
  double v[3] = {0.0, 0.0, 0.0};
  int c[4] = {0, 0, 0, 0};
  vortex_velocity_rare<LEGS>(R, px, py, pz, v, c);
  vx += v[0];
  vy += v[1];
  vz += v[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) cnt[i] += c[i];
}

template <int LEGS>
__global__ void __launch_bounds__(kCollSlices* kCollThreads) collapsed_kernel(SegArgs A) {
  __shared__ __align__(128) RawTile raw[2];
  __shared__ __align__(16) VortexRec rec[kTile];
  __shared__ __align__(16) RingX3 recx[kTile];
  __shared__ double other[3][kCollThreads];  // the second slice's sums
  __shared__ __align__(8) uint64_t bar[2];
  const int slice = threadIdx.x / kCollThreads, lt = threadIdx.x % kCollThreads;

  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  const int64_t blocks = (A.n_points + kCollThreads - 1) / kCollThreads;
  int64_t pos = static_cast<int64_t>(blockIdx.x) * A.runs.share;
  const int64_t end = min64(pos + A.runs.share, blocks * A.n_vort);
  int64_t blk = div_small(pos, A.n_vort);
  int cnt[4] = {0, 0, 0, 0};
  uint32_t phase[2] = {0u, 0u};
  int buf = 0;
  for (; pos < end; ++blk) {
    const int64_t vb = pos - blk * A.n_vort;
    const int64_t ve = min64(vb + (end - pos), A.n_vort);
    const int ntiles = static_cast<int>((ve - vb + kTile - 1) / kTile);
    const int64_t i = blk * kCollThreads + lt;
    const bool active = i < A.n_points;
    double px = 0.0, py = 0.0, pz = 0.0;
    if (active) {
      px = A.points[3 * i + 0];
      py = A.points[3 * i + 1];
      pz = A.points[3 * i + 2];
    }
    const x3::F3 p[3] = {x3::split_fast(px), x3::split_fast(py), x3::split_fast(pz)};
    const bool in_range = x3_range(px) && x3_range(py) && x3_range(pz);
    double vx = 0.0, vy = 0.0, vz = 0.0;
    if (threadIdx.x == 0)
      issue_tile(A, raw[buf], vb, static_cast<int>(min64(kTile, ve - vb)), &bar[buf]);
    for (int t = 0; t < ntiles; ++t, buf ^= 1) {
      const int64_t v0 = vb + static_cast<int64_t>(t) * kTile;
      const int n = static_cast<int>(min64(kTile, ve - v0));
      if (t + 1 < ntiles && threadIdx.x == 0) {
        const int64_t v1 = v0 + kTile;
        issue_tile(A, raw[buf ^ 1], v1, static_cast<int>(min64(kTile, ve - v1)),
                   &bar[buf ^ 1]);
      }
      const bool got = mbar_wait(&bar[buf], phase[buf]);
      if (!__syncthreads_and(got)) {
        flag_status(kStatusTimeout);
        // Drain the copy that may still be in flight into the other buffer.
        if (threadIdx.x == 0 && t + 1 < ntiles) mbar_wait(&bar[buf ^ 1], phase[buf ^ 1]);
        return;
      }
      phase[buf] ^= 1u;
      if (A.use_tma)
        tail_tile(A, raw[buf], v0, n);
      else
        load_tile(A, raw[buf], v0, n);
      __syncthreads();
      for (int k = threadIdx.x; k < n; k += kCollSlices * kCollThreads) {
        prep_vortex<LEGS>(rec[k], &raw[buf].c[0][3 * k], &raw[buf].c[1][3 * k],
                          &raw[buf].c[2][3 * k], &raw[buf].c[3][3 * k], raw[buf].strength[k],
                          raw[buf].rc0[k], A.ages ? raw[buf].age[k] : 0.0, A.nu);
        prep_x3<LEGS>(recx[k], rec[k]);
      }
      __syncthreads();
      if (active) {
#pragma unroll 1
        for (int k = slice; k < n; k += kCollSlices) {
          if (!in_range || recx[k].near > kNoX3) {  // nothing of the three-float path is run
            add_general<LEGS>(rec[k], px, py, pz, vx, vy, vz, cnt);
            continue;
          }
          vortex_velocity_x3<LEGS>(RingView{recx[k]}, p, vx, vy, vz, cnt,
                                   [&](double* v, int* c) {
                                     vortex_velocity_rare<LEGS>(rec[k], px, py, pz, v, c);
                                   });
        }
      }
      __syncthreads();
    }
    if (slice == 1) {
      other[0][lt] = vx;
      other[1][lt] = vy;
      other[2][lt] = vz;
    }
    __syncthreads();
    if (slice == 0 && active) {
      double* o = vb == 0 ? A.out + 3 * i : A.partial + 3 * (A.runs.row(blockIdx.x) + lt);
      o[0] = vx + other[0][lt];
      o[1] = vy + other[1][lt];
      o[2] = vz + other[2][lt];
    }
    pos += ve - vb;
  }
  flush_counts(cnt, A.counts);
}

// dst[v] = out[v] + the partial sums of value v = 3 row + component, in a fixed order:
// kReduceLanes lanes per value take the block's CTAs in turn, then a shuffle
// tree.  (One thread per value waits for one load after another: 12 us for 200
// points split 50 ways.)
constexpr int kReduceLanes = 8;

// dst_counts, if not null, receives the skip counts, which start again at zero.
__global__ void reduce_runs_kernel(const double* __restrict__ partial, int64_t n_points, Runs R,
                                   const double* out, double* dst, int64_t* counts,
                                   int64_t* dst_counts) {
  if (dst_counts != nullptr && blockIdx.x == 0 && threadIdx.x < 4) {
    dst_counts[threadIdx.x] = counts[threadIdx.x];
    counts[threadIdx.x] = 0;
  }
  const int64_t v =
      (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / kReduceLanes;
  const int lane = threadIdx.x % kReduceLanes;
  const bool active = v < 3 * n_points;
  double s = 0.0;
  if (active) {
    const int64_t i = v / 3, blk = i / kCollThreads;
    const int64_t at = 3 * (i - blk * kCollThreads) + v % 3;
    // the CTAs that start inside the block
    const int64_t c_end = div_small((blk + 1) * R.n_vort + R.share - 1, R.share);
    for (int64_t c = div_small(blk * R.n_vort, R.share) + 1 + lane; c < c_end; c += kReduceLanes)
      s += partial[3 * R.row(c) + at];
  }
#pragma unroll
  for (int off = kReduceLanes / 2; off >= 1; off >>= 1)
    s += __shfl_down_sync(0xffffffffu, s, off, kReduceLanes);
  if (active && lane == 0) dst[v] = out[v] + s;
}

// The general path of one (point, vortex) pair of an expanded call.
template <int LEGS>
__device__ __noinline__ void expanded_rare(const SegArgs& A, int64_t m, int64_t p, double* v,
                                           int* cnt) {
  VortexRec R;
  prep_vortex<LEGS>(R, A.corner[0] + 3 * m, A.corner[1] + 3 * m, A.corner[2] + 3 * m,
                    A.corner[3] + 3 * m, A.strengths[m], A.rc0s[m], A.ages ? A.ages[m] : 0.0,
                    A.nu);
  vortex_velocity_rare<LEGS>(R, A.points[3 * p], A.points[3 * p + 1], A.points[3 * p + 2], v, cnt);
}

// The general path for a thread's vortex at all points of the CTA.  One preparation
// for all of them (501 points x 1,003 rings in millimetres: 216 us, 319 us with one
// per pair after the three-float path; 252 us is the reference's sequence
// throughout).
template <int LEGS>
__device__ __noinline__ void expanded_general(const SegArgs& A, int64_t m, int64_t p0, int np,
                                              int* cnt) {
  VortexRec R;
  prep_vortex<LEGS>(R, A.corner[0] + 3 * m, A.corner[1] + 3 * m, A.corner[2] + 3 * m,
                    A.corner[3] + 3 * m, A.strengths[m], A.rc0s[m], A.ages ? A.ages[m] : 0.0,
                    A.nu);
#pragma unroll 1
  for (int k = 0; k < np; ++k) {
    const double* p = A.points + 3 * (p0 + k);
    double v[3] = {0.0, 0.0, 0.0};
    vortex_velocity_rare<LEGS>(R, p[0], p[1], p[2], v, cnt);
    double* o = A.out + ((p0 + k) * A.n_vort + m) * 3;
    o[0] = v[0];
    o[1] = v[1];
    o[2] = v[2];
  }
}

// A thread's own vortex in shared memory, word w of thread t at [w][t] (no bank
// conflicts; the legs' loop indexes corners and legs, which registers cannot).
constexpr int kRingWords = 48;  // 12 coordinates and 4 leg lengths as three floats
struct RingColumn {
  const float* w;
  const double* c;  // [c2 x 4][half c1]
  float near_;
  __device__ __forceinline__ x3::F3 f3(int i) const {
    return x3::F3{w[3 * i * kExpThreads], w[(3 * i + 1) * kExpThreads],
                  w[(3 * i + 2) * kExpThreads]};
  }
  __device__ __forceinline__ x3::F3 corner(int c_, int k) const { return f3(3 * c_ + k); }
  __device__ __forceinline__ x3::F3 r0sq(int l) const { return f3(12 + l); }
  __device__ __forceinline__ double c2(int l) const { return c[l * kExpThreads]; }
  __device__ __forceinline__ double half_c1() const { return c[4 * kExpThreads]; }
  __device__ __forceinline__ float near() const { return near_; }
};

template <int LEGS>
__global__ void __launch_bounds__(kExpThreads) expanded_kernel(SegArgs A, int points_per_cta) {
  extern __shared__ x3::F3 pts[];  // points_per_cta x 3
  __shared__ float words[kRingWords * kExpThreads];
  __shared__ double consts[5 * kExpThreads];
  const int64_t m = static_cast<int64_t>(blockIdx.x) * kExpThreads + threadIdx.x;
  const int64_t p0 = static_cast<int64_t>(blockIdx.y) * points_per_cta;
  const int np = static_cast<int>(min64(points_per_cta, A.n_points - p0));
  bool far = false;  // a point out of the three-float range
  for (int k = threadIdx.x; k < 3 * np; k += kExpThreads) {
    const double x = A.points[3 * p0 + k];
    pts[k] = x3::split_fast(x);
    far = far || !x3_range(x);
  }
  RingColumn col{words + threadIdx.x, consts + threadIdx.x, 0.0f};
  if (m < A.n_vort) {
    VortexRec R;
    RingX3 X;
    prep_vortex<LEGS>(R, A.corner[0] + 3 * m, A.corner[1] + 3 * m, A.corner[2] + 3 * m,
                      A.corner[3] + 3 * m, A.strengths[m], A.rc0s[m],
                      A.ages ? A.ages[m] : 0.0, A.nu);
    prep_x3<LEGS>(X, R);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const x3::F3 v = i < 12 ? X.c[i / 3][i % 3] : X.r0sq[i & 3];
      words[(3 * i) * kExpThreads + threadIdx.x] = v.h;
      words[(3 * i + 1) * kExpThreads + threadIdx.x] = v.m;
      words[(3 * i + 2) * kExpThreads + threadIdx.x] = v.l;
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) consts[l * kExpThreads + threadIdx.x] = X.c2[l];
    consts[4 * kExpThreads + threadIdx.x] = X.half_c1;
    col.near_ = X.near;
  }
  // a CTA with a point or a warp with a vortex out of range takes the general path
  // as a whole: its lanes would have to run both
  const bool general = __syncthreads_or(far) || __any_sync(0xffffffffu, col.near_ > kNoX3);
  if (np <= 0) return;
  int cnt[4] = {0, 0, 0, 0};
  if (m < A.n_vort && general) {
    int c[4] = {0, 0, 0, 0};
    expanded_general<LEGS>(A, m, p0, np, c);
#pragma unroll
    for (int i = 0; i < 4; ++i) cnt[i] = c[i];
  } else if (m < A.n_vort) {
#pragma unroll 1
    for (int k = 0; k < np; ++k) {
      double vx = 0.0, vy = 0.0, vz = 0.0;
      vortex_velocity_x3<LEGS>(col, pts + 3 * k, vx, vy, vz, cnt, [&](double* v, int* c) {
        expanded_rare<LEGS>(A, m, p0 + k, v, c);
      });
      double* o = A.out + ((p0 + k) * A.n_vort + m) * 3;
      o[0] = vx;
      o[1] = vy;
      o[2] = vz;
    }
  }
  flush_counts(cnt, A.counts);
}

// Split of the vortex range for a collapsed call: enough CTAs for about two
// per SM, at least two vortices (and an even count) per split.  The scratch
// holds one row of partial sums per point and split; a run of collapsed_share
// is no shorter than a split, so its CTAs need no more.
int collapsed_splits(int64_t n_points, int64_t n_vort, int64_t* chunk) {
  const int64_t gx = (n_points + kCollThreads - 1) / kCollThreads;
  const int64_t want = 2LL * device_sm_count();
  int64_t s = gx >= want ? 1 : (want + gx - 1) / gx;
  int64_t maxs = (n_vort + 1) / 2;
  if (s > maxs) s = maxs;
  if (s < 1) s = 1;
  int64_t c = (n_vort + s - 1) / s;
  c = (c + 1) & ~int64_t(1);
  s = (n_vort + c - 1) / c;
  *chunk = c;
  return static_cast<int>(s);
}

// Work per CTA: an equal share of all (block, vortex) work for two CTAs per SM, or
// whole blocks where those fill the GPU.  Shares are even, so that with an even
// number of vortices a run starts on a 16-byte boundary of their arrays; from an
// odd vortex on no bulk copy runs, which costs nothing that shows (reading the
// first tile in one go and the others in bulk: 200 points x 101 rings 28.5 us
// against 28.3, 1,000 x 1,001 155.8 against 155.5).
int64_t collapsed_share(int64_t n_points, int64_t n_vort) {
  int64_t chunk = 0;
  if (collapsed_splits(n_points, n_vort, &chunk) == 1) return n_vort;
  const int64_t total = (n_points + kCollThreads - 1) / kCollThreads * n_vort;
  const int64_t want = 2LL * device_sm_count();
  const int64_t even = ((total + want - 1) / want + 1) & ~int64_t(1);
  return even > chunk ? even : chunk;
}

int check_legs(int leg_set) {
  return leg_set == FVX_LEGS_RING || leg_set == FVX_LEGS_CHORDWISE ||
         leg_set == FVX_LEGS_HORSESHOE;
}

}  // namespace

// Internal launcher shared by the device, host and scratch-free entry points.
// host: the inputs are in page-locked host memory, read as they are, and the
// result (out being device memory) and the skip counts go to host->out and
// host->counts there, the device's counters restarting at zero; asked for only
// where segments_collapsed_scratch is not 0.
int segments_collapsed_launch(const double* points, int64_t n_points, const double* br,
                              const double* fr, const double* fl, const double* bl,
                              const double* strengths, const double* r_c0s, const double* ages,
                              double nu, int64_t n_vort, int leg_set, double* out,
                              int64_t* counts, void* scratch, size_t scratch_bytes,
                              const SegmentsHostIO* host, cudaStream_t stream) {
  FVX_ARG_CHECK(check_legs(leg_set), "unknown leg set %d", leg_set);
  FVX_ARG_CHECK(n_points >= 0 && n_vort >= 0, "negative size");
  if (n_points == 0) return FVX_OK;
  FVX_ARG_CHECK(points && out, "null points/out");
  if (n_vort == 0) {
    FVX_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * 3 * n_points, stream));
    return FVX_OK;
  }
  FVX_ARG_CHECK(br && fr && fl && bl && strengths && r_c0s, "null vortex array");
  int64_t chunk = 0;
  const int splits = collapsed_splits(n_points, n_vort, &chunk);
  const size_t need = splits > 1 ? sizeof(double) * 3 * n_points * splits : 0;
  if (need > 0 && (scratch == nullptr || scratch_bytes < need)) {
    set_last_error("segments_collapsed needs %zu scratch bytes, got %zu", need, scratch_bytes);
    return FVX_ERR_SCRATCH;
  }
  SegArgs A;
  A.points = points;
  A.corner[0] = br;
  A.corner[1] = fr;
  A.corner[2] = fl;
  A.corner[3] = bl;
  A.strengths = strengths;
  A.rc0s = r_c0s;
  A.ages = ages;
  A.nu = nu;
  A.n_points = n_points;
  A.n_vort = n_vort;
  const int64_t blocks = (n_points + kCollThreads - 1) / kCollThreads;
  Runs& R = A.runs;
  R.share = collapsed_share(n_points, n_vort);
  R.n_vort = n_vort;
  const int64_t ctas = (blocks * n_vort + R.share - 1) / R.share;
  FVX_ARG_CHECK(ctas < (1LL << 31), "too many target points");
  R.c_last = static_cast<int>((blocks - 1) * n_vort / R.share + 1);
  R.last_rows = static_cast<int>(n_points - (blocks - 1) * kCollThreads);
  A.out = out;
  A.partial = static_cast<double*>(scratch);
  A.counts = counts;
  A.use_tma = host == nullptr && aligned16(br) && aligned16(fr) && aligned16(fl) && aligned16(bl) &&
              aligned16(strengths) && aligned16(r_c0s) && (!ages || aligned16(ages));
  const unsigned grid = static_cast<unsigned>(ctas);
  switch (leg_set) {
    case FVX_LEGS_RING:
      collapsed_kernel<FVX_LEGS_RING><<<grid, kCollSlices * kCollThreads, 0, stream>>>(A);
      break;
    case FVX_LEGS_CHORDWISE:
      collapsed_kernel<FVX_LEGS_CHORDWISE><<<grid, kCollSlices * kCollThreads, 0, stream>>>(A);
      break;
    default:
      collapsed_kernel<FVX_LEGS_HORSESHOE><<<grid, kCollSlices * kCollThreads, 0, stream>>>(A);
      break;
  }
  FVX_LAUNCH_CHECK();
  if (splits > 1) {
    const int64_t lanes = 3 * n_points * kReduceLanes;
    reduce_runs_kernel<<<static_cast<unsigned>((lanes + 255) / 256), 256, 0, stream>>>(
        A.partial, n_points, R, out, host ? host->out : out, counts,
        host ? host->counts : nullptr);
    FVX_LAUNCH_CHECK();
  }
  return FVX_OK;
}

size_t segments_collapsed_scratch(int64_t n_points, int64_t n_vort) {
  if (n_points <= 0 || n_vort <= 0) return 0;
  int64_t chunk = 0;
  const int splits = collapsed_splits(n_points, n_vort, &chunk);
  return splits > 1 ? sizeof(double) * 3 * n_points * splits : 0;
}

int segments_expanded_launch(const double* points, int64_t n_points, const double* br,
                             const double* fr, const double* fl, const double* bl,
                             const double* strengths, const double* r_c0s, const double* ages,
                             double nu, int64_t n_vort, int leg_set, double* out,
                             int64_t* counts, cudaStream_t stream) {
  FVX_ARG_CHECK(check_legs(leg_set), "unknown leg set %d", leg_set);
  FVX_ARG_CHECK(n_points >= 0 && n_vort >= 0, "negative size");
  if (n_points == 0 || n_vort == 0) return FVX_OK;  // (N,M,3) is empty
  FVX_ARG_CHECK(points && out && br && fr && fl && bl && strengths && r_c0s, "null array");
  SegArgs A;
  A.points = points;
  A.corner[0] = br;
  A.corner[1] = fr;
  A.corner[2] = fl;
  A.corner[3] = bl;
  A.strengths = strengths;
  A.rc0s = r_c0s;
  A.ages = ages;
  A.nu = nu;
  A.n_points = n_points;
  A.n_vort = n_vort;
  A.runs = Runs{};
  A.out = out;
  A.partial = nullptr;
  A.counts = counts;
  A.use_tma = 0;
  const int64_t gx = (n_vort + kExpThreads - 1) / kExpThreads;
  // eight CTAs per SM: fewer leave the FP32 pipe waiting, more repeat the prologue.
  // Rings with 4, 6, 8, 10 and 12, us: 200 points x 501 rings 28.9, 28.8, 28.8, 28.7,
  // 40.3; 200 x 3,000 128, 107, 93, 98, 111; 501 x 1,003 96, 83, 83, 86, 97; 1,500 x 501
  // 132, 121, 112, 112, 128; 3,000 x 3,000 1,674, 1,385, 1,305, 1,330, 1,246; horseshoes
  // alike; ten is better at 501 x 3,000 (293, 252, 240, 203, 223)
  const int64_t want = 8LL * device_sm_count();
  int64_t gy = gx >= want ? 1 : (want + gx - 1) / gx;
  if (gy > n_points) gy = n_points;
  int ppc = static_cast<int>((n_points + gy - 1) / gy);
  if (ppc > 512) ppc = 512;
  gy = (n_points + ppc - 1) / ppc;
  FVX_ARG_CHECK(gy <= 65535, "too many target points for one expanded launch");
  dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy));
  size_t smem = sizeof(x3::F3) * 3 * ppc;
  switch (leg_set) {
    case FVX_LEGS_RING:
      expanded_kernel<FVX_LEGS_RING><<<grid, kExpThreads, smem, stream>>>(A, ppc);
      break;
    case FVX_LEGS_CHORDWISE:
      expanded_kernel<FVX_LEGS_CHORDWISE><<<grid, kExpThreads, smem, stream>>>(A, ppc);
      break;
    default:
      expanded_kernel<FVX_LEGS_HORSESHOE><<<grid, kExpThreads, smem, stream>>>(A, ppc);
      break;
  }
  FVX_LAUNCH_CHECK();
  return FVX_OK;
}

}  // namespace fvx

extern "C" {

size_t fvx_segments_collapsed_scratch_bytes(int64_t n_points, int64_t n_vortices, int) {
  return fvx::segments_collapsed_scratch(n_points, n_vortices);
}

int fvx_segments_collapsed(const double* points, int64_t n_points, const double* br,
                           const double* fr, const double* fl, const double* bl,
                           const double* strengths, const double* r_c0s, const double* ages,
                           double nu, int64_t n_vortices, int leg_set, double* out,
                           int64_t* singularity_counts, void* scratch, size_t scratch_bytes,
                           void* stream) {
  return fvx::segments_collapsed_launch(points, n_points, br, fr, fl, bl, strengths, r_c0s,
                                        ages, nu, n_vortices, leg_set, out, singularity_counts,
                                        scratch, scratch_bytes, nullptr,
                                        static_cast<cudaStream_t>(stream));
}

int fvx_segments_expanded(const double* points, int64_t n_points, const double* br,
                          const double* fr, const double* fl, const double* bl,
                          const double* strengths, const double* r_c0s, const double* ages,
                          double nu, int64_t n_vortices, int leg_set, double* out,
                          int64_t* singularity_counts, void* stream) {
  return fvx::segments_expanded_launch(points, n_points, br, fr, fl, bl, strengths, r_c0s,
                                       ages, nu, n_vortices, leg_set, out, singularity_counts,
                                       static_cast<cudaStream_t>(stream));
}

}  // extern "C"
