// Batched bundle adjustment of many small independent problems (triplets, small submodels) in
// one persistent launch.
//
// The reference solves its triplets one after another on one CPU core, 5 LM iterations each
// (SfM/generate_triples/src/generate_triples.cpp:403-415; submodels likewise,
// SfM/generate_submodels_L1/src/generate_submodels_L1.cpp:330-337).  Here one thread block owns
// one problem at a time and runs the whole SparseLevenbergOptimizer::minimize loop
// (V3D/src/Math/v3d_optimization.cpp:719-1250) for it with the reference's semantics: Huber
// weights frozen across a trial, initial lambda = tau * max diagonal, the gradient / update
// stopping tests, the gain ratio, the lambda schedule, the status codes.  Blocks take problems
// from a queue ordered by decreasing size (longest-processing-time first).
//
// Model: StdMetricBundleOptimizer, up to kMaxCams = 4 cameras per problem (reduced system up to
// 24 x 24), any number of points, each point observed by up to kMaxTrack cameras.  Everything
// is FP64.  Per-point quantities are recomputed from the parameters in every pass over the
// points instead of being stored: one pass per iteration linearises and builds the damped reduced
// system on the FP64 tensor cores, a warp solves it, and a second pass takes the step
// (back-substitution, trial points, trial cost with frozen weights).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "lm.cuh"
#include "model.cuh"
#include "structure.cuh"

namespace v3dba {
namespace {

constexpr int kMaxCams = 4;
constexpr int kMaxTrack = 16;

struct BatchDev {
  int count = 0;
  // per problem
  int* cam_off = nullptr;   // first camera of the problem
  int* n_cams = nullptr;
  int* pt_off = nullptr;    // first point
  int* n_pts = nullptr;
  int* order = nullptr;     // processing order (decreasing size)
  double* thr = nullptr;    // Huber threshold
  // per camera (current parameters, updated in place)
  double* R = nullptr;      // 9
  double* T = nullptr;      // 3
  double* K = nullptr;      // 9
  // per point
  double* X = nullptr;      // 3 (current, updated in place)
  double* Xt = nullptr;     // 3 (trial)
  int* ptr = nullptr;       // [total points + 1] observations of global point g
  // per observation (point-major inside each problem)
  double* meas = nullptr;   // 2
  unsigned char* cam = nullptr;  // camera index inside the problem
  double* w = nullptr;      // Huber weights of the last linearisation
  // results
  int* status = nullptr;
  int* iterations = nullptr;
  int* rejected = nullptr;
  double* cost = nullptr;       // cost at the last linearisation
  double* init_cost = nullptr;
  double* lambda_out = nullptr;
  unsigned* queue = nullptr;    // work counter
};

struct BatchOpts {
  double tau, grad_thr, upd_thr;
  int max_iter;
};

template <int NT>
__device__ __forceinline__ double block_max(double v, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_max(v);
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double m = red[0];
  for (int w = 1; w < NT / 32; ++w) m = fmax(m, red[w]);
  __syncthreads();
  return m;
}

struct CamS {
  double R[9], T[3], K[9];
  double f, fy;   // focal lengths of the Jacobian rows: K00 and (K11 / K00) K00
  int affine;     // the last row of K is 0 0 1: the projection divides by the depth itself
};

// ---- one problem per block: the pieces of k_batched_lm -----------------------------------------

// Columns of the per-warp operand tiles: 32 points x 2 residual rows, padded so that the eight rows
// that a fragment load touches fall into different banks (a row is 4 double banks after the last).
constexpr int kTileK = 64, kTileLd = kTileK + 4;

template <int NC>
struct BatchLay {
  static constexpr int kPairs = NC * (NC + 1) / 2;
  static constexpr int kA = NC * 6 * kTileLd;    // A_c, column per (point, residual row)
  static constexpr int kZ = 8 * kTileLd;         // right operand of one camera pair
  static constexpr int kWarp = kA + kZ;          // doubles per warp (the A part also holds its sums)
  static constexpr int kTile = kPairs * 64;      // doubles of a slot's block sums
  static constexpr int kDim = 6 * NC;
  static constexpr int kSld = kDim + 1;
  static_assert(2 * kTile <= kA, "a warp's block sums, of two slots with four warps, take the place of its A tiles");
};

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// One observation at (cam, X): the residual, v = R X, the depth's point and d proj / d XX, whose
// nonzero entries are {P00, P02, P11, P12}.
struct ObsLin {
  double e[2], v[3], P[4];
};
__device__ __forceinline__ void project_obs(const CamS& c, const double X[3], double mx, double my, ObsLin& o) {
#pragma unroll
  for (int r = 0; r < 3; ++r) o.v[r] = c.R[3 * r] * X[0] + c.R[3 * r + 1] * X[1] + c.R[3 * r + 2] * X[2];
  const double y0 = o.v[0] + c.T[0], y1 = o.v[1] + c.T[1], y2 = o.v[2] + c.T[2];
  const double iz = 1.0 / y2;
  double ih = iz;
  if (!c.affine) ih = 1.0 / (c.K[6] * y0 + c.K[7] * y1 + c.K[8] * y2);
  o.e[0] = (c.K[0] * y0 + c.K[1] * y1 + c.K[2] * y2) * ih - mx;
  o.e[1] = (c.K[3] * y0 + c.K[4] * y1 + c.K[5] * y2) * ih - my;
  o.P[0] = c.f * iz;
  o.P[1] = -o.P[0] * y0 * iz;
  o.P[2] = c.fy * iz;
  o.P[3] = -o.P[2] * y1 * iz;
}
__device__ __forceinline__ void weigh(ObsLin& o, double w, double r[2]) {
  r[0] = -w * o.e[0];
  r[1] = -w * o.e[1];
#pragma unroll
  for (int t = 0; t < 4; ++t) o.P[t] *= w;
}
__device__ __forceinline__ void point_block(const CamS& c, const ObsLin& o, double B[2][3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    B[0][q] = o.P[0] * c.R[q] + o.P[1] * c.R[6 + q];
    B[1][q] = o.P[2] * c.R[3 + q] + o.P[3] * c.R[6 + q];
  }
}
__device__ __forceinline__ void camera_block(const ObsLin& o, double A[2][6]) {
  A[0][0] = o.P[0]; A[0][1] = 0.0; A[0][2] = o.P[1];
  A[1][0] = 0.0; A[1][1] = o.P[2]; A[1][2] = o.P[3];
  A[0][3] = o.P[1] * o.v[1];
  A[0][4] = o.P[0] * o.v[2] - o.P[1] * o.v[0];
  A[0][5] = -o.P[0] * o.v[1];
  A[1][3] = o.P[3] * o.v[1] - o.P[2] * o.v[2];
  A[1][4] = -o.P[3] * o.v[0];
  A[1][5] = o.P[2] * o.v[0];
}

__device__ __forceinline__ void add_point(const double B[2][3], const double r[2], double V[6], double gb[3]) {
#pragma unroll
  for (int rr = 0; rr < 2; ++rr) {
    V[0] += B[rr][0] * B[rr][0]; V[1] += B[rr][0] * B[rr][1]; V[2] += B[rr][0] * B[rr][2];
    V[3] += B[rr][1] * B[rr][1]; V[4] += B[rr][1] * B[rr][2]; V[5] += B[rr][2] * B[rr][2];
#pragma unroll
    for (int c = 0; c < 3; ++c) gb[c] += B[rr][c] * r[rr];
  }
}

// (V + lambda I)^-1 by cofactors; *det tells a singular point (0) from a non-finite one.
__device__ __forceinline__ bool invert_point(const double V[6], double lam, double vi[6], double* det_out) {
  const double a0 = V[0] + lam, a3 = V[3] + lam, a5 = V[5] + lam;
  const double c00 = a3 * a5 - V[4] * V[4], c01 = V[2] * V[4] - V[1] * a5, c02 = V[1] * V[4] - V[2] * a3;
  const double det = a0 * c00 + V[1] * c01 + V[2] * c02;
  *det_out = det;
  if (!(det != 0.0) || !isfinite(det)) return false;
  const double id = 1.0 / det;
  vi[0] = c00 * id; vi[1] = c01 * id; vi[2] = c02 * id;
  vi[3] = (a0 * a5 - V[2] * V[2]) * id;
  vi[4] = (V[1] * V[2] - a0 * V[4]) * id;
  vi[5] = (a0 * a3 - V[1] * V[1]) * id;
  return true;
}
__device__ __forceinline__ void mul_sym3(const double vi[6], const double x[3], double y[3]) {
  y[0] = vi[0] * x[0] + vi[1] * x[1] + vi[2] * x[2];
  y[1] = vi[1] * x[0] + vi[3] * x[1] + vi[4] * x[2];
  y[2] = vi[2] * x[0] + vi[4] * x[1] + vi[5] * x[2];
}

__device__ __forceinline__ void store_a(double* Ac, int lane, const double A[2][6]) {
#pragma unroll
  for (int a = 0; a < 6; ++a) *reinterpret_cast<double2*>(Ac + a * kTileLd + 2 * lane) = make_double2(A[0][a], A[1][a]);
}

// acc += A Z^T over the warp's 32 points: rows 0..5 of the left tile against `rows` rows of the right
// one; the other rows are read from `zero`.  Four accumulators in turn (one chain of 16 DMMAs measured
// the same: the other warps of the SM fill it).
__device__ __forceinline__ void tile_product(const double* Ac, const double* Z, const double* zero, int rows, int lane,
                                             double (&acc)[2]) {
  const int r = lane >> 2, k = lane & 3;
  const double* ap = (r < 6 ? Ac + r * kTileLd : zero) + k;
  const double* zp = (r < rows ? Z + r * kTileLd : zero) + k;
  double part[4][2];
#pragma unroll
  for (int t = 0; t < 4; ++t) part[t][0] = part[t][1] = 0.0;
#pragma unroll 1
  for (int s = 0; s < kTileK; s += 16)
#pragma unroll
    for (int t = 0; t < 4; ++t) dmma884(part[t][0], part[t][1], ap[s + 4 * t], zp[s + 4 * t]);
#pragma unroll
  for (int t = 0; t < 2; ++t) acc[t] += (part[0][t] + part[1][t]) + (part[2][t] + part[3][t]);
}

// Z = (delta I - BV_t B_u^T) A_u for the lane's point (zero unless `use`); A_u is read back from the
// lane's own columns of its tile.
__device__ __forceinline__ void store_z(double* Z, const double* Au, int lane, const double BV[2][3], const double Bu[2][3],
                                        bool diag, bool use) {
  double P[2][2];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      P[r][c] = ((diag && r == c) ? 1.0 : 0.0) - (BV[r][0] * Bu[c][0] + BV[r][1] * Bu[c][1] + BV[r][2] * Bu[c][2]);
      if (!use) P[r][c] = 0.0;
    }
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    const double2 u = *reinterpret_cast<const double2*>(Au + a * kTileLd + 2 * lane);
    *reinterpret_cast<double2*>(Z + a * kTileLd + 2 * lane) =
        make_double2(P[0][0] * u.x + P[0][1] * u.y, P[1][0] * u.x + P[1][1] * u.y);
  }
}
__device__ __forceinline__ void store_row(double* Z, int row, int lane, double x, double y) {
  *reinterpret_cast<double2*>(Z + row * kTileLd + 2 * lane) = make_double2(x, y);
}

// Warp Cholesky of the reduced system (order 6 NC, identity beyond the problem's cameras) with the
// right-hand side as one more row, then the back-substitution: lane r keeps row r in registers and a
// step exchanges one column through shared memory.  False when a pivot is not positive.
template <int NC>
__device__ __forceinline__ bool warp_solve(double* S, const double* rhs, double* x, double* colb /* [2][32] */, int n6) {
  constexpr int ND = BatchLay<NC>::kDim, LD = BatchLay<NC>::kSld;
  const int lane = threadIdx.x & 31;
  double row[ND];
#pragma unroll
  for (int c = 0; c < ND; ++c) {
    double v = lane == c ? 1.0 : 0.0;
    if (lane < n6 && c <= lane) v = S[lane * LD + c];
    if (lane == ND) v = c < n6 ? rhs[c] : 0.0;
    row[c] = v;
  }
  bool ok = true;
  double inv_own = 1.0;
#pragma unroll
  for (int k = 0; k < ND; ++k) {
    const double d = __shfl_sync(0xffffffffu, row[k], k);
    if (!(d > 0.0)) ok = false;
    const double inv = rsqrt(d > 0.0 ? d : 1.0);
    if (lane == k) inv_own = inv;
    const double l = row[k] * inv;
    row[k] = l;
    if (k + 1 < ND) {
      double* cb = colb + 32 * (k & 1);   // two buffers: one barrier a step
      cb[lane] = l;
      __syncwarp();
#pragma unroll
      for (int c = k + 1; c < ND; ++c) row[c] -= l * cb[c];
    }
  }
  __syncwarp();
  if (lane < ND) {
#pragma unroll
    for (int c = 0; c < ND; ++c)
      if (c <= lane) S[lane * LD + c] = row[c];
  }
  if (lane == ND) {
#pragma unroll
    for (int c = 0; c < ND; ++c) colb[c] = row[c];
  }
  __syncwarp();
  double y = lane < ND ? colb[lane] : 0.0;
#pragma unroll
  for (int k = 0; k < ND; ++k) row[k] = (lane < k) ? S[k * LD + lane] : 0.0;   // column `lane` of L
#pragma unroll
  for (int k = ND - 1; k >= 0; --k) {
    const double xk = __shfl_sync(0xffffffffu, y * inv_own, k);
    if (lane == k) x[k] = xk;
    y -= row[k] * xk;
  }
  return ok;
}

// One point of a pass: its track, and the measurement of each camera that sees it.  `mask` is empty
// for a track that names a camera twice (it takes the general way) and beyond the last point.
template <int NC>
struct Track {
  double X[3];
  double2 m[NC];
  int o0, n;
  unsigned slot, mask;   // track position of camera c in bits 4c..4c+3 of slot, if bit c of mask
  bool twice;
};
template <int NC>
__device__ __forceinline__ Track<NC> load_track(const BatchDev& b, const double* Xc, int pt0, int M, int j) {
  Track<NC> t;
  const bool in = j < M;
  const size_t g = (size_t)(pt0 + (in ? j : 0));
  t.o0 = in ? b.ptr[g] : 0;
  t.n = in ? b.ptr[g + 1] - t.o0 : 0;
  t.slot = t.mask = 0;
  t.twice = false;
  for (int k = 0; k < t.n; ++k) {
    const int c = b.cam[t.o0 + k];
    t.twice |= (t.mask >> c) & 1u;
    t.mask |= 1u << c;
    t.slot |= (unsigned)k << (4 * c);
  }
  if (t.twice) t.mask = 0;
#pragma unroll
  for (int q = 0; q < 3; ++q) t.X[q] = in ? Xc[3 * g + q] : 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c)
    t.m[c] = ((t.mask >> c) & 1u)
                 ? *reinterpret_cast<const double2*>(b.meas + 2 * (size_t)(t.o0 + (int)((t.slot >> (4 * c)) & 15u)))
                 : make_double2(0.0, 0.0);
  return t;
}

// The sums over a problem's points have one order for every block size: tile c of 32 points belongs to slot
// c % kSlots, one warp sums a slot's tiles in order, and the slots add up as slots_sum has it.  So a problem's
// result does not depend on the threads that its batch gets, nor on the problems beside it.
constexpr int kSlots = 8;   // the warps of the largest block

template <typename F>
__device__ __forceinline__ double slots_sum(F v) {
  return (((v(0) + v(2)) + v(4)) + v(6)) + (((v(1) + v(3)) + v(5)) + v(7));
}
// A warp's sum of per-lane values of the slots.
__device__ __forceinline__ double slots_warp_sum(const double (*v)[32]) {
  const int lane = threadIdx.x & 31;
  return warp_sum(slots_sum([&](int sl) { return v[sl][lane]; }));
}

// One thread block per problem at a time.  A pass over the points gives each warp 32 points, one per
// lane.  The reduced system is a product on the FP64 tensor cores: with residual rows 2p, 2p+1 of a
// point's cameras as the inner dimension, block (i, l) is
//     sum_p A_i^T (delta_il I - B_i (V + lambda I)^-1 B_l^T) A_l,
// so one pass builds U, the Schur complement, the reduced rhs (a seventh column r_i - B_i q) and the
// gradient (an eighth, r_i) from one linearisation of every observation; each warp sums its points in
// eight-by-eight accumulators and the slots' sums are added in order (deterministic, no atomics).
// Bound by FP64 latency: 14 KB of operand tiles per warp and 168 registers (a few spill: 60 bytes a thread
// with three cameras, about 550 with four) leave 12 warps per SM, the FP64 pipe is active 24% and the DMMA
// pipe 16% of the cycles.  Of the 2.2 ms that 4096 triplets of 50-800 points take for 4 iterations the products
// are 0.8, the step pass 0.5, the solve 0.25 (timed by leaving each out).  Loading the next tile's tracks
// during the products took 24 registers more and, with the slots, 2.43 ms.  A pass per camera pair that linearised each point again for it (39
// linearisations per point and iteration instead of 6) took 6.7 ms; the same for 61 triplets 1.29 ms
// against 0.17.
template <int NT, int NC>
__global__ void __launch_bounds__(NT, NT > 128 ? 1 : 384 / NT) k_batched_lm(BatchDev b, BatchOpts o, int first, int last) {
  using L = BatchLay<NC>;
  constexpr int NW = NT / 32, ND = L::kDim, LD = L::kSld, OWN = kSlots / NW;   // slots of a warp
  extern __shared__ double dyn[];   // [NW][L::kWarp]
  __shared__ CamS cams[NC], tcams[NC];
  __shared__ double S[ND * LD], rhs[ND], da[ND], ga[ND], udiag[ND], colb[64], red[NW], zrow[kTileK];
  __shared__ double sc[8];    // 0 err, 1 lambda, 2 nu, 3 newErr, 4 d2, 5 dg, 6 plen
  __shared__ int si[8];       // 0 problem, 1 stop, 3 fail, 4 accept, 5 status, 7 rejected
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* Aw = dyn + wid * L::kWarp;
  double* Zw = Aw + L::kA;
  double(*part)[kSlots][32] = reinterpret_cast<double(*)[kSlots][32]>(dyn);   // per-lane sums of the slots
  // The total of what the warps left at v for their slots, one (of several, summed) or two `second` apart.
  auto slots_total = [&](const double* v, int second) {
    if (OWN > 2) return v[0] + v[L::kWarp];
    return slots_sum([&](int sl) { return v[(sl % NW) * L::kWarp + (sl / NW) * second]; });
  };
  for (int e = tid; e < kTileK; e += NT) zrow[e] = 0.0;   // read after the barrier below
  for (;;) {
    if (tid == 0) {
      const unsigned slot = atomicAdd(b.queue, 1u);
      si[0] = (first + (int)slot < last) ? b.order[first + slot] : -1;
    }
    __syncthreads();
    const int p = si[0];
    if (p < 0) return;
    const int N = b.n_cams[p], M = b.n_pts[p], c0 = b.cam_off[p], pt0 = b.pt_off[p];
    const double thr = b.thr[p];
    const int chunks = (M + 31) / 32;
    const double* Xc = b.X;   // current and trial points; an accepted step swaps them
    double* Xt = b.Xt;
    if (tid < N) {
      CamS& c = cams[tid];
      for (int q = 0; q < 9; ++q) { c.R[q] = b.R[9 * (c0 + tid) + q]; c.K[q] = b.K[9 * (c0 + tid) + q]; }
      for (int q = 0; q < 3; ++q) c.T[q] = b.T[3 * (c0 + tid) + q];
      c.f = c.K[0];
      c.fy = (c.K[4] / c.K[0]) * c.K[0];
      c.affine = c.K[6] == 0.0 && c.K[7] == 0.0 && c.K[8] == 1.0;
    }
    // cached parameter length (v3d_metricbundle.h:37-45)
    {
      for (int sl = wid; sl < kSlots; sl += NW) {
        double v = 0.0;
        for (int j = 32 * sl + lane; j < M; j += 32 * kSlots) {
          const double* X = Xc + 3 * (size_t)(pt0 + j);
          v += X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
        }
        if (sl == 0 && lane < N) {
          const double* T = b.T + 3 * (size_t)(c0 + lane);
          v += T[0] * T[0] + T[1] * T[1] + T[2] * T[2] + 3.0;
        }
        part[0][sl][lane] = v;
      }
      __syncthreads();
      const double s = wid == 0 ? slots_warp_sum(part[0]) : 0.0;
      if (tid == 0) {
        sc[6] = sqrt(s);
        sc[1] = 1e-3;   // lambda of a new optimizer object
        sc[2] = 2.0;    // _nu
        si[1] = 0; si[5] = V3DBA_STATUS_TIMEOUT; si[7] = 0;
      }
      __syncthreads();
    }
    int it = 0;
    for (it = 0; it < o.max_iter; ++it) {
      // Sums of one pass over the points.  mode 0: the first iteration's linearisation, for the
      // initial lambda (diagonal of U beside the gradient); mode 1: the damped reduced system.
      // After a rejected step the parameters, and so the weights and sums, are the same again.
      for (int mode = it == 0 ? 0 : 1; mode < 2; ++mode) {
        const double lam = sc[1];
        double acc[L::kPairs][2], err = 0.0, gbmax = 0.0, vdmax = -1e30;
#pragma unroll
        for (int t = 0; t < L::kPairs; ++t) acc[t][0] = acc[t][1] = 0.0;
        // The sums of the warp's earlier slots, one after another (two warps) or each for itself (four); kept in
        // memory, as they are touched once a slot.
        volatile double kept[L::kPairs][2], kept_err;
#pragma unroll 1
        for (int sl = wid; sl < kSlots; sl += NW) {
          if (OWN > 1 && sl > wid && sl < chunks) {
#pragma unroll
            for (int t = 0; t < L::kPairs; ++t)
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                kept[t][u] = OWN > 2 && sl > wid + NW ? kept[t][u] + acc[t][u] : acc[t][u];
                acc[t][u] = 0.0;
              }
            kept_err = OWN > 2 && sl > wid + NW ? kept_err + err : err;
            err = 0.0;
          }
#pragma unroll 1
          for (int ch = sl; ch < chunks; ch += kSlots) {
            Track<NC> tr = load_track<NC>(b, Xc, pt0, M, 32 * ch + lane);
            const double X[3] = {tr.X[0], tr.X[1], tr.X[2]};
            const int o0 = tr.o0, n = tr.n;
            const bool twice = tr.twice;
            double V[6] = {0, 0, 0, 0, 0, 0}, gb[3] = {0, 0, 0}, B[NC][2][3], r[NC][2];
            // no branch on the presence of a camera (with branches it measured the same)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              if (c >= N) {
#pragma unroll
                for (int q = 0; q < 3; ++q) B[c][0][q] = B[c][1][q] = 0.0;
                r[c][0] = r[c][1] = 0.0;
                continue;
              }
              const bool has = (tr.mask >> c) & 1u;
              ObsLin ol;
              project_obs(cams[c], X, tr.m[c].x, tr.m[c].y, ol);
              const double w = huber_weight(thr, ol.e);
              if (has) b.w[o0 + (int)((tr.slot >> (4 * c)) & 15u)] = w;
              weigh(ol, w, r[c]);
              if (!has) ol.P[0] = ol.P[1] = ol.P[2] = ol.P[3] = r[c][0] = r[c][1] = 0.0;
              const double cost = w * w * (ol.e[0] * ol.e[0] + ol.e[1] * ol.e[1]);
              err += has ? cost : 0.0;
              point_block(cams[c], ol, B[c]);
              double A[2][6];
              camera_block(ol, A);
              add_point(B[c], r[c], V, gb);
              store_a(Aw + c * 6 * kTileLd, lane, A);
            }
            if (tr.mask) {
              gbmax = fmax(gbmax, fmax(fabs(gb[0]), fmax(fabs(gb[1]), fabs(gb[2]))));
              vdmax = fmax(vdmax, fmax(V[0], fmax(V[3], V[5])));
            }
            // without the elimination (mode 0) the same product is U, and its right-hand side the gradient
            double vi[6] = {0, 0, 0, 0, 0, 0}, q[3], det;
            bool ok = true;
            if (mode == 1) {
              ok = invert_point(V, lam, vi, &det);
              const bool dead = !ok && !isfinite(det);
              // A point at infinity enters the gradient (column 7 of the cameras' own blocks), where it is no
              // number unless the camera sees it well, but not the system.
              if (__any_sync(0xffffffffu, dead)) {
                const double zero2[2][6] = {};
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                  if (c >= N) continue;
                  for (int a = 0; a < 6; ++a) {
                    const double2 u = *reinterpret_cast<const double2*>(Aw + (6 * c + a) * kTileLd + 2 * lane);
                    const double g = warp_sum(dead ? u.x * r[c][0] + u.y * r[c][1] : 0.0);
                    if (lane == 4 * a + 3) acc[c * NC - c * (c - 1) / 2][1] += g;
                  }
                  if (dead) {
                    store_a(Aw + c * 6 * kTileLd, lane, zero2);
                    r[c][0] = r[c][1] = 0.0;
                  }
                }
              }
            }
            mul_sym3(vi, gb, q);
            int pr = 0;
#pragma unroll
            for (int i = 0; i < NC; ++i) {
              double BV[2][3];
              mul_sym3(vi, B[i][0], BV[0]);
              mul_sym3(vi, B[i][1], BV[1]);
#pragma unroll
              for (int l = i; l < NC; ++l, ++pr) {
                if (l >= N || (l != i && mode == 0)) continue;
                store_z(Zw, Aw + l * 6 * kTileLd, lane, BV, B[l], i == l, ok);
                if (i == l) {
                  const double e0 = r[i][0] - (B[i][0][0] * q[0] + B[i][0][1] * q[1] + B[i][0][2] * q[2]);
                  const double e1 = r[i][1] - (B[i][1][0] * q[0] + B[i][1][1] * q[1] + B[i][1][2] * q[2]);
                  store_row(Zw, 6, lane, ok ? e0 : 0.0, ok ? e1 : 0.0);
                  store_row(Zw, 7, lane, r[i][0], r[i][1]);
                }
                __syncwarp();
                tile_product(Aw + i * 6 * kTileLd, Zw, zrow, i == l ? 8 : 6, lane, acc[pr]);
                __syncwarp();
              }
            }
            // tracks that name a camera twice: their observation pairs one per round and point
            if (__any_sync(0xffffffffu, twice)) {
              double vi[6] = {0, 0, 0, 0, 0, 0}, q[3] = {0, 0, 0};
              bool ok = false, dead = false;
              const int nt = twice ? n : 0;
              {
                double V2[6] = {0, 0, 0, 0, 0, 0}, gb2[3] = {0, 0, 0}, det;
                for (int t = 0; t < nt; ++t) {
                  const int k = o0 + t;
                  const CamS& cm = cams[b.cam[k]];
                  ObsLin ol;
                  double rr[2], Bt[2][3];
                  project_obs(cm, X, b.meas[2 * (size_t)k], b.meas[2 * (size_t)k + 1], ol);
                  const double w = huber_weight(thr, ol.e);
                  b.w[k] = w;
                  err += w * w * (ol.e[0] * ol.e[0] + ol.e[1] * ol.e[1]);
                  weigh(ol, w, rr);
                  point_block(cm, ol, Bt);
                  add_point(Bt, rr, V2, gb2);
                }
                if (twice) {
                  gbmax = fmax(gbmax, fmax(fabs(gb2[0]), fmax(fabs(gb2[1]), fabs(gb2[2]))));
                  vdmax = fmax(vdmax, fmax(V2[0], fmax(V2[3], V2[5])));
                  ok = invert_point(V2, lam, vi, &det);
                  dead = mode == 1 && !ok && !isfinite(det);
                  mul_sym3(vi, gb2, q);
                }
              }
#pragma unroll 1
              for (int i = 0; i < N; ++i)
#pragma unroll 1
                for (int l = i; l < N; ++l) {
                  if (mode == 0 && l != i) continue;
                  double* Ac = Aw + i * 6 * kTileLd;
                  int t = 0, u = -1;
                  for (;;) {
                    // the lane's next pair (t, u) of an observation in camera i with one in camera l; the
                    // diagonal's U term and gradient come with t == u (mode 0 has only those)
                    bool have = false;
                    while (!have) {
                      if (++u >= nt) { u = 0; ++t; }
                      if (t >= nt) break;
                      have = b.cam[o0 + t] == i && b.cam[o0 + u] == l && (mode == 1 || t == u);
                    }
                    if (!__any_sync(0xffffffffu, have)) break;
                    const int at = i * NC - i * (i - 1) / 2 + (l - i);
                    double At[2][6] = {}, Z[8][2] = {};
                    if (i == l && __any_sync(0xffffffffu, have && dead && t == u)) {   // (as above)
                      double g[6] = {};
                      if (have && dead && t == u) {
                        double rt[2];
                        ObsLin ol;
                        project_obs(cams[i], X, b.meas[2 * (size_t)(o0 + t)], b.meas[2 * (size_t)(o0 + t) + 1], ol);
                        weigh(ol, b.w[o0 + t], rt);
                        camera_block(ol, At);
                        for (int a = 0; a < 6; ++a) {
                          g[a] = At[0][a] * rt[0] + At[1][a] * rt[1];
                          At[0][a] = At[1][a] = 0.0;
                        }
                      }
                      for (int a = 0; a < 6; ++a) {
                        const double v = warp_sum(g[a]);
#pragma unroll
                        for (int pr = 0; pr < L::kPairs; ++pr)
                          if (pr == at && lane == 4 * a + 3) acc[pr][1] += v;
                      }
                    }
                    if (have && !dead) {
                      double Au[2][6], Bt[2][3], Bu[2][3], rt[2], ru[2], BV[2][3];
                      ObsLin ol;
                      project_obs(cams[i], X, b.meas[2 * (size_t)(o0 + t)], b.meas[2 * (size_t)(o0 + t) + 1], ol);
                      weigh(ol, b.w[o0 + t], rt);
                      point_block(cams[i], ol, Bt);
                      camera_block(ol, At);
                      project_obs(cams[l], X, b.meas[2 * (size_t)(o0 + u)], b.meas[2 * (size_t)(o0 + u) + 1], ol);
                      weigh(ol, b.w[o0 + u], ru);
                      point_block(cams[l], ol, Bu);
                      camera_block(ol, Au);
                      mul_sym3(vi, Bt[0], BV[0]);
                      mul_sym3(vi, Bt[1], BV[1]);
                      for (int rr = 0; rr < 2; ++rr) {
                        double P[2];
                        for (int cc = 0; cc < 2; ++cc)
                          P[cc] = ((t == u && rr == cc) ? 1.0 : 0.0) -
                                  (mode == 1 ? BV[rr][0] * Bu[cc][0] + BV[rr][1] * Bu[cc][1] + BV[rr][2] * Bu[cc][2] : 0.0);
                        const bool use = mode == 0 || ok;
                        for (int a = 0; a < 6; ++a) Z[a][rr] = use ? P[0] * Au[0][a] + P[1] * Au[1][a] : 0.0;
                        if (t == u) {
                          if (mode == 1 && ok) Z[6][rr] = rt[rr] - (Bt[rr][0] * q[0] + Bt[rr][1] * q[1] + Bt[rr][2] * q[2]);
                          Z[7][rr] = rt[rr];
                        }
                      }
                    }
                    store_a(Ac, lane, At);
                    for (int a = 0; a < 8; ++a) store_row(Zw, a, lane, Z[a][0], Z[a][1]);
                    __syncwarp();
                    double add[2] = {0.0, 0.0};
                    tile_product(Ac, Zw, zrow, 8, lane, add);
#pragma unroll
                    for (int pr = 0; pr < L::kPairs; ++pr)
                      if (pr == at) { acc[pr][0] += add[0]; acc[pr][1] += add[1]; }
                    __syncwarp();
                  }
                }
            }
          }
        }
        // the slots' sums
        __syncwarp();
        const bool more = OWN > 1 && wid + NW < chunks;   // something was kept
#pragma unroll
        for (int t = 0; t < L::kPairs; ++t) {
          double2* at = reinterpret_cast<double2*>(Aw + t * 64 + (lane >> 2) * 8 + 2 * (lane & 3));
          if (OWN == 2) {
            at[0] = more ? make_double2(kept[t][0], kept[t][1]) : make_double2(acc[t][0], acc[t][1]);
            at[L::kTile / 2] = more ? make_double2(acc[t][0], acc[t][1]) : make_double2(0.0, 0.0);
          } else {
            at[0] = more ? make_double2(kept[t][0] + acc[t][0], kept[t][1] + acc[t][1]) : make_double2(acc[t][0], acc[t][1]);
          }
        }
        if (OWN == 2) {
          Zw[lane] = more ? kept_err : err;
          Zw[32 + lane] = more ? err : 0.0;
        } else {
          Zw[lane] = more ? kept_err + err : err;
        }
        const double gm = block_max<NT>(gbmax, red);
        const double vm = block_max<NT>(vdmax, red);
        for (int e = tid; e < L::kTile; e += NT) {
          const double s = slots_total(dyn + e, L::kTile);
          int i = 0, t = e >> 6;
          while (t >= NC - i) { t -= NC - i; ++i; }
          const int l = i + t, a = (e >> 3) & 7, c = e & 7;
          if (a >= 6 || l >= N) continue;
          // S_il[a][c] is element (6l + c, 6i + a); only the lower triangle is stored
          if (c < 6) {
            if (mode == 0) { if (i == l && a == c) udiag[6 * i + a] = s; }
            else if (i != l || c >= a) S[(6 * l + c) * LD + 6 * i + a] = s + ((i == l && a == c) ? lam : 0.0);
          } else if (i == l) {
            if (c == 7) ga[6 * i + a] = s;
            else if (mode == 1) rhs[6 * i + a] = s;
          }
        }
        __syncthreads();
        if (wid == 0) {
          const double errs = warp_sum(slots_total(dyn + L::kA + lane, 32));
          // (fmax leaves out what is no number)
          double gx = lane < 6 * N ? fmax(fabs(ga[lane]), 0.0) : 0.0;
          double dx = (mode == 0 && lane < 6 * N) ? fmax(udiag[lane], -1e30) : -1e30;
          gx = warp_max(gx);
          dx = warp_max(dx);
          if (lane == 0) {
            sc[0] = errs;
            if (fmax(gx, gm) < o.grad_thr) { si[5] = V3DBA_STATUS_CONVERGED; si[1] = 1; }
            if (mode == 0) {
              if (b.init_cost) b.init_cost[p] = errs;
              if (!si[1]) sc[1] = o.tau * fmax(dx, vm);
            }
          }
        }
        __syncthreads();
        if (si[1]) break;
      }
      if (si[1]) break;
      const double lam = sc[1];
      if (wid == 0) {
        const bool ok = warp_solve<NC>(S, rhs, da, colb, 6 * N);
        if (lane == 0) si[3] = ok ? 0 : 1;
        __syncwarp();
        if (ok && lane < N) {   // trial cameras
          CamS c = cams[lane];
          const double* d = da + 6 * lane;
          c.T[0] += d[0]; c.T[1] += d[1]; c.T[2] += d[2];
          rotate_update(d + 3, c.R);
          tcams[lane] = c;
        }
      }
      __syncthreads();
      if (!si[3]) {
        // ---- points: back-substitution, trial points, trial cost with frozen weights ----
        for (int sl = wid; sl < kSlots; sl += NW) {
          double nerr = 0.0, d2 = 0.0, dg = 0.0;
          for (int j = 32 * sl + lane; j < M; j += 32 * kSlots) {
            const size_t g = (size_t)(pt0 + j);
            const int o0 = b.ptr[g], n = b.ptr[g + 1] - o0;
            const double X[3] = {Xc[3 * g], Xc[3 * g + 1], Xc[3 * g + 2]};
            double V[6] = {0, 0, 0, 0, 0, 0}, gb[3] = {0, 0, 0}, s[3] = {0, 0, 0}, vi[6], db[3] = {0, 0, 0}, det;
            for (int t = 0; t < n; ++t) {
              const int k = o0 + t;
              const int c = b.cam[k];
              const double2 m = *reinterpret_cast<const double2*>(b.meas + 2 * (size_t)k);
              const CamS& cm = cams[c];
              ObsLin ol;
              double r[2], B[2][3];
              project_obs(cm, X, m.x, m.y, ol);
              weigh(ol, b.w[k], r);
              point_block(cm, ol, B);
              add_point(B, r, V, gb);
              // A da = P (dT + omega x v)
              const double* d = da + 6 * c;
              const double t0 = d[0] + (d[4] * ol.v[2] - d[5] * ol.v[1]);
              const double t1 = d[1] + (d[5] * ol.v[0] - d[3] * ol.v[2]);
              const double t2 = d[2] + (d[3] * ol.v[1] - d[4] * ol.v[0]);
              const double a0 = ol.P[0] * t0 + ol.P[1] * t2, a1 = ol.P[2] * t1 + ol.P[3] * t2;
#pragma unroll
              for (int q = 0; q < 3; ++q) s[q] += B[0][q] * a0 + B[1][q] * a1;
            }
            if (invert_point(V, lam, vi, &det)) {
#pragma unroll
              for (int q = 0; q < 3; ++q) s[q] = gb[q] - s[q];
              mul_sym3(vi, s, db);
              d2 += db[0] * db[0] + db[1] * db[1] + db[2] * db[2];
              dg += db[0] * gb[0] + db[1] * gb[1] + db[2] * gb[2];
            }
            const double Xn[3] = {X[0] + db[0], X[1] + db[1], X[2] + db[2]};
            Xt[3 * g] = Xn[0];
            Xt[3 * g + 1] = Xn[1];
            Xt[3 * g + 2] = Xn[2];
            for (int t = 0; t < n; ++t) {
              const int k = o0 + t;
              const double2 m = *reinterpret_cast<const double2*>(b.meas + 2 * (size_t)k);
              ObsLin ol;
              project_obs(tcams[b.cam[k]], Xn, m.x, m.y, ol);
              const double wk = b.w[k];
              nerr += wk * wk * (ol.e[0] * ol.e[0] + ol.e[1] * ol.e[1]);
            }
          }
          part[0][sl][lane] = nerr;
          part[1][sl][lane] = d2;
          part[2][sl][lane] = dg;
        }
        __syncthreads();
        if (wid == 0) {
          const double dl = lane < 6 * N ? da[lane] : 0.0, gl = lane < 6 * N ? ga[lane] : 0.0;
          const double nerr = slots_warp_sum(part[0]);
          const double d2 = slots_warp_sum(part[1]) + warp_sum(dl * dl), dg = slots_warp_sum(part[2]) + warp_sum(dl * gl);
          if (lane == 0) {
            si[4] = 0;
            if (sqrt(d2) < o.upd_thr * (sc[6] + o.upd_thr)) {
              si[5] = V3DBA_STATUS_SMALL_UPDATE;
              si[1] = 1;
            } else {
              const double rho = (sc[0] - nerr) / (lam * d2 + dg);
              if (rho > 0.0) {
                const double r = 2.0 * rho - 1.0;
                sc[1] = fmax(lam * fmax(1.0 / 3.0, 1.0 - r * r * r), 1e-10);
                si[4] = 1;
              }
            }
          }
        }
      } else if (tid == 0) {
        si[4] = 0;
      }
      __syncthreads();
      if (si[1]) break;
      if (si[4]) {
        if (tid < N) cams[tid] = tcams[tid];
        double* const was = const_cast<double*>(Xc);
        Xc = Xt;
        Xt = was;
        if (tid == 0) sc[2] = 2.0;
      } else if (tid == 0) {
        sc[1] *= sc[2];
        sc[2] *= 2.0;
        si[7]++;
      }
      __syncthreads();
    }
    // write back
    if (Xc != b.X)
      for (int e = tid; e < 3 * M; e += NT) b.X[3 * (size_t)pt0 + e] = Xc[3 * (size_t)pt0 + e];
    if (tid < N) {
      for (int q = 0; q < 9; ++q) b.R[9 * (c0 + tid) + q] = cams[tid].R[q];
      for (int q = 0; q < 3; ++q) b.T[3 * (c0 + tid) + q] = cams[tid].T[q];
    }
    if (tid == 0) {
      b.status[p] = si[5];
      b.iterations[p] = it;
      b.rejected[p] = si[7];
      b.cost[p] = sc[0];
      b.lambda_out[p] = sc[1];
    }
    __syncthreads();
  }
}

// ---- layout of a batch from flat arrays ----------------------------------------------------------

constexpr int kBadIndex = 1, kUnsorted = 2, kLongTrack = 4;

// One block per problem: the camera bytes and the start of every point's observations, for problems whose
// observations are in point order; *flag tells an index out of range and observations out of order
// (nothing is written through either).
__global__ void __launch_bounds__(256) k_batch_layout(BatchDev b, const int* __restrict__ obs_off,
                                                      const int* __restrict__ view, const int* __restrict__ point,
                                                      int* flag) {
  const int p = blockIdx.x;
  const int o0 = obs_off[p], n = obs_off[p + 1] - o0, N = b.n_cams[p], M = b.n_pts[p];
  int* ptr = b.ptr + b.pt_off[p];
  int bad = 0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const int v = view[o0 + k], j = point[o0 + k], before = k > 0 ? point[o0 + k - 1] : -1;
    const bool ok = (unsigned)v < (unsigned)N && (unsigned)j < (unsigned)M;
    if (!ok) bad |= kBadIndex;
    if (j < before) bad |= kUnsorted;
    b.cam[o0 + k] = (unsigned char)v;
    if (ok && before >= -1 && j >= before)
      for (int t = before + 1; t <= j; ++t) ptr[t] = o0 + k;
    if (ok && k == n - 1)
      for (int t = j + 1; t <= M; ++t) ptr[t] = o0 + n;   // (the next problem's first point starts there too)
  }
  if (n == 0)
    for (int t = threadIdx.x; t <= M; t += blockDim.x) ptr[t] = o0;
  if (bad) atomicOr(flag, bad);
}

__global__ void __launch_bounds__(256) k_batch_tracks(const int* __restrict__ ptr, int n, int* flag) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n && ptr[j + 1] - ptr[j] > kMaxTrack) atomicOr(flag, kLongTrack);
}

}  // namespace
}  // namespace v3dba

using namespace v3dba;

// ---- host ----------------------------------------------------------------------------------

struct v3dba_batch_s {
  BatchDev d;
  std::vector<void*> allocs;
  std::vector<int> h_cam_off, h_n_cams, h_pt_off, h_n_pts, h_order, h_size;
  int total_cams = 0, total_pts = 0, total_obs = 0;
  int max_cams = 0;               // cameras of the largest problem
  double* d_init = nullptr;       // initial R, T, X (for reset)
  CallRes res;                    // owns the stream and the events
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int small_threads = 0, large_threads = 0;   // block sizes: set or autotuned, else 0 (default_threads)
  int split = 0;                  // problems [0, split) of the order use large_threads
};

namespace {

template <typename T>
int balloc(v3dba_batch_t h, T** p, size_t n) {
  // stream-ordered, from the device's pool (which keeps what a destroyed batch freed): a batch
  // created per call does not pay cudaMalloc / cudaFree each time
  void* q = nullptr;
  int rc0 = ensure_pool();
  if (rc0) return rc0;
  if (injected_alloc_failure()) return V3DBA_ERR_OUT_OF_MEMORY;
  cudaError_t e = cudaMallocAsync(&q, std::max<size_t>(n, 1) * sizeof(T), h->stream);
  if (e != cudaSuccess) { cudaGetLastError(); return V3DBA_ERR_OUT_OF_MEMORY; }
  h->allocs.push_back(q);
  *p = static_cast<T*>(q);
  return V3DBA_OK;
}

template <typename T>
int bupload(v3dba_batch_t h, T** p, const std::vector<T>& v) {
  int rc = balloc(h, p, v.size());
  if (rc) return rc;
  // the host vector outlives the copy: v3dba_batch_create synchronises the stream before returning
  if (!v.empty()) V3DBA_CUDA_TRY(cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
  return V3DBA_OK;
}

void batch_free(v3dba_batch_t h) {
  if (!h) return;
  if (h->stream)
    for (void* p : h->allocs) cudaFreeAsync(p, h->stream);
  h->res.release();
  delete h;
}

struct BatchKernel {
  void (*fn)(BatchDev, BatchOpts, int, int);
  size_t smem;
};
template <int NT, int NC>
BatchKernel batch_kernel_of() {
  return {k_batched_lm<NT, NC>, sizeof(double) * (NT / 32) * BatchLay<NC>::kWarp};
}
// Triplets (three cameras, the usual problem) have their own instances: a fourth camera costs four
// more camera pairs of accumulators and a third more shared memory per warp.
BatchKernel batch_kernel(int threads, int max_cams) {
  if (max_cams <= 3)
    return threads == 64 ? batch_kernel_of<64, 3>() : threads == 128 ? batch_kernel_of<128, 3>() : batch_kernel_of<256, 3>();
  return threads == 64 ? batch_kernel_of<64, 4>() : threads == 128 ? batch_kernel_of<128, 4>() : batch_kernel_of<256, 4>();
}

// Threads per problem of a batch that sets no schedule; they set the time alone, not the results.  A problem's
// passes take time in inverse proportion to its warps as far as it has tiles of 32 points for them, but the
// 256-thread instance runs one block per SM where the others keep 12 warps.  Measured (4 iterations, triplets
// of 20-90, 50-300 and 50-800 points; ms with 64 / 128 / 256 threads), the lines lie where the best changes:
//    148 problems  .103 .075 .066   .223 .137 .100   .488 .285 .170
//    296           .113 .079 .123   .236 .164 .156   .510 .327 .227
//    420           .130 .089 .177   .270 .186 .217   .578 .378 .325
//    500           .131 .141 .230   .279 .186 .252   .608 .382 .381
//   1000           .170 .214 .400   .338 .328 .463   .748 .565 .706
//   1184           .194 .225 .464   .354 .371 .547   .751 .661 .823
//   4096           .561 .729 1.57   1.16 1.22 1.88   2.24 2.19 2.88
// With four cameras the second line is the same, and from 256 points a problem on 256 threads are the best
// at every count (50-800 points, 600 problems 1.03 .661 .626, 4096 4.16 4.24 3.95).
int default_threads(int count, int sms, int points, int max_cams) {
  const int per_sm = (count + sms - 1) / sms;
  if (points >= 256) return per_sm <= 3 || max_cams > 3 ? 256 : 128;
  if (points >= 128) return per_sm <= 2 ? 256 : per_sm <= 7 ? 128 : 64;
  return per_sm <= 1 ? 256 : per_sm <= 3 ? 128 : 64;
}

int batch_resources(v3dba_batch_t h) {
  const int rc = h->res.acquire();
  h->stream = h->res.st;
  h->ev0 = h->res.ev0;
  h->ev1 = h->res.ev1;
  return rc;
}

int launch_range(v3dba_batch_t h, int threads, int first, int last, const BatchOpts& o) {
  if (last <= first) return V3DBA_OK;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (threads == 0) threads = default_threads(last - first, sms, h->total_pts / h->d.count, h->max_cams);
  V3DBA_CUDA_TRY(cudaMemsetAsync(h->d.queue, 0, sizeof(unsigned), h->stream));
  const BatchKernel k = batch_kernel(threads, h->max_cams);
  V3DBA_CUDA_TRY(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem));
  int per_sm = 1;
  V3DBA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.fn, threads, k.smem));
  const int grid = std::max(1, std::min(last - first, sms * std::max(per_sm, 1)));
  k.fn<<<grid, threads, k.smem, h->stream>>>(h->d, o, first, last);
  V3DBA_LAUNCH_CHECK();
  return V3DBA_OK;
}

int batch_run(v3dba_batch_t h, const v3dba_options* opts) {
  BatchOpts o;
  o.tau = opts->tau;
  o.grad_thr = opts->gradient_threshold;
  o.upd_thr = opts->update_threshold;
  o.max_iter = opts->max_iterations;
  int rc = launch_range(h, h->large_threads, 0, h->split, o);
  if (rc) return rc;
  return launch_range(h, h->small_threads, h->split, h->d.count, o);
}

}  // namespace

extern "C" {

int v3dba_batch_create(const v3dba_problem* problems, int count, v3dba_batch_t* out) {
  if (!problems || count <= 0 || !out) return V3DBA_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  int total_cams = 0, total_pts = 0, total_obs = 0;
  for (int p = 0; p < count; ++p) {
    const v3dba_problem& q = problems[p];
    if (q.model != V3DBA_MODEL_STD) return V3DBA_ERR_UNSUPPORTED;
    if (q.n_cameras <= 0 || q.n_cameras > kMaxCams || q.n_points < 0 || q.n_measurements < 0) return V3DBA_ERR_UNSUPPORTED;
    if (!q.K || !q.R || !q.T || (q.n_points && !q.X) || (q.n_measurements && (!q.measurements || !q.view || !q.point)))
      return V3DBA_ERR_INVALID_ARGUMENT;
    if (!(q.inlier_threshold > 0.0)) return V3DBA_ERR_INVALID_INPUT;
    std::vector<int> cnt(q.n_points, 0);
    for (int k = 0; k < q.n_measurements; ++k) {
      if (q.view[k] < 0 || q.view[k] >= q.n_cameras || q.point[k] < 0 || q.point[k] >= q.n_points) return V3DBA_ERR_INVALID_INPUT;
      if (++cnt[q.point[k]] > kMaxTrack) return V3DBA_ERR_UNSUPPORTED;
      if (!std::isfinite(q.measurements[2 * k]) || !std::isfinite(q.measurements[2 * k + 1])) return V3DBA_ERR_INVALID_INPUT;
    }
    for (int t = 0; t < 9 * q.n_cameras; ++t)
      if (!std::isfinite(q.K[t]) || !std::isfinite(q.R[t])) return V3DBA_ERR_INVALID_INPUT;
    for (int t = 0; t < 3 * q.n_points; ++t)
      if (!std::isfinite(q.X[t])) return V3DBA_ERR_INVALID_INPUT;
    total_cams += q.n_cameras;
    total_pts += q.n_points;
    total_obs += q.n_measurements;
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return V3DBA_ERR_NO_DEVICE; }
  v3dba_batch_t h = new (std::nothrow) v3dba_batch_s();
  if (!h) return V3DBA_ERR_OUT_OF_MEMORY;
  h->total_cams = total_cams; h->total_pts = total_pts; h->total_obs = total_obs;
  std::vector<double> R(9 * (size_t)total_cams), T(3 * (size_t)total_cams), K(9 * (size_t)total_cams);
  std::vector<double> X(3 * (size_t)total_pts), meas(2 * (size_t)total_obs), thr(count);
  std::vector<int> ptr(total_pts + 1, 0);
  std::vector<unsigned char> cam(total_obs);
  int co = 0, po = 0, oo = 0;
  for (int p = 0; p < count; ++p) {
    const v3dba_problem& q = problems[p];
    h->h_cam_off.push_back(co); h->h_n_cams.push_back(q.n_cameras);
    h->h_pt_off.push_back(po); h->h_n_pts.push_back(q.n_points);
    h->h_size.push_back(q.n_measurements);
    h->max_cams = std::max(h->max_cams, q.n_cameras);
    thr[p] = q.inlier_threshold;
    std::copy(q.R, q.R + 9 * q.n_cameras, R.begin() + 9 * (size_t)co);
    std::copy(q.T, q.T + 3 * q.n_cameras, T.begin() + 3 * (size_t)co);
    std::copy(q.K, q.K + 9 * q.n_cameras, K.begin() + 9 * (size_t)co);
    std::copy(q.X, q.X + 3 * q.n_points, X.begin() + 3 * (size_t)po);
    // point-major observations (stable); inputs already in point order (a triplet stage's, or
    // any BundlePointStructure's) are copied as they are
    bool sorted = true;
    for (int k = 1; k < q.n_measurements && sorted; ++k) sorted = q.point[k] >= q.point[k - 1];
    if (sorted) {
      int k = 0;
      for (int j = 0; j < q.n_points; ++j) {
        ptr[po + j] = oo + k;
        while (k < q.n_measurements && q.point[k] == j) ++k;
      }
      ptr[po + q.n_points] = oo + q.n_measurements;
      std::copy(q.measurements, q.measurements + 2 * (size_t)q.n_measurements, meas.begin() + 2 * (size_t)oo);
      for (int k2 = 0; k2 < q.n_measurements; ++k2) cam[oo + k2] = (unsigned char)q.view[k2];
    } else {
      std::vector<int> c(q.n_points + 1, 0);
      for (int k = 0; k < q.n_measurements; ++k) c[q.point[k] + 1]++;
      for (int j = 0; j < q.n_points; ++j) c[j + 1] += c[j];
      for (int j = 0; j <= q.n_points; ++j) ptr[po + j] = oo + c[j];
      std::vector<int> fill(c.begin(), c.end() - 1);
      for (int k = 0; k < q.n_measurements; ++k) {
        const int dst = oo + fill[q.point[k]]++;
        meas[2 * (size_t)dst] = q.measurements[2 * k];
        meas[2 * (size_t)dst + 1] = q.measurements[2 * k + 1];
        cam[dst] = (unsigned char)q.view[k];
      }
    }
    co += q.n_cameras; po += q.n_points; oo += q.n_measurements;
  }
  ptr[total_pts] = oo;
  // longest-processing-time order
  h->h_order.resize(count);
  std::iota(h->h_order.begin(), h->h_order.end(), 0);
  std::stable_sort(h->h_order.begin(), h->h_order.end(), [&](int a, int b2) { return h->h_size[a] > h->h_size[b2]; });
  h->split = 0;
  int rc;
#define BTRY(x) do { if ((rc = (x)) != V3DBA_OK) { batch_free(h); return rc; } } while (0)
  BTRY(batch_resources(h));
  h->d.count = count;
  BTRY(bupload(h, &h->d.cam_off, h->h_cam_off));
  BTRY(bupload(h, &h->d.n_cams, h->h_n_cams));
  BTRY(bupload(h, &h->d.pt_off, h->h_pt_off));
  BTRY(bupload(h, &h->d.n_pts, h->h_n_pts));
  BTRY(bupload(h, &h->d.order, h->h_order));
  BTRY(bupload(h, &h->d.thr, thr));
  BTRY(bupload(h, &h->d.R, R));
  BTRY(bupload(h, &h->d.T, T));
  BTRY(bupload(h, &h->d.K, K));
  BTRY(bupload(h, &h->d.X, X));
  BTRY(balloc(h, &h->d.Xt, 3 * (size_t)total_pts));
  BTRY(bupload(h, &h->d.ptr, ptr));
  BTRY(bupload(h, &h->d.meas, meas));
  BTRY(bupload(h, &h->d.cam, cam));
  BTRY(balloc(h, &h->d.w, (size_t)total_obs));
  BTRY(balloc(h, &h->d.status, count));
  BTRY(balloc(h, &h->d.iterations, count));
  BTRY(balloc(h, &h->d.rejected, count));
  BTRY(balloc(h, &h->d.cost, count));
  BTRY(balloc(h, &h->d.init_cost, count));
  BTRY(balloc(h, &h->d.lambda_out, count));
  BTRY(balloc(h, &h->d.queue, 1));
  // the initial parameters (for v3dba_batch_reset), copied on the device
  BTRY(balloc(h, &h->d_init, 9 * (size_t)total_cams + 3 * (size_t)total_cams + 3 * (size_t)total_pts));
  if (cudaMemcpyAsync(h->d_init, h->d.R, sizeof(double) * 9 * total_cams, cudaMemcpyDeviceToDevice, h->stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(h->d_init + 9 * (size_t)total_cams, h->d.T, sizeof(double) * 3 * total_cams,
                      cudaMemcpyDeviceToDevice, h->stream) != cudaSuccess ||
      cudaMemcpyAsync(h->d_init + 12 * (size_t)total_cams, h->d.X, sizeof(double) * 3 * total_pts,
                      cudaMemcpyDeviceToDevice, h->stream) != cudaSuccess ||
      cudaStreamSynchronize(h->stream) != cudaSuccess) {
    cudaGetLastError();
    batch_free(h);
    return V3DBA_ERR_CUDA;
  }
#undef BTRY
  *out = h;
  return V3DBA_OK;
}

}  // extern "C"

namespace {

// The flat arrays straight to the device: the checks, the camera bytes and the point offsets are made
// there (4096 triplets, 1.7M points: 86 -> 6.5 ms against the host's loops).  Returns V3DBA_OK with
// *out == nullptr where the host's way has to be taken: an index or value that it then refuses with its
// own code, or observations that are not in point order (a look at the first problems, in_point_order, keeps
// most of those from the upload).
int batch_create_device(int count, const int* n_cameras, const int* n_points, const int* n_measurements,
                        const double* thr, const double* K, const double* R, const double* T, const double* X,
                        const double* measurements, const int* view, const int* point, v3dba_batch_t* out) {
  *out = nullptr;
  v3dba_batch_t h = new (std::nothrow) v3dba_batch_s();
  if (!h) return V3DBA_ERR_OUT_OF_MEMORY;
  std::vector<int> obs_off(1, 0);
  int co = 0, po = 0;
  for (int p = 0; p < count; ++p) {
    h->h_cam_off.push_back(co); h->h_n_cams.push_back(n_cameras[p]);
    h->h_pt_off.push_back(po); h->h_n_pts.push_back(n_points[p]);
    h->h_size.push_back(n_measurements[p]);
    h->max_cams = std::max(h->max_cams, n_cameras[p]);
    co += n_cameras[p];
    po += n_points[p];
    obs_off.push_back(obs_off.back() + n_measurements[p]);
  }
  const size_t nc = h->total_cams = co, np = h->total_pts = po, no = h->total_obs = obs_off.back();
  h->h_order.resize(count);
  std::iota(h->h_order.begin(), h->h_order.end(), 0);
  std::stable_sort(h->h_order.begin(), h->h_order.end(), [&](int a, int b2) { return h->h_size[a] > h->h_size[b2]; });
  int rc;
#define BTRY(x) do { if ((rc = (x)) != V3DBA_OK) { batch_free(h); return rc; } } while (0)
#define BCUDA(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) { cudaGetLastError(); batch_free(h); \
    return _e == cudaErrorMemoryAllocation ? V3DBA_ERR_OUT_OF_MEMORY : V3DBA_ERR_CUDA; } } while (0)
  BTRY(batch_resources(h));
  h->d.count = count;
  BatchDev& d = h->d;
  int *d_off, *d_view, *d_point, *d_flag;
  BTRY(balloc(h, &d.cam_off, count));
  BTRY(balloc(h, &d.n_cams, count));
  BTRY(balloc(h, &d.pt_off, count));
  BTRY(balloc(h, &d.n_pts, count));
  BTRY(balloc(h, &d.order, count));
  BTRY(balloc(h, &d.thr, count));
  BTRY(balloc(h, &d.R, 9 * nc));
  BTRY(balloc(h, &d.T, 3 * nc));
  BTRY(balloc(h, &d.K, 9 * nc));
  BTRY(balloc(h, &d.X, 3 * np));
  BTRY(balloc(h, &d.Xt, 3 * np));
  BTRY(balloc(h, &d.ptr, np + 1));
  BTRY(balloc(h, &d.meas, 2 * no));
  BTRY(balloc(h, &d.cam, no));
  BTRY(balloc(h, &d.w, no));
  BTRY(balloc(h, &d.status, count));
  BTRY(balloc(h, &d.iterations, count));
  BTRY(balloc(h, &d.rejected, count));
  BTRY(balloc(h, &d.cost, count));
  BTRY(balloc(h, &d.init_cost, count));
  BTRY(balloc(h, &d.lambda_out, count));
  BTRY(balloc(h, &d.queue, 1));
  BTRY(balloc(h, &h->d_init, 12 * nc + 3 * np));
  BTRY(balloc(h, &d_off, (size_t)count + 1));
  BTRY(balloc(h, &d_flag, 1));
  BTRY(balloc(h, &d_view, no));
  BTRY(balloc(h, &d_point, no));
  const size_t I = sizeof(int), D = sizeof(double), cnt = (size_t)count;
  BTRY(copy_up({{d.cam_off, h->h_cam_off.data(), I * cnt},
                {d.n_cams, n_cameras, I * cnt},
                {d.pt_off, h->h_pt_off.data(), I * cnt},
                {d.n_pts, n_points, I * cnt},
                {d.order, h->h_order.data(), I * cnt},
                {d_off, obs_off.data(), I * (cnt + 1)},
                {d.thr, thr, D * cnt},
                {d.R, R, D * 9 * nc},
                {d.T, T, D * 3 * nc},
                {d.K, K, D * 9 * nc},
                {d.X, X, D * 3 * np},
                {d.meas, measurements, D * 2 * no},
                {d_view, view, I * no},
                {d_point, point, I * no}},
               h->stream));
  BCUDA(cudaMemsetAsync(d_flag, 0, I, h->stream));
  BTRY(check_device({{d.K, 9 * (int64_t)nc, kCheckDouble, 0},
                     {d.R, 9 * (int64_t)nc, kCheckDouble, 0},
                     {d.X, 3 * (int64_t)np, kCheckDouble, 0},
                     {d.meas, 2 * (int64_t)no, kCheckDouble, 0}},
                    d_flag, h->stream));
  k_batch_layout<<<count, 256, 0, h->stream>>>(d, d_off, d_view, d_point, d_flag);
  note_launches(1);
  BCUDA(cudaPeekAtLastError());
  int flag = 0;
  BCUDA(cudaMemcpyAsync(&flag, d_flag, I, cudaMemcpyDeviceToHost, h->stream));
  BCUDA(cudaStreamSynchronize(h->stream));
  if (!flag && np > 0) {   // (the offsets are complete)
    k_batch_tracks<<<(unsigned)((np + 255) / 256), 256, 0, h->stream>>>(d.ptr, (int)np, d_flag);
    note_launches(1);
    BCUDA(cudaPeekAtLastError());
    BCUDA(cudaMemcpyAsync(&flag, d_flag, I, cudaMemcpyDeviceToHost, h->stream));
  }
  BCUDA(cudaMemcpyAsync(h->d_init, d.R, D * 9 * nc, cudaMemcpyDeviceToDevice, h->stream));
  BCUDA(cudaMemcpyAsync(h->d_init + 9 * nc, d.T, D * 3 * nc, cudaMemcpyDeviceToDevice, h->stream));
  BCUDA(cudaMemcpyAsync(h->d_init + 12 * nc, d.X, D * 3 * np, cudaMemcpyDeviceToDevice, h->stream));
  BCUDA(cudaStreamSynchronize(h->stream));
#undef BTRY
#undef BCUDA
  if (flag) {
    batch_free(h);
    return V3DBA_OK;
  }
  *out = h;
  return V3DBA_OK;
}

// Whether the first kDeviceCheckMin observations of flat problems are in point order (10 us).  A program's
// problems mostly are or are not, all alike: without this look 4096 triplets out of order were uploaded for
// nothing (created in 127-157 ms instead of 121).
bool in_point_order(int count, const int* n_measurements, const int* point) {
  int64_t left = kDeviceCheckMin;
  for (int p = 0; p < count && left > 0; ++p) {
    const int n = (int)std::min<int64_t>(n_measurements[p], left);
    for (int k = 1; k < n; ++k)
      if (point[k] < point[k - 1]) return false;
    point += n_measurements[p];
    left -= n;
  }
  return true;
}

}  // namespace

extern "C" {

int v3dba_batch_create_flat(int count, const int* n_cameras, const int* n_points, const int* n_measurements,
                            const double* inlier_threshold, const double* K, const double* R, const double* T,
                            const double* X, const double* measurements, const int* view, const int* point,
                            v3dba_batch_t* out) {
  if (count <= 0 || !n_cameras || !n_points || !n_measurements || !inlier_threshold || !K || !R || !T || !out)
    return V3DBA_ERR_INVALID_ARGUMENT;
  std::vector<v3dba_problem> probs((size_t)count);
  size_t co = 0, po = 0, oo = 0;
  bool usual = true;   // nothing that the host's way refuses for its counts or threshold
  for (int p = 0; p < count; ++p) {
    if (n_cameras[p] < 0 || n_points[p] < 0 || n_measurements[p] < 0) return V3DBA_ERR_INVALID_ARGUMENT;
    if ((n_points[p] && !X) || (n_measurements[p] && (!measurements || !view || !point)))
      return V3DBA_ERR_INVALID_ARGUMENT;
    v3dba_problem q;
    std::memset(&q, 0, sizeof(q));
    q.model = V3DBA_MODEL_STD;
    q.n_cameras = n_cameras[p];
    q.n_points = n_points[p];
    q.n_measurements = n_measurements[p];
    q.inlier_threshold = inlier_threshold[p];
    q.K = K + 9 * co;
    q.R = R + 9 * co;
    q.T = T + 3 * co;
    q.X = X ? X + 3 * po : nullptr;
    q.measurements = measurements ? measurements + 2 * oo : nullptr;
    q.view = view ? view + oo : nullptr;
    q.point = point ? point + oo : nullptr;
    probs[p] = q;
    usual &= n_cameras[p] > 0 && n_cameras[p] <= kMaxCams && inlier_threshold[p] > 0.0;
    co += (size_t)n_cameras[p];
    po += (size_t)n_points[p];
    oo += (size_t)n_measurements[p];
  }
  *out = nullptr;
  int ndev = 0;
  const bool device = cudaGetDeviceCount(&ndev) == cudaSuccess && ndev > 0;
  if (!device) cudaGetLastError();
  if (usual && device && oo + po >= (size_t)kDeviceCheckMin && oo <= 0x7fffffff && po <= 0x7fffffff - 1 &&
      in_point_order(count, n_measurements, point)) {
    const int rc = batch_create_device(count, n_cameras, n_points, n_measurements, inlier_threshold, K, R, T, X,
                                       measurements, view, point, out);
    if (rc || *out) return rc;
  }
  return v3dba_batch_create(probs.data(), count, out);
}

int v3dba_batch_destroy(v3dba_batch_t h) {
  if (!h) return V3DBA_ERR_INVALID_ARGUMENT;
  batch_free(h);
  return V3DBA_OK;
}

int v3dba_batch_reset(v3dba_batch_t h) {
  if (!h) return V3DBA_ERR_INVALID_ARGUMENT;
  const size_t nc = h->total_cams, np = h->total_pts;
  V3DBA_CUDA_TRY(cudaMemcpyAsync(h->d.R, h->d_init, 9 * nc * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  V3DBA_CUDA_TRY(cudaMemcpyAsync(h->d.T, h->d_init + 9 * nc, 3 * nc * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  V3DBA_CUDA_TRY(cudaMemcpyAsync(h->d.X, h->d_init + 12 * nc, 3 * np * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  V3DBA_CUDA_TRY(cudaStreamSynchronize(h->stream));
  return V3DBA_OK;
}

int v3dba_batch_set_schedule(v3dba_batch_t h, int large_threads, int small_threads, int split) {
  if (!h) return V3DBA_ERR_INVALID_ARGUMENT;
  auto ok = [](int t) { return t == 64 || t == 128 || t == 256; };
  if (!ok(large_threads) || !ok(small_threads) || split < 0 || split > h->d.count) return V3DBA_ERR_INVALID_ARGUMENT;
  h->large_threads = large_threads;
  h->small_threads = small_threads;
  h->split = split;
  return V3DBA_OK;
}

int v3dba_batch_minimize(v3dba_batch_t h, const v3dba_options* opts, v3dba_result* results, double* device_ms) {
  if (!h) return V3DBA_ERR_INVALID_ARGUMENT;
  v3dba_options o;
  if (opts) o = *opts; else v3dba_default_options(&o);
  V3DBA_CUDA_TRY(cudaEventRecord(h->ev0, h->stream));
  int rc = batch_run(h, &o);
  if (rc) return rc;
  V3DBA_CUDA_TRY(cudaEventRecord(h->ev1, h->stream));
  V3DBA_CUDA_TRY(cudaEventSynchronize(h->ev1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, h->ev0, h->ev1);
  if (device_ms) *device_ms = ms;
  if (results) {
    const int n = h->d.count;
    std::vector<int> st(n), it(n), rj(n);
    std::vector<double> c(n), ic(n), lm(n);
    if ((rc = copy_down({{st.data(), h->d.status, n * sizeof(int)},
                         {it.data(), h->d.iterations, n * sizeof(int)},
                         {rj.data(), h->d.rejected, n * sizeof(int)},
                         {c.data(), h->d.cost, n * sizeof(double)},
                         {ic.data(), h->d.init_cost, n * sizeof(double)},
                         {lm.data(), h->d.lambda_out, n * sizeof(double)}},
                        h->stream)))
      return rc;
    for (int p = 0; p < n; ++p) {
      v3dba_result& r = results[p];
      std::memset(&r, 0, sizeof(r));
      r.status = st[p]; r.iterations = it[p]; r.n_rejected = rj[p];
      r.cost = c[p]; r.initial_cost = ic[p]; r.lambda = lm[p];
      r.device_ms = ms; r.fp64_from_iteration = -1;
    }
  }
  return V3DBA_OK;
}

int v3dba_batch_get_params(v3dba_batch_t h, int index, double* R, double* T, double* X) {
  if (!h || index < 0 || index >= h->d.count) return V3DBA_ERR_INVALID_ARGUMENT;
  const size_t c0 = h->h_cam_off[index], nc = h->h_n_cams[index];
  const size_t p0 = h->h_pt_off[index], np = h->h_n_pts[index];
  if (R) V3DBA_CUDA_TRY(cudaMemcpy(R, h->d.R + 9 * c0, 9 * nc * sizeof(double), cudaMemcpyDeviceToHost));
  if (T) V3DBA_CUDA_TRY(cudaMemcpy(T, h->d.T + 3 * c0, 3 * nc * sizeof(double), cudaMemcpyDeviceToHost));
  if (X) V3DBA_CUDA_TRY(cudaMemcpy(X, h->d.X + 3 * p0, 3 * np * sizeof(double), cudaMemcpyDeviceToHost));
  return V3DBA_OK;
}

int v3dba_batch_get_all_params(v3dba_batch_t h, double* R, double* T, double* X) {
  if (!h) return V3DBA_ERR_INVALID_ARGUMENT;
  std::vector<HostCopy> list;
  if (R) list.push_back({R, h->d.R, 9 * (size_t)h->total_cams * sizeof(double)});
  if (T) list.push_back({T, h->d.T, 3 * (size_t)h->total_cams * sizeof(double)});
  if (X) list.push_back({X, h->d.X, 3 * (size_t)h->total_pts * sizeof(double)});
  return copy_down(list, h->stream);
}

int v3dba_batch_autotune(v3dba_batch_t h, const v3dba_options* opts, int* large_threads, int* small_threads,
                         int* split) {
  if (!h) return V3DBA_ERR_INVALID_ARGUMENT;
  v3dba_options o;
  if (opts) o = *opts; else v3dba_default_options(&o);
  const int n = h->d.count;
  const int cand_threads[2][2] = {{128, 64}, {256, 128}};
  const int splits[4] = {0, n / 8, n / 4, n / 2};
  double best = 1e30;
  int bl = h->large_threads, bs = h->small_threads, bp = h->split;
  for (int c = 0; c < 2; ++c)
    for (int q = 0; q < 4; ++q) {
      const int lt = cand_threads[c][0], st = cand_threads[c][1];
      for (int alt = 0; alt < 2; ++alt) {
        const int small = alt ? lt : st;   // also try one block size for everything
        int rc = v3dba_batch_set_schedule(h, lt, small, splits[q]);
        if (rc) return rc;
        if ((rc = v3dba_batch_reset(h))) return rc;
        double ms = 0.0;
        if ((rc = v3dba_batch_minimize(h, &o, nullptr, &ms))) return rc;
        if (ms < best) { best = ms; bl = lt; bs = small; bp = splits[q]; }
      }
    }
  int rc = v3dba_batch_set_schedule(h, bl, bs, bp);
  if (rc) return rc;
  if ((rc = v3dba_batch_reset(h))) return rc;
  if (large_threads) *large_threads = bl;
  if (small_threads) *small_threads = bs;
  if (split) *split = bp;
  return V3DBA_OK;
}

int v3dba_minimize_batched(const v3dba_problem* problems, int count, const v3dba_options* opts,
                           double* const* K, double* const* R, double* const* T, double* const* dist,
                           double* const* X, v3dba_result* results) {
  (void)K;
  (void)dist;
  v3dba_batch_t h = nullptr;
  int rc = v3dba_batch_create(problems, count, &h);
  if (rc) return rc;
  rc = v3dba_batch_minimize(h, opts, results, nullptr);
  if (rc == V3DBA_OK && (R || T || X)) {
    std::vector<double> Ra(9 * (size_t)h->total_cams), Ta(3 * (size_t)h->total_cams), Xa(3 * (size_t)h->total_pts);
    rc = v3dba_batch_get_all_params(h, Ra.data(), Ta.data(), Xa.data());
    for (int p = 0; rc == V3DBA_OK && p < count; ++p) {
      const size_t c0 = h->h_cam_off[p], nc = h->h_n_cams[p], p0 = h->h_pt_off[p], np = h->h_n_pts[p];
      if (R && R[p]) std::copy(Ra.begin() + 9 * c0, Ra.begin() + 9 * (c0 + nc), R[p]);
      if (T && T[p]) std::copy(Ta.begin() + 3 * c0, Ta.begin() + 3 * (c0 + nc), T[p]);
      if (X && X[p]) std::copy(Xa.begin() + 3 * p0, Xa.begin() + 3 * (p0 + np), X[p]);
    }
  }
  v3dba_batch_destroy(h);
  return rc;
}

}  // extern "C"

// ---- triplet stage ---------------------------------------------------------------------------
//
// The steps either side of the triplet adjustment (SfM/generate_triples/src/generate_triples.cpp:
// 380-415) for all triplets of a call: k_triplet_prepare (one thread per track) triangulates and
// filters, k_triplet_assemble (one block per triplet) applies the survival tests and packs the
// surviving points and measurements point-major into the batch layout, k_batched_lm adjusts every
// accepted triplet, k_triplet_scatter returns each track's point.

namespace v3dba {
namespace {

struct StageDev {
  int n_trk = 0;
  const int* trk_tri = nullptr;     // [n_trk] triplet of each track
  const int* tptr = nullptr;        // [n_trk+1] measurements of each track (global)
  const int* mview = nullptr;       // [n_meas] triple view
  const float* mpos = nullptr;      // [2 n_meas]
  const double* focal = nullptr;    // [3 count]
  const int* trk_off = nullptr;     // [count] first track of each triplet
  const int* n_trk_of = nullptr;    // [count]
  double* Xtri = nullptr;           // [3 n_trk] linear triangulation
  unsigned char* kept = nullptr;    // [n_meas]
  int* keptcnt = nullptr;           // [n_trk] surviving measurements of a surviving track, else 0
  int* slot = nullptr;              // [n_trk] point slot inside its triplet's problem, or -1
  int* verdict = nullptr;           // [count]
  int* n_surv = nullptr;            // [count]
  int* pt_track = nullptr;          // [total point slots]
  double max_err, min_ratio;
  int min_points;
};

// Least squares of the 2K x 3 system A x = b by Householder QR (the algorithm of TNT's QR,
// V3D/include/Math/v3d_linear_tnt.h:1589-1629 and its solve, :1734-1771): column norms by hypot,
// reflector sign from the diagonal, R's diagonal kept apart.  Returns false when rank deficient.
__device__ bool qr_least_squares3(double (*A)[3], double* b, int m, double x[3]) {
  double rdiag[3];
  for (int k = 0; k < 3; ++k) {
    double nrm = 0.0;
    for (int i = k; i < m; ++i) nrm = hypot(nrm, A[i][k]);
    if (nrm != 0.0) {
      if (A[k][k] < 0.0) nrm = -nrm;
      for (int i = k; i < m; ++i) A[i][k] /= nrm;
      A[k][k] += 1.0;
      for (int j = k + 1; j < 3; ++j) {
        double s = 0.0;
        for (int i = k; i < m; ++i) s += A[i][k] * A[i][j];
        s = -s / A[k][k];
        for (int i = k; i < m; ++i) A[i][j] += s * A[i][k];
      }
    }
    rdiag[k] = -nrm;
  }
  if (rdiag[0] == 0.0 || rdiag[1] == 0.0 || rdiag[2] == 0.0) return false;
  for (int k = 0; k < 3; ++k) {
    double s = 0.0;
    for (int i = k; i < m; ++i) s += A[i][k] * b[i];
    s = -s / A[k][k];
    for (int i = k; i < m; ++i) b[i] += s * A[i][k];
  }
  for (int k = 2; k >= 0; --k) {
    b[k] /= rdiag[k];
    for (int i = 0; i < k; ++i) b[i] -= b[k] * A[i][k];
  }
  x[0] = b[0];
  x[1] = b[1];
  x[2] = b[2];
  return true;
}

// One thread per track: triangulateLinear (v3d_mviewutilities.h:260-303) and filterTripleModel
// (generate_triples.cpp:44-81).  The filter mirrors the reference's arithmetic: the projection
// rounded to float, the float difference and sum of squares, the float square root, times the
// view's focal length in double (no fused multiply-adds, so the decision is the host's).
__global__ void __launch_bounds__(128) k_triplet_prepare(BatchDev b, StageDev s) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= s.n_trk) return;
  const int t = s.trk_tri[g];
  const int c0 = b.cam_off[t];
  const int m0 = s.tptr[g], K = s.tptr[g + 1] - m0;
  double A[2 * kMaxTrack][3], rhs[2 * kMaxTrack], X[3];
  for (int q = 0; q < K; ++q) {
    const int v = s.mview[m0 + q];
    const double* R = b.R + 9 * (size_t)(c0 + v);
    const double* T = b.T + 3 * (size_t)(c0 + v);
    const double x = (double)s.mpos[2 * (m0 + q)], y = (double)s.mpos[2 * (m0 + q) + 1];
    for (int c = 0; c < 3; ++c) {
      A[2 * q][c] = __dsub_rn(__dmul_rn(x, R[6 + c]), R[c]);
      A[2 * q + 1][c] = __dsub_rn(__dmul_rn(y, R[6 + c]), R[3 + c]);
    }
    rhs[2 * q] = __dsub_rn(T[0], __dmul_rn(x, T[2]));
    rhs[2 * q + 1] = __dsub_rn(T[1], __dmul_rn(y, T[2]));
  }
  const bool ok = K > 0 && qr_least_squares3(A, rhs, 2 * K, X);
  if (!ok) X[0] = X[1] = X[2] = nan("");
  int cnt = 0;
  for (int q = 0; q < K; ++q) {
    const int v = s.mview[m0 + q];
    const double* R = b.R + 9 * (size_t)(c0 + v);
    const double* T = b.T + 3 * (size_t)(c0 + v);
    double Y[3];
    for (int r = 0; r < 3; ++r) {
      double acc = __dmul_rn(R[3 * r], X[0]);
      acc = __dadd_rn(acc, __dmul_rn(R[3 * r + 1], X[1]));
      acc = __dadd_rn(acc, __dmul_rn(R[3 * r + 2], X[2]));
      Y[r] = __dadd_rn(acc, T[r]);
    }
    const float px = (float)__ddiv_rn(Y[0], Y[2]), py = (float)__ddiv_rn(Y[1], Y[2]);
    const float dx = __fsub_rn(px, s.mpos[2 * (m0 + q)]), dy = __fsub_rn(py, s.mpos[2 * (m0 + q) + 1]);
    const float n = (float)sqrt((double)__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
    const double err = __dmul_rn(s.focal[3 * t + v], (double)n);
    const bool keep = err < s.max_err;   // false for NaN
    s.kept[m0 + q] = keep ? 1 : 0;
    cnt += keep ? 1 : 0;
  }
  s.keptcnt[g] = cnt >= 3 ? cnt : 0;
  s.Xtri[3 * (size_t)g] = X[0];
  s.Xtri[3 * (size_t)g + 1] = X[1];
  s.Xtri[3 * (size_t)g + 2] = X[2];
}

// Exclusive block-wide scan of one int per thread (256 threads); returns the prefix and the
// block total in *total.
__device__ __forceinline__ int block_scan256(int v, int* sm /* [8] */, int* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sm[wid] = x;
  __syncthreads();
  int base = 0, tot = 0;
  for (int w = 0; w < 8; ++w) {
    if (w < wid) base += sm[w];
    tot += sm[w];
  }
  __syncthreads();
  *total = tot;
  return base + x - v;
}

// One block (256 threads) per triplet: survival tests (generate_triples.cpp:393-398) and the
// bundle problem of the survivors, point-major as BundlePointStructure builds it
// (v3d_mviewutilities.h:136-158).
__global__ void __launch_bounds__(256) k_triplet_assemble(BatchDev b, StageDev s) {
  __shared__ int sm[8];
  const int t = blockIdx.x;
  const int g0 = s.trk_off[t], n = s.n_trk_of[t];
  int surv = 0;
  for (int base = 0; base < n; base += 256) {
    const int g = g0 + base + threadIdx.x;
    int tot;
    block_scan256((base + (int)threadIdx.x < n && s.keptcnt[g] > 0) ? 1 : 0, sm, &tot);
    surv += tot;
  }
  int verdict = V3DBA_TRIPLET_ACCEPTED;
  if (surv < s.min_points) verdict = V3DBA_TRIPLET_TOO_FEW_POINTS;
  else if ((double)surv < s.min_ratio * (double)n) verdict = V3DBA_TRIPLET_POINTS_DROPPED;
  const int pt0 = b.pt_off[t];
  const int ob0 = s.tptr[g0];   // the triplet's measurement range bounds its kept measurements
  if (threadIdx.x == 0) {
    s.verdict[t] = verdict;
    s.n_surv[t] = surv;
    b.n_pts[t] = verdict == V3DBA_TRIPLET_ACCEPTED ? surv : 0;
    b.ptr[pt0] = ob0;
  }
  int q_run = 0, o_run = 0;
  for (int base = 0; base < n; base += 256) {
    const int g = g0 + base + threadIdx.x;
    const bool in = base + (int)threadIdx.x < n;
    const int kc = in ? s.keptcnt[g] : 0;
    const bool sv = kc > 0 && verdict == V3DBA_TRIPLET_ACCEPTED;
    int tq, to;
    const int q = q_run + block_scan256(sv ? 1 : 0, sm, &tq);
    const int o = o_run + block_scan256(sv ? kc : 0, sm, &to);
    if (in) s.slot[g] = sv ? q : -1;
    if (sv) {
      const int p = pt0 + q;
      b.X[3 * (size_t)p] = s.Xtri[3 * (size_t)g];
      b.X[3 * (size_t)p + 1] = s.Xtri[3 * (size_t)g + 1];
      b.X[3 * (size_t)p + 2] = s.Xtri[3 * (size_t)g + 2];
      b.ptr[p + 1] = ob0 + o + kc;
      s.pt_track[p] = g;
      int w = ob0 + o;
      for (int m = s.tptr[g]; m < s.tptr[g + 1]; ++m) {
        if (!s.kept[m]) continue;
        b.meas[2 * (size_t)w] = (double)s.mpos[2 * m];
        b.meas[2 * (size_t)w + 1] = (double)s.mpos[2 * m + 1];
        b.cam[w] = (unsigned char)s.mview[m];
        ++w;
      }
    }
    q_run += tq;
    o_run += to;
  }
}

// One thread per track: the point after the stage.
__global__ void __launch_bounds__(256) k_triplet_scatter(BatchDev b, StageDev s, double* __restrict__ Xout) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= s.n_trk) return;
  const int t = s.trk_tri[g], q = s.slot[g];
  const double* src = (q >= 0) ? b.X + 3 * (size_t)(b.pt_off[t] + q) : s.Xtri + 3 * (size_t)g;
  Xout[3 * (size_t)g] = src[0];
  Xout[3 * (size_t)g + 1] = src[1];
  Xout[3 * (size_t)g + 2] = src[2];
}

// Per-triplet bookkeeping filled on the device: the triplet of every track, the batch layout's
// camera / point offsets, identity intrinsics and the adjustment's threshold.
__global__ void __launch_bounds__(256) k_triplet_setup(BatchDev b, int* __restrict__ trk_tri, const int* __restrict__ trk_off,
                                                       int* __restrict__ n_trk_of, double thr) {
  const int t = blockIdx.x;
  const int g0 = trk_off[t], g1 = trk_off[t + 1];
  for (int g = g0 + threadIdx.x; g < g1; g += blockDim.x) trk_tri[g] = t;
  if (threadIdx.x < 27) b.K[27 * (size_t)t + threadIdx.x] = (threadIdx.x % 9 == 0 || threadIdx.x % 9 == 4 || threadIdx.x % 9 == 8) ? 1.0 : 0.0;
  if (threadIdx.x == 0) {
    b.cam_off[t] = 3 * t;
    b.n_cams[t] = 3;
    b.pt_off[t] = g0 + t;   // one spare point slot per triplet keeps the end pointers apart
    b.thr[t] = thr;
    n_trk_of[t] = g1 - g0;
  }
}

}  // namespace
}  // namespace v3dba

namespace {

// The stage on flat inputs (all triplets concatenated); outputs flat.  See v3dba_triplet_stage_flat.
int triplet_stage_core(int count, const double* R, const double* T, const double* focal, const int32_t* tracks_of,
                       const int32_t* track_ptr, const int32_t* view, const float* pos,
                       const v3dba_triplet_stage_options& o, int32_t* verdict_out, int32_t* npts_out,
                       int32_t* status_out, int32_t* iters_out, double* cost_out, double* R_out, double* T_out,
                       double* X_out, uint8_t* kept_out, double* device_ms, bool verify) {
  const size_t n_trk = (size_t)tracks_of[count];
  const size_t n_meas = n_trk > 0 ? (size_t)track_ptr[n_trk] : 0;
  if (n_trk > 0x7fffffffull - (size_t)count || n_meas > 0x7fffffffull) return V3DBA_ERR_UNSUPPORTED;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return V3DBA_ERR_NO_DEVICE; }
  // longest-processing-time order of the adjustments (by raw measurement count)
  std::vector<int> size(count), order(count);
  for (int t = 0; t < count; ++t) size[t] = track_ptr[tracks_of[t + 1]] - track_ptr[tracks_of[t]];
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return size[a] > size[c]; });
  const size_t n_slots = n_trk + count;

  PhaseTrace trace("V3DBA_TRACE_STAGE", "v3dba_triplet_stage");
  v3dba_batch_t h = new (std::nothrow) v3dba_batch_s();
  if (!h) return V3DBA_ERR_OUT_OF_MEMORY;
  h->total_cams = 3 * count;
  h->max_cams = 3;
  h->total_pts = (int)n_slots;
  h->total_obs = (int)n_meas;
  int rc;
  Arena ar;
  auto done = [&]() {
    ar.release(h->stream);
    batch_free(h);   // synchronises the stream before destroying it
  };
#define BTRY(x) do { if ((rc = (x)) != V3DBA_OK) { done(); return rc; } } while (0)
#define BCUDA(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) { cudaGetLastError(); done(); \
    return _e == cudaErrorMemoryAllocation ? V3DBA_ERR_OUT_OF_MEMORY : V3DBA_ERR_CUDA; } } while (0)
#define BLAUNCH() do { note_launches(1); BCUDA(cudaPeekAtLastError()); } while (0)
#define BUP(dst, src, n) up.push_back({dst, src, sizeof(*(src)) * (n)})
#define BDOWN(dst, src, n) down.push_back({dst, src, sizeof(*(src)) * (n)})
  BTRY(batch_resources(h));
  h->d.count = count;
  StageDev s;
  int *d_trk_tri, *d_tptr, *d_trk_off, *d_n_trk_of, *d_view;
  float* d_mpos;
  double* d_focal;
  double* d_Xout;
  ar.add(&h->d.cam_off, count);
  ar.add(&h->d.n_cams, count);
  ar.add(&h->d.pt_off, count);
  ar.add(&h->d.n_pts, count);
  ar.add(&h->d.order, count);
  ar.add(&h->d.thr, count);
  ar.add(&h->d.R, 27 * (size_t)count);
  ar.add(&h->d.T, 9 * (size_t)count);
  ar.add(&h->d.K, 27 * (size_t)count);
  ar.add(&h->d.X, 3 * n_slots);
  ar.add(&h->d.Xt, 3 * n_slots);
  ar.add(&h->d.ptr, n_slots + 1);
  ar.add(&h->d.meas, 2 * n_meas);
  ar.add(&h->d.cam, n_meas);
  ar.add(&h->d.w, n_meas);
  ar.add(&h->d.status, count);
  ar.add(&h->d.iterations, count);
  ar.add(&h->d.rejected, count);
  ar.add(&h->d.cost, count);
  ar.add(&h->d.init_cost, count);
  ar.add(&h->d.lambda_out, count);
  ar.add(&h->d.queue, 1);
  ar.add(&d_trk_tri, n_trk);
  ar.add(&d_tptr, n_trk + 1);
  ar.add(&d_trk_off, (size_t)count + 1);
  ar.add(&d_n_trk_of, count);
  ar.add(&d_view, n_meas);
  ar.add(&d_mpos, 2 * n_meas);
  ar.add(&d_focal, 3 * (size_t)count);
  ar.add(&s.Xtri, 3 * n_trk);
  ar.add(&s.kept, n_meas);
  ar.add(&s.keptcnt, n_trk);
  ar.add(&s.slot, n_trk);
  ar.add(&s.verdict, count);
  ar.add(&s.n_surv, count);
  ar.add(&s.pt_track, n_slots);
  ar.add(&d_Xout, 3 * n_trk);
  BTRY(ar.commit(h->stream));
  trace.mark("alloc", h->stream);
  // inputs: one copy of each caller array
  std::vector<HostCopy> up;
  BUP(h->d.R, R, 27 * (size_t)count);
  BUP(h->d.T, T, 9 * (size_t)count);
  BUP(d_focal, focal, 3 * (size_t)count);
  BUP(d_trk_off, tracks_of, (size_t)count + 1);
  BUP(d_tptr, track_ptr, n_trk + 1);
  BUP(d_view, view, n_meas);
  BUP(d_mpos, pos, 2 * n_meas);
  BUP(h->d.order, order.data(), (size_t)count);
  BTRY(copy_up(up, h->stream));
  if (verify) {   // views and positions, before anything uses them
    int bad = 0;
    int* flag = reinterpret_cast<int*>(h->d.queue);
    BCUDA(cudaMemsetAsync(flag, 0, sizeof(int), h->stream));
    BTRY(check_device({{d_view, (int64_t)n_meas, kCheckIndex, 3}, {d_mpos, 2 * (int64_t)n_meas, kCheckFloat, 0}}, flag,
                      h->stream));
    BCUDA(cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    BCUDA(cudaStreamSynchronize(h->stream));
    if (bad) {
      done();
      return V3DBA_ERR_INVALID_INPUT;
    }
  }
  trace.mark("upload", h->stream);
  s.n_trk = (int)n_trk;
  s.trk_tri = d_trk_tri;
  s.tptr = d_tptr;
  s.mview = d_view;
  s.mpos = d_mpos;
  s.focal = d_focal;
  s.trk_off = d_trk_off;
  s.n_trk_of = d_n_trk_of;
  s.max_err = o.max_reproj_error;
  s.min_ratio = o.min_point_ratio;
  s.min_points = o.min_points;
  BCUDA(cudaEventRecord(h->ev0, h->stream));
  k_triplet_setup<<<count, 256, 0, h->stream>>>(h->d, d_trk_tri, d_trk_off, d_n_trk_of, o.inlier_threshold);
  BLAUNCH();
  if (n_trk > 0) {
    k_triplet_prepare<<<(unsigned)((n_trk + 127) / 128), 128, 0, h->stream>>>(h->d, s);
    BLAUNCH();
  }
  k_triplet_assemble<<<count, 256, 0, h->stream>>>(h->d, s);
  BLAUNCH();
  BatchOpts bo;
  bo.tau = o.tau;
  bo.grad_thr = 1e-10;
  bo.upd_thr = 1e-10;
  bo.max_iter = o.max_iterations;
  BTRY(launch_range(h, 0, 0, count, bo));
  if (n_trk > 0) {
    k_triplet_scatter<<<(unsigned)((n_trk + 255) / 256), 256, 0, h->stream>>>(h->d, s, d_Xout);
    BLAUNCH();
  }
  BCUDA(cudaEventRecord(h->ev1, h->stream));
  trace.mark("kernels", h->stream);
  std::vector<HostCopy> down;
  BDOWN(verdict_out, s.verdict, (size_t)count);
  BDOWN(npts_out, s.n_surv, (size_t)count);
  BDOWN(status_out, h->d.status, (size_t)count);
  BDOWN(iters_out, h->d.iterations, (size_t)count);
  BDOWN(cost_out, h->d.cost, (size_t)count);
  BDOWN(R_out, h->d.R, 27 * (size_t)count);
  BDOWN(T_out, h->d.T, 9 * (size_t)count);
  if (X_out) BDOWN(X_out, d_Xout, 3 * n_trk);
  if (kept_out) BDOWN(kept_out, s.kept, n_meas);
  BTRY(copy_down(down, h->stream));
  trace.mark("download");
  if (device_ms) {
    float ms = 0.f;
    BCUDA(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
    *device_ms = ms;
  }
  done();
  trace.mark("free");
#undef BTRY
#undef BCUDA
#undef BLAUNCH
#undef BUP
#undef BDOWN
  return V3DBA_OK;
}

// Shared validation of one triplet's tracks (track_ptr relative to the triplet); without `values` the
// views and positions are left to the caller.
int check_tracks(int n_tracks, const int32_t* track_ptr, const int32_t* view, const float* pos, bool values = true) {
  if (n_tracks < 0 || (n_tracks > 0 && (!track_ptr || !view || !pos))) return V3DBA_ERR_INVALID_ARGUMENT;
  if (n_tracks == 0) return V3DBA_OK;
  if (track_ptr[0] != 0) return V3DBA_ERR_INVALID_INPUT;
  unsigned odd = 0;   // no early exit, so that the loop runs on vectors; the second one finds the first fault
  for (int k = 0; k < n_tracks; ++k) odd |= (unsigned)(track_ptr[k + 1] - track_ptr[k]) > (unsigned)kMaxTrack ? 1u : 0u;
  for (int k = 0; k < n_tracks && odd; ++k) {
    const int len = track_ptr[k + 1] - track_ptr[k];
    if (len < 0) return V3DBA_ERR_INVALID_INPUT;
    if (len > kMaxTrack) return V3DBA_ERR_UNSUPPORTED;
  }
  if (!values) return V3DBA_OK;
  const int nm = track_ptr[n_tracks];
  unsigned bad = 0;
  for (int m = 0; m < nm; ++m) bad |= (unsigned)view[m] > 2u ? 1u : 0u;
  if (bad) return V3DBA_ERR_INVALID_INPUT;
  if (!all_finite_f(pos, 2 * (size_t)nm)) return V3DBA_ERR_INVALID_INPUT;
  return V3DBA_OK;
}

int stage_options(const v3dba_triplet_stage_options* opts, v3dba_triplet_stage_options* o) {
  v3dba_default_triplet_stage_options(o);
  if (opts) *o = *opts;
  if (!(o->inlier_threshold > 0.0) || o->max_iterations < 0 || !(o->tau >= 0.0)) return V3DBA_ERR_INVALID_ARGUMENT;
  return V3DBA_OK;
}

}  // namespace

extern "C" {

void v3dba_default_triplet_stage_options(v3dba_triplet_stage_options* o) {
  if (!o) return;
  o->max_reproj_error = 1.0;
  o->min_points = 50;
  o->min_point_ratio = 0.5;
  o->inlier_threshold = 1.0;
  o->tau = 1e-3;
  o->max_iterations = 5;
}

int v3dba_triplet_stage_flat(int count, const double* R, const double* T, const double* focal, const int32_t* tracks_of,
                             const int32_t* track_ptr, const int32_t* view, const float* pos,
                             const v3dba_triplet_stage_options* opts, int32_t* verdict, int32_t* n_points,
                             int32_t* status, int32_t* iterations, double* cost, double* R_out, double* T_out,
                             double* X_out, uint8_t* kept, double* device_ms) {
  if (count <= 0 || !R || !T || !focal || !tracks_of || !track_ptr || !verdict || !n_points || !status ||
      !iterations || !cost || !R_out || !T_out)
    return V3DBA_ERR_INVALID_ARGUMENT;
  v3dba_triplet_stage_options o;
  int rc = stage_options(opts, &o);
  if (rc) return rc;
  if (!all_finite(R, 27 * (size_t)count) || !all_finite(T, 9 * (size_t)count) || !all_finite(focal, 3 * (size_t)count))
    return V3DBA_ERR_INVALID_INPUT;
  if (tracks_of[0] != 0) return V3DBA_ERR_INVALID_INPUT;
  for (int t = 0; t < count; ++t)
    if (tracks_of[t + 1] < tracks_of[t]) return V3DBA_ERR_INVALID_INPUT;
  const int n_trk = tracks_of[count];
  if (n_trk > 0 && (!view || !pos)) return V3DBA_ERR_INVALID_ARGUMENT;
  if (track_ptr[0] != 0) return V3DBA_ERR_INVALID_INPUT;
  // the global track_ptr is one list: check it in one pass, as one triplet of n_trk tracks; the views and
  // positions of large calls on the device
  int ndev = 0;
  const bool device = cudaGetDeviceCount(&ndev) == cudaSuccess && ndev > 0;
  if (!device) cudaGetLastError();
  const bool verify = device && (int64_t)n_trk >= kDeviceCheckMin;
  if ((rc = check_tracks(n_trk, track_ptr, view, pos, !verify))) return rc;
  return triplet_stage_core(count, R, T, focal, tracks_of, track_ptr, view, pos, o, verdict, n_points, status,
                            iterations, cost, R_out, T_out, X_out, kept, device_ms, verify);
}

int v3dba_triplet_stage(const v3dba_triplet* trips, int count, const v3dba_triplet_stage_options* opts,
                        v3dba_triplet_result* results, double* const* Xout, uint8_t* const* keptout,
                        double* device_ms) {
  if (!trips || count <= 0 || !results) return V3DBA_ERR_INVALID_ARGUMENT;
  v3dba_triplet_stage_options o;
  int rc = stage_options(opts, &o);
  if (rc) return rc;
  size_t n_trk = 0, n_meas = 0;
  for (int t = 0; t < count; ++t) {
    const v3dba_triplet& q = trips[t];
    if ((rc = check_tracks(q.n_tracks, q.track_ptr, q.view, q.pos))) return rc;
    if (!all_finite(q.R, 27) || !all_finite(q.T, 9) || !all_finite(q.focal, 3)) return V3DBA_ERR_INVALID_INPUT;
    n_trk += q.n_tracks;
    n_meas += q.n_tracks > 0 ? q.track_ptr[q.n_tracks] : 0;
  }
  if (n_trk > 0x7fffffffull - (size_t)count || n_meas > 0x7fffffffull) return V3DBA_ERR_UNSUPPORTED;
  // concatenate
  std::vector<double> R(27 * (size_t)count), T(9 * (size_t)count), focal(3 * (size_t)count);
  std::vector<int32_t> tracks_of((size_t)count + 1), tptr(n_trk + 1), view(n_meas);
  std::vector<float> pos(2 * n_meas);
  size_t g = 0, mm = 0;
  for (int t = 0; t < count; ++t) {
    const v3dba_triplet& q = trips[t];
    std::copy(q.R, q.R + 27, R.begin() + 27 * (size_t)t);
    std::copy(q.T, q.T + 9, T.begin() + 9 * (size_t)t);
    std::copy(q.focal, q.focal + 3, focal.begin() + 3 * (size_t)t);
    tracks_of[t] = (int32_t)g;
    const int nm = q.n_tracks > 0 ? q.track_ptr[q.n_tracks] : 0;
    for (int k = 0; k < q.n_tracks; ++k) tptr[g + k] = (int32_t)mm + q.track_ptr[k];
    if (nm) {
      std::copy(q.view, q.view + nm, view.begin() + mm);
      std::copy(q.pos, q.pos + 2 * nm, pos.begin() + 2 * mm);
    }
    g += q.n_tracks;
    mm += nm;
  }
  tracks_of[count] = (int32_t)g;
  tptr[n_trk] = (int32_t)mm;
  std::vector<int32_t> verdict(count), npts(count), status(count), iters(count);
  std::vector<double> cost(count), Ro(27 * (size_t)count), To(9 * (size_t)count), Xo(3 * n_trk);
  std::vector<uint8_t> kept(n_meas);
  rc = triplet_stage_core(count, R.data(), T.data(), focal.data(), tracks_of.data(), tptr.data(), view.data(),
                          pos.data(), o, verdict.data(), npts.data(), status.data(), iters.data(), cost.data(),
                          Ro.data(), To.data(), Xo.data(), kept.data(), device_ms, false);
  if (rc) return rc;
  size_t gg = 0, m2 = 0;
  for (int t = 0; t < count; ++t) {
    v3dba_triplet_result& r = results[t];
    r.verdict = verdict[t];
    r.n_tracks = trips[t].n_tracks;
    r.n_points = npts[t];
    const bool acc = verdict[t] == V3DBA_TRIPLET_ACCEPTED;
    r.status = acc ? status[t] : V3DBA_STATUS_TIMEOUT;
    r.iterations = acc ? iters[t] : 0;
    r.cost = acc ? cost[t] : 0.0;
    const double* Rs = acc ? Ro.data() + 27 * (size_t)t : trips[t].R;
    const double* Ts = acc ? To.data() + 9 * (size_t)t : trips[t].T;
    std::copy(Rs, Rs + 27, r.R);
    std::copy(Ts, Ts + 9, r.T);
    const int nt = trips[t].n_tracks, nm = nt > 0 ? trips[t].track_ptr[nt] : 0;
    if (Xout && Xout[t]) std::copy(Xo.begin() + 3 * gg, Xo.begin() + 3 * (gg + nt), Xout[t]);
    if (keptout && keptout[t]) std::copy(kept.begin() + m2, kept.begin() + m2 + nm, keptout[t]);
    gg += nt;
    m2 += nm;
  }
  return V3DBA_OK;
}

}  // extern "C"
