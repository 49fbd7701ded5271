// LM kernels of the B200 bundle adjuster: linearisation, point elimination (Schur complement),
// back-substitution, parameter update and cost.  See lm.cuh for the data layout.
//
// The arithmetic restates V3D/src/Math/v3d_optimization.cpp:784-1187 (weighting, J^T e, the
// U/V/W/X/Y/Z blocks, damping, update, cost with the old weights) on a point-eliminated system.
// Residuals, weights, gradient and cost are FP64.  The normal-equation blocks are stored in
// `Real` (float in mixed mode, double in FP64 mode); their sums are taken in FP64, except the
// camera-pair Schur sums of the mixed mode, which accumulate in FP32.  All reductions run in a
// fixed order (no floating-point atomics), so results are bit-reproducible run to run.
//
// Per-observation storage differs by precision.  FP32 blocks store the products W_k = A_k^T B_k
// and T_k = W_k Vinv_j (two 4-byte 6x3 blocks), which the Schur, rhs and back-substitution
// kernels gather.  FP64 blocks store B_k instead (2x3) and apply W_k and T_k factor by factor
// (W_k x = A_k^T (B_k x), T_k^T y = Vinv_j B_k^T (A_k y)): the linearisation writes 96 bytes less
// per observation and the point elimination writes no per-observation block at all, against
// 126 instead of 108 FMAs and one more point-block gather per Schur pair.
#include <algorithm>
#include <atomic>
#include <cstdio>

#include "common.cuh"
#include "async_copy.cuh"
#include "lm.cuh"
#include "model.cuh"

namespace v3dba {

// ---- layout ---------------------------------------------------------------------------------

__host__ __device__ constexpr int round4(int x) { return (x + 3) & ~3; }
__host__ __device__ constexpr int nsym(int n) { return n * (n + 1) / 2; }

// x elements of T rounded up to whole 16-byte vectors (4 floats, 2 doubles).
template <typename T>
__host__ __device__ constexpr int vround(int x) {
  return sizeof(T) == 4 ? (x + 3) & ~3 : (x + 1) & ~1;
}

// Strides of the blocks stored in `Real`, in whole 16-byte vectors.
template <int DA, int DC, typename Real = float>
struct Lay {
  static constexpr int DCc = DC > 0 ? DC : 1;
  static constexpr int SA = vround<Real>(2 * DA);    // A_k, Real
  static constexpr int SW = round4(3 * DA);          // W_k / T_k, float (FP32 blocks only)
  static constexpr int SC = vround<Real>(2 * DCc);   // C_k, Real
  static constexpr int SG = (DA + 1) & ~1;           // A_k^T r_k, double
  static constexpr int SV = vround<Real>(6);         // V_j / Vinv_j upper triangle, Real
  static constexpr int SY = vround<Real>(3 * DCc);   // Y_j / Vinv_j Y_j, Real
  static constexpr int SU = vround<Real>(DA * DA);   // U_i, Real
  static constexpr int SX = vround<Real>(DA * DCc);  // X_i, Real
  static constexpr int NZ = nsym(DC);
};

// symmetric 3x3 index of the packed upper triangle (00,01,02,11,12,22)
__device__ __forceinline__ int s3(int r, int c) {
  const int a = r < c ? r : c, b = r < c ? c : r;
  return a == 0 ? b : (a == 1 ? 2 + b : 5);
}

template <int N>
__device__ __forceinline__ void vload(const float* __restrict__ p, float (&v)[N]) {
  static_assert(N % 4 == 0, "float vectors are loaded 4 at a time");
  const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
  for (int t = 0; t < N / 4; ++t) {
    const float4 u = __ldg(q + t);
    v[4 * t] = u.x; v[4 * t + 1] = u.y; v[4 * t + 2] = u.z; v[4 * t + 3] = u.w;
  }
}
template <int N>
__device__ __forceinline__ void vload(const double* __restrict__ p, double (&v)[N]) {
  static_assert(N % 2 == 0, "double vectors are loaded 2 at a time");
  const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
  for (int t = 0; t < N / 2; ++t) {
    const double2 u = __ldg(q + t);
    v[2 * t] = u.x; v[2 * t + 1] = u.y;
  }
}
template <int N>
__device__ __forceinline__ void vstore(float* p, const float (&v)[N]) {
  float4* q = reinterpret_cast<float4*>(p);
#pragma unroll
  for (int t = 0; t < N / 4; ++t) q[t] = make_float4(v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3]);
}
template <int N>
__device__ __forceinline__ void vstore(double* p, const double (&v)[N]) {
  double2* q = reinterpret_cast<double2*>(p);
#pragma unroll
  for (int t = 0; t < N / 2; ++t) q[t] = make_double2(v[2 * t], v[2 * t + 1]);
}

// One warp's fold of n partials (summed or maxed) in a fixed order, eight loads in flight per lane; every
// lane receives the result.
template <bool SUM>
__device__ __forceinline__ double warp_fold(const double* __restrict__ p, int n) {
  constexpr double kNone = SUM ? 0.0 : -1e30;
  const int lane = threadIdx.x & 31;
  double acc = kNone;
  for (int b = lane; b < n; b += 256) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = b + 32 * u < n ? p[b + 32 * u] : kNone;
#pragma unroll
    for (int u = 0; u < 8; ++u) acc = SUM ? acc + v[u] : fmax(acc, v[u]);
  }
  return SUM ? warp_sum(acc) : warp_max(acc);
}

// The single-block folds run on kFoldWarps warps: the blocks of a value are cut into as many contiguous
// segments as there are warps for it.  Folds NV values of nblk partials each (the first NS summed, the
// rest maxed), stored value-major: part[t * nblk + b] (see store_partials).  Every thread receives the
// results; smem needs NV * fold_segs(NV) doubles.  One warp per value took 53 and 96 us where 2,000 cameras
// and 1M points leave 15,600 and 21,300 partials; see k_relin_finalize and k_trial_finalize for the rest.
constexpr int kFoldWarps = 32;
__host__ __device__ constexpr int fold_segs(int nv) { return nv >= kFoldWarps ? 1 : kFoldWarps / nv; }
template <int NV, int NS>
__device__ void fold_partials(const double* __restrict__ part, int nblk, double (&out)[NV], double* smem) {
  constexpr int SEG = fold_segs(NV);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int len = (nblk + SEG - 1) / SEG;
  for (int q = wid; q < NV * SEG; q += nw) {
    const int t = q / SEG, b0 = min((q - t * SEG) * len, nblk);
    const double* p = part + (size_t)t * nblk + b0;
    const int n = min(len, nblk - b0);
    const double v = t < NS ? warp_fold<true>(p, n) : warp_fold<false>(p, n);
    if (lane == 0) smem[q] = v;
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    double v = smem[t * SEG];
#pragma unroll
    for (int u = 1; u < SEG; ++u) v = t < NS ? v + smem[t * SEG + u] : fmax(v, smem[t * SEG + u]);
    out[t] = v;
  }
  __syncthreads();   // smem may be reused right away
}

// The block's NV partials (valid in thread 0) to part[t * nblk + bid] (by default the launch's
// block index and count; a stage run as a block range of a merged launch passes its own).
template <int NV>
__device__ __forceinline__ void store_partials(double* __restrict__ part, const double (&v)[NV], int bid, int nblk) {
  if (threadIdx.x == 0) {
#pragma unroll
    for (int t = 0; t < NV; ++t) part[(size_t)t * nblk + bid] = v[t];
  }
}
template <int NV>
__device__ __forceinline__ void store_partials(double* __restrict__ part, const double (&v)[NV]) {
  store_partials(part, v, (int)blockIdx.x, (int)gridDim.x);
}

// Warp-wide sum of V values (V a multiple of 32) by recursive halving: each of the five
// butterfly stages exchanges half of the remaining values, V - V/32 shuffles in total instead
// of 5V.  Afterwards lane L holds the totals of values [L*V/32, (L+1)*V/32) in v[0 .. V/32).
template <int H, typename T, int V>
__device__ __forceinline__ void rt_stage(T (&v)[V], int lane, int m) {
#pragma unroll
  for (int t = 0; t < H; ++t) {
    const bool up = (lane & m) != 0;
    const T send = up ? v[t] : v[t + H];
    const T keep = up ? v[t + H] : v[t];
    v[t] = keep + __shfl_xor_sync(0xffffffffu, send, m);
  }
}
template <int V, typename T>
__device__ __forceinline__ void warp_reduce_transpose(T (&v)[V]) {
  static_assert(V % 32 == 0, "pad the value count to a multiple of 32");
  const int lane = threadIdx.x & 31;
  rt_stage<V / 2>(v, lane, 16);
  rt_stage<V / 4>(v, lane, 8);
  rt_stage<V / 8>(v, lane, 4);
  rt_stage<V / 16>(v, lane, 2);
  rt_stage<V / 32>(v, lane, 1);
}

__host__ __device__ constexpr int round32(int x) { return (x + 31) & ~31; }

// value layout of the per-camera sums: U (packed upper triangle), ga, X
template <int DA, int DC>
struct CamV {
  static constexpr int NU = nsym(DA);
  static constexpr int NX = DC > 0 ? DA * DC : 0;
  static constexpr int NV = NU + DA + NX;
  static constexpr int VP = round32(NV);
};
// value layout of the per-camera reduced rhs / border sums: W q, T Y
template <int DA, int DC>
struct RhsV {
  static constexpr int NX = DC > 0 ? DA * DC : 0;
  static constexpr int NV = DA + NX;
  static constexpr int VP = round32(NV);
};
template <int DA>
struct SchurV {
  static constexpr int NV = DA * DA;
  static constexpr int VP = round32(NV);
};

// sum[t] += values lane + 32 t of the partials [c0, c1) of VP values each, in order, eight partials in
// flight (one after another, a camera's 24 partials took 7 us).
template <int PER, int VP>
__device__ __forceinline__ void sum_chunks(double (&sum)[PER], const double* __restrict__ part, int c0, int c1, int lane) {
  constexpr int U = PER <= 2 ? 8 : 4;
  for (int c = c0; c < c1; c += U) {
    double v[U][PER];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int t = 0; t < PER; ++t) v[u][t] = c + u < c1 ? part[(size_t)(c + u) * VP + lane + 32 * t] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int t = 0; t < PER; ++t) sum[t] += v[u][t];
  }
}

// row / column of the packed upper-triangle index u of a DA x DA matrix
template <int DA>
__device__ __forceinline__ void unpack_sym(int u, int& r, int& c) {
  r = 0;
  int start = 0;
  while (u >= start + (DA - r)) { start += DA - r; ++r; }
  c = r + (u - start);
}

// ---- staged blocks ---------------------------------------------------------------------------
// The chunk kernels contract small blocks over long lists (observations of a camera, observation pairs of
// a camera pair).  A lane that loads its own blocks touches a cache line per lane and instruction, and the
// L1's wavefronts, not bandwidth, set the time.  So a warp copies the blocks of 32 list entries to shared
// memory together, consecutive lanes on consecutive 16 bytes of a block, and contracts them with DMMA where
// the sums are FP64: two doubles of accumulator per lane and tile instead of 28 to 112.

// Copies block `idx` (each lane's own; negative: zeros) of STRIDE values for the warp's 32 pairs:
// dst[pair * STRIDE + t] = src[idx(pair) * STRIDE + t].
template <int STRIDE, typename T>
__device__ __forceinline__ void stage_blocks(T* dst, const T* __restrict__ src, int idx, int lane) {
  constexpr int E = 16 / sizeof(T), V = STRIDE / E;   // values per copy, copies per block
  static_assert(STRIDE % E == 0, "blocks are whole 16-byte vectors");
#pragma unroll
  for (int t = 0; t < V; ++t) {
    const int e = lane + 32 * t, rec = e / V, off = e - rec * V;
    const int k = __shfl_sync(0xffffffffu, idx, rec);
    cp16(dst + E * e, src + (size_t)max(k, 0) * STRIDE + E * off, k >= 0);
  }
}

// Writes the lanes' blocks v (of lanes with k >= 0) to dst[k * STRIDE + t], consecutive lanes on consecutive 16
// bytes of a block (STAGED; buf: 32 blocks of the warp), or every lane its own.
template <bool STAGED, int STRIDE, typename T>
__device__ __forceinline__ void put_block(T* __restrict__ dst, void* buf, const T (&v)[STRIDE], int k, int lane) {
  constexpr int E = 16 / sizeof(T), V = STRIDE / E;
  if constexpr (!STAGED) {
    vstore(dst + (size_t)k * STRIDE, v);
    return;
  }
  static_assert(STRIDE % E == 0, "blocks are whole 16-byte vectors");
  if (k >= 0) vstore(reinterpret_cast<T*>(buf) + lane * STRIDE, v);
  __syncwarp();
#pragma unroll
  for (int t = 0; t < V; ++t) {
    const int e = lane + 32 * t, rec = e / V, off = e - rec * V;
    const int kk = __shfl_sync(0xffffffffu, k, rec);
    if (kk >= 0) reinterpret_cast<float4*>(dst + (size_t)kk * STRIDE)[off] = reinterpret_cast<const float4*>(buf)[e];
  }
  __syncwarp();
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// ---- relinearisation --------------------------------------------------------------------

constexpr int kPtThreads = 128;
constexpr int kCamWarps = 4;
// Lanes per point of the track kernels that store or load one block per observation: the lanes of
// a group take the observations of one track in turn, so a warp's 16-byte stores / loads of one
// trip hit runs of consecutive blocks instead of 32 scattered ones (the observations of a track
// are contiguous in the point-major order), at the price of idle lanes on short tracks and of
// the group sums.  Measured on the 200-camera scene (375k observations, tracks of 3-12), in µs
// per launch for 1 / 2 / 4 / 8 lanes: k_linearize FP32 53.8 / 51.3 / 61.1 / 86.8, FP64 105.6 /
// 87.9 / 92.1 / 113.3; k_point_backsub FP32 13.5 / 16.6 / 14.8 / 14.6, FP64 30.2 / 17.7 / 20.8 /
// 21.0; k_point_eliminate was fastest with one lane (23.1 / 49.7) and keeps one.
constexpr int kLinLanes = 2;
template <typename Real>
__host__ __device__ constexpr int backsub_lanes() { return sizeof(Real) == 8 ? 2 : 1; }
constexpr int kMaxPtLanes = 2;

// Sum over the G consecutive lanes of a group (all lanes of the warp take part).
template <int G, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// FP32 blocks store W_k and T_k per observation; FP64 blocks store B_k (see the file header).
template <typename Real>
__host__ __device__ constexpr bool stores_products() { return sizeof(Real) == 4; }
constexpr int kSB = 6;   // stride of B_k (2 x 3 row-major) in doubles

template <int DC>
struct RelinNV {
  static constexpr int NZ = nsym(DC);
  static constexpr int NS = 1 + NZ + DC;   // cost, Z (packed), gc
  static constexpr int NV = NS + 2;        // + max |gb|, max diag V
};

// 16-byte units of the largest block that k_linearize stores per observation.
template <int DA, int DC, typename Real>
__host__ __device__ constexpr int obs_block_units() {
  using L = Lay<DA, DC, Real>;
  int m = L::SA * (int)sizeof(Real);
  const int w = stores_products<Real>() ? L::SW * 4 : kSB * 8, g = L::SG * 8, c = DC > 0 ? L::SC * (int)sizeof(Real) : 0;
  m = m > w ? m : w;
  m = m > g ? m : g;
  m = m > c ? m : c;
  return m / 16;
}

// kLinLanes lanes per point: each linearises every kLinLanes-th observation of the track (FP64),
// stores the weighted blocks, and accumulates its share of V_j, gb_j, Y_j, summed over the group
// at the end in a fixed order; Z, gc and the cost go to per-block partials.  The cameras come as packed
// records, half as many loads: 2000 cameras, 5.5M observations, 531 -> 503 us (FP64 blocks 551 -> 505); copying
// the records to shared memory by the whole warp instead took 561, for the registers that it held.
template <int MODEL, int DA, int DC, typename Real>
__global__ void __launch_bounds__(kPtThreads) k_linearize(DevState s, double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  using L = Lay<DA, DC, Real>;
  constexpr int DCc = L::DCc;
  constexpr int NS = RelinNV<DC>::NS, NV = RelinNV<DC>::NV, NZ = L::NZ;
  __shared__ double red[(kPtThreads / 32) * NV];
  constexpr int kBlk = obs_block_units<DA, DC, Real>();
  const Dims& D = s.d;
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  const int tp = gt / kLinLanes, lig = gt % kLinLanes;
  const int j = tp < D.M ? (s.p_order ? s.p_order[tp] : tp) : D.M;   // longest tracks first (p_order)
  double v[NV];
#pragma unroll
  for (int t = 0; t < NV; ++t) v[t] = (t < NS) ? 0.0 : -1e30;
  double V[6] = {0, 0, 0, 0, 0, 0}, gb[3] = {0, 0, 0}, Y[3][DCc];
#pragma unroll
  for (int b = 0; b < 3; ++b)
#pragma unroll
    for (int c = 0; c < DCc; ++c) Y[b][c] = 0.0;
  const bool fixB = j < D.nnB;
  int k0 = 0, k1 = 0;
  double X[3] = {0, 0, 0};
  if (j < D.M) {
#pragma unroll
    for (int t = 0; t < 3; ++t) X[t] = s.cur.X[3 * (size_t)j + t];
    k0 = s.p_ptr[j];
    k1 = s.p_ptr[j + 1];
  }
  // With FP64 blocks (216 to 340 bytes an observation) the warp writes its 32 observations' blocks together,
  // through shared memory: 375,000 observations with 7 global intrinsics 64.5 -> 59.4 us, 460,000 of a rig
  // 42.0 -> 38.3; 5.5M 504 -> 523, and with FP32 blocks the first 48.7 -> 51.9 and the last 501 -> 599 (the
  // blocks wait in registers for the warp), so those are written lane by lane.
  constexpr bool STAGED = !stores_products<Real>();
  __shared__ float4 stage[STAGED ? kPtThreads * kBlk : 1];
  const int lane = threadIdx.x & 31;
  float4* buf = stage + (threadIdx.x & ~31) * kBlk;
  const int own = (k1 - k0 - lig + kLinLanes - 1) / kLinLanes, trips = STAGED ? __reduce_max_sync(0xffffffffu, own) : own;
  for (int u = 0; u < trips; ++u) {
    const int kt = k0 + lig + kLinLanes * u, k = !STAGED || kt < k1 ? kt : -1;
    double A[2][DA], B[2][3], C[2][DCc], r0 = 0.0, r1 = 0.0;
    if (k >= 0) {
      const int i = s.o_cam[k];
      const bool fixA = i < D.nnA;
      Cam cam;
      load_cam_packed<MODEL>(cam, s.cur.pack, s.cur.K, s.cur.dist, i);
      if (MODEL == kModelStereo) load_rig(cam, s.rig, s.o_sub[k]);
      double e[2];
      linearize_obs<MODEL, DA, DC>(cam, X, s.o_meas[2 * k], s.o_meas[2 * k + 1], D.mode, D.cached_ar, e, A, B, C);
      const double w = huber_weight(D.thr, e);
      s.o_w[k] = w;
      v[0] += w * w * (e[0] * e[0] + e[1] * e[1]);
      r0 = -w * e[0];
      r1 = -w * e[1];
      const double wa = fixA ? 0.0 : w, wb = fixB ? 0.0 : w;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int q = 0; q < DA; ++q) A[r][q] *= wa;
#pragma unroll
        for (int q = 0; q < 3; ++q) B[r][q] *= wb;
#pragma unroll
        for (int q = 0; q < DCc; ++q) C[r][q] = (DC > 0 && q >= D.nnC) ? C[r][q] * w : 0.0;
      }
      // point sums
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = r; c < 3; ++c) V[s3(r, c)] += B[0][r] * B[0][c] + B[1][r] * B[1][c];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        gb[b] += B[0][b] * r0 + B[1][b] * r1;
#pragma unroll
        for (int c = 0; c < DCc; ++c) Y[b][c] += B[0][b] * C[0][c] + B[1][b] * C[1][c];
      }
      if (DC > 0) {
        int z = 0;
#pragma unroll
        for (int r = 0; r < DCc; ++r)
#pragma unroll
          for (int c = r; c < DCc; ++c) v[1 + z++] += C[0][r] * C[0][c] + C[1][r] * C[1][c];
#pragma unroll
        for (int c = 0; c < DCc; ++c) v[1 + NZ + c] += C[0][c] * r0 + C[1][c] * r1;
      }
    }
    // per-observation blocks
    {
      Real a[L::SA];
#pragma unroll
      for (int t = 0; t < L::SA; ++t) a[t] = Real(0);
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < DA; ++q) a[r * DA + q] = Real(A[r][q]);
      put_block<STAGED, L::SA>(reinterpret_cast<Real*>(s.o_A), buf, a, k, lane);
    }
    if constexpr (stores_products<Real>()) {
      float wv[L::SW];
#pragma unroll
      for (int t = 0; t < L::SW; ++t) wv[t] = 0.f;
#pragma unroll
      for (int q = 0; q < DA; ++q)
#pragma unroll
        for (int b = 0; b < 3; ++b) wv[q * 3 + b] = float(A[0][q] * B[0][b] + A[1][q] * B[1][b]);
      put_block<STAGED, L::SW>(s.o_W, buf, wv, k, lane);
    } else {
      double bv[kSB];
#pragma unroll
      for (int t = 0; t < kSB; ++t) bv[t] = 0.0;
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int b = 0; b < 3; ++b) bv[r * 3 + b] = B[r][b];
      put_block<STAGED, kSB>(s.o_B, buf, bv, k, lane);
    }
    if (DC > 0) {
      Real cv[L::SC];
#pragma unroll
      for (int t = 0; t < L::SC; ++t) cv[t] = Real(0);
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < DCc; ++q) cv[r * DCc + q] = Real(C[r][q]);
      put_block<STAGED, L::SC>(reinterpret_cast<Real*>(s.o_C), buf, cv, k, lane);
    }
    {
      double g[L::SG];
#pragma unroll
      for (int t = 0; t < L::SG; ++t) g[t] = 0.0;
#pragma unroll
      for (int q = 0; q < DA; ++q) g[q] = A[0][q] * r0 + A[1][q] * r1;
      put_block<STAGED, L::SG>(s.o_ga, buf, g, k, lane);
    }
  }
  // the group's sums (every lane takes part in the shuffles)
#pragma unroll
  for (int t = 0; t < 6; ++t) V[t] = group_sum<kLinLanes>(V[t]);
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    gb[b] = group_sum<kLinLanes>(gb[b]);
#pragma unroll
    for (int c = 0; c < DCc; ++c) Y[b][c] = DC > 0 ? group_sum<kLinLanes>(Y[b][c]) : 0.0;
  }
  if (j < D.M && lig == 0) {
    Real vv[L::SV];
#pragma unroll
    for (int t = 0; t < L::SV; ++t) vv[t] = t < 6 ? Real(V[t]) : Real(0);
    vstore(reinterpret_cast<Real*>(s.p_V) + (size_t)j * L::SV, vv);
    double g4[4] = {gb[0], gb[1], gb[2], 0.0};
    vstore(s.p_gb + (size_t)j * 4, g4);
    if (DC > 0) {
      Real yv[L::SY];
#pragma unroll
      for (int t = 0; t < L::SY; ++t) yv[t] = Real(0);
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < DCc; ++c) yv[b * DCc + c] = Real(Y[b][c]);
      vstore(reinterpret_cast<Real*>(s.p_Y) + (size_t)j * L::SY, yv);
    }
    if (!fixB && k1 > k0) {
      v[NS] = fmax(fabs(gb[0]), fmax(fabs(gb[1]), fabs(gb[2])));
      v[NS + 1] = fmax(V[0], fmax(V[3], V[5]));
    } else if (!fixB) {
      v[NS] = 0.0;
      v[NS + 1] = 0.0;
    }
  }
  block_reduce<NV, NS>(v, red);
  store_partials(part, v);
}

// Shared memory of a warp of k_camera_chunks, in bytes.
template <int DA, int DC, typename Real>
__host__ __device__ constexpr int camera_stage_bytes() {
  using L = Lay<DA, DC, Real>;
  return 32 * ((L::SA + (DC > 0 ? L::SC : 0)) * (int)sizeof(Real) + L::SG * (int)sizeof(double));
}

// One warp per chunk of a camera's observation list: partial U = sum A^T A, ga = sum A^T r,
// X = sum A^T C (FP64 sums); the partials of a camera are folded in chunk order afterwards.  The inner
// dimension of the products is the residual rows of 32 observations (of ga, the observations).
// 200 cameras, 375,000 observations, DC = 7: FP32 blocks 25 -> 13.7 us, FP64 35 -> 21 (216 registers held 7
// warps on an SM); the copies' latency bounds it, at 4.5 TB/s.
template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(kCamWarps * 32) k_camera_chunks(DevState s, double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  using L = Lay<DA, DC, Real>;
  using CV = CamV<DA, DC>;
  constexpr int DCc = L::DCc, NT = (DA + 7) / 8;
  extern __shared__ double stage_sm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = lane >> 2, kk = lane & 3;
  const int ch = blockIdx.x * kCamWarps + w;
  if (ch >= s.nch_cam) return;
  char* sm = reinterpret_cast<char*>(stage_sm) + w * camera_stage_bytes<DA, DC, Real>();
  double* G = reinterpret_cast<double*>(sm);
  Real* A = reinterpret_cast<Real*>(G + 32 * L::SG);
  Real* C = A + 32 * L::SA;
  double u[NT][NT][2], g[NT][2], x[NT][2];
#pragma unroll
  for (int a = 0; a < NT; ++a) {
    g[a][0] = g[a][1] = x[a][0] = x[a][1] = 0.0;
#pragma unroll
    for (int c = 0; c < NT; ++c) u[a][c][0] = u[a][c][1] = 0.0;
  }
  constexpr int RD = kCamChunk / 32;
  const int beg = s.cc_beg[ch], n = s.cc_end[ch] - beg;
  int ks[RD];   // the chunk's indices first
#pragma unroll
  for (int v = 0; v < RD; ++v) ks[v] = 32 * v + lane < n ? s.c_obs[beg + 32 * v + lane] : -1;
#pragma unroll
  for (int v = 0; v < RD; ++v) {
    if (32 * v >= n) break;
    const int k = ks[v];
    stage_blocks<L::SA>(A, reinterpret_cast<const Real*>(s.o_A), k, lane);
    stage_blocks<L::SG>(G, (const double*)s.o_ga, k, lane);
    if (DC > 0) stage_blocks<L::SC>(C, reinterpret_cast<const Real*>(s.o_C), k, lane);
    cp_join();
#pragma unroll
    for (int st = 0; st < 16; ++st) {   // two observations a step
      const int q = 2 * st + (kk >> 1), rr = kk & 1;
      double a[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) a[t] = 8 * t + r < DA ? double(A[q * L::SA + rr * DA + 8 * t + r]) : 0.0;
#pragma unroll
      for (int ta = 0; ta < NT; ++ta)
#pragma unroll
        for (int tc = ta; tc < NT; ++tc) dmma884(u[ta][tc], a[ta], a[tc]);
      if (DC > 0) {
        const double c = r < DC ? double(C[q * L::SC + rr * DCc + r]) : 0.0;
#pragma unroll
        for (int ta = 0; ta < NT; ++ta) dmma884(x[ta], a[ta], c);
      }
    }
#pragma unroll
    for (int st = 0; st < 8; ++st)      // four observations a step, against ones
#pragma unroll
      for (int t = 0; t < NT; ++t) dmma884(g[t], 8 * t + r < DA ? G[(4 * st + kk) * L::SG + 8 * t + r] : 0.0, 1.0);
    __syncwarp();
  }
  double* out = part + (size_t)ch * CV::VP;
#pragma unroll
  for (int ta = 0; ta < NT; ++ta) {
    const int R = 8 * ta + r;
    if (R >= DA) continue;
    if (kk == 0) out[CV::NU + R] = g[ta][0];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (DC > 0 && 2 * kk + t < DC) out[CV::NU + DA + R * DCc + 2 * kk + t] = x[ta][t];
#pragma unroll
      for (int tc = ta; tc < NT; ++tc) {
        const int Cc = 8 * tc + 2 * kk + t;
        if (Cc < DA && R <= Cc) out[R * DA - R * (R - 1) / 2 + (Cc - R)] = u[ta][tc][t];
      }
    }
  }
}

// One warp per camera: folds its chunk partials in order and stores U_i, ga_i, X_i; gradient
// max and max diagonal of the varying cameras go to per-block partials.
template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(kCamWarps * 32) k_camera_finish(DevState s, const double* __restrict__ cpart,
                                                                   double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  using L = Lay<DA, DC, Real>;
  using CV = CamV<DA, DC>;
  constexpr int DCc = L::DCc;
  constexpr int PER = CV::VP / 32;
  __shared__ double red[kCamWarps * 2];
  const Dims& D = s.d;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * kCamWarps + (threadIdx.x >> 5);
  double v[2] = {-1e30, -1e30};
  if (i < D.N) {
    double sum[PER];
#pragma unroll
    for (int t = 0; t < PER; ++t) sum[t] = 0.0;
    sum_chunks<PER, CV::VP>(sum, cpart, s.cam_cc_ptr[i], s.cam_cc_ptr[i + 1], lane);
    Real* cU = reinterpret_cast<Real*>(s.c_U) + (size_t)i * L::SU;
    Real* cX = reinterpret_cast<Real*>(s.c_X) + (size_t)i * L::SX;
    double gm = 0.0, dm = -1e30;
#pragma unroll
    for (int t = 0; t < PER; ++t) {
      const int vi = lane + 32 * t;
      if (vi < CV::NU) {
        int r, c;
        unpack_sym<DA>(vi, r, c);
        cU[r * DA + c] = Real(sum[t]);
        cU[c * DA + r] = Real(sum[t]);
        if (r == c) dm = fmax(dm, sum[t]);
      } else if (vi < CV::NU + DA) {
        s.c_ga[(size_t)i * L::SG + (vi - CV::NU)] = sum[t];
        gm = fmax(gm, fabs(sum[t]));
      } else if (vi < CV::NV) {
        const int x = vi - CV::NU - DA;
        cX[(x / DCc) * DCc + x % DCc] = Real(sum[t]);
      }
    }
    gm = warp_max(gm);
    dm = warp_max(dm);
    if (i >= D.nnA) {
      v[0] = gm;
      v[1] = dm;
    }
  }
  block_reduce<2, 0>(v, red);
  store_partials(part, v);
}

// Sums the relinearisation partials: cost, Z, gc, gradient max, max diagonal, initial lambda.
template <int DC>
__global__ void __launch_bounds__(32 * kFoldWarps) k_relin_finalize(DevState s, const double* __restrict__ part_pt, int nbp,
                                                        const double* __restrict__ part_cam, int nbc,
                                                        int init_lambda, double tau) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  constexpr int NS = RelinNV<DC>::NS, NV = RelinNV<DC>::NV, NZ = nsym(DC);
  constexpr int DCc = DC > 0 ? DC : 1;
  __shared__ double red[NV * fold_segs(NV) > kFoldWarps ? NV * fold_segs(NV) : kFoldWarps];
  double a[NV];
  fold_partials<NV, NS>(part_pt, nbp, a, red);
  double b[2];
  fold_partials<2, 0>(part_cam, nbc, b, red);
  if (threadIdx.x == 0) {
    const Dims& D = s.d;
    double gmax = fmax(fmax(a[NS], b[0]), 0.0);
    double dmax = fmax(a[NS + 1], b[1]);
    if (DC > 0) {
      int z = 0;
      for (int r = 0; r < DCc; ++r)
        for (int c = r; c < DCc; ++c, ++z) {
          s.g_Z[r * DCc + c] = a[1 + z];
          s.g_Z[c * DCc + r] = a[1 + z];
          if (r == c && r >= D.nnC) dmax = fmax(dmax, a[1 + z]);
        }
      for (int c = 0; c < DCc; ++c) {
        s.g_gc[c] = a[1 + NZ + c];
        if (c >= D.nnC) gmax = fmax(gmax, fabs(a[1 + NZ + c]));
      }
    }
    s.d_relin[0] = a[0];
    s.d_relin[1] = gmax;
    s.d_relin[2] = dmax;
    if (init_lambda) *s.d_lambda = tau * dmax;
  }
}

// ---- reduced system ---------------------------------------------------------------------

template <int DC>
struct ElimNV {
  static constexpr int NZ = nsym(DC);
  static constexpr int NV = (DC > 0) ? NZ + DC : 1;
};

__device__ __forceinline__ bool inv3(const double a[6], double o[6]) {
  // inverse of the symmetric matrix [[a0,a1,a2],[a1,a3,a4],[a2,a4,a5]] by cofactors
  const double c00 = a[3] * a[5] - a[4] * a[4];
  const double c01 = a[2] * a[4] - a[1] * a[5];
  const double c02 = a[1] * a[4] - a[2] * a[3];
  const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
  if (!(det != 0.0) || !isfinite(det)) return false;
  const double id = 1.0 / det;
  o[0] = c00 * id;
  o[1] = c01 * id;
  o[2] = c02 * id;
  o[3] = (a[0] * a[5] - a[2] * a[2]) * id;
  o[4] = (a[1] * a[2] - a[0] * a[4]) * id;
  o[5] = (a[0] * a[3] - a[1] * a[1]) * id;
  return true;
}

// T_k = W_k Vinv_j of the FP32 blocks for kPtThreads consecutive observations, one per thread.  The blocks
// move through shared memory, so that all global accesses are whole lines; a thread inverts its point's
// V + lambda I itself (as k_point_eliminate's point blocks do, the same bits), which costs less than waiting
// for them.  One thread per point walking its track's blocks took 23 us for 375,000 observations and 368
// for 5.5M (2.1 of the copy's 6.5 TB/s); with these blocks in the same launch 19.5
// and about 140.
template <int DA, int DC>
__device__ __forceinline__ void products_body(const DevState& s, int bid) {
  using L = Lay<DA, DC, float>;
  __shared__ float4 sm[kPtThreads * L::SW / 4];
  const int tid = threadIdx.x, k0 = bid * kPtThreads, n = min(kPtThreads, s.d.K - k0), nv = n * L::SW / 4;
  const float4* src = reinterpret_cast<const float4*>(s.o_W + (size_t)k0 * L::SW);
  for (int e = tid; e < nv; e += kPtThreads) sm[e] = __ldg(src + e);
  double vi[6] = {0, 0, 0, 0, 0, 0};
  if (tid < n) {
    const int j = s.o_pt[k0 + tid];
    const double lam = *s.d_lambda;
    float vv[L::SV];
    vload(reinterpret_cast<const float*>(s.p_V) + (size_t)j * L::SV, vv);
    const double a[6] = {double(vv[0]) + lam, double(vv[1]), double(vv[2]), double(vv[3]) + lam, double(vv[4]),
                         double(vv[5]) + lam};
    if (j < s.d.nnB || !inv3(a, vi)) vi[0] = vi[1] = vi[2] = vi[3] = vi[4] = vi[5] = 0.0;
  }
  __syncthreads();
  if (tid < n) {
    float w[L::SW], t[L::SW];
    float4* own = sm + tid * (L::SW / 4);
#pragma unroll
    for (int q = 0; q < L::SW / 4; ++q) {
      const float4 x = own[q];
      w[4 * q] = x.x; w[4 * q + 1] = x.y; w[4 * q + 2] = x.z; w[4 * q + 3] = x.w;
    }
#pragma unroll
    for (int x = 0; x < L::SW; ++x) t[x] = 0.f;
#pragma unroll
    for (int r = 0; r < DA; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        t[r * 3 + c] = float(double(w[r * 3]) * vi[s3(0, c)] + double(w[r * 3 + 1]) * vi[s3(1, c)] +
                             double(w[r * 3 + 2]) * vi[s3(2, c)]);
#pragma unroll
    for (int q = 0; q < L::SW / 4; ++q) own[q] = make_float4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
  }
  __syncthreads();
  float4* dst = reinterpret_cast<float4*>(s.o_T + (size_t)k0 * L::SW);
  for (int e = tid; e < nv; e += kPtThreads) dst[e] = sm[e];
}

// One thread per point: Vinv_j = (V_j + lambda I)^-1, q_j = Vinv gb, Vinv Y_j; Y^T Vinv Y and Y^T q go to
// per-block partials.  With FP32 blocks, the blocks from nbp on form the observations' T_k.
template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(kPtThreads) k_point_eliminate(DevState s, double* __restrict__ part, int nbp) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  if constexpr (stores_products<Real>()) {
    if ((int)blockIdx.x >= nbp) {
      products_body<DA, DC>(s, blockIdx.x - nbp);
      return;
    }
  }
  using L = Lay<DA, DC, Real>;
  constexpr int DCc = L::DCc;
  constexpr int NV = ElimNV<DC>::NV;
  __shared__ double red[(kPtThreads / 32) * NV];
  const Dims& D = s.d;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  double v[NV];
#pragma unroll
  for (int t = 0; t < NV; ++t) v[t] = 0.0;
  if (j < D.M) {
    const double lam = *s.d_lambda;
    Real vv[L::SV];
    vload(reinterpret_cast<const Real*>(s.p_V) + (size_t)j * L::SV, vv);
    double a[6] = {double(vv[0]) + lam, double(vv[1]), double(vv[2]), double(vv[3]) + lam, double(vv[4]),
                   double(vv[5]) + lam};
    double vi[6] = {0, 0, 0, 0, 0, 0};
    const bool fixB = j < D.nnB;
    if (!fixB && !inv3(a, vi)) {
      *s.d_fail = 1;
      vi[0] = vi[1] = vi[2] = vi[3] = vi[4] = vi[5] = 0.0;
    }
    Real vo[L::SV];
#pragma unroll
    for (int t = 0; t < L::SV; ++t) vo[t] = t < 6 ? Real(vi[t]) : Real(0);
    vstore(reinterpret_cast<Real*>(s.p_Vinv) + (size_t)j * L::SV, vo);
    double gb[4];
    vload(s.p_gb + (size_t)j * 4, gb);
    double q[4] = {0, 0, 0, 0};
#pragma unroll
    for (int r = 0; r < 3; ++r) q[r] = vi[s3(r, 0)] * gb[0] + vi[s3(r, 1)] * gb[1] + vi[s3(r, 2)] * gb[2];
    vstore(s.p_q + (size_t)j * 4, q);
    if (DC > 0) {
      Real yv[L::SY];
      vload(reinterpret_cast<const Real*>(s.p_Y) + (size_t)j * L::SY, yv);
      double YV[3][DCc];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < DCc; ++c)
          YV[r][c] = vi[s3(r, 0)] * double(yv[c]) + vi[s3(r, 1)] * double(yv[DCc + c]) + vi[s3(r, 2)] * double(yv[2 * DCc + c]);
      Real yo[L::SY];
#pragma unroll
      for (int t = 0; t < L::SY; ++t) yo[t] = Real(0);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < DCc; ++c) yo[r * DCc + c] = Real(YV[r][c]);
      vstore(reinterpret_cast<Real*>(s.p_YV) + (size_t)j * L::SY, yo);
      int z = 0;
#pragma unroll
      for (int r = 0; r < DCc; ++r)
#pragma unroll
        for (int c = r; c < DCc; ++c, ++z)
          v[z] = double(yv[r]) * YV[0][c] + double(yv[DCc + r]) * YV[1][c] + double(yv[2 * DCc + r]) * YV[2][c];
#pragma unroll
      for (int c = 0; c < DCc; ++c)
        v[nsym(DC) + c] = double(yv[c]) * q[0] + double(yv[DCc + c]) * q[1] + double(yv[2 * DCc + c]) * q[2];
    }
  }
  block_reduce<NV, NV>(v, red);
  store_partials(part, v, (int)blockIdx.x, nbp);
}

// ---- Schur sums over the pair lists ------------------------------------------------------------
// One warp per chunk of a camera-pair block's observation pairs: partial sum T_k W_m^T (FP32 blocks: the
// stored T_k and W_m; FP64 blocks: A_k^T (B_k Vinv_j B_m^T) A_m).  The blocks of 32 pairs are copied to
// shared memory by the warp together, consecutive lanes on consecutive 16 bytes of a block.  Loads of a
// lane's own blocks touch a cache line per lane and instruction: the L1's wavefronts were 82% busy, at 5.1
// TB/s from L2 and 16% of the FP64 pipe.  Staged, FP32 blocks read at 8 TB/s from L2, which is the bound: the
// launch with the rhs chunks went 1,487 -> 929 us on 2,000 cameras (35M pairs), the sums alone 60 -> 48 us on
// 200 (1.8M pairs, FP64 118 -> 103).

// Shared memory of a warp, in bytes.
template <int DA, typename Real>
__host__ __device__ constexpr int schur_stage_bytes() {
  using L = Lay<DA, 0, Real>;
  return stores_products<Real>() ? 2 * 32 * 2 * L::SW * (int)sizeof(float)
                                 : 32 * (2 * L::SA + 2 * kSB + L::SV + 4) * (int)sizeof(double);
}

template <int DA>
__device__ __forceinline__ void schur_chunk_fp32(const DevState& s, double* __restrict__ part, float* sm, int ch, int lane) {
  using L = Lay<DA, 0, float>;
  using SV = SchurV<DA>;
  float acc[SV::VP];
#pragma unroll
  for (int t = 0; t < SV::VP; ++t) acc[t] = 0.f;
  // the chunk's indices first, then the blocks of the next 32 pairs in flight during the current ones
  constexpr int R = kPairChunk / 32, kBuf = 32 * 2 * L::SW;
  const int beg = s.bc_beg[ch], n = s.bc_end[ch] - beg;
  int k[R], m[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const bool in = 32 * u + lane < n;
    k[u] = in ? s.pr_k[beg + 32 * u + lane] : -1;
    m[u] = in ? s.pr_m[beg + 32 * u + lane] : -1;
  }
  auto fetch = [&](int u) {
    float* b = sm + (u & 1) * kBuf;
    stage_blocks<L::SW>(b, (const float*)s.o_T, k[u], lane);
    stage_blocks<L::SW>(b + 32 * L::SW, (const float*)s.o_W, m[u], lane);
    cp_commit();
  };
  fetch(0);
#pragma unroll
  for (int u = 0; u < R; ++u) {
    if (32 * u >= n) break;
    if (u + 1 < R && 32 * (u + 1) < n) {
      fetch(u + 1);
      cp_join_but_last();
    } else {
      cp_join();
    }
    if (32 * u + lane < n) {
      const float* b = sm + (u & 1) * kBuf + lane * L::SW;
      float t[L::SW], w[L::SW];
#pragma unroll
      for (int q = 0; q < L::SW / 4; ++q) {
        const float4 x = reinterpret_cast<const float4*>(b)[q], y = reinterpret_cast<const float4*>(b + 32 * L::SW)[q];
        t[4 * q] = x.x; t[4 * q + 1] = x.y; t[4 * q + 2] = x.z; t[4 * q + 3] = x.w;
        w[4 * q] = y.x; w[4 * q + 1] = y.y; w[4 * q + 2] = y.z; w[4 * q + 3] = y.w;
      }
#pragma unroll
      for (int a = 0; a < DA; ++a)
#pragma unroll
        for (int c = 0; c < DA; ++c)
          acc[a * DA + c] += t[a * 3] * w[c * 3] + t[a * 3 + 1] * w[c * 3 + 1] + t[a * 3 + 2] * w[c * 3 + 2];
    }
    __syncwarp();
  }
  warp_reduce_transpose(acc);
#pragma unroll
  for (int t = 0; t < SV::VP / 32; ++t) part[(size_t)ch * SV::VP + lane * (SV::VP / 32) + t] = double(acc[t]);
}

// With the residual rows of the 32 pairs as the inner dimension, sum A_k^T M A_m on DMMA, M = B_k Vinv_j
// B_m^T from a lane's own pair.
template <int DA>
__device__ __forceinline__ void schur_chunk_fp64(const DevState& s, double* __restrict__ part, double* sm, int ch, int lane) {
  using L = Lay<DA, 0, double>;
  using SV = SchurV<DA>;
  constexpr int NT = (DA + 7) / 8, SA = L::SA;
  double* Ak = sm;
  double* Am = Ak + 32 * SA;
  double* Bk = Am + 32 * SA;
  double* Bm = Bk + 32 * kSB;
  double* Vi = Bm + 32 * kSB;
  double* Mx = Vi + 32 * L::SV;    // [32][2][2]
  double acc[2][NT][NT][2];        // two sets, for even and odd steps (shorter DMMA chains)
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int a = 0; a < NT; ++a)
#pragma unroll
      for (int c = 0; c < NT; ++c) acc[u][a][c][0] = acc[u][a][c][1] = 0.0;
  const int beg = s.bc_beg[ch], n = s.bc_end[ch] - beg, r = lane >> 2, kk = lane & 3;
  constexpr int R = kPairChunk / 32;
  int ks[R], ms[R], js[R];   // the chunk's indices first
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const bool in = 32 * u + lane < n;
    ks[u] = in ? s.pr_k[beg + 32 * u + lane] : -1;
    ms[u] = in ? s.pr_m[beg + 32 * u + lane] : -1;
  }
#pragma unroll
  for (int u = 0; u < R; ++u) js[u] = ks[u] >= 0 ? s.o_pt[ks[u]] : -1;
#pragma unroll
  for (int u = 0; u < R; ++u) {
    if (32 * u >= n) break;
    const int k = ks[u], m = ms[u], j = js[u];
    stage_blocks<SA>(Ak, reinterpret_cast<const double*>(s.o_A), k, lane);
    stage_blocks<kSB>(Bk, (const double*)s.o_B, k, lane);
    stage_blocks<SA>(Am, reinterpret_cast<const double*>(s.o_A), m, lane);
    stage_blocks<kSB>(Bm, (const double*)s.o_B, m, lane);
    stage_blocks<L::SV>(Vi, reinterpret_cast<const double*>(s.p_Vinv), j, lane);
    cp_join();
    {
      double bk[6], bm[6], vi[6];
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const double2 x = reinterpret_cast<const double2*>(Bk + kSB * lane)[t], y = reinterpret_cast<const double2*>(Bm + kSB * lane)[t],
                      z = reinterpret_cast<const double2*>(Vi + L::SV * lane)[t];
        bk[2 * t] = x.x; bk[2 * t + 1] = x.y;
        bm[2 * t] = y.x; bm[2 * t + 1] = y.y;
        vi[2 * t] = z.x; vi[2 * t + 1] = z.y;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        double Q[3];   // row q of B_k Vinv_j
#pragma unroll
        for (int c = 0; c < 3; ++c) Q[c] = bk[3 * q] * vi[s3(0, c)] + bk[3 * q + 1] * vi[s3(1, c)] + bk[3 * q + 2] * vi[s3(2, c)];
        reinterpret_cast<double2*>(Mx)[2 * lane + q] =
            make_double2(Q[0] * bm[0] + Q[1] * bm[1] + Q[2] * bm[2], Q[0] * bm[3] + Q[1] * bm[4] + Q[2] * bm[5]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int st = 0; st < 16; ++st) {   // two pairs a step: inner index kk = 2 (pair) + (residual row)
      const int q = 2 * st + (kk >> 1);
      const double2 mm = reinterpret_cast<const double2*>(Mx)[2 * q + (kk & 1)];
      double a[NT], z[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int row = 8 * t + r;
        const bool ok = row < DA;
        const double* am = Am + q * SA + (ok ? row : 0);
        a[t] = ok ? Ak[q * SA + (kk & 1) * DA + row] : 0.0;
        z[t] = ok ? mm.x * am[0] + mm.y * am[DA] : 0.0;
      }
#pragma unroll
      for (int ta = 0; ta < NT; ++ta)
#pragma unroll
        for (int tc = 0; tc < NT; ++tc) dmma884(acc[st & 1][ta][tc], a[ta], z[tc]);
    }
    __syncwarp();
  }
#pragma unroll
  for (int ta = 0; ta < NT; ++ta)
#pragma unroll
    for (int tc = 0; tc < NT; ++tc)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int row = 8 * ta + r, col = 8 * tc + 2 * kk + t;
        if (row < DA && col < DA) part[(size_t)ch * SV::VP + row * DA + col] = acc[0][ta][tc][t] + acc[1][ta][tc][t];
      }
}

// The same sums from a lane's own loads (DIRECT): where tracks see a camera more than once (a rig's two
// cameras in one pose), neighbouring pairs share their blocks, and the shared lines and the L1 serve them
// (300 rig poses, 3.2M pairs, FP32 blocks: 64 us, staged 68); and for a launch of a single wave, where a
// chunk's latency counts and the copies add to it (20 cameras, 268 chunks, FP64: 7.1 us, staged 8.7).
constexpr int kDirectChunks = 1184;   // two blocks of four chunks on each of 148 SMs
// (the direct FP64 sums of more than 9 unknowns per camera spill their accumulators)
template <int DA, typename Real>
__host__ __device__ constexpr bool has_direct() { return stores_products<Real>() || DA <= 9; }
template <int DA, typename Real>
bool schur_direct(const DevState& s) { return has_direct<DA, Real>() && (s.repeats || s.nch_blk <= kDirectChunks); }

// FP32 blocks: the sums in the same order as schur_chunk_fp32.  Two pairs a trip, so both pairs' gathers
// are in flight, except with 13 unknowns per camera, whose blocks already fill the register file.
template <int DA>
__device__ __forceinline__ void schur_chunk_fp32_direct(const DevState& s, double* __restrict__ part, int ch, int lane) {
  using L = Lay<DA, 0, float>;
  using SV = SchurV<DA>;
  constexpr int U = DA <= 11 ? 2 : 1;
  float acc[SV::VP];
#pragma unroll
  for (int t = 0; t < SV::VP; ++t) acc[t] = 0.f;
  const int end = s.bc_end[ch];
  for (int p = s.bc_beg[ch] + lane; p < end; p += 32 * U) {
    float t[U][L::SW], w[U][L::SW];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = p + 32 * u < end ? p + 32 * u : p;   // a missing second pair re-reads the first
      vload(s.o_T + (size_t)s.pr_k[q] * L::SW, t[u]);
      vload(s.o_W + (size_t)s.pr_m[q] * L::SW, w[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u > 0 && p + 32 * u >= end) break;
#pragma unroll
      for (int a = 0; a < DA; ++a)
#pragma unroll
        for (int c = 0; c < DA; ++c)
          acc[a * DA + c] += t[u][a * 3] * w[u][c * 3] + t[u][a * 3 + 1] * w[u][c * 3 + 1] +
                             t[u][a * 3 + 2] * w[u][c * 3 + 2];
    }
  }
  warp_reduce_transpose(acc);
#pragma unroll
  for (int t = 0; t < SV::VP / 32; ++t) part[(size_t)ch * SV::VP + lane * (SV::VP / 32) + t] = double(acc[t]);
}

template <int DA>
__device__ __forceinline__ void schur_chunk_fp64_direct(const DevState& s, double* __restrict__ part, int ch, int lane) {
  using L = Lay<DA, 0, double>;
  using SV = SchurV<DA>;
  double acc[SV::VP];
#pragma unroll
  for (int t = 0; t < SV::VP; ++t) acc[t] = 0.0;
  const double* oA = reinterpret_cast<const double*>(s.o_A);
  const int end = s.bc_end[ch];
  for (int p = s.bc_beg[ch] + lane; p < end; p += 32) {
    const int k = s.pr_k[p], m = s.pr_m[p];
    const int j = s.o_pt[k];
    double Ak[L::SA], Am[L::SA], Bk[kSB], Bm[kSB], vi[L::SV];
    vload(oA + (size_t)k * L::SA, Ak);
    vload(s.o_B + (size_t)k * kSB, Bk);
    vload(oA + (size_t)m * L::SA, Am);
    vload(s.o_B + (size_t)m * kSB, Bm);
    vload(reinterpret_cast<const double*>(s.p_Vinv) + (size_t)j * L::SV, vi);
    double Q[2][3];   // B_k Vinv_j
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        Q[r][c] = Bk[3 * r] * vi[s3(0, c)] + Bk[3 * r + 1] * vi[s3(1, c)] + Bk[3 * r + 2] * vi[s3(2, c)];
    double Mx[2][2];  // B_k Vinv_j B_m^T
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int t = 0; t < 2; ++t) Mx[r][t] = Q[r][0] * Bm[3 * t] + Q[r][1] * Bm[3 * t + 1] + Q[r][2] * Bm[3 * t + 2];
#pragma unroll
    for (int c = 0; c < DA; ++c) {
      const double n0 = Mx[0][0] * Am[c] + Mx[0][1] * Am[DA + c];
      const double n1 = Mx[1][0] * Am[c] + Mx[1][1] * Am[DA + c];
#pragma unroll
      for (int a = 0; a < DA; ++a) acc[a * DA + c] += Ak[a] * n0 + Ak[DA + a] * n1;
    }
  }
  warp_reduce_transpose(acc);
#pragma unroll
  for (int t = 0; t < SV::VP / 32; ++t) part[(size_t)ch * SV::VP + lane * (SV::VP / 32) + t] = acc[t];
}

template <int DA, typename Real, bool DIRECT>
__device__ __forceinline__ void schur_chunks_body(DevState s, double* __restrict__ part, int bid, int nblk) {
  extern __shared__ double stage_sm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ch = bid * 4 + w;
  if (ch >= s.nch_blk) return;
  if constexpr (DIRECT && has_direct<DA, Real>()) {
    if constexpr (stores_products<Real>()) schur_chunk_fp32_direct<DA>(s, part, ch, lane);
    else schur_chunk_fp64_direct<DA>(s, part, ch, lane);
  } else {
    char* sm = reinterpret_cast<char*>(stage_sm) + w * schur_stage_bytes<DA, Real>();
    if constexpr (stores_products<Real>()) schur_chunk_fp32<DA>(s, part, reinterpret_cast<float*>(sm), ch, lane);
    else schur_chunk_fp64<DA>(s, part, reinterpret_cast<double*>(sm), ch, lane);
  }
}

// FP64 blocks, points grouped by their cameras: one block per chunk of up to 32 points that the same L
// cameras see.  With (V + lambda I)^-1 = F N F^T and G_k = A_k^T (B_k F) the chunk's part of the whole L x L
// block matrix is G N G^T, G one row per camera unknown and three columns per point, formed in shared memory
// (observations of a point in the same camera add up first) and multiplied with DMMA; N multiplies the left
// fragment, nine FMAs for nine DMMAs.
// F is C^-T of the Cholesky factor of V + lambda I and N = I, while every pivot keeps kGroupPivot of its diagonal
// entry: the rounding of G then counts by B C^-T, whose entries are at most 1, and not by the condition number
// of V (F = I throughout gave 24-iteration runs of 200 cameras 8% more error).  Below that rounding decides about
// the pivot, and F = I with N = k_point_eliminate's own inverse, which the pair lists, the right-hand side and
// the step use: the system stays one and the same.  (C^-T there left a point out, or turned a pivot's sign, that
// the other parts kept.)
// Every observation's blocks are read once per trial instead of once per pair (144 bytes instead of 340
// times the pairs of its track), the gathers that bound the pair lists: their L2 to L1 traffic was 870
// MB at 5.8 TB/s (pairs staged through shared memory and multiplied with DMMA reached 9.4 TB/s, and no
// more).  200 cameras, 50,000 points, 1.8M pairs: 118.6 -> 49.6 us (finish 4.3 -> 8.5); 300 rig poses,
// 40,000 points, 3.2M pairs (two observations per pose): 118 -> 48 us (5.7 -> 6.8).  Bound by the
// latency of a chunk (pattern, blocks, product): the DMMAs are 14 us of it.
constexpr int kGroupThreads = 256;
constexpr double kGroupPivot = 1e-8;
template <int DA>
__device__ __forceinline__ void schur_group_body(const DevState& s, int ch) {
  using L_ = Lay<DA, 0, double>;
  extern __shared__ double group_sm[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int4 d = reinterpret_cast<const int4*>(s.gr_desc)[ch];
  const int p0 = d.x, np = d.y, e0 = d.z, L = d.w;
  const int rows = DA * L, ld = group_ld(rows), nq = group_pad(np);
  double* Gs = group_sm;
  double* Ns = Gs + 3 * nq * ld + 8;                     // [nq][6] N (00 01 02 11 12 22)
  double* Fs = Ns + 6 * nq;                              // [np][6] F^T (00 10 11 20 21 22)
  int* first = reinterpret_cast<int*>(Fs + 6 * nq);      // [np] first observation of the point
  int* rank = first + kGroupPoints;                      // [track] rank of the observation's camera
  int* head = rank + kGroupTrack;                        // [L] first observation in the camera ...
  int* next = head + kGroupTrack;                        // [track] ... and the next one, or -1
  if (tid < np) {
    const int j = s.gr_pt[p0 + tid];
    first[tid] = s.p_ptr[j];
    const double lam = *s.d_lambda;
    double V[L_::SV], vi[L_::SV];   // (vi: zero for a fixed point and a singular one, which k_point_eliminate reports)
    vload(reinterpret_cast<const double*>(s.p_V) + (size_t)j * L_::SV, V);
    vload(reinterpret_cast<const double*>(s.p_Vinv) + (size_t)j * L_::SV, vi);
    const double i0 = rsqrt(V[0] + lam), l10 = V[1] * i0, l20 = V[2] * i0;
    const double d1 = V[3] + lam - l10 * l10, i1 = rsqrt(d1), l21 = (V[4] - l20 * l10) * i1;
    const double d2 = V[5] + lam - l20 * l20 - l21 * l21, i2 = rsqrt(d2);
    const bool plain = V[0] + lam > 0.0 && d1 > kGroupPivot * (V[3] + lam) && d2 > kGroupPivot * (V[5] + lam) &&
                       isfinite(i0) && isfinite(i1) && isfinite(i2) && vi[0] != 0.0;
    const double c10 = -l10 * i0 * i1;
    const double F[6] = {i0, c10, i1, -(l20 * i0 + l21 * c10) * i2, -l21 * i1 * i2, i2};
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      Fs[6 * tid + t] = plain ? F[t] : (t == 0 || t == 2 || t == 5) ? 1.0 : 0.0;
      Ns[6 * tid + t] = !plain ? vi[t] : (t == 0 || t == 3 || t == 5) ? 1.0 : 0.0;
    }
  } else if (tid < nq) {                                 // the last DMMA steps' padding
#pragma unroll
    for (int t = 0; t < 6; ++t) Ns[6 * tid + t] = 0.0;
  } else if (tid >= kGroupThreads - kGroupTrack) {       // two other warps: the pattern
    const int t = tid - (kGroupThreads - kGroupTrack), j = s.gr_pt[p0], k0 = s.p_ptr[j], n = s.p_ptr[j + 1] - k0;
    rank[t] = t < n ? (int)s.gr_rank[k0 + t] : -1;
  }
  for (int e = 3 * np * ld + tid; e < 3 * nq * ld; e += kGroupThreads) Gs[e] = 0.0;   // (padding too)
  __syncthreads();
  if (tid < kGroupTrack) {
    int h = -1, nx = -1;
    const int mine = rank[tid];
    for (int u = kGroupTrack - 1; u >= 0; --u) {
      const int ru = rank[u];
      if (ru == tid) h = u;
      if (u > tid && ru == mine) nx = u;
    }
    head[tid] = h;
    next[tid] = nx;
  }
  __syncthreads();
  // one column (of three) of a point's rows in one camera per thread
  for (int idx = tid; idx < 3 * np * L; idx += kGroupThreads) {
    const int q = idx / (3 * L), rest = idx - q * 3 * L, sl = rest / 3, u = rest - 3 * sl;
    const double* f = Fs + 6 * q;
    const double f0 = u == 0 ? f[0] : u == 1 ? f[1] : f[3], f1 = u == 0 ? 0.0 : u == 1 ? f[2] : f[4], f2 = u == 2 ? f[5] : 0.0;
    double g[DA];
#pragma unroll
    for (int a = 0; a < DA; ++a) g[a] = 0.0;
    for (int t = head[sl]; t >= 0; t = next[t]) {
      const size_t k = (size_t)(first[q] + t);
      double A[L_::SA], B[kSB];
      vload(reinterpret_cast<const double*>(s.o_A) + k * L_::SA, A);
      vload(s.o_B + k * kSB, B);
      const double h0 = B[0] * f0 + B[1] * f1 + B[2] * f2, h1 = B[3] * f0 + B[4] * f1 + B[5] * f2;   // of B_k F
#pragma unroll
      for (int a = 0; a < DA; ++a) g[a] += A[a] * h0 + A[DA + a] * h1;
    }
    double* out = Gs + (3 * q + u) * ld + DA * sl;
#pragma unroll
    for (int a = 0; a < DA; ++a) out[a] = g[a];
  }
  __syncthreads();
  // lower tiles of G N G^T, up to three of a tile row at a time (they share the row's fragment); three DMMA
  // steps take four points, lane kk = 0..3 of a step one column of point kk
  const int T = (rows + 7) / 8, r = lane >> 2, kk = lane & 3;
  int unit = 0;
  for (int ti = T - 1; ti >= 0; --ti)
    for (int tj = 0; tj <= ti; tj += 3, ++unit) {
      if (unit % (kGroupThreads / 32) != (tid >> 5)) continue;
      const int nt = min(3, ti - tj + 1);
      double acc[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
      const double* ga = Gs + 3 * kk * ld + 8 * ti + r;
      const double* gb = Gs + 3 * kk * ld + 8 * tj + r;
      const double2* vp = reinterpret_cast<const double2*>(Ns + 6 * kk);
      for (int q = 0; q < nq; q += 4, ga += 12 * ld, gb += 12 * ld, vp += 12) {
        const double2 v0 = vp[0], v1 = vp[1], v2 = vp[2];   // 00 01, 02 11, 12 22
        const double g0 = ga[0], g1 = ga[ld], g2 = ga[2 * ld];
        const double a[3] = {v0.x * g0 + v0.y * g1 + v1.x * g2, v0.y * g0 + v1.y * g1 + v2.x * g2,
                             v1.x * g0 + v2.x * g1 + v2.y * g2};
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          dmma884(acc[0], a[u], gb[u * ld]);
          if (nt > 1) dmma884(acc[1], a[u], gb[u * ld + 8]);
          if (nt > 2) dmma884(acc[2], a[u], gb[u * ld + 16]);
        }
      }
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        if (t >= nt) break;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int R = 8 * ti + r, C = 8 * (tj + t) + 2 * kk + u;
          if (R >= rows || C > R) continue;
          const int sr = R / DA, sc = C / DA;
          s.gr_part[(size_t)(e0 + sr * (sr + 1) / 2 + sc) * (DA * DA) + (R - sr * DA) * DA + (C - sc * DA)] = acc[t][u];
        }
      }
    }
}

template <int DA>
__global__ void __launch_bounds__(kGroupThreads, DA <= 9 ? 3 : 2) k_schur_groups(DevState s) {
  pdl_wait();
  pdl_trigger();
  schur_group_body<DA>(s, blockIdx.x);
}

template <int DA, typename Real, bool DIRECT>
__global__ void __launch_bounds__(128) k_schur_chunks(DevState s, double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  schur_chunks_body<DA, Real, DIRECT>(s, part, blockIdx.x, gridDim.x);
}

// One warp per camera-pair block (i <= l): S_il = delta_il (U_i + lambda I) - sum of its chunk
// partials, written into the lower triangle of the dense column-major S.
template <int DA, typename Real>
__device__ __forceinline__ void schur_finish_body(DevState s, const double* __restrict__ part, int bid, int nblk,
                                                  bool skip_fixed_diag = false) {
  using L = Lay<DA, 0, Real>;
  using SV = SchurV<DA>;
  constexpr int PER = SV::VP / 32;
  const int lane = threadIdx.x & 31;
  const bool grouped = !stores_products<Real>() && s.gr_n > 0;
  const int b = grouped ? bid : bid * 4 + (threadIdx.x >> 5);
  if (b >= s.nb) return;
  const int i = s.b_i[b], l = s.b_l[b];
  // beside rhs_finish in one launch, the identity block of a fixed camera is rhs_finish's alone
  if (skip_fixed_diag && i == l && i < s.d.nnA) return;
  double sum[PER];
#pragma unroll
  for (int t = 0; t < PER; ++t) sum[t] = 0.0;
  if (grouped) {
    // Grouped points: the four warps take the block's partial sums in turn, four in flight each (a
    // camera's own block has one per chunk that the camera is in), and add up in warp order.  A partial
    // sum holds the rows of the later camera; of a camera with itself, the lower triangle.
    __shared__ double ws[3][SV::VP];
    const int w = threadIdx.x >> 5;
    int at[PER];
#pragma unroll
    for (int t = 0; t < PER; ++t) {
      const int e = min(lane + 32 * t, SV::NV - 1), a = e / DA, c = e % DA;
      at[t] = (i == l && a > c) ? a * DA + c : c * DA + a;
    }
    const int e1 = s.gr_bptr[b + 1];
    for (int e = s.gr_bptr[b] + w; e < e1; e += 16) {
      double v[4][PER];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double* p = s.gr_part + (size_t)s.gr_ent[min(e + 4 * u, e1 - 1)] * (DA * DA);
#pragma unroll
        for (int t = 0; t < PER; ++t) v[u][t] = p[at[t]];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int t = 0; t < PER; ++t) sum[t] += e + 4 * u < e1 ? v[u][t] : 0.0;
    }
    if (w > 0)
#pragma unroll
      for (int t = 0; t < PER; ++t) ws[w - 1][lane + 32 * t] = sum[t];
    __syncthreads();
    if (w > 0) return;
#pragma unroll
    for (int t = 0; t < PER; ++t) sum[t] += ws[0][lane + 32 * t] + ws[1][lane + 32 * t] + ws[2][lane + 32 * t];
  } else {
    sum_chunks<PER, SV::VP>(sum, part, s.blk_bc_ptr[b], s.blk_bc_ptr[b + 1], lane);
  }
  const double lam = *s.d_lambda;
  const Real* cU = reinterpret_cast<const Real*>(s.c_U) + (size_t)i * L::SU;
  const size_t ld = s.ld;
#pragma unroll
  for (int t = 0; t < PER; ++t) {
    const int e = lane + 32 * t;
    if (e >= SV::NV) continue;
    const int a = e / DA, c = e % DA;
    double val = -sum[t];
    if (i == l) val += double(cU[a * DA + c]) + (a == c ? lam : 0.0);
    if (s.Sb) {
      reinterpret_cast<Real*>(s.Sb)[(size_t)b * DA * DA + a * DA + c] = Real(val);
    } else {
      // element (row l*DA + c, col i*DA + a) of the lower triangle holds S_il[a][c]
      s.S[(size_t)(i * DA + a) * ld + (l * DA + c)] = val;
    }
  }
}

template <int DA, typename Real>
__global__ void __launch_bounds__(128) k_schur_finish(DevState s, const double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  schur_finish_body<DA, Real>(s, part, blockIdx.x, gridDim.x);
}

// Whether the rhs chunks are staged: FP64 blocks stay with a lane's own loads where the sums are 32 values
// or less and the tile mostly padding: few border columns (158 cameras, DC = 1: 8.2 us against 12.5
// staged), or more unknowns than a tile's eight rows (30 cameras, DA = 11: 188 us an iteration against 198).
template <int DA, int DC, typename Real>
__host__ __device__ constexpr bool rhs_staged() {
  return stores_products<Real>() || RhsV<DA, DC>::VP > 32 || (DC == 0 && DA <= 8);
}
// Shared memory of a warp of the rhs chunks, in bytes.
template <int DA, int DC, typename Real>
__host__ __device__ constexpr int rhs_stage_bytes() {
  using L = Lay<DA, DC, Real>;
  return !rhs_staged<DA, DC, Real>() ? 0 : 32 * (4 * (int)sizeof(double) + (DC > 0 ? L::SY * (int)sizeof(Real) : 0) +
               (stores_products<Real>() ? L::SW * (int)sizeof(float) : (L::SA + kSB) * (int)sizeof(double)));
}

// One warp per chunk of a camera's observations: partial sum_k W_k q_j(k) and sum_k T_k Y_j(k),
// the latter as sum_k W_k (Vinv Y)_j(k), together the product of the W_k with the 1 + DC <= 8 columns
// [q Vinv Y] of their points: with FP32 blocks the inner dimension is the points' three coordinates (four
// observations in three DMMA steps), with FP64 blocks the residual rows (W_k x = A_k^T (B_k x)).  200 cameras,
// DC = 7: FP32 blocks 25 -> 14 us, FP64 32 -> 26.
template <int DA, int DC, typename Real, int WARPS = kCamWarps>
__device__ __forceinline__ void rhs_chunks_body(DevState s, double* __restrict__ part, int bid, int nblk) {
  using L = Lay<DA, DC, Real>;
  using RV = RhsV<DA, DC>;
  constexpr int DCc = L::DCc, NT = (DA + 7) / 8;
  static_assert(DC <= 7, "the right-hand side and the border are eight columns");
  extern __shared__ double stage_sm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = lane >> 2, kk = lane & 3;
  const int ch = bid * WARPS + w;
  if (w >= WARPS || ch >= s.nch_cam) return;
  if constexpr (!rhs_staged<DA, DC, Real>()) {
    double acc[RV::VP];
#pragma unroll
    for (int t = 0; t < RV::VP; ++t) acc[t] = 0.0;
    for (int idx = s.cc_beg[ch] + lane; idx < s.cc_end[ch]; idx += 32) {
      const int k = s.c_obs[idx];
      const int j = s.o_pt[k];
      double q[4], A[L::SA], B[kSB];
      vload(s.p_q + (size_t)j * 4, q);
      vload(reinterpret_cast<const double*>(s.o_A) + (size_t)k * L::SA, A);
      vload(s.o_B + (size_t)k * kSB, B);
      const double bq0 = B[0] * q[0] + B[1] * q[1] + B[2] * q[2];
      const double bq1 = B[3] * q[0] + B[4] * q[1] + B[5] * q[2];
#pragma unroll
      for (int a = 0; a < DA; ++a) acc[a] += A[a] * bq0 + A[DA + a] * bq1;
      if (DC > 0) {
        double yv[L::SY];
        vload(reinterpret_cast<const double*>(s.p_YV) + (size_t)j * L::SY, yv);
#pragma unroll
        for (int c = 0; c < DCc; ++c) {
          const double by0 = B[0] * yv[c] + B[1] * yv[DCc + c] + B[2] * yv[2 * DCc + c];
          const double by1 = B[3] * yv[c] + B[4] * yv[DCc + c] + B[5] * yv[2 * DCc + c];
#pragma unroll
          for (int a = 0; a < DA; ++a) acc[DA + a * DCc + c] += A[a] * by0 + A[DA + a] * by1;
        }
      }
    }
    warp_reduce_transpose(acc);
#pragma unroll
    for (int t = 0; t < RV::VP / 32; ++t) part[(size_t)ch * RV::VP + lane * (RV::VP / 32) + t] = acc[t];
    return;
  }
  char* sm = reinterpret_cast<char*>(stage_sm) + w * rhs_stage_bytes<DA, DC, Real>();
  double* Q = reinterpret_cast<double*>(sm);
  Real* Y = reinterpret_cast<Real*>(Q + 32 * 4);
  char* rest = reinterpret_cast<char*>(Y + (DC > 0 ? 32 * L::SY : 0));
  float* W = reinterpret_cast<float*>(rest);           // FP32 blocks
  double* A = reinterpret_cast<double*>(rest);         // FP64 blocks
  double* B = A + 32 * L::SA;
  double acc[2][NT][2];   // two sets in turn (shorter DMMA chains)
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int a = 0; a < NT; ++a) acc[v][a][0] = acc[v][a][1] = 0.0;
  // element c of column r of an entry's [q Vinv Y]
  auto column = [&](int q, int c) -> double {
    return r == 0 ? Q[4 * q + c] : (DC > 0 && r <= DC) ? double(Y[q * L::SY + c * DCc + r - 1]) : 0.0;
  };
  constexpr int RD = kCamChunk / 32;
  const int beg = s.cc_beg[ch], n = s.cc_end[ch] - beg;
  int ks[RD], js[RD];   // the chunk's indices first
#pragma unroll
  for (int v = 0; v < RD; ++v) ks[v] = 32 * v + lane < n ? s.c_obs[beg + 32 * v + lane] : -1;
#pragma unroll
  for (int v = 0; v < RD; ++v) js[v] = ks[v] >= 0 ? s.o_pt[ks[v]] : -1;
#pragma unroll
  for (int v = 0; v < RD; ++v) {
    if (32 * v >= n) break;
    const int k = ks[v], j = js[v];
    stage_blocks<4>(Q, (const double*)s.p_q, j, lane);
    if (DC > 0) stage_blocks<L::SY>(Y, reinterpret_cast<const Real*>(s.p_YV), j, lane);
    if constexpr (stores_products<Real>()) {
      stage_blocks<L::SW>(W, (const float*)s.o_W, k, lane);
    } else {
      stage_blocks<L::SA>(A, reinterpret_cast<const double*>(s.o_A), k, lane);
      stage_blocks<kSB>(B, (const double*)s.o_B, k, lane);
    }
    cp_join();
    if constexpr (stores_products<Real>()) {
#pragma unroll
      for (int st = 0; st < 24; ++st) {
        const int i = 4 * (st % 3) + kk, q = 4 * (st / 3) + i / 3, c = i % 3;
        const double z = column(q, c);
#pragma unroll
        for (int t = 0; t < NT; ++t)
          dmma884(acc[st & 1][t], 8 * t + r < DA ? double(W[q * L::SW + (8 * t + r) * 3 + c]) : 0.0, z);
      }
    } else {
#pragma unroll
      for (int st = 0; st < 16; ++st) {
        const int q = 2 * st + (kk >> 1), rr = kk & 1;
        const double* b = B + kSB * q + 3 * rr;
        const double z = b[0] * column(q, 0) + b[1] * column(q, 1) + b[2] * column(q, 2);
#pragma unroll
        for (int t = 0; t < NT; ++t)
          dmma884(acc[st & 1][t], 8 * t + r < DA ? A[q * L::SA + rr * DA + 8 * t + r] : 0.0, z);
      }
    }
    __syncwarp();
  }
  double* out = part + (size_t)ch * RV::VP;
#pragma unroll
  for (int ta = 0; ta < NT; ++ta) {
    const int R = 8 * ta + r;
    if (R >= DA) continue;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int col = 2 * kk + t;
      const double v = acc[0][ta][t] + acc[1][ta][t];
      if (col == 0) out[R] = v;
      else if (DC > 0 && col <= DC) out[DA + R * DCc + col - 1] = v;
    }
  }
}

template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(kCamWarps * 32) k_rhs_chunks(DevState s, double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  rhs_chunks_body<DA, DC, Real>(s, part, blockIdx.x, gridDim.x);
}

// One warp per camera: rhs_i = ga_i - sum W q and the camera/global border X_i - sum T Y into S;
// identity block, zero rhs and zero border for fixed cameras.
template <int DA, int DC, typename Real>
__device__ __forceinline__ void rhs_finish_body(DevState s, const double* __restrict__ cpart, int bid, int nblk) {
  using L = Lay<DA, DC, Real>;
  using RV = RhsV<DA, DC>;
  constexpr int DCc = L::DCc;
  constexpr int PER = RV::VP / 32;
  const Dims& D = s.d;
  const int lane = threadIdx.x & 31;
  const int i = bid * kCamWarps + (threadIdx.x >> 5);
  if (i >= D.N) return;
  const size_t ld = s.ld, rs = s.rhs_stride;
  const int c0 = D.N * DA;
  if (i < D.nnA) {
    for (int t = lane; t < DA * DA; t += 32) {
      const int a = t / DA, c = t % DA;
      if (s.Sb) reinterpret_cast<Real*>(s.Sb)[(size_t)s.diag_blk[i] * DA * DA + t] = Real(a == c ? 1.0 : 0.0);
      else s.S[(size_t)(i * DA + a) * ld + (i * DA + c)] = (a == c) ? 1.0 : 0.0;
    }
    for (int a = lane; a < DA; a += 32) s.rhs[(size_t)(i * DA + a) * rs] = 0.0;
    if (!s.Sb)
      for (int t = lane; t < RV::NX; t += 32) s.S[(size_t)(i * DA + t / DCc) * ld + c0 + t % DCc] = 0.0;
    return;
  }
  double sum[PER];
#pragma unroll
  for (int t = 0; t < PER; ++t) sum[t] = 0.0;
  sum_chunks<PER, RV::VP>(sum, cpart, s.cam_cc_ptr[i], s.cam_cc_ptr[i + 1], lane);
  const Real* cX = reinterpret_cast<const Real*>(s.c_X) + (size_t)i * L::SX;
#pragma unroll
  for (int t = 0; t < PER; ++t) {
    const int e = lane + 32 * t;
    if (e < DA) {
      s.rhs[(size_t)(i * DA + e) * rs] = s.c_ga[(size_t)i * L::SG + e] - sum[t];
    } else if (e < RV::NV) {
      const int x = e - DA, a = x / DCc, c = x % DCc;
      const double val = (c >= D.nnC) ? double(cX[a * DCc + c]) - sum[t] : 0.0;
      s.S[(size_t)(i * DA + a) * ld + (c0 + c)] = val;  // row c0+c, col i*DA+a
    }
  }
}

template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(kCamWarps * 32) k_rhs_finish(DevState s, const double* __restrict__ cpart) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  rhs_finish_body<DA, DC, Real>(s, cpart, blockIdx.x, gridDim.x);
}

// Global block: S_cc = Z + lambda I - sum_j Y_j^T Vinv_j Y_j, rhs_c = gc - sum_j Y_j^T q_j.  One warp per
// value (the elements are independent): global_blocks(DC) blocks of four warps instead of one block for
// all 35 values of DC = 7, whose fold was the longest part of the finishing launch.
__host__ __device__ constexpr int global_blocks(int DC) { return DC > 0 ? (nsym(DC) + DC + 3) / 4 : 0; }
template <int DA, int DC>
__device__ __forceinline__ void global_block_body(DevState s, const double* __restrict__ part, int nbp, int bid, int nblk) {
  constexpr int NV = ElimNV<DC>::NV;
  constexpr int DCc = DC > 0 ? DC : 1;
  const int t = 4 * bid + (threadIdx.x >> 5);
  if (DC == 0 || t >= NV) return;
  const double a = warp_fold<true>(part + (size_t)t * nbp, nbp);
  if ((threadIdx.x & 31) != 0) return;
  const Dims& D = s.d;
  const int c0 = D.N * DA;
  if (t < nsym(DC)) {
    int r, c;
    unpack_sym<DCc>(t, r, c);
    double val;
    if (r < D.nnC || c < D.nnC) val = (r == c) ? 1.0 : 0.0;
    else val = s.g_Z[r * DCc + c] - a + (r == c ? *s.d_lambda : 0.0);
    s.S[(size_t)(c0 + r) * s.ld + (c0 + c)] = val;   // row c0+c >= col c0+r
  } else {
    const int c = t - nsym(DC);
    s.rhs[(size_t)(c0 + c) * s.rhs_stride] = (c < D.nnC) ? 0.0 : s.g_gc[c] - a;
  }
}

template <int DA, int DC>
__global__ void __launch_bounds__(128) k_global_block(DevState s, const double* __restrict__ part, int nbp) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  global_block_body<DA, DC>(s, part, nbp, blockIdx.x, gridDim.x);
}

// ---- trial step ----------------------------------------------------------------------------

// Camera i's part of the reduced solution, in 16-byte loads where its offset is a multiple of 16 bytes
// (k_update_merged's points, 5.5M observations of 2000 cameras: 192 -> 170 us).
template <int DA>
__device__ __forceinline__ void load_step(double (&da)[DA], const double* __restrict__ x, int i) {
  if constexpr (DA % 2 == 0) {
    vload(x + (size_t)i * DA, da);
  } else {
#pragma unroll
    for (int a = 0; a < DA; ++a) da[a] = x[i * DA + a];
  }
}

// G lanes per point: db_j = q_j - sum_k T_k^T da_i(k) - (Vinv Y_j) dc; X' = X + db.  With FP64
// blocks the sum is Vinv_j sum_k B_k^T (A_k da_i(k)).
template <int DA, int DC, typename Real>
__device__ __forceinline__ void point_backsub_body(DevState s, double* __restrict__ part, int bid, int nblk) {
  using L = Lay<DA, DC, Real>;
  constexpr int DCc = L::DCc;
  __shared__ double red[(kPtThreads / 32) * 2];
  const Dims& D = s.d;
  constexpr int G = backsub_lanes<Real>();
  const int gt = bid * blockDim.x + threadIdx.x;
  const int j = gt / G, lig = gt % G;
  const bool active = j < D.M && j >= D.nnB;
  double v[2] = {0.0, 0.0};
  double acc[3] = {0, 0, 0};
  const double* x = s.x;
  if (active) {
    // this lane's share of sum_k T_k^T dc_i over the track (FP64 blocks: of sum_k B_k^T A_k dc_i,
    // multiplied by Vinv_j below)
    for (int k = s.p_ptr[j] + lig; k < s.p_ptr[j + 1]; k += G) {
      const int i = s.o_cam[k];
      if constexpr (stores_products<Real>()) {
        float t[L::SW];
        vload(s.o_T + (size_t)k * L::SW, t);
        double da[DA];
        load_step<DA>(da, x, i);
#pragma unroll
        for (int a = 0; a < DA; ++a)
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[c] += double(t[a * 3 + c]) * da[a];
      } else {
        double A[L::SA], B[kSB];
        vload(reinterpret_cast<const double*>(s.o_A) + (size_t)k * L::SA, A);
        vload(s.o_B + (size_t)k * kSB, B);
        double ad0 = 0.0, ad1 = 0.0, da[DA];
        load_step<DA>(da, x, i);
#pragma unroll
        for (int a = 0; a < DA; ++a) {
          ad0 += A[a] * da[a];
          ad1 += A[DA + a] * da[a];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += B[c] * ad0 + B[3 + c] * ad1;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) acc[c] = group_sum<G>(acc[c]);
  if (j < D.M && lig == 0) {
    double db[3] = {0, 0, 0};
    if (active) {
      double q[4];
      vload(s.p_q + (size_t)j * 4, q);
      if constexpr (!stores_products<Real>()) {
        double vi[L::SV];
        vload(reinterpret_cast<const double*>(s.p_Vinv) + (size_t)j * L::SV, vi);
        const double a0 = acc[0], a1 = acc[1], a2 = acc[2];
#pragma unroll
        for (int r = 0; r < 3; ++r) acc[r] = vi[s3(r, 0)] * a0 + vi[s3(r, 1)] * a1 + vi[s3(r, 2)] * a2;
      }
      if (DC > 0) {
        Real yv[L::SY];
        vload(reinterpret_cast<const Real*>(s.p_YV) + (size_t)j * L::SY, yv);
        const int c0 = D.N * DA;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < DCc; ++c) acc[r] += double(yv[r * DCc + c]) * x[c0 + c];
      }
      double gb[4];
      vload(s.p_gb + (size_t)j * 4, gb);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        db[r] = q[r] - acc[r];
        v[0] += db[r] * db[r];
        v[1] += db[r] * gb[r];
      }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) s.trial.X[3 * j + r] = s.cur.X[3 * j + r] + db[r];
  }
  block_reduce<2, 2>(v, red);
  store_partials(part, v, bid, nblk);
}

template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(kPtThreads) k_point_backsub(DevState s, double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  point_backsub_body<DA, DC, Real>(s, part, blockIdx.x, gridDim.x);
}

// One thread per camera (plus the globals on thread 0 of block 0): trial parameters.
template <int MODEL, int DA, int DC>
__device__ __forceinline__ void camera_update_body(DevState s, double* __restrict__ part, int bid, int nblk) {
  __shared__ double red[4 * 2];
  const Dims& D = s.d;
  const int i = bid * blockDim.x + threadIdx.x;
  const double* x = s.x;
  double v[2] = {0.0, 0.0};
  if (i < D.N) {
    double R[9], T[3];
#pragma unroll
    for (int t = 0; t < 9; ++t) R[t] = s.cur.R[9 * i + t];
#pragma unroll
    for (int t = 0; t < 3; ++t) T[t] = s.cur.T[3 * i + t];
    double K[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double dist[4] = {0, 0, 0, 0};
    if (MODEL == kModelStd || MODEL == kModelVarying) {   // per-camera K (STEREO has none)
#pragma unroll
      for (int t = 0; t < 9; ++t) K[t] = s.cur.K[9 * i + t];
    }
    if (MODEL == kModelVarying) {
#pragma unroll
      for (int t = 0; t < 4; ++t) dist[t] = s.cur.dist[4 * i + t];
    }
    if (i >= D.nnA) {
      double d[DA];
#pragma unroll
      for (int a = 0; a < DA; ++a) {
        d[a] = x[i * DA + a];
        v[0] += d[a] * d[a];
        v[1] += d[a] * s.c_ga[(size_t)i * Lay<DA, DC>::SG + a];
      }
      T[0] += d[0]; T[1] += d[1]; T[2] += d[2];
      rotate_update(d + 3, R);
      if (MODEL == kModelVarying && DA > 6) {
        double di[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int a = 6; a < DA; ++a) di[a - 6] = d[a];
        intrinsic_update(D.mode, di, K, dist, -1.0);
      }
    }
#pragma unroll
    for (int t = 0; t < 9; ++t) s.trial.R[9 * i + t] = R[t];
#pragma unroll
    for (int t = 0; t < 3; ++t) s.trial.T[3 * i + t] = T[t];
    if (MODEL == kModelStd || MODEL == kModelVarying) {
#pragma unroll
      for (int t = 0; t < 9; ++t) s.trial.K[9 * i + t] = K[t];
    }
    if (MODEL == kModelVarying) {
#pragma unroll
      for (int t = 0; t < 4; ++t) s.trial.dist[4 * i + t] = dist[t];
    }
    store_cam_packed<MODEL>(s.trial.pack, i, R, T, K, dist);
  }
  if (MODEL == kModelCommon && bid == 0 && threadIdx.x == 0) {
    double K[9], dist[4];
    for (int t = 0; t < 9; ++t) K[t] = s.cur.K[t];
    for (int t = 0; t < 4; ++t) dist[t] = s.cur.dist[t];
    if (DC > D.nnC) {
      double di[7] = {0, 0, 0, 0, 0, 0, 0};
      const int c0 = D.N * DA;
      for (int c = 0; c < DC; ++c) {
        di[c] = (c >= D.nnC) ? x[c0 + c] : 0.0;
        v[0] += di[c] * di[c];
        v[1] += di[c] * s.g_gc[c];
      }
      intrinsic_update(D.mode, di, K, dist, D.cached_ar);
    }
    for (int t = 0; t < 9; ++t) s.trial.K[t] = K[t];
    for (int t = 0; t < 4; ++t) s.trial.dist[t] = dist[t];
  }
  block_reduce<2, 2>(v, red);
  store_partials(part, v, bid, nblk);
}

template <int MODEL, int DA, int DC>
__global__ void __launch_bounds__(128) k_camera_update(DevState s, double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  camera_update_body<MODEL, DA, DC>(s, part, blockIdx.x, gridDim.x);
}

// ---- merged launches of independent stages (the LM path) -------------------------------------
// Stages that do not read each other's output run as block ranges of one launch: one kernel
// boundary (drain and fill) less each.  Every block runs the same code on the same data as in the
// stage's own kernel (block index and count of its range), so the results are the same bits.

// Schur chunks (blocks [0, g1)) and reduced-rhs chunks: both read only the elimination's output.
template <int DA, int DC, typename Real, bool DIRECT>
__global__ void __launch_bounds__(128) k_chunks_merged(DevState s, int g1, int g2) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x < g1) schur_chunks_body<DA, Real, DIRECT>(s, s.part_bc, blockIdx.x, g1);
  else rhs_chunks_body<DA, DC, Real>(s, s.part_cc, blockIdx.x - g1, g2);
}

// Grouped Schur sums (blocks [0, g1)) and reduced-rhs chunks, FP64 blocks.  A block of rhs chunks uses the
// first warps that find room for their tiles in the shared memory of a group.
template <int DA, int DC>
__host__ __device__ constexpr int group_rhs_warps() {
  constexpr int bytes = rhs_stage_bytes<DA, DC, double>(), most = kGroupThreads / 32;
  return bytes * most <= kGroupSmem ? most : kGroupSmem / (bytes > 0 ? bytes : 1);
}
template <int DA, int DC>
__global__ void __launch_bounds__(kGroupThreads, DA <= 9 ? 3 : 2) k_groups_merged(DevState s, int g1, int g2) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x < g1) schur_group_body<DA>(s, blockIdx.x);
  else rhs_chunks_body<DA, DC, double, group_rhs_warps<DA, DC>()>(s, s.part_cc, blockIdx.x - g1, g2);
}

// Schur finish (blocks [0, g1)), rhs / border finish ([g1, g1 + g2)) and, with global
// parameters, the global block (the last blocks): they write disjoint parts of S and rhs.
template <int DA, int DC, typename Real>
__global__ void __launch_bounds__(128) k_finish_merged(DevState s, int g1, int g2, const double* __restrict__ pelim,
                                                       int nbp) {
  pdl_wait();
  pdl_trigger();
  const int b = blockIdx.x;
  if (b < g1) schur_finish_body<DA, Real>(s, s.part_bc, b, g1, true);
  else if (b < g1 + g2) rhs_finish_body<DA, DC, Real>(s, s.part_cc, b - g1, g2);
  else global_block_body<DA, DC>(s, pelim, nbp, b - g1 - g2, global_blocks(DC));
}

// Camera (and global) update (blocks [0, g1)) and point back-substitution: both read the
// reduced solution and the current parameters and write different parts of the trial ones.  At most 64
// registers: the few camera blocks would take 80 to 120 and leave the points, which need 32 to 42 and wait for
// their loads, half the warps (5.5M observations, the whole iteration 2341 -> 2275 us; 375,000, FP64 blocks 497
// -> 495).  Camera blocks with a K of their own then spill (88 bytes, 120 to 284 with a distortion of their own),
// which small scenes do not feel: 20 cameras 111 us an iteration, 25 with their own intrinsics 187, either way
// (at 40 registers 20 cameras took 3 us more).
template <int MODEL, int DA, int DC, typename Real>
__global__ void __launch_bounds__(128, 8) k_update_merged(DevState s, int g1, int g2, double* __restrict__ pcam,
                                                       double* __restrict__ ppt) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x < g1) camera_update_body<MODEL, DA, DC>(s, pcam, blockIdx.x, g1);
  else point_backsub_body<DA, DC, Real>(s, ppt, blockIdx.x - g1, g2);
}

template <int MODEL>
__global__ void __launch_bounds__(128) k_pack_cameras(DevState s, ParamSet P) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.d.N) return;
  Cam c;
#pragma unroll
  for (int t = 0; t < 9; ++t) c.K[t] = 0.0;
  load_cam<MODEL>(c, P.R, P.T, P.K, P.dist, i);
  store_cam_packed<MODEL>(P.pack, i, c.R, c.T, c.K, c.d);
}

// One thread per observation: sum |w e|^2 at parameters P, with the stored (frozen) weights or
// with weights recomputed at P.  Bound by the camera records that a warp's 32 cameras take from L2 (192
// bytes an observation in sectors): 2000 cameras, 5.5M observations, 179 us with the parameters as separate
// doubles, 143 as records; records copied to shared memory by the whole warp took 137 there but 12.5 instead
// of 8.4 at 375,000 observations of 200 cameras, and observations in camera order 12.4 (their points and
// weights are then scattered).
constexpr int kCostThreads = 256;
template <int MODEL>
__global__ void __launch_bounds__(kCostThreads) k_obs_cost(DevState s, ParamSet P, int recompute_w,
                                                           double* __restrict__ part) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  __shared__ double red[kCostThreads / 32];
  const Dims& D = s.d;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double v[1] = {0.0}, X[3] = {0, 0, 0}, m[2] = {0, 0}, w = 0.0;
  if (k < D.K) {
    const int i = s.o_cam[k], j = s.o_pt[k];
#pragma unroll
    for (int t = 0; t < 3; ++t) X[t] = P.X[3 * (size_t)j + t];
    vload(s.o_meas + 2 * (size_t)k, m);
    if (!recompute_w) w = s.o_w[k];
    Cam cam;
    load_cam_packed<MODEL>(cam, P.pack, P.K, P.dist, i);
    if (MODEL == kModelStereo) load_rig(cam, s.rig, s.o_sub[k]);
    double XX[3], e[2];
    residual<MODEL>(cam, X, m[0], m[1], XX, e);
    if (recompute_w) w = huber_weight(D.thr, e);
    v[0] = w * w * (e[0] * e[0] + e[1] * e[1]);
  }
  block_reduce<1, 1>(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// The trial's scalars: the points' |db|^2 and db.gb (two values of nbp partials), the cameras' (two of
// nbc) and the cost (nbo), folded side by side by eight, one and fourteen warps a value.
__global__ void __launch_bounds__(32 * kFoldWarps) k_trial_finalize(DevState s, const double* __restrict__ pb, int nbp,
                                                                    const double* __restrict__ pc, int nbc,
                                                                    const double* __restrict__ po, int nbo) {
  pdl_wait();      // the previous stage's writes are visible
  pdl_trigger();   // the next stage may be scheduled once all blocks of this one are resident
  __shared__ double red[kFoldWarps];
  const int w = threadIdx.x >> 5;
  const double* p = w < 16 ? pb + (size_t)(w >> 3) * nbp : w < 18 ? pc + (size_t)(w - 16) * nbc : po;
  const int n = w < 16 ? nbp : w < 18 ? nbc : nbo, segs = w < 16 ? 8 : w < 18 ? 1 : 14;
  const int at = w < 16 ? (w & 7) : w < 18 ? 0 : w - 18;
  const int len = (n + segs - 1) / segs, b0 = min(at * len, n);
  const double v = warp_fold<true>(p + b0, min(len, n - b0));
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double d2 = 0.0, dg = 0.0, c = 0.0;
    for (int u = 0; u < 8; ++u) {
      d2 += red[u];
      dg += red[8 + u];
    }
    for (int u = 18; u < kFoldWarps; ++u) c += red[u];
    s.d_trial[0] = c;
    s.d_trial[1] = d2 + red[16];
    s.d_trial[2] = dg + red[17];
    s.d_trial[3] = *s.d_fail != 0 ? 1.0 : 0.0;   // every kernel that can fail ran before this one
  }
}

__global__ void __launch_bounds__(32 * kFoldWarps) k_sum_to(const double* __restrict__ po, int nbo, double* out) {
  __shared__ double red[kFoldWarps];
  double c[1];
  fold_partials<1, 1>(po, nbo, c, red);
  if (threadIdx.x == 0) *out = c[0];
}

// ---- host launchers ----------------------------------------------------------------------

inline int cdiv(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// partial-buffer regions (in doubles)
struct PartLayout {
  size_t relin_pt, relin_cam, elim, backsub, camupd, obs;
};

// blocks of k_obs_cost
inline int cost_blocks(const DevState& s) { return cdiv(std::max(s.d.K, 1), kCostThreads); }
// blocks of a track kernel with `lanes` lanes per point (the partial regions are sized for the most)
inline int lane_blocks(int M, int lanes = kMaxPtLanes) { return cdiv((int64_t)std::max(M, 1) * lanes, kPtThreads); }

template <int DA, int DC>
inline PartLayout part_layout(const DevState& s) {
  PartLayout p;
  const int bl = lane_blocks(s.d.M);
  const int bc = cdiv(std::max(s.d.N, 1), kCamWarps);
  const int bu = cdiv(std::max(s.d.N, 1), 128);
  p.relin_pt = 0;
  p.relin_cam = p.relin_pt + (size_t)bl * RelinNV<DC>::NV;
  p.elim = p.relin_cam + (size_t)bc * 2;
  p.backsub = p.elim + (size_t)bl * ElimNV<DC>::NV;
  p.camupd = p.backsub + (size_t)bl * 2;
  p.obs = p.camupd + (size_t)bu * 2;
  return p;
}

template <int MODEL, int DA, int DC, typename Real>
struct Ops {
  // Shared memory of the staged kernels, allowed in the handle's context the first time it is asked for.
  static constexpr size_t kCamSmem = (size_t)kCamWarps * camera_stage_bytes<DA, DC, Real>();
  static constexpr size_t kRhsSmem = (size_t)kCamWarps * rhs_stage_bytes<DA, DC, Real>();
  static constexpr size_t kSchurSmem = (size_t)4 * schur_stage_bytes<DA, Real>();
  static constexpr size_t kBothSmem = kRhsSmem > kSchurSmem ? kRhsSmem : kSchurSmem;
  static void allow_stages(uint64_t ctx) {
    static std::atomic<uint64_t> allowed[8];   // contexts, by the last bits of their number
    if (ctx != 0 && allowed[ctx % 8].load() == ctx) return;
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(k_camera_chunks<DA, DC, Real>, attr, (int)kCamSmem);
    cudaFuncSetAttribute(k_rhs_chunks<DA, DC, Real>, attr, (int)kRhsSmem);
    cudaFuncSetAttribute(k_schur_chunks<DA, Real, false>, attr, (int)kSchurSmem);
    cudaFuncSetAttribute(k_chunks_merged<DA, DC, Real, false>, attr, (int)kBothSmem);
    cudaFuncSetAttribute(k_chunks_merged<DA, DC, Real, true>, attr, (int)kRhsSmem);
    if (!stores_products<Real>()) {
      cudaFuncSetAttribute(k_schur_groups<DA>, attr, kGroupSmem);
      cudaFuncSetAttribute(k_groups_merged<DA, DC>, attr, kGroupSmem);
    }
    allowed[ctx % 8].store(ctx);
  }
  static bool grouped(const DevState& s) { return !stores_products<Real>() && s.gr_n > 0; }
  // shared memory of the grouped launches: a group's, or the rhs chunks' of one block if that is more
  static size_t group_smem(const DevState& s) {
    constexpr size_t rhs = (size_t)group_rhs_warps<DA, DC>() * rhs_stage_bytes<DA, DC, double>();
    return std::max((size_t)s.gr_smem, rhs);
  }
  // Launches one stage of the LM iteration (see LmStage in lm.cuh).
  static int stage(DevState& s, int id, int init_lambda, double tau, cudaStream_t st) {
    allow_stages(s.ctx);
    const PartLayout pl = part_layout<DA, DC>(s);
    const int bp = cdiv(std::max(s.d.M, 1), kPtThreads);                  // one lane per point
    const int bl = lane_blocks(s.d.M, kLinLanes);                          // the linearisation
    const int bb = lane_blocks(s.d.M, backsub_lanes<Real>());              // the back-substitution
    const int bc = cdiv(std::max(s.d.N, 1), kCamWarps);
    const int bu = cdiv(std::max(s.d.N, 1), 128);
    const int bo = cost_blocks(s);
    cudaError_t e = cudaSuccess;
    switch (id) {
      case kStageLinearize:
        e = launch_pdl(k_linearize<MODEL, DA, DC, Real>, dim3(bl), dim3(kPtThreads), 0, st, s, s.part + pl.relin_pt);
        break;
      case kStageCameraChunks:
        if (s.nch_cam == 0) return V3DBA_OK;
        e = launch_pdl(k_camera_chunks<DA, DC, Real>, dim3(cdiv(s.nch_cam, kCamWarps)), dim3(kCamWarps * 32), kCamSmem, st, s,
                       s.part_cc);
        break;
      case kStageCameraFinish:
        e = launch_pdl(k_camera_finish<DA, DC, Real>, dim3(bc), dim3(kCamWarps * 32), 0, st, s, (const double*)s.part_cc,
                       s.part + pl.relin_cam);
        break;
      case kStageRelinFinalize:
        e = launch_pdl(k_relin_finalize<DC>, dim3(1), dim3(32 * kFoldWarps), 0, st, s, (const double*)(s.part + pl.relin_pt), bl,
                       (const double*)(s.part + pl.relin_cam), bc, init_lambda, tau);
        break;
      case kStagePointEliminate:
        e = launch_pdl(k_point_eliminate<DA, DC, Real>,
                       dim3(bp + (stores_products<Real>() ? cdiv(s.d.K, kPtThreads) : 0)), dim3(kPtThreads), 0, st, s,
                       s.part + pl.elim, bp);
        break;
      case kStageSchurChunks:
        if (grouped(s)) {
          e = launch_pdl(k_schur_groups<DA>, dim3(s.gr_n), dim3(kGroupThreads), (size_t)s.gr_smem, st, s);
          break;
        }
        if (s.nch_blk == 0) return V3DBA_OK;
        if (schur_direct<DA, Real>(s))
          e = launch_pdl(k_schur_chunks<DA, Real, true>, dim3(cdiv(s.nch_blk, 4)), dim3(128), 0, st, s, s.part_bc);
        else
          e = launch_pdl(k_schur_chunks<DA, Real, false>, dim3(cdiv(s.nch_blk, 4)), dim3(128), kSchurSmem, st, s,
                         s.part_bc);
        break;
      case kStageSchurFinish:
        if (s.nb == 0) return V3DBA_OK;
        e = launch_pdl(k_schur_finish<DA, Real>, dim3(grouped(s) ? s.nb : cdiv(s.nb, 4)), dim3(128), 0, st, s,
                       (const double*)s.part_bc);
        break;
      case kStageRhsChunks:
        if (s.nch_cam == 0) return V3DBA_OK;
        e = launch_pdl(k_rhs_chunks<DA, DC, Real>, dim3(cdiv(s.nch_cam, kCamWarps)), dim3(kCamWarps * 32), kRhsSmem, st, s,
                       s.part_cc);
        break;
      case kStageRhsFinish:
        e = launch_pdl(k_rhs_finish<DA, DC, Real>, dim3(bc), dim3(kCamWarps * 32), 0, st, s, (const double*)s.part_cc);
        break;
      case kStageGlobalBlock:
        if (DC == 0) return V3DBA_OK;
        e = launch_pdl(k_global_block<DA, DC>, dim3(global_blocks(DC)), dim3(128), 0, st, s, (const double*)(s.part + pl.elim), bp);
        break;
      case kStagePointBacksub:
        e = launch_pdl(k_point_backsub<DA, DC, Real>, dim3(bb), dim3(kPtThreads), 0, st, s, s.part + pl.backsub);
        break;
      case kStageCameraUpdate:
        e = launch_pdl(k_camera_update<MODEL, DA, DC>, dim3(bu), dim3(128), 0, st, s, s.part + pl.camupd);
        break;
      case kStageTrialCost:
        e = launch_pdl(k_obs_cost<MODEL>, dim3(bo), dim3(kCostThreads), 0, st, s, (ParamSet)s.trial, 0, s.part + pl.obs);
        break;
      case kStageTrialFinalize:
        e = launch_pdl(k_trial_finalize, dim3(1), dim3(32 * kFoldWarps), 0, st, s, (const double*)(s.part + pl.backsub), bb,
                       (const double*)(s.part + pl.camupd), bu, (const double*)(s.part + pl.obs), bo);
        break;
      default:
        return V3DBA_ERR_INVALID_ARGUMENT;
    }
    if (e != cudaSuccess) {
      fprintf(stderr, "v3dba: launch of stage %d failed: %s\n", id, cudaGetErrorString(e));
      cudaGetLastError();
      return V3DBA_ERR_CUDA;
    }
    V3DBA_LAUNCH_CHECK();
    return V3DBA_OK;
  }
  static int run(DevState& s, int first, int last, int init_lambda, double tau, cudaStream_t st) {
    for (int id = first; id <= last; ++id) {
      const int rc = stage(s, id, init_lambda, tau, st);
      if (rc) return rc;
    }
    return V3DBA_OK;
  }
  static int relinearize(DevState& s, bool init_lambda, double tau, cudaStream_t st) {
    return run(s, kStageLinearize, kStageRelinFinalize, init_lambda ? 1 : 0, tau, st);
  }
  static int launched(cudaError_t e) {
    if (e != cudaSuccess) {
      fprintf(stderr, "v3dba: merged launch failed: %s\n", cudaGetErrorString(e));
      cudaGetLastError();
      return V3DBA_ERR_CUDA;
    }
    V3DBA_LAUNCH_CHECK();
    return V3DBA_OK;
  }
  // elimination, then the Schur and rhs chunks in one launch, then the three finishing stages in
  // one launch (the same work as the stages kStagePointEliminate .. kStageGlobalBlock)
  static int build_reduced(DevState& s, cudaStream_t st) {
    int rc = stage(s, kStagePointEliminate, 0, 0.0, st);
    if (rc) return rc;
    const PartLayout pl = part_layout<DA, DC>(s);
    if (grouped(s)) {
      const int g2 = cdiv(s.nch_cam, group_rhs_warps<DA, DC>());
      if ((rc = launched(launch_pdl(k_groups_merged<DA, DC>, dim3(s.gr_n + g2), dim3(kGroupThreads), group_smem(s), st, s,
                                    s.gr_n, g2))))
        return rc;
    } else {
      const int g1 = s.nch_blk > 0 ? cdiv(s.nch_blk, 4) : 0, g2 = s.nch_cam > 0 ? cdiv(s.nch_cam, kCamWarps) : 0;
      const bool direct = g1 == 0 || schur_direct<DA, Real>(s);   // (without Schur chunks, the smaller shared memory)
      const cudaError_t e =
          g1 + g2 == 0 ? cudaSuccess
          : direct ? launch_pdl(k_chunks_merged<DA, DC, Real, true>, dim3(g1 + g2), dim3(128), kRhsSmem, st, s, g1, g2)
                   : launch_pdl(k_chunks_merged<DA, DC, Real, false>, dim3(g1 + g2), dim3(128), kBothSmem, st, s, g1, g2);
      if (g1 + g2 > 0 && (rc = launched(e))) return rc;
    }
    const int f1 = grouped(s) ? s.nb : s.nb > 0 ? cdiv(s.nb, 4) : 0, f2 = cdiv(std::max(s.d.N, 1), kCamWarps);
    const int bp = cdiv(std::max(s.d.M, 1), kPtThreads);
    return launched(launch_pdl(k_finish_merged<DA, DC, Real>, dim3(f1 + f2 + global_blocks(DC)), dim3(128), 0, st, s,
                               f1, f2, (const double*)(s.part + pl.elim), bp));
  }
  // camera update and point back-substitution in one launch, then the trial cost and the step
  // statistics (the stages kStagePointBacksub .. kStageTrialFinalize)
  static int finish_trial(DevState& s, cudaStream_t st) {
    const PartLayout pl = part_layout<DA, DC>(s);
    const int bu = cdiv(std::max(s.d.N, 1), 128), bb = lane_blocks(s.d.M, backsub_lanes<Real>());
    int rc = launched(launch_pdl(k_update_merged<MODEL, DA, DC, Real>, dim3(bu + bb), dim3(128), 0, st, s, bu, bb,
                                 s.part + pl.camupd, s.part + pl.backsub));
    if (rc) return rc;
    return run(s, kStageTrialCost, kStageTrialFinalize, 0, 0.0, st);
  }
  static int cost(DevState& s, const ParamSet& P, double* d_out, cudaStream_t st) {
    const PartLayout pl = part_layout<DA, DC>(s);
    const int bo = cost_blocks(s);
    k_obs_cost<MODEL><<<bo, kCostThreads, 0, st>>>(s, P, 1, s.part + pl.obs);
    V3DBA_LAUNCH_CHECK();
    k_sum_to<<<1, 32 * kFoldWarps, 0, st>>>(s.part + pl.obs, bo, d_out);
    V3DBA_LAUNCH_CHECK();
    return V3DBA_OK;
  }
  static int pack(DevState& s, const ParamSet& P, cudaStream_t st) {
    if (s.d.N == 0) return V3DBA_OK;
    k_pack_cameras<MODEL><<<cdiv(s.d.N, 128), 128, 0, st>>>(s, P);
    V3DBA_LAUNCH_CHECK();
    return V3DBA_OK;
  }
  static const LmOps* table() {
    static const LmOps t = {&relinearize, &build_reduced, &finish_trial, &pack, &cost, &stage};
    return &t;
  }
};

size_t camera_chunk_values(int DA, int DC) {
  const int nu = DA * (DA + 1) / 2 + DA + DA * DC;
  const int nr = DA + DA * DC;
  return (size_t)round32(std::max(nu, nr));
}
size_t block_chunk_values(int DA) { return (size_t)round32(DA * DA); }

// size (in doubles) of the partial buffer for the given dims
size_t partial_doubles(const DevState& s) {
  const int bc = cdiv(std::max(s.d.N, 1), kCamWarps);
  const int bu = cdiv(std::max(s.d.N, 1), 128);
  const int bo = cost_blocks(s);
  const size_t maxNV = RelinNV<7>::NV;
  const int bl = lane_blocks(s.d.M);
  return (size_t)bl * maxNV + (size_t)bc * 2 + (size_t)bl * ElimNV<7>::NV + (size_t)bl * 2 + (size_t)bu * 2 + bo + 64;
}

template <typename Real>
const LmOps* ops_for(int model, int DA, int DC) {
  if (model == kModelStd) return DA == 6 && DC == 0 ? Ops<kModelStd, 6, 0, Real>::table() : nullptr;
  if (model == kModelStereo) return DA == 6 && DC == 0 ? Ops<kModelStereo, 6, 0, Real>::table() : nullptr;
  if (model == kModelCommon) {
    if (DA != 6) return nullptr;
    switch (DC) {
      case 0: return Ops<kModelCommon, 6, 0, Real>::table();
      case 1: return Ops<kModelCommon, 6, 1, Real>::table();
      case 3: return Ops<kModelCommon, 6, 3, Real>::table();
      case 5: return Ops<kModelCommon, 6, 5, Real>::table();
      case 7: return Ops<kModelCommon, 6, 7, Real>::table();
    }
    return nullptr;
  }
  if (model == kModelVarying) {
    if (DC != 0) return nullptr;
    switch (DA) {
      case 6: return Ops<kModelVarying, 6, 0, Real>::table();
      case 7: return Ops<kModelVarying, 7, 0, Real>::table();
      case 9: return Ops<kModelVarying, 9, 0, Real>::table();
      case 11: return Ops<kModelVarying, 11, 0, Real>::table();
      case 13: return Ops<kModelVarying, 13, 0, Real>::table();
    }
  }
  return nullptr;
}

const LmOps* lm_ops(int model, int DA, int DC, bool fp64) {
  return fp64 ? ops_for<double>(model, DA, DC) : ops_for<float>(model, DA, DC);
}

}  // namespace v3dba
