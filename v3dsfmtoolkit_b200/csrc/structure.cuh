// Device construction of a problem's structure (structure.cu).
#pragma once

#include <cstdint>
#include <functional>
#include <vector>

#include "common.cuh"

namespace v3dba {

struct DevState;

// Allocates `bytes` of device memory that the caller owns (the handle's buffers).
using DevAlloc = std::function<int(void**, size_t)>;

// Checks of a call's arrays once they are on the device, for calls of kDeviceCheckMin items and more:
// the scan of the caller's arrays by one thread took 0.65 ms for 375,000 observations, 0.03 here with the
// read-back of the answer.  Smaller calls are checked on the host, before the device is touched.
constexpr int64_t kDeviceCheckMin = 32768;
enum CheckKind { kCheckIndex, kCheckDouble, kCheckFloat };
struct CheckSeg {
  const void* p;
  int64_t n;
  int kind;    // kCheckIndex: every int in [0, hi); else every value finite
  int hi;
};
constexpr int kCheckSegs = 8;
// *d_flag |= 1 where a value of any segment (at most kCheckSegs) fails its check.
int check_device(const std::vector<CheckSeg>& segs, int* d_flag, cudaStream_t st);
// *out = sum of the n squares of x, in an order fixed by n; part: kSumBlocks doubles.
constexpr int kSumBlocks = 256;
int sum_squares_device(const double* x, int64_t n, double* part, double* out, cudaStream_t st);

struct DeviceStructure {
  // device, allocated through the DevAlloc
  int* o_orig = nullptr;   // [K] caller's index of each point-major observation
  int* o_pt = nullptr;     // [K] point of each observation
  int* o_cam = nullptr;    // [K] camera of each observation
  double* o_meas = nullptr;   // [2K]
  int* p_ptr = nullptr;    // [M+1] observations of each point
  int* c_ptr = nullptr;    // [N+1] observations of each camera ...
  int* c_obs = nullptr;    // [K]   ... in point-major order
  int* b_i = nullptr;      // [nb] camera-pair blocks (i <= l), (i, l) order
  int* b_l = nullptr;
  int* b_ptr = nullptr;    // [nb+1] pairs of each block
  int* pr_k = nullptr;     // [P] observation of camera i in each pair
  int* pr_m = nullptr;     // [P] observation of camera l
  int64_t P = 0;
  // host copies of the small arrays
  std::vector<int> h_c_ptr, h_b_i, h_b_l, h_b_ptr;
};

// Builds the structure of `p` on the device, on stream `st`.  With `verify` the indices and measurements
// are checked there first, together with the segments in *verify, and V3DBA_ERR_INVALID_INPUT is returned
// where a check fails (nothing has used the arrays then); without, they have been checked.
int build_structure_device(const v3dba_problem* p, const DevAlloc& alloc, cudaStream_t st, DeviceStructure& S,
                           const std::vector<CheckSeg>* verify = nullptr);

// Groups the points of a problem by their cameras (the camera sequence of the track) for the grouped
// Schur complement and fills the gr_ fields of `s`; leaves gr_n = 0 where the pair lists are the better
// way.  V3DBA_SCHUR=groups|pairs in the environment forces either where the limits allow it.
int build_schur_groups(DevState& s, const DevAlloc& alloc, cudaStream_t st);

// Stable grouping of n items by device int keys in [0, nv): perm[t] is the t-th item in key
// order (input order among equal keys), items ptr[v] .. ptr[v+1]-1 of perm have key v.  perm
// ([n]) and ptr ([nv+1]) are caller-owned device buffers; the scratch is stream-ordered.
int group_by_key_device(const int* keys, int n, int nv, int* perm, int* ptr, cudaStream_t st);

}  // namespace v3dba
