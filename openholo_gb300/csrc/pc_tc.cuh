// Point-cloud sums on the tensor cores: what pointcloud.cu needs of them, and
// what the FP32 (pc_tc.cu) and FP64 (pc_tc64.cu) forms share.
#pragma once
#include "context.h"
#include "tc_common.cuh"

namespace oh {

struct PCGeom {
  double k, px, py, hlx, hly, sx, sy, sz, off, stx, sty, lambda;
  int nx, ny;
};

// True when the tensor-core form takes the sum (sm_103, enough work that its
// launches do not matter, 32-bit sizes).
bool pc_tc_wants(const PCGeom& g, int n, bool fp64);

// Sums the points of one chunk (n points) whose phase is separable over plane
// regions (see pc_tc.cu) into field / fringe (field is added to when accumulate,
// else overwritten; fringe is always added to).  The other points are left in
// slow[0, *slow_n) (device) for the caller; the order within both groups is the
// input's.  FP64: field double2, fringe double.
oh_status pc_tc_enqueue(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, float2* field, float* fringe,
                        bool accumulate, const float4** slow, const int** slow_n, cudaStream_t st);
oh_status pc_tc64_enqueue(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, double2* field, double* fringe,
                          bool accumulate, const float4** slow, const int** slow_n, cudaStream_t st);

namespace pctc {

constexpr int kRows = 128, kCols = 64;                // plane region
constexpr int kPts = 4;                                // points per operand stage
constexpr int kBatch = 32;                             // points per record batch
constexpr long long kWaitCycles = 2000000000LL;

struct PcPt { double x, y, z; float a; int fast; };
struct Counts { int fast, slow; unsigned amax; int aborted; };

// A chunk's points, sorted into separable and other ones (device memory).
struct Sorted {
  PcPt* pts;
  int* list;                       // separable points, unless every point is
  float4* slow;
  Counts* cnt;
};
size_t sorted_bytes(int n);
// base: sorted_bytes(n) of scratch
oh_status sort_points(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, bool fp64, void* base, Sorted* out,
                      cudaStream_t st);

// Splits of the points (one CTA per region and split) that fill the last wave of
// `slots` CTAs best: the fewest up to 8 that reach 95 %, `batches` record batches
// each at least.
int point_splits(int regions, int n, int slots, int batches);

__device__ __forceinline__ bool wait_live(uint64_t* b, uint32_t parity, const int* abort) {
  const long long t0 = clock64();
  while (!tc::mb_try(b, parity)) {
    if (*((volatile const int*)abort) || clock64() - t0 > kWaitCycles) return false;
  }
  return true;
}
// the whole warp waits: lane 0 polls; false (and the abort flag) on timeout
__device__ __forceinline__ bool warp_wait(uint64_t* b, uint32_t parity, int* abort, int lane) {
  bool ok = true;
  if (lane == 0) {
    ok = wait_live(b, parity, abort);
    if (!ok) atomicExch(abort, 1);
  }
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  __syncwarp();
  return ok;
}
__device__ __forceinline__ void arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::su32(b)) : "memory");
}

// 2^-(e+1) and its inverse, e the exponent of the largest amplitude (kept to
// normal scales)
__device__ __forceinline__ float amp_scale(unsigned amax, float* inv) {
  int e = (int)(amax >> 23) - 126;
  e = amax == 0u ? 0 : max(-100, min(100, e));
  *inv = __int_as_float((127 + e) << 23);
  return __int_as_float((127 - e) << 23);
}

}  // namespace pctc

}  // namespace oh
