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
                        bool accumulate, bool fine, const float4** slow, const int** slow_n, cudaStream_t st);
oh_status pc_tc64_enqueue(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, double2* field, double* fringe,
                          bool accumulate, const float4** slow, const int** slow_n, cudaStream_t st);

namespace pctc {

constexpr int kRows = 128, kCols = 64;                // plane region
constexpr int kPts = 4;                                // points per operand stage
constexpr int kBatch = 32;                             // points per record batch
constexpr long long kWaitCycles = 2000000000LL;

constexpr int kMaxCls = 12;

struct PcPt { double x, y, z; float a; int fast; };
// A chunk's points as pc_tc_split orders them.  The separable ones come in classes of
// like amplitude, each with a scale of its own (operands are fixed point): class c
// has the batches [batch[c], batch[c + 1]) and amplitudes below 2^(exp[c] - 126).
struct Counts {
  int fast;                        // list slots; every class but the last fills whole batches
  int slow, aborted, ncls;
  int batch[kMaxCls + 1], exp[kMaxCls];
  int hist[256];                   // separable points by the exponent of their amplitude
};

// A chunk's points, sorted into separable and other ones (device memory).
struct Sorted {
  PcPt* pts;
  int* list;                       // separable points (-1: none), unless all are in one class
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

// A CTA's batches [b, b1) in groups: at most `most` batches of one class.
struct Groups {
  const int* batch;                // Counts::batch
  int ncls, b1, most;
  int c, end;                      // class and end of the current group
  __device__ __forceinline__ void start(int b) {
    while (c + 1 < ncls && batch[c + 1] <= b) ++c;
    end = min(b1, b + most);
    if (c + 1 < ncls) end = min(end, batch[c + 1]);
  }
};

// Exponent of a class's scale: amplitudes times 2^-class_exp are at most one (kept to
// normal scales).
__device__ __forceinline__ int class_exp(int exp) { return max(-100, min(100, exp - 126)); }
__device__ __forceinline__ float pow2f(int e) { return __int_as_float(max(127 + e, 0) << 23); }

}  // namespace pctc

}  // namespace oh
