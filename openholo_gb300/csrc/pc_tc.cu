// Point-cloud hologram (exact distances) as a contraction on the tensor cores.
//
// Over a plane region of 128 rows x 64 columns around (Xc, Yc), with r0 the
// distance from a point to the region's centre, u, v the offsets from it and
//   p = (2 dx u + u^2) / r0^2,  q = (2 dy v + v^2) / r0^2,
// the distance is r = r0 sqrt(1 + p + q), and
//   sqrt(1 + p + q) = sqrt(1 + p) + sqrt(1 + q) - 1 - P Q / 4 + O(p^2 q^2 / 10),
//   P = 2 (1 - 1 / sqrt(1 + p)),  Q = 2 (1 - 1 / sqrt(1 + q))
// (the terms linear in p or in q are exact).  So the phase k r is separable up
// to the cross term chi = -(k r0 / 4) P Q, a few hundredths of a radian, and
//   exp(i k r) = sum_n [E(v) Qh^n] [E(u) (i kq P)^n / n!],  chi = kq P Qh,
// four terms (n < 4) in all: W[y][x] = sum over points and n of L_n[y] R_n[x], a
// complex matrix product with K = 4 per point.  Embedded in reals (K column 2k,
// 2k+1 = Re, Im of term k; B rows 2x, 2x+1 give Re, Im of column x) it is a
// product C = A B^T with M = 128, N = 128 and K = 8 per point.
//
// Operands (amplitudes scaled by a power of two to at most one) are split into
// a multiple of 2^-8 and an FP16 remainder (absolute error 2^-21) and, where FINE asks
// for it, the FP16 rest of that (2^-25; six products instead of four, sine and cosine
// to 2^-23 instead of 2^-21: 1.2e-7 against 7.3e-7 of the L2 norm).  The tensor
// core truncates each FP32 accumulation (a plain FP16 high/low split in one
// accumulator lost 2e-5 over 700 points that way), so the products of the
// multiples of 2^-8 have an accumulator of their own, in which sums up to 256
// are exact, and the three products with a remainder, 2^-8 of that, another.  A
// term adds at most 1.09 (sum over n of chi^n / n!, chi < 0.07, and the rounding),
// so every 224 points the producers add both accumulators into the partial plane
// in global memory (L2), which rounds to nearest: in one accumulator 32768
// points in phase lost 4e-4, now 1.4e-6 (1024 x 1024, 5000 points: 727 -> 745 us).
//
// A point's operand error is 2^-22 of the scale, whatever its amplitude.  pc_tc_split
// therefore cuts clouds of uneven amplitude into classes with scales S of their own,
// until sum S^2 over the points is at most 8 times a lower bound of sum a^2: octaves
// from the largest amplitude down, the last class whatever is left.  Amplitudes spread
// evenly over 0..1 stay one class.  10000 points at 1 / 100 of one bright point:
// 3.9e-5 with one scale, 7e-7 with two.
//
// pc_tc_prep decides in FP64 per point whether the dropped terms stay below
// 1e-6 rad at the worst corner of the plane; other points (near or strongly
// off-axis scenes) go to a list that the caller sums directly.
//
// One CTA per region and split of the points, 320 threads, two CTAs per SM: warp
// 9 forms the per-region records of 32 points at a time (FP64 phases reduced to
// 32-bit fractions of a turn), warps 0-7 build the operands of four points (K =
// 32) per stage straight into shared memory in the 64-byte-swizzled layout a TMA
// load would give, warp 8 issues tcgen05.mma; warps 0-7 read the accumulators
// between stages, while the tensor core waits.  Splits write partial planes that
// pc_tc_sum adds in order, so the result does not depend on timing.  Waits are
// bounded: on timeout the CTA sets the device error word and the outputs stay
// unwritten.
//
// What bounds it: the operand producers (53 % of the issue slots) and shared
// memory (63 %: their stores and the tensor core's operand reads).  16 producer
// warps in two groups were 8 % slower (spills and spinning waits).  1024 x 1024 x 5000
// points: 790 us with two-part operands (5.74 ms directly), 988 with three; the phase
// in whole numbers takes 45 us of it, in floats its square term left 1.3e-6.
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include "pc_tc.cuh"
#include "tc_common.cuh"

namespace oh {

namespace {

using namespace pctc;
using tc::su32;

constexpr int kBK = 8 * kPts;                          // K per stage
constexpr int kStages = 2;
constexpr int kTile = 128 * kBK * 2;                   // 8 KB: 128 rows x 32 FP16
template <bool FINE> constexpr int kParts = FINE ? 3 : 2;         // parts of an operand
template <bool FINE> constexpr int kStageBytes = 2 * kParts<FINE> * kTile;         // A's parts, then B's
constexpr int kAccCols = 128, kTmemCols = 2 * kAccCols;   // exact products, products with remainders
constexpr int kProducers = 8, kThreads = 32 * (kProducers + 2);
constexpr int kMinBatches = 2;                         // of a split (see point_splits)
constexpr int kGroup = 7;                              // batches (224 points) between additions to the partial plane
constexpr int kPer = kBatch / kPts;                    // stages per batch
constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // FP16 in, FP32 out

// One point as a region sees it: phase in turns = frac(t0 + m (cy + m c2y)) + m^2 qy +
// rest(m) along the rows (m = row - 64), the same with cx, c2x, qx along the columns
// (m = column - 32, no t0).
struct alignas(16) PcRec {
  int t0, cx, cy;
  float amp;
  float c0, ax, bx, ay;            // r0 / lambda; p = m (ax + bx m), q = m (ay + by m)
  float by, iqs, kq;               // 1 / max |Q|; cross factor kq (rad)
  int c2x, c2y;
  float qx, qy, pad;               // what c2x and c2y round off
};

struct PcTcArgs {
  PCGeom g;
  const PcPt* pts;
  const int* list;                 // fast points by class, unless every point is fast and of one class
  Counts* cnt;
  int regions_x, splits;
  float2* part;                    // [splits][ny][nx]
  int* err;
};

// FP64 position of a point, and whether the separable form holds over the whole
// plane: every dropped term below 1e-6 rad at the plane's worst corner (see the
// head of this file), fp64: near 1e-10 rad there (see pc_tc64.cu).
__device__ __forceinline__ PcPt prep_point(const PCGeom& g, float4 p, int fp64) {
  PcPt o;
  o.x = (double)p.x * g.sx; o.y = (double)p.y * g.sy; o.z = (double)p.z * g.sz + g.off;
  o.a = p.w;
  const double az = fabs(o.z);
  const float U = (float)(0.5 * kCols * g.px), V = (float)(0.5 * kRows * g.py), zf = (float)az, kf = (float)g.k;
  // |p| r0^2 = |(dx + u)^2 - dx^2| over the plane's pixels: with D the farthest
  // pixel, a region that ends at the edge gives 2 D U - U^2, one that runs past
  // it 2 D U + U^2 at most
  const float DX = (float)(g.hlx + fabs(o.x)), DY = (float)(g.hly + fabs(o.y));
  const float eu = g.nx % kCols ? U : -U, ev = g.ny % kRows ? V : -V;
  const float iz = 1.f / zf, iz2 = iz * iz;
  const float pm = fminf((2.f * DX + eu) * U * iz2, U * iz + U * U * iz2);
  const float qm = fminf((2.f * DY + ev) * V * iz2, V * iz + V * V * iz2);
  const float r0 = sqrtf((DX + U) * (DX + U) + (DY + V) * (DY + V) + zf * zf);
  const float chi = 0.25f * kf * r0 * pm * qm, m = fmaxf(pm, qm);
  const float turns = kf * r0 * 0.15915494f;
  // separable form: rank-four remainder, p^2 q^2 term, series ends (phase of
  // one axis, P and Q), and the float part of the axis phases below 4 turns
  bool ok = m < 0.01f && chi * chi * chi * chi < 24e-6f && 0.1f * kf * r0 * pm * pm * qm * qm < 2e-7f &&
            0.0273f * m * m * m * m * m * turns < 3e-8f && chi * 0.55f * m * m * m < 2e-7f &&
            turns * 0.5f * fmaxf(U, V) * fmaxf(U, V) * iz2 < 4.f && fminf(U, V) * fminf(U, V) * iz2 > 1e-25f && fabsf(p.w) < 1e30f &&
            fabs(o.x) < 1e3 && fabs(o.y) < 1e3 && az < 1e3;
  if (fp64) {
    // rank-six remainder; terms past p^2 q^2; the axis series' m^7 term; the column
    // factor (scaled by the row factor's maximum over whole regions) below 0.088
    const float c3 = chi * chi * chi, t = fmaxf(U, V) * iz, t3 = t * t * t;
    const float qf = fminf((2.f * DY + (g.ny % kRows ? 3.f * V : -V)) * V * iz2, V * iz + V * V * iz2);
    ok = ok && 0.25f * kf * r0 * pm * qf < 0.086f && c3 * c3 < 720.f * 1.2e-10f && kf * r0 * (pm * qm) * (pm * qm) * (pm + qm) < 1e-10f &&
         turns * t3 * t3 * t < 3e-11f;
  }
  o.fast = ok ? 1 : 0;
  return o;
}

__global__ void __launch_bounds__(128) pc_tc_prep(PCGeom g, const float4* __restrict__ in, int n, int fp64,
                                                  PcPt* __restrict__ pts, Counts* __restrict__ cnt) {
  __shared__ int hist[256];
  for (int i = threadIdx.x; i < 256; i += 128) hist[i] = 0;
  __syncthreads();
  int slow = 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const PcPt o = prep_point(g, in[j], fp64);
    if (o.fast) atomicAdd(&hist[__float_as_uint(fabsf(o.a)) >> 23], 1);
    else ++slow;
    pts[j] = o;
  }
  slow = __reduce_add_sync(0xffffffffu, slow);
  if ((threadIdx.x & 31) == 0 && slow) atomicAdd(&cnt->slow, slow);
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += 128)
    if (hist[i]) atomicAdd(&cnt->hist[i], hist[i]);
}

// One block: the classes (see Counts and the head of this file), then the fast points'
// indices by class and the slow points, both in input order.  With one class and no
// slow point the index list stays unwritten (and unread).  PREP (n <= 1024): forms the
// points as well, two launches fewer: where every point is refused the form is all
// overhead (147 -> 163 us at 300 points on 512 x 512).
template <bool PREP>
__global__ void __launch_bounds__(1024) pc_tc_split(PCGeom g, int fp64, const float4* __restrict__ in, PcPt* pts, int n,
                                                    int* __restrict__ list, float4* __restrict__ slow,
                                                    Counts* cnt) {
  __shared__ int hist[256], exps[kMaxCls], first[kMaxCls + 1], count[kMaxCls], next[kMaxCls + 1], wsum[32][kMaxCls + 1];
  __shared__ int s_ncls;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int nslow;
  if constexpr (PREP) {
    if (threadIdx.x < 256) hist[threadIdx.x] = 0;
    __syncthreads();
    bool refused = false;
    if (threadIdx.x < n) {
      const PcPt o = prep_point(g, in[threadIdx.x], fp64);
      if (o.fast) atomicAdd(&hist[__float_as_uint(fabsf(o.a)) >> 23], 1);
      refused = !o.fast;
      pts[threadIdx.x] = o;
    }
    nslow = __syncthreads_count(refused);
    if (threadIdx.x == 0) { cnt->slow = nslow; cnt->aborted = 0; }
  } else {
    if (threadIdx.x < 256) hist[threadIdx.x] = cnt->hist[threadIdx.x];
    nslow = cnt->slow;
    __syncthreads();
  }
  if (warp == 0) {
    unsigned word[8];                                   // the exponents that occur
#pragma unroll
    for (int i = 0; i < 8; ++i) word[i] = __ballot_sync(0xffffffffu, hist[32 * i + lane] != 0);
    if (lane == 0) {
      auto each = [&](auto f) {                         // from the largest down, until f is false
#pragma unroll
        for (int i = 7; i >= 0; --i)
          for (unsigned m = word[i]; m; m &= ~(0x80000000u >> __clz(m)))
            if (!f(32 * i + 31 - __clz(m))) return;
      };
      int top = -1, rest = 0, c = 0, slot = 0;
      float left = 0.f;                                 // of sum S^2, in units of 4^top
      each([&](int e) {
        if (top < 0) top = e;
        rest += hist[e];
        left += 8.f * (float)hist[e] * pow2f(2 * (e - top));
        return true;
      });
      each([&](int e) {
        const float S2 = 4.f * pow2f(2 * (e - top));
        const bool all = S2 * (float)rest <= left || c == kMaxCls - 1;
        exps[c] = e;
        first[c] = slot;
        count[c] = all ? rest : hist[e];
        cnt->exp[c] = e;
        cnt->batch[c] = slot / kBatch;
        slot += all ? rest : (hist[e] + kBatch - 1) / kBatch * kBatch;
        left -= S2 * (float)hist[e];
        rest -= count[c];
        ++c;
        return !all;
      });
      s_ncls = c;
      cnt->ncls = c;
      cnt->batch[c] = (slot + kBatch - 1) / kBatch;
      cnt->fast = slot;
    }
  }
  __syncthreads();
  const int ncls = s_ncls;
  if (nslow == 0 && ncls <= 1) return;
  if (nslow == n) {                                     // (nothing to sort)
    for (int j = threadIdx.x; j < n; j += 1024) slow[j] = in[j];
    return;
  }
  if (threadIdx.x <= kMaxCls) next[threadIdx.x] = threadIdx.x < ncls ? first[threadIdx.x] : 0;     // [kMaxCls]: slow points
  for (int c = 0; c + 1 < ncls; ++c)
    for (int i = first[c] + count[c] + threadIdx.x; i < first[c + 1]; i += 1024) list[i] = -1;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int j = base + threadIdx.x;
    int c = kMaxCls + 1;                                // none
    if (j < n) {
      c = kMaxCls;
      if (pts[j].fast) {
        const int e = (int)(__float_as_uint(fabsf(pts[j].a)) >> 23);
        for (c = 0; c + 1 < ncls && exps[c + 1] >= e;) ++c;
      }
    }
    const unsigned same = __match_any_sync(0xffffffffu, c);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (lane <= kMaxCls) wsum[warp][lane] = 0;
    __syncwarp();
    if (rank == 0 && c <= kMaxCls) wsum[warp][c] = __popc(same);
    __syncthreads();
    if (c <= kMaxCls) {
      int at = next[c] + rank;
      for (int w = 0; w < warp; ++w) at += wsum[w][c];
      if (c < kMaxCls) list[at] = j;
      else slow[at] = in[j];
    }
    __syncthreads();
    if (threadIdx.x <= kMaxCls) {
      int t = next[threadIdx.x];
      for (int w = 0; w < 32; ++w) t += wsum[w][threadIdx.x];
      next[threadIdx.x] = t;
    }
    __syncthreads();
  }
}

// Byte offset of 16-byte chunk c of row r in a [128][32] FP16 tile with 64-byte swizzle.
__device__ __forceinline__ int sw_off(int r, int c) { return r * 64 + ((c ^ ((r >> 1) & 3)) << 4); }

__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
// Parts of (a, b), |a|, |b| <= 1: the multiples of 2^-8 nearest them (adding 6 in FP16
// rounds to them), FP16 remainders and, where wanted, FP16 rests of those.
template <bool THIRD>
__device__ __forceinline__ void split(float a, float b, uint32_t* hi, uint32_t* lo, uint32_t* rest) {
  const __half2 six = __floats2half2_rn(6.f, 6.f);
  const __half2 h = __hsub2(__hadd2(__floats2half2_rn(a, b), six), six);
  const float2 f = __half22float2(h);
  a -= f.x;
  b -= f.y;
  const __half2 l = __floats2half2_rn(a, b);
  *hi = h2u(h);
  *lo = h2u(l);
  if constexpr (THIRD) {
    const float2 g = __half22float2(l);
    *rest = h2u(__floats2half2_rn(a - g.x, b - g.y));
  }
}

// w[k] of lane i of four <- w[i] of lane k
__device__ __forceinline__ void quad_transpose(float4* w, int lane) {
  auto swap = [&](float4& keep0, float4& keep1, bool up, int mask) {   // the upper lane sends keep0, the lower keep1
    const float4 s = up ? keep0 : keep1;
    const float4 r = make_float4(__shfl_xor_sync(0xffffffffu, s.x, mask), __shfl_xor_sync(0xffffffffu, s.y, mask),
                                 __shfl_xor_sync(0xffffffffu, s.z, mask), __shfl_xor_sync(0xffffffffu, s.w, mask));
    if (up) keep0 = r; else keep1 = r;
  };
  swap(w[0], w[1], lane & 1, 1);
  swap(w[2], w[3], lane & 1, 1);
  swap(w[0], w[2], lane & 2, 2);
  swap(w[1], w[3], lane & 2, 2);
}
__device__ __forceinline__ void red_add4(float2* p, float4 v) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void put2(float2* p, float2 v, bool add) {
  if (add) asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
  else *p = v;
}

// turns -> (cos, sin)
template <bool FINE>
__device__ __forceinline__ void cis(float t, float* c, float* s) {
  t -= rintf(t);
  if constexpr (FINE) {
    sincospif(2.f * t, s, c);
  } else {
    t *= 6.28318530717958647692f;
    *c = __cosf(t);
    *s = __sinf(t);
  }
}
// Phase at offset m of one axis, (r0 / lambda) (sqrt(1 + w) - 1) and t0, without most of
// its whole turns; *w = m (a + b m).  The terms in m and m^2 are whole numbers of 2^-32
// turns (in floats the second, of up to two turns, was off by 1e-6 rad).
__device__ __forceinline__ float axis_turns(int t0, int c1, int c2, float q, float c0, float a, float b, int m, float* w) {
  const float mf = (float)m, m2 = mf * mf, bm = b * mf, abm = a + bm;
  const unsigned um = (unsigned)m;
  *w = mf * abm;
  const float w2 = *w * *w;
  // -w^2 / 8 without its term in m^2, then w^3 / 16 - 5 w^4 / 128
  const float rest = fmaf(w2 * *w, fmaf(*w, -0.0390625f, 0.0625f), (-0.125f * m2 * mf) * b * (abm + a));
  return (float)(int)((unsigned)t0 + um * ((unsigned)c1 + um * (unsigned)c2)) * 2.3283064365386963e-10f + fmaf(c0, rest, q * m2);
}
__device__ __forceinline__ float cross_arg(float w) { return w * fmaf(w, fmaf(w, 0.625f, -0.75f), 1.f); }

template <bool FINE>
__global__ void __launch_bounds__(kThreads, 2) pc_tc_regions(PcTcArgs a) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ PcRec recs[2][kBatch];
  __shared__ int cls_batch[kMaxCls + 1], cls_e[kMaxCls];
  const uint32_t raw = su32(smem_dyn);
  unsigned char* base = smem_dyn + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kStages * kStageBytes<FINE>);
  uint64_t* full = bars;                  // [kStages], one arrival per producer warp
  uint64_t* empty = bars + kStages;       // [kStages], tcgen05.commit
  uint64_t* rfull = bars + 2 * kStages;   // [2], the record warp's
  uint64_t* rempty = rfull + 2;           // [2], one arrival per producer warp
  uint64_t* gdone = rfull + 4;            // a group's products are done (tcgen05.commit)
  uint64_t* gfree = rfull + 5;            // a group's accumulators are read, one arrival per producer warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rfull + 6);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int X0 = (blockIdx.x % a.regions_x) * kCols, Y0 = (blockIdx.x / a.regions_x) * kRows;
  const int nx = a.g.nx, ny = a.g.ny;
  const int nfast = a.cnt->fast;
  const int ncls = a.cnt->ncls;
  const bool identity = a.cnt->slow == 0 && ncls == 1;
  const int nbatch = (nfast + kBatch - 1) / kBatch;
  const int b0 = (int)((long long)blockIdx.y * nbatch / a.splits), b1 = (int)((long long)(blockIdx.y + 1) * nbatch / a.splits);
  const int first = b0 * kBatch, last = min(b1 * kBatch, nfast);
  const int nst = (last - first + kPts - 1) / kPts;
  float2* part = a.part + (size_t)blockIdx.y * nx * ny;
  if (nfast == 0) return;                 // pc_tc_sum reads no partial plane then
  if (nst <= 0) {
    for (int i = threadIdx.x; i < kRows * kCols; i += kThreads) {
      const int r = Y0 + i / kCols, c = X0 + i % kCols;
      if (r < ny && c < nx) part[(size_t)r * nx + c] = make_float2(0.f, 0.f);
    }
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { tc::mb_init(&full[s], kProducers); tc::mb_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { tc::mb_init(&rfull[s], 1); tc::mb_init(&rempty[s], kProducers); }
    tc::mb_init(gdone, 1);
    tc::mb_init(gfree, kProducers);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x <= ncls) cls_batch[threadIdx.x] = a.cnt->batch[threadIdx.x];
  if (threadIdx.x < ncls) cls_e[threadIdx.x] = class_exp(a.cnt->exp[threadIdx.x]);
  if (warp == 1) tc::tmem_alloc(tmem_slot, kTmemCols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < kProducers) {
    // point slot j of the stage, A rows rb and rb + 64, B column rb
    const int j = threadIdx.x & 3, rb = threadIdx.x >> 2;
    const int offA0 = sw_off(rb, j), offA1 = sw_off(rb + 64, j);
    // the two B rows of a column, in an order that spreads a quarter-warp over the banks
    const int par = rb & 1;
    const int offB0 = sw_off(2 * rb + par, j), offB1 = sw_off(2 * rb + 1 - par, j);
    // group g's sums into the partial plane: TMEM lanes 32 (warp % 4) .. (region
    // rows), 32 complex columns per warp / 4, turned so that four lanes write 64
    // bytes of a row.  Every value has one writer, so the reductions (no wait for the
    // old value) keep its order.
    const int Yq = Y0 + 32 * (warp & 3) + (lane & ~3), Xw = X0 + 32 * (warp >> 2);
    auto flush = [&](int g, float rel) -> bool {         // rel: the group's scale over the first class's
      if (!warp_wait(gdone, (uint32_t)(g & 1), abort_flag, lane)) return false;
      tc::fence_after();
      const uint32_t at = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(64 * (warp >> 2));
#pragma unroll 1
      for (int c = 0; c < 32; c += 8) {
        uint32_t v[32];                                  // exact products' sums, then the others'
        tc::tmem_ld16x2(at + 2 * c, at + kAccCols + 2 * c, v);
        float4 w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          auto sum = [&](int i) { return rel * (__uint_as_float(v[4 * q + i]) + __uint_as_float(v[16 + 4 * q + i])); };
          w[q] = make_float4(sum(0), sum(1), sum(2), sum(3));
        }
        quad_transpose(w, lane);
        const int X = Xw + c + 2 * (lane & 3);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (Yq + k >= ny || X >= nx) continue;
          float2* dst = part + (size_t)(Yq + k) * nx + X;
          if (nx % 2 == 0) {
            if (g) red_add4(dst, w[k]);
            else *reinterpret_cast<float4*>(dst) = w[k];
          } else {
            put2(dst, make_float2(w[k].x, w[k].y), g);
            if (X + 1 < nx) put2(dst + 1, make_float2(w[k].z, w[k].w), g);
          }
        }
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) arrive(gfree);
      return true;
    };
    Groups gr{cls_batch, ncls, b1, kGroup, 0, 0};       // the oldest group not read out
    gr.start(b0);
    int g = 0;
    bool ok = true;
    for (int it = 0; it < nst && ok; ++it) {
      const int s = it % kStages, batch = it / kPer, rs = batch & 1;
      if (it % kPer == 0) ok = warp_wait(&rfull[rs], (uint32_t)((batch >> 1) & 1), abort_flag, lane);
      ok = ok && warp_wait(&empty[s], (uint32_t)(((it / kStages) & 1) ^ 1), abort_flag, lane);
      if (!ok) break;
      const PcRec q = recs[rs][(it % kPer) * kPts + j];
      unsigned char* sA = base + s * kStageBytes<FINE>;
      unsigned char* sB = sA + kParts<FINE> * kTile;
      auto put = [&](unsigned char* tile, int off, uint4 v) { *reinterpret_cast<uint4*>(tile + off) = v; };
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float c, sn, w;
        cis<FINE>(axis_turns(q.t0, q.cy, q.c2y, q.qy, q.c0, q.ay, q.by, rb - 64 + 64 * h, &w), &c, &sn);
        const float Qh = cross_arg(w) * q.iqs;
        float re = q.amp * c, im = q.amp * sn;
        uint4 hi, lo, rest = make_uint4(0u, 0u, 0u, 0u);
        split<FINE>(re, im, &hi.x, &lo.x, &rest.x);
        // (the other terms' rests meet columns below 0.07)
        re *= Qh; im *= Qh;
        split<false>(re, im, &hi.y, &lo.y, nullptr);
        re *= Qh; im *= Qh;
        split<false>(re, im, &hi.z, &lo.z, nullptr);
        re *= Qh; im *= Qh;
        split<false>(re, im, &hi.w, &lo.w, nullptr);
        const int off = h ? offA1 : offA0;
        put(sA, off, hi);
        put(sA + kTile, off, lo);
        if constexpr (FINE) put(sA + 2 * kTile, off, rest);
      }
      {
        float c, sn, w;
        cis<FINE>(axis_turns(0, q.cx, q.c2x, q.qx, q.c0, q.ax, q.bx, rb - 32, &w), &c, &sn);
        const float x = q.kq * cross_arg(w);
        const float x2 = 0.5f * x * x, x3 = x * x2 * 0.33333333333f;
        // R_n = (c + i s) (i x)^n / n!
        uint4 v[3];
        split<FINE>(c, sn, &v[0].x, &v[1].x, &v[2].x);
        split<FINE>(-x * sn, x * c, &v[0].y, &v[1].y, &v[2].y);
        split<FINE>(-x2 * c, -x2 * sn, &v[0].z, &v[1].z, &v[2].z);
        split<FINE>(x3 * sn, -x3 * c, &v[0].w, &v[1].w, &v[2].w);
        // row 2x takes (Re, -Im) of each term, row 2x + 1 (Im, Re)
        const uint32_t neg = 0x80000000u;
#pragma unroll
        for (int k = 0; k < kParts<FINE>; ++k) {
          const uint4 u = v[k];
          const uint4 r0 = make_uint4(u.x ^ neg, u.y ^ neg, u.z ^ neg, u.w ^ neg);
          const uint4 r1 = make_uint4(__byte_perm(u.x, 0, 0x1032), __byte_perm(u.y, 0, 0x1032),
                                      __byte_perm(u.z, 0, 0x1032), __byte_perm(u.w, 0, 0x1032));
          put(sB + k * kTile, offB0, par ? r1 : r0);
          put(sB + k * kTile, offB1, par ? r0 : r1);
        }
      }
      // generic-proxy writes -> visible to the tensor core's async proxy
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        arrive(&full[s]);
        if (it % kPer == kPer - 1) arrive(&rempty[rs]);
      }
      // a group is read out while its successor's first stages wait for the
      // tensor core
      const int next = (gr.end - b0) * kPer;
      if (it >= next && (it == next + 1 || it == nst - 1)) {
        ok = flush(g++, pow2f(cls_e[gr.c] - cls_e[0]));
        gr.start(gr.end);
      }
    }
    if (ok) flush(g, pow2f(cls_e[gr.c] - cls_e[0]));
  } else if (warp == kProducers) {
    if (lane == 0) {
      Groups gr{cls_batch, ncls, b1, kGroup, 0, 0};
      gr.start(b0);
      int next = min(nst, (gr.end - b0) * kPer);
      uint32_t add = 0u, gph = 0u;        // the group's first stage starts its accumulators
      for (int it = 0; it < nst; ++it) {
        const int s = it % kStages;
        bool ok = true;
        if (it == next) {
          ok = wait_live(gfree, gph, abort_flag);
          gph ^= 1u;
          gr.start(gr.end);
          next = min(nst, (gr.end - b0) * kPer);
          add = 0u;
        }
        ok = ok && wait_live(&full[s], (uint32_t)((it / kStages) & 1), abort_flag);
        if (!ok) {
          atomicExch(abort_flag, 1);
          break;
        }
        tc::fence_after();
        // part k of an operand kTile further on
        const uint32_t st0 = su32(base + s * kStageBytes<FINE>);
        const uint64_t da = tc::desc_sw64(st0, 16, 512), db = tc::desc_sw64(st0 + kParts<FINE> * kTile, 16, 512);
#pragma unroll
        for (int kk = 0; kk < kBK / 16; ++kk) {
          auto mma = [&](uint32_t acc, int i, int j, uint32_t on) {
            tc::umma_bf16(acc, da + (uint64_t)((i * kTile + kk * 32) >> 4), db + (uint64_t)((j * kTile + kk * 32) >> 4), kIdesc, on);
          };
          mma(tmem, 0, 0, kk ? 1u : add);
          mma(tmem + kAccCols, 0, 1, kk ? 1u : add);
          mma(tmem + kAccCols, 1, 0, 1u);
          mma(tmem + kAccCols, 1, 1, 1u);
          if constexpr (FINE) {
            mma(tmem + kAccCols, 0, 2, 1u);
            mma(tmem + kAccCols, 2, 0, 1u);
          }
        }
        add = 1u;
        tc::umma_commit(&empty[s]);
        if (it == next - 1) tc::umma_commit(gdone);
      }
    }
  } else {
    // record warp: lane k forms point k of each batch
    const double il = a.g.k * 0.15915494309189533576888376337251;      // 1 / lambda
    const double Xc = ((double)(X0 + kCols / 2) + 0.5) * a.g.px - a.g.hlx;
    const double Yc = a.g.hly - ((double)(Y0 + kRows / 2) + 0.5) * a.g.py;
    const double ref = Xc * a.g.stx + Yc * a.g.sty;
    int c = 0;
    auto frac32 = [](double t) { return (int)__double2ll_rn((t - rint(t)) * 4294967296.0); };
    const int batches = b1 - b0;
    for (int b = 0; b < batches; ++b) {
      const int rs = b & 1;
      if (!warp_wait(&rempty[rs], (uint32_t)(((b >> 1) & 1) ^ 1), abort_flag, lane)) break;
      const int k = first + b * kBatch + lane;
      PcRec r{};
      while (c + 1 < ncls && cls_batch[c + 1] <= b0 + b) ++c;
      const int at = k < last ? identity ? k : a.list[k] : -1;
      if (at >= 0) {
        const PcPt p = a.pts[at];
        const double dx = Xc - p.x, dy = Yc - p.y;
        const double r2 = fma(dx, dx, fma(dy, dy, p.z * p.z));
        const double ri = rsqrt(r2), r0 = r2 * ri;
        const double sx = dx * ri, sy = dy * ri;
        r.t0 = frac32((r0 - ref) * il);
        r.cx = frac32((sx - a.g.stx) * a.g.px * il);
        r.cy = frac32((a.g.sty - sy) * a.g.py * il);
        // (r0 / lambda) (1 - s^2) t^2 / 2 per squared pixel, t = pitch / r0
        auto square = [&](double sn, double pitch, int* c2, float* q) {
          const double t = pitch * ri, e = 2147483648.0 * (r0 * il) * fma(-sn, sn, 1.0) * t * t, n = rint(e);
          *c2 = (int)n;
          *q = (float)(e - n) * 2.3283064365386963e-10f;
        };
        square(sx, a.g.px, &r.c2x, &r.qx);
        square(sy, a.g.py, &r.c2y, &r.qy);
        const float rif = (float)ri, pxr = (float)a.g.px * rif, pyr = (float)a.g.py * rif;
        r.amp = p.a * pow2f(-cls_e[c]);
        r.c0 = (float)(r0 * il);
        r.ax = 2.f * (float)sx * pxr; r.bx = pxr * pxr;
        r.ay = -2.f * (float)sy * pyr; r.by = pyr * pyr;
        const float qs = fabsf(r.ay) * (kRows / 2) + r.by * (kRows / 2) * (kRows / 2);
        r.iqs = 1.f / qs;
        r.kq = -1.57079632679f * r.c0 * qs;
      }
      recs[rs][lane] = r;
      __syncwarp();
      if (lane == 0) arrive(&rfull[rs]);
    }
  }
  __syncwarp();
  const bool good = __syncthreads_and(!*((volatile int*)abort_flag));
  if (!good && threadIdx.x == 0) {
    atomicOr(a.err, 8);
    atomicOr(&a.cnt->aborted, 1);
  }
  // after a timeout the issuer's products must have let go of shared memory and
  // TMEM: one more commit tracks all of them
  if (!good && threadIdx.x == 32 * kProducers) {
    tc::mb_init(full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::umma_commit(full);
    tc::mb_wait(full, 0, kWaitCycles);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, kTmemCols);
  }
}

// The splits' partial planes added in order, unscaled, into the outputs.  After
// a timeout nothing is written.
__global__ void __launch_bounds__(256) pc_tc_sum(const float2* __restrict__ part, int splits, size_t n,
                                                 const Counts* __restrict__ cnt,
                                                 float2* __restrict__ field, float* __restrict__ fringe, int accumulate) {
  if (cnt->aborted) return;
  const bool none = cnt->fast == 0;
  const float unscale = pow2f(class_exp(cnt->exp[0]));
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float2 v = make_float2(0.f, 0.f);
    if (!none)
      for (int s = 0; s < splits; ++s) v = cadd(v, part[(size_t)s * n + i]);
    v = cscale(v, unscale);
    if (field) field[i] = accumulate ? cadd(field[i], v) : v;
    if (fringe) fringe[i] += v.x;
  }
}

}  // namespace

namespace pctc {

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t sorted_bytes(int n) {
  return align256(sizeof(Counts)) + align256((size_t)n * sizeof(PcPt)) +
         align256(((size_t)n + kMaxCls * kBatch) * sizeof(int)) + align256((size_t)n * sizeof(float4));
}

oh_status sort_points(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, bool fp64, void* base, Sorted* out,
                      cudaStream_t st) {
  char* p = static_cast<char*>(base);
  out->cnt = (Counts*)p;
  p += align256(sizeof(Counts));
  out->pts = (PcPt*)p;
  p += align256((size_t)n * sizeof(PcPt));
  out->list = (int*)p;
  p += align256(((size_t)n + kMaxCls * kBatch) * sizeof(int));
  out->slow = (float4*)p;
  KernelTimer kt(ctx, "pc_tc_prep", st);
  if (n <= 1024) {
    pc_tc_split<true><<<1, 1024, 0, st>>>(g, fp64 ? 1 : 0, pts, out->pts, n, out->list, out->slow, out->cnt);
    OH_LAUNCH_CHECK();
    return OH_OK;
  }
  OH_CUDA_TRY(cudaMemsetAsync(out->cnt, 0, sizeof(Counts), st));
  pc_tc_prep<<<std::min((n + 127) / 128, sm_count() * 8), 128, 0, st>>>(g, pts, n, fp64 ? 1 : 0, out->pts, out->cnt);
  OH_LAUNCH_CHECK();
  pc_tc_split<false><<<1, 1024, 0, st>>>(g, 0, pts, out->pts, n, out->list, out->slow, out->cnt);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

int point_splits(int regions, int n, int slots, int batches) {
  int splits = 1;
  double best = 0.0;
  for (int s = 1; s <= 8 && (s == 1 || n / (kBatch * s) >= batches); ++s) {
    const double waves = (double)regions * s / slots, fill = waves / std::ceil(waves);
    if (fill > best + 1e-9) { best = fill; splits = s; }
    if (best >= 0.95) break;
  }
  return splits;
}

}  // namespace pctc

bool pc_tc_wants(const PCGeom& g, int n, bool fp64) {
  // FP32: the direct kernels take about 0.24 us per point (a block's serial
  // chain) or 1.1e-6 us per term, whichever sum is due; below 60 us they beat the
  // launches and part-filled regions here (1024x1024 x 60 points: 87 us direct, 48
  // here; x 120: 148 and 69; 128x128 x 500: 128 and 58).
  // FP64: directly 3 to 7 us per point (a block's serial chain) or 73 ps per term
  // (the FP64 pipe); here 55 us at least (100x100 x 30 points: 90 us directly, 57
  // us here; 300x300 x 30: 262 and 61).
  const double terms = (double)n * g.nx * g.ny;
  const double direct = fp64 ? 7.0 * n + 7.3e-5 * terms : 0.24 * n + 1.1e-6 * terms;
  if (direct < (fp64 ? 150.0 : 60.0)) return false;
  const long long regions = (long long)((g.nx + kCols - 1) / kCols) * ((g.ny + kRows - 1) / kRows);
  if (regions >= (1 << 24)) return false;
  if (!fp64 && n < 4096) {
    // Small planes have few regions, and small clouds few points to split among more
    // CTAs: 45 us, then 0.22 us for each point of a CTA alone on its SM (128x128 x 250
    // points: 69 us directly, 110 here in one split).
    const int splits = point_splits((int)regions, n, 2 * sm_count(), kMinBatches);
    const double ctas = (double)regions * splits;
    const double share = ctas > sm_count() ? 2.0 * std::ceil(ctas / (2.0 * sm_count())) : 1.0;
    if (direct < 1.1 * (45.0 + 0.22 * share * n / splits)) return false;
  }
  int dev = 0, major = 0, minor = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return major == 10 && minor == 3;
}

oh_status pc_tc_enqueue(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, float2* field, float* fringe,
                        bool accumulate, bool fine, const float4** slow, const int** slow_n, cudaStream_t st) {
  const int rx = (g.nx + kCols - 1) / kCols, ry = (g.ny + kRows - 1) / kRows, regions = rx * ry;
  const int splits = point_splits(regions, n, 2 * sm_count(), kMinBatches);
  const size_t plane = (size_t)g.nx * g.ny, o_part = sorted_bytes(n);
  void* ptr;
  OH_TRY(scratch(ctx, "pc.tc", o_part + plane * splits * sizeof(float2), &ptr));
  float2* part = (float2*)((char*)ptr + o_part);
  Sorted s;
  OH_TRY(sort_points(ctx, g, pts, n, false, ptr, &s, st));
  PcTcArgs a{g, s.pts, s.list, s.cnt, rx, splits, part, ctx->dev_err};
  auto launch = [&](auto kern, int stage_bytes) -> oh_status {
    const int smem = kStages * stage_bytes + 1024 + 256;
    OH_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    KernelTimer kt(ctx, "pc_tc_regions", st);
    kern<<<dim3(regions, splits), kThreads, smem, st>>>(a);
    OH_LAUNCH_CHECK();
    return OH_OK;
  };
  OH_TRY(fine ? launch(pc_tc_regions<true>, kStageBytes<true>) : launch(pc_tc_regions<false>, kStageBytes<false>));
  KernelTimer kt(ctx, "pc_tc_sum", st);
  pc_tc_sum<<<(int)std::min<size_t>((plane + 255) / 256, (size_t)sm_count() * 16), 256, 0, st>>>(
      part, splits, plane, s.cnt, field, fringe, accumulate ? 1 : 0);
  OH_LAUNCH_CHECK();
  *slow = s.slow;
  *slow_n = &s.cnt->slow;
  return OH_OK;
}

}  // namespace oh
