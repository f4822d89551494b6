// FP64 point-cloud hologram as a contraction on the tensor cores.
//
// The region form of pc_tc.cu carried further.  Beyond the term -P Q / 4 the
// distance over r0 has -(3/32) P^2 Q^2 (and terms below 5e-13 rad for 512 um
// regions at 0.1 m), so the cross phase is a function of the product P Q alone,
//   chi + mu,  chi = -(k r0 / 4) P Q,  mu = -1.5 chi^2 / (k r0),
// and exp(i (chi + mu)) six separable terms (n < 6; chi^6 / 720 is below
// 1.2e-10 where pc_tc_prep lets a point in, at the plane's corner, and mostly far
// less).
// Axis phases are 64-bit fractions of a turn (a quartic in the pixel offset in
// exact integer arithmetic, its coefficients from FP64 once per point and
// region), their sines and cosines and the factors two-float numbers
// (pc_ff.cuh, about 2e-13).
//
// The products run on BF16 operands without rounding error: terms 0, 1 are
// split into multiples of 2^-8, 2^-16 and 2^-24 of at most 256 steps each and two
// BF16 rests, terms 2, 3 the same from 2^-16 on their small side, terms 4, 5 into
// two BF16 parts.  The products of slices i and j, i + j <= 4, go to four FP32
// accumulators in TMEM: level i + j = 0, 1 and 2, whose sums over 96 points stay
// within 24 bits of their common step and are exact, and one for the rest
// (2^-25 and below).  Every 96 points the producers add the four into a
// two-float partial plane in global memory (L2); pc_tc_sum64 adds the splits'
// planes and converts.  Steps are fixed relative to a class's scale (pc_tc_split): clouds of
// uneven amplitude get a scale per class.  Against a 64-bit sum with r / lambda to extended
// precision: 1.4e-12 (1024x1024, 5000 points; the direct kernel 8e-11).
//
// One CTA per region and split of the points, one per SM (TMEM full), 26 warps:
// warps 0-15 build the row operands (A) of four points per stage, warps 16-23
// the column operands (B), warp 24 issues tcgen05.mma (28 per stage: M 128, N
// 128, K 16 = 4 points x 2 terms x (Re, Im)), warp 25 forms the records of 32
// points at a time.  Waits are bounded: on timeout the CTA sets the device
// error word and the outputs stay unwritten.
//
// 1024x1024, 5000 points: 382 ms directly (FP64 pipe) -> 3.8 ms.  What bounds it:
// the producers' dependent two-float chains (about 2.3 ms of it), then the group
// additions (0.65 ms) and the products (28 x 64 clocks a stage, mostly hidden).
// The products issued from a run-time table took 225 clocks each (6.1 ms).
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include "pc_ff.cuh"
#include "pc_tc.cuh"
#include "tc_common.cuh"

namespace oh {

namespace {

using namespace pctc;
using tc::su32;

constexpr int kTiles = 6;                              // 8 KB tiles of 128 rows x 32 BF16 per operand
constexpr int kTile = 128 * 32 * 2;
constexpr int kStages = 2, kStageBytes = 2 * kTiles * kTile;
constexpr int kAccCols = 128, kTmemCols = 4 * kAccCols;
constexpr int kAWarps = 16, kBWarps = 8, kThreads = 32 * (kAWarps + kBWarps + 2);
constexpr int kGroup = 3;                              // batches (96 points) between additions to the partial plane
constexpr uint32_t kIdesc = tc::idesc_bf16(128, 128, 0, 0);

struct alignas(16) RecA { uint64_t t0, c1, c2, c3, c4; float c5, c6; ff a, b; float amp, qs; };
struct alignas(16) RecB { uint64_t c1, c2, c3, c4; float c5, c6; ff a, b, kq; float cmu, pad; };

struct Args {
  PCGeom g;
  const PcPt* pts;
  const int* list;
  Counts* cnt;
  int regions_x, splits;
  double il, il_lo;                // 1 / lambda = il + il_lo
  float4* part;                    // [splits][ny][nx] (Re h, Re l, Im h, Im l)
  int* err;
};

// Byte offset of point j's 8 bytes (two terms' Re, Im) in K block blk of row r:
// 64-byte swizzled rows of two blocks of 16 BF16.
__device__ __forceinline__ int sw_off(int r, int blk, int j) {
  return r * 64 + (((2 * blk + (j >> 1)) ^ ((r >> 1) & 3)) << 4) + ((j & 1) << 3);
}
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void put(unsigned char* tile, int off, uint32_t a, uint32_t b) {
  *reinterpret_cast<uint2*>(tile + off) = make_uint2(a, b);
}

// (tile, K block) of a pair of terms' slice: terms 0, 1 slice k: tile k block 0;
// terms 2, 3: A slices 0-3 tile k block 1, B slices 1-4 tile k block 1; terms 4,
// 5: part 0 in the free block (A tile 4, B tile 0, block 1), part 1 tile 5 block 0.
struct Op { int at, ab, bt, bb, acc; };
__device__ __forceinline__ constexpr Op product(int o) {
  constexpr Op ops[28] = {
    {0, 0, 0, 0, 0},
    {0, 0, 1, 0, 1}, {1, 0, 0, 0, 1}, {0, 1, 1, 1, 1},
    {0, 0, 2, 0, 2}, {1, 0, 1, 0, 2}, {2, 0, 0, 0, 2}, {0, 1, 2, 1, 2}, {1, 1, 1, 1, 2},
    {0, 0, 3, 0, 3}, {1, 0, 2, 0, 3}, {2, 0, 1, 0, 3}, {3, 0, 0, 0, 3},
    {0, 0, 4, 0, 3}, {1, 0, 3, 0, 3}, {2, 0, 2, 0, 3}, {3, 0, 1, 0, 3}, {4, 0, 0, 0, 3},
    {0, 1, 3, 1, 3}, {1, 1, 2, 1, 3}, {2, 1, 1, 1, 3},
    {0, 1, 4, 1, 3}, {1, 1, 3, 1, 3}, {2, 1, 2, 1, 3}, {3, 1, 1, 1, 3},
    {4, 1, 0, 1, 3}, {5, 0, 0, 1, 3}, {4, 1, 5, 0, 3}};
  return ops[o];
}

__global__ void __launch_bounds__(kThreads, 1) pc_tc64_regions(Args a) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ float4 tab[256];
  __shared__ RecA recA[2][kBatch];
  __shared__ RecB recB[2][kBatch];
  __shared__ int cls_batch[kMaxCls + 1], cls_e[kMaxCls];
  const uint32_t raw = su32(smem_dyn);
  unsigned char* base = smem_dyn + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + kStages * kStageBytes);   // [2], one arrival per producer warp
  uint64_t* empty = full + 2;             // [2], tcgen05.commit
  uint64_t* rfull = full + 4;             // [2], the record warp's
  uint64_t* rempty = full + 6;            // [2], one arrival per producer warp
  uint64_t* gdone = full + 8;             // a group's products are done (tcgen05.commit)
  uint64_t* gfree = full + 9;             // a group's accumulators are read, one arrival per A warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full + 10);
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
  constexpr int kPer = kBatch / kPts;     // stages per record batch
  float4* part = a.part + (size_t)blockIdx.y * nx * ny;
  if (nfast == 0) return;                 // pc_tc_sum64 reads no partial plane then
  if (nst <= 0) {
    for (int i = threadIdx.x; i < kRows * kCols; i += kThreads) {
      const int r = Y0 + i / kCols, c = X0 + i % kCols;
      if (r < ny && c < nx) part[(size_t)r * nx + c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      tc::mb_init(&full[s], kAWarps + kBWarps);
      tc::mb_init(&empty[s], 1);
      tc::mb_init(&rfull[s], 1);
      tc::mb_init(&rempty[s], kAWarps + kBWarps);
    }
    tc::mb_init(gdone, 1);
    tc::mb_init(gfree, kAWarps);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  ff_directions(tab, threadIdx.x, kThreads);
  if (threadIdx.x <= ncls) cls_batch[threadIdx.x] = a.cnt->batch[threadIdx.x];
  if (threadIdx.x < ncls) cls_e[threadIdx.x] = class_exp(a.cnt->exp[threadIdx.x]);
  if (warp == 1) tc::tmem_alloc(tmem_slot, kTmemCols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < kAWarps) {
    // A: point slot j of row r; a half-warp's rows r, r + 1, r + 4, r + 5 spread
    // its 8-byte stores over all banks
    const int j = threadIdx.x & 3, q = threadIdx.x >> 2;
    const int row = (q & 1) | ((q & 2) << 1) | ((q & 4) >> 1) | (q & ~7);
    const int m = row - kRows / 2;
    const int off0 = sw_off(row, 0, j), off1 = sw_off(row, 1, j);
    // group g's sums into the partial plane: TMEM lanes 32 (warp % 4) .. (region
    // rows), 16 complex columns per warp / 4
    const int Y = Y0 + 32 * (warp & 3) + lane, c0 = 16 * (warp >> 2);
    auto flush = [&](int g, float rel) -> bool {         // rel: the group's scale over the first class's
      if (!warp_wait(gdone, (uint32_t)(g & 1), abort_flag, lane)) return false;
      tc::fence_after();
      float4* dst = part + (size_t)Y * nx + X0 + c0;
      const uint32_t at = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(2 * c0);
#pragma unroll 1
      for (int c = 0; c < 16; c += 4) {
        uint32_t v[32];                                  // eight columns of each accumulator
        tc::tmem_ld8x4(at + 2 * c, at + kAccCols + 2 * c, at + 2 * kAccCols + 2 * c, at + 3 * kAccCols + 2 * c, v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (Y >= ny || X0 + c0 + c + i >= nx) continue;
          float4 o = g ? dst[c + i] : make_float4(0.f, 0.f, 0.f, 0.f);
          auto add = [&](int k, float h, float l) -> ff {
            const ff s = ff_sum(__uint_as_float(v[k]), __uint_as_float(v[8 + k]));
            const float tail = __uint_as_float(v[16 + k]) + __uint_as_float(v[24 + k]);
            const ff t = ff_sum(h, OH_FMUL(rel, s.h));
            return ff_quick(t.h, OH_FADD(OH_FADD(t.l, l), OH_FMUL(rel, OH_FADD(s.l, tail))));
          };
          const ff re = add(2 * i, o.x, o.y), im = add(2 * i + 1, o.z, o.w);
          dst[c + i] = make_float4(re.h, re.l, im.h, im.l);
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
      const int s = it & 1, batch = it / kPer, rs = batch & 1;
      if (it % kPer == 0) ok = warp_wait(&rfull[rs], (uint32_t)((batch >> 1) & 1), abort_flag, lane);
      ok = ok && warp_wait(&empty[s], (uint32_t)(((it >> 1) & 1) ^ 1), abort_flag, lane);
      if (!ok) break;
      unsigned char* A = base + s * kStageBytes;
      const RecA& r = recA[rs][(it % kPer) * kPts + j];
      const AxisRec ax{r.t0, r.c1, r.c2, r.c3, r.c4, r.c5, r.c6, r.a, r.b};
      const ffc E = axis_cis(ax, m, tab);
      const ff Q = axis_cross(ax, m, r.qs);
      ff re = ff_mulf(E.x, r.amp), im = ff_mulf(E.y, r.amp);
      const ff r1 = re * Q, i1 = im * Q;
      {
        float a0[5], a1[5], b0_[5], b1_[5];
        ff_slices<true>(re, a0);
        ff_slices<true>(im, a1);
        ff_slices<true>(r1, b0_);
        ff_slices<true>(i1, b1_);
#pragma unroll
        for (int k = 0; k < 5; ++k) put(A + k * kTile, off0, pack(a0[k], a1[k]), pack(b0_[k], b1_[k]));
      }
      re = r1 * Q;
      im = i1 * Q;
      const float r3 = re.h * Q.h, i3 = im.h * Q.h;
      {
        float a0[5], a1[5], b0_[5], b1_[5];
        ff_slices<true>(re, a0);
        ff_slices<true>(im, a1);
        ff_slices<true>(ff{r3, 0.f}, b0_);
        ff_slices<true>(ff{i3, 0.f}, b1_);
#pragma unroll
        for (int k = 0; k < 4; ++k) put(A + k * kTile, off1, pack(a0[k], a1[k]), pack(b0_[k], b1_[k]));
      }
      {
        const float r4 = r3 * Q.h, i4 = i3 * Q.h, r5 = r4 * Q.h, i5 = i4 * Q.h;
        const float r4h = bf16_round(r4), i4h = bf16_round(i4), r5h = bf16_round(r5), i5h = bf16_round(i5);
        put(A + 4 * kTile, off1, pack(r4h, i4h), pack(r5h, i5h));
        put(A + 5 * kTile, off0, pack(r4 - r4h, i4 - i4h), pack(r5 - r5h, i5 - i5h));
      }
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
  } else if (warp < kAWarps + kBWarps) {
    // B: point slot j of column x; rows 2x (Re, -Im) and 2x + 1 (Im, Re)
    const int t = threadIdx.x - 32 * kAWarps, j = t & 3, x = t >> 2, m = x - kCols / 2;
    const int o0 = sw_off(2 * x, 0, j), o1 = sw_off(2 * x + 1, 0, j), p0 = sw_off(2 * x, 1, j), p1 = sw_off(2 * x + 1, 1, j);
    auto put2 = [&](unsigned char* tile, int e, int o, float ar, float ai, float br, float bi) {
      put(tile, e, pack(ar, -ai), pack(br, -bi));
      put(tile, o, pack(ai, ar), pack(bi, br));
    };
    bool ok = true;
    for (int it = 0; it < nst && ok; ++it) {
      const int s = it & 1, batch = it / kPer, rs = batch & 1;
      if (it % kPer == 0) ok = warp_wait(&rfull[rs], (uint32_t)((batch >> 1) & 1), abort_flag, lane);
      ok = ok && warp_wait(&empty[s], (uint32_t)(((it >> 1) & 1) ^ 1), abort_flag, lane);
      if (!ok) break;
      unsigned char* B = base + s * kStageBytes + kTiles * kTile;
      const RecB& r = recB[rs][(it % kPer) * kPts + j];
      const AxisRec ax{0ull, r.c1, r.c2, r.c3, r.c4, r.c5, r.c6, r.a, r.b};
      const ffc E = axis_cis(ax, m, tab);
      const ff ch = r.kq * axis_cross(ax, m, 1.f);
      const ff R1r = -E.y * ch, R1i = E.x * ch;            // i chi E
      {
        float a0[5], a1[5], b0_[5], b1_[5];
        ff_slices<true>(E.x, a0);
        ff_slices<true>(E.y, a1);
        ff_slices<true>(R1r, b0_);
        ff_slices<true>(R1i, b1_);
#pragma unroll
        for (int k = 0; k < 5; ++k) put2(B + k * kTile, o0, o1, a0[k], a1[k], b0_[k], b1_[k]);
      }
      // (-chi^2 / 2 + i mu) E,  (-i chi^3 / 6 - chi mu) E,  chi^4 / 24 E,  i chi^5 / 120 E
      const ff hc{0.5f * ch.h, 0.5f * ch.l};
      ff R2r = -R1i * hc, R2i = R1r * hc;
      const float c2 = ch.h * ch.h, c3 = c2 * ch.h, mu = r.cmu * c2;
      R2r.l = OH_FFMA(-mu, E.y.h, R2r.l);
      R2i.l = OH_FFMA(mu, E.x.h, R2i.l);
      const float k3 = c3 * 0.16666667f, m3 = -c3 * r.cmu;
      {
        float a0[5], a1[5], b0_[5], b1_[5];
        ff_slices<false>(R2r, a0);
        ff_slices<false>(R2i, a1);
        ff_slices<false>(ff{E.x.h * m3 + E.y.h * k3, 0.f}, b0_);
        ff_slices<false>(ff{E.y.h * m3 - E.x.h * k3, 0.f}, b1_);
#pragma unroll
        for (int k = 1; k < 5; ++k) put2(B + k * kTile, p0, p1, a0[k], a1[k], b0_[k], b1_[k]);
      }
      {
        const float k4 = c2 * c2 * 0.041666668f, k5 = c3 * c2 * 0.0083333333f;
        const float r4 = E.x.h * k4, i4 = E.y.h * k4, r5 = -E.y.h * k5, i5 = E.x.h * k5;
        const float r4h = bf16_round(r4), i4h = bf16_round(i4), r5h = bf16_round(r5), i5h = bf16_round(i5);
        put2(B, p0, p1, r4h, i4h, r5h, i5h);
        put2(B + 5 * kTile, o0, o1, r4 - r4h, i4 - i4h, r5 - r5h, i5 - i5h);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        arrive(&full[s]);
        if (it % kPer == kPer - 1) arrive(&rempty[rs]);
      }
    }
  } else if (warp == kAWarps + kBWarps) {
    if (lane == 0) {
      Groups gr{cls_batch, ncls, b1, kGroup, 0, 0};
      gr.start(b0);
      int next = min(nst, (gr.end - b0) * kPer);
      uint32_t add = 0u, gph = 0u;        // the group's first stage starts its accumulators
      for (int it = 0; it < nst; ++it) {
        const int s = it & 1;
        bool ok = true;
        if (it == next) {
          ok = wait_live(gfree, gph, abort_flag);
          gph ^= 1u;
          gr.start(gr.end);
          next = min(nst, (gr.end - b0) * kPer);
          add = 0u;
        }
        ok = ok && wait_live(&full[s], (uint32_t)((it >> 1) & 1), abort_flag);
        if (!ok) {
          atomicExch(abort_flag, 1);
          break;
        }
        tc::fence_after();
        const uint32_t A = su32(base + s * kStageBytes), B = A + kTiles * kTile;
        const uint64_t dA = tc::desc_sw64(A, 16, 512), dB = tc::desc_sw64(B, 16, 512);
        // (unrolled: 28 products a stage, 64 clocks each, leave one thread no
        // time for address arithmetic)
#pragma unroll
        for (int o = 0; o < 28; ++o) {
          const Op op = product(o);
          const bool start = o == 0 || o == 1 || o == 4 || o == 9;       // first product of its accumulator
          tc::umma_bf16(tmem + op.acc * kAccCols, dA + (uint64_t)(op.at * (kTile >> 4) + op.ab * 2),
                        dB + (uint64_t)(op.bt * (kTile >> 4) + op.bb * 2), kIdesc, start ? add : 1u);
        }
        add = 1u;
        tc::umma_commit(&empty[s]);
        if (it == next - 1) tc::umma_commit(gdone);
      }
    }
  } else {
    // record warp: lane k forms point k of each batch
    const double Xc = ((double)(X0 + kCols / 2) + 0.5) * a.g.px - a.g.hlx;
    const double Yc = a.g.hly - ((double)(Y0 + kRows / 2) + 0.5) * a.g.py;
    const double ref = (Xc * a.g.stx + Yc * a.g.sty) * a.il;
    int c = 0;
    auto fix64 = [](double t) { return (uint64_t)__double2ll_rn((t - rint(t)) * 9223372036854775808.0) << 1; };
    const int batches = b1 - b0;
    for (int b = 0; b < batches; ++b) {
      const int rs = b & 1;
      if (!warp_wait(&rempty[rs], (uint32_t)(((b >> 1) & 1) ^ 1), abort_flag, lane)) break;
      const int k = first + b * kBatch + lane;
      RecA ra{};
      RecB rb{};
      ra.qs = 1.f;
      while (c + 1 < ncls && cls_batch[c + 1] <= b0 + b) ++c;
      const int at = k < last ? identity ? k : a.list[k] : -1;
      if (at >= 0) {
        const PcPt p = a.pts[at];
        const double dx = Xc - p.x, dy = Yc - p.y, az = fabs(p.z);
        const double rho2 = fma(dx, dx, dy * dy), r2 = fma(az, az, rho2);
        const double ri = rsqrt(r2), r0 = r2 * ri;
        // r0 / lambda = |z| / lambda (to twice FP64) + rho^2 / (r0 + |z|) / lambda
        const double w = az * a.il, wl = fma(az, a.il, -w) + az * a.il_lo;
        const double v = rho2 / (r0 + az) * a.il - ref;
        ra.t0 = fix64((w - rint(w)) + wl + (v - rint(v)));
        const double C = r0 * a.il;
        // (r0 / lambda) (sqrt(1 + 2 s t + t^2) - 1), t = m tau: the terms in m .. m^6
        auto axis = [&](double s, double tilt, double pitch, uint64_t* c1, uint64_t* c2, uint64_t* c3, uint64_t* c4,
                        float* c5, float* c6) {
          const double tau = pitch * ri, t2 = tau * tau, s2 = s * s, e2 = C * (1.0 - s2) * 0.5 * t2, e3 = e2 * tau, e4 = e2 * t2;
          *c1 = fix64((s - tilt) * pitch * a.il);
          *c2 = fix64(e2);
          *c3 = fix64(-s * e3);
          *c4 = fix64(e4 * (1.25 * s2 - 0.25));
          const float f5 = (float)(e3 * t2), sf = (float)s, sf2 = sf * sf;
          *c5 = f5 * sf * (0.75f - 1.75f * sf2);
          *c6 = f5 * (float)tau * (0.125f - 1.75f * sf2 + 2.625f * sf2 * sf2);
        };
        const double sx = dx * ri, sy = -dy * ri;       // rows run against y
        axis(sx, a.g.stx, a.g.px, &rb.c1, &rb.c2, &rb.c3, &rb.c4, &rb.c5, &rb.c6);
        axis(sy, -a.g.sty, a.g.py, &ra.c1, &ra.c2, &ra.c3, &ra.c4, &ra.c5, &ra.c6);
        const double tx = a.g.px * ri, ty = a.g.py * ri;
        const double ay = 2.0 * sy * ty, by = ty * ty;
        // scale of the row factor: its maximum over the region (1 % for its curvature),
        // so that |Q| <= 1 and the column factor is no larger than chi: above 0.088
        // its second term would leave the 256 steps that BF16 holds (a power of
        // two above the maximum did, 3e-6 off at the corners of 1920 x 1080)
        const double qs = (double)(float)(1.01 * (fabs(ay) * (kRows / 2) + by * (kRows / 2) * (kRows / 2))), iqs = 1.0 / qs;
        ra.a = ff(ay * iqs); ra.b = ff(by * iqs);
        ra.qs = (float)qs;
        ra.amp = p.a * pow2f(-cls_e[c]);
        rb.a = ff(2.0 * sx * tx); rb.b = ff(tx * tx);
        const double kr = 6.283185307179586476925286766559 * C;
        rb.kq = ff(-0.25 * kr * qs);
        rb.cmu = -1.5f / (float)kr;
      }
      recA[rs][lane] = ra;
      recB[rs][lane] = rb;
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
  if (!good && threadIdx.x == 32 * (kAWarps + kBWarps)) {
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

// The splits' partial planes added in order (two-float), converted and unscaled.
__global__ void __launch_bounds__(256) pc_tc_sum64(const float4* __restrict__ part, int splits, size_t n,
                                                   const Counts* __restrict__ cnt, double2* __restrict__ field,
                                                   double* __restrict__ fringe, int accumulate) {
  if (cnt->aborted) return;
  const bool none = cnt->fast == 0;
  const float unscale = pow2f(class_exp(cnt->exp[0]));
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    ff re{0.f, 0.f}, im{0.f, 0.f};
    if (!none)
      for (int s = 0; s < splits; ++s) {
        const float4 p = part[(size_t)s * n + i];
        const ff u = ff_sum(re.h, p.x), v = ff_sum(im.h, p.z);
        re = ff_quick(u.h, OH_FADD(u.l, OH_FADD(re.l, p.y)));
        im = ff_quick(v.h, OH_FADD(v.l, OH_FADD(im.l, p.w)));
      }
    // an exact scale per part; the sum rounds once
    const double x = (double)re.h * unscale + (double)re.l * unscale, y = (double)im.h * unscale + (double)im.l * unscale;
    if (field) {
      double2 f = make_double2(x, y);
      if (accumulate) { const double2 b = field[i]; f.x += b.x; f.y += b.y; }
      field[i] = f;
    }
    if (fringe) fringe[i] += x;
  }
}

}  // namespace

oh_status pc_tc64_enqueue(oh_ctx* ctx, const PCGeom& g, const float4* pts, int n, double2* field, double* fringe,
                          bool accumulate, const float4** slow, const int** slow_n, cudaStream_t st) {
  const int rx = (g.nx + kCols - 1) / kCols, ry = (g.ny + kRows - 1) / kRows, regions = rx * ry;
  const int splits = point_splits(regions, n, sm_count(), 3);
  const size_t plane = (size_t)g.nx * g.ny, o_part = sorted_bytes(n);
  void* ptr;
  OH_TRY(scratch(ctx, "pc.tc", o_part + plane * splits * sizeof(float4), &ptr));
  float4* part = (float4*)((char*)ptr + o_part);
  Sorted s;
  OH_TRY(sort_points(ctx, g, pts, n, true, ptr, &s, st));
  const int smem = kStages * kStageBytes + 1024 + 256;
  OH_CUDA_TRY(cudaFuncSetAttribute(pc_tc64_regions, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const double il = 1.0 / g.lambda;
  Args a{g, s.pts, s.list, s.cnt, rx, splits, il, std::fma(-g.lambda, il, 1.0) * il, part, ctx->dev_err};
  {
    KernelTimer kt(ctx, "pc_tc64_regions", st);
    pc_tc64_regions<<<dim3(regions, splits), kThreads, smem, st>>>(a);
    OH_LAUNCH_CHECK();
  }
  KernelTimer kt(ctx, "pc_tc_sum64", st);
  pc_tc_sum64<<<(int)std::min<size_t>((plane + 255) / 256, (size_t)sm_count() * 16), 256, 0, st>>>(
      part, splits, plane, s.cnt, field, fringe, accumulate ? 1 : 0);
  OH_LAUNCH_CHECK();
  *slow = s.slow;
  *slow_n = &s.cnt->slow;
  return OH_OK;
}

}  // namespace oh
