// Implicit-GEMM convolutions on the tcgen05 tensor cores (BF16 operands,
// FP32 accumulation in TMEM), the compute core of the learned surrogate.
//
// Activations are NHWC BF16 with a channel stride that is a multiple of 32
// (64 bytes), so 32 channels of one pixel are one 64-byte line of a
// 64-byte-swizzled shared-memory tile.
//
// conv_fwd_tc: Y[p][co] = sum_{tap, ci} X[p + s*off(tap)][ci] W[co][tap*cin + ci]
//   GEMM with M = 128 pixels (a bx x by patch), N = BN output channels,
//   K = taps x cin in 32-channel steps.  The A tile of a K step is one TMA
//   load of the 4-D activation map at the tap's offset: out-of-range pixels
//   read as zero, which is the convolution's zero padding.  s = +1 is the
//   forward convolution; s = -1 with the transposed weight matrix
//   Wt[ci][tap*cout + co] is the gradient with respect to the input (dgrad).
//   Epilogue: + bias, ReLU, multiplication by (mask > 0) (the ReLU derivative
//   of the layer below, for dgrad), BF16 store with an output channel stride
//   (so a layer can write straight into one half of a concatenation buffer).
// conv_wgrad_tc: dW^T[tap*cin + ci][co] += sum_p X[p + off(tap)][ci] dZ[p][co]
//   GEMM with M = 128 rows of the (tap, ci) space (four 32-channel groups,
//   each its own TMA load at its tap's offset), N = cout, K = pixels in
//   64-pixel steps; both operands are MN-major (channels contiguous), K split
//   across CTAs, partial sums added with vector reductions.
//
// Roles: one or more warps issue TMA loads into a ring of stages, one or more
// issue tcgen05.mma and release stages with tcgen05.commit, four or eight read the
// accumulators (warp w TMEM lanes 32 (w % 4) .. + 31).  Every
// mbarrier wait gives up after about one second of SM clock: the CTA then
// sets the device error word, lets its copies and MMAs land, frees TMEM and
// returns.  Pipeline waits (a stage's copies, a stage's release) also give
// up as soon as the other role has aborted; the final waits for the MMAs and
// for copies still in flight keep the full bound.
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdlib>
#include "context.h"
#include "tc_common.cuh"
#include "unet.cuh"

namespace oh {

namespace {

constexpr int kConvThreads = 128;
constexpr long long kWaitCycles = 2000000000LL;      // ~1 s at 2 GHz

__device__ __forceinline__ bool wait_live(uint64_t* b, uint32_t parity, const int* abort) {
  const long long t0 = clock64();
  while (!tc::mb_try(b, parity)) {
    if (*((volatile const int*)abort) || clock64() - t0 > kWaitCycles) return false;
  }
  return true;
}

// Waits for the copies of each stage's last use, which two loaders arrive on
// (uses[2][n]: loads issued): after an abort one may be a use ahead of the other,
// whose arrival is made up here.
__device__ __forceinline__ void land_pairs(uint64_t* full, const int* uses, int n) {
  for (int i = 0; i < n; ++i) {
    const int u = uses[i], v = uses[n + i];
    if (u != v) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::su32(&full[i])) : "memory");
    if (max(u, v)) tc::mb_wait(&full[i], (uint32_t)((max(u, v) - 1) & 1), kWaitCycles);
  }
}

constexpr int pow2_at_least(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512; }

template <int BN> struct FwdCfg {
  static constexpr int kA = 128 * 64;                  // 128 pixels x 32 channels
  static constexpr int kB = BN * 64;                   // BN rows x 32 K
  static constexpr int kSteps = 3;                     // K steps per stage: a wait and a commit per six MMAs
  static constexpr int kStage = kSteps * (kA + kB);
  static constexpr int kStages = BN <= 64 ? 3 : BN == 96 ? 5 : BN == 128 ? 4 : 3;
  static constexpr int kTmemBuf = pow2_at_least(BN);  // columns of one accumulator
  static constexpr int kTmem = 2 * kTmemBuf;          // two accumulators: MMA and epilogue overlap
  static constexpr int kThreads = 224;                // warps 0, 1 TMA, warp 2 MMA, warps 3-6 epilogue
  static constexpr int kSmem = kStages * kStage + 1024 + 256;
};

// 32 output channels cb.. of pixel pix from the accumulator's columns r: bias,
// ReLU, mask, BF16 store.
__device__ __forceinline__ void conv_store32(const ConvArgs& a, const uint32_t* r, const float* bias, size_t pix,
                                             int cb) {
  float v[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(r[e]);
#pragma unroll
  for (int e = 0; e < 32; ++e) v[e] += bias[e];
  if (a.relu) {
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = fmaxf(v[e], 0.f);
  }
  if (a.mask) {
    const uint4* mp = reinterpret_cast<const uint4*>(a.mask + pix * a.mask_cs + cb);
#pragma unroll
    for (int g4 = 0; g4 < 4; ++g4) {
      const uint4 mv = __ldg(mp + g4);
      const __nv_bfloat162* mb = reinterpret_cast<const __nv_bfloat162*>(&mv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(mb[e]);
        if (!(f.x > 0.f)) v[g4 * 8 + 2 * e] = 0.f;
        if (!(f.y > 0.f)) v[g4 * 8 + 2 * e + 1] = 0.f;
      }
    }
  }
  uint4* op = reinterpret_cast<uint4*>(a.out + pix * a.out_cs + cb);
#pragma unroll
  for (int g4 = 0; g4 < 4; ++g4) {
    uint4 o;
    __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) ob[e] = __floats2bfloat162_rn(v[g4 * 8 + 2 * e], v[g4 * 8 + 2 * e + 1]);
    op[g4] = o;
  }
}

// Persistent CTAs: CTA i takes pixel tiles i, i + gridDim.x, ... of output
// channel tile blockIdx.y.  Two loading warps stream the K steps of all its
// tiles (one the pixels, one the weights) through one ring of stages; the MMA
// issuer accumulates tile j into TMEM buffer j & 1 and commits it to the epilogue
// warps, which drain it (bias, ReLU, mask, BF16 store) while the next tile
// accumulates in the other buffer.
//
// What bounds it: the layers that come here are narrow (less than 128 pixels),
// often one tile per CTA, and its K steps run in series: about 350 clocks for each
// when every step had its own wait and commit.
template <int BN>
__global__ void __launch_bounds__(FwdCfg<BN>::kThreads) conv_fwd_tc(const __grid_constant__ CUtensorMap mX,
                                                                    const __grid_constant__ CUtensorMap mW,
                                                                    ConvArgs a) {
  typedef FwdCfg<BN> Cfg;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = tc::su32(smem_raw);
  unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + Cfg::kStages * Cfg::kStage);
  uint64_t* empty = full + Cfg::kStages;
  uint64_t* tfull = empty + Cfg::kStages;              // [2] accumulator ready (MMA commit)
  uint64_t* tempty = tfull + 2;                        // [2] accumulator drained (4 epilogue warps)
  uint64_t* done = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* uses = abort_flag + 1;                          // [2][kStages] loads issued per stage: pixels, weights
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const long long tiles = (long long)a.n * a.tiles_y * a.tiles_x;
  const int ntl = blockIdx.x < tiles ? (int)((tiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  const int co0 = blockIdx.y * BN;
  const int cchunks = a.cin >> 5;
  const int nk = a.taps * cchunks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      tc::mb_init(&full[s], 2); tc::mb_init(&empty[s], 1);
      uses[s] = uses[Cfg::kStages + s] = 0;
    }
    for (int b = 0; b < 2; ++b) { tc::mb_init(&tfull[b], 1); tc::mb_init(&tempty[b], 4); }
    tc::mb_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __shared__ float sbias[BN];               // this CTA's output-channel biases (0 without bias)
  for (int c = threadIdx.x; c < BN; c += blockDim.x)
    sbias[c] = (a.bias && co0 + c < a.cout) ? a.bias[co0 + c] : 0.f;
  if (warp == 2) tc::tmem_alloc(tmem_slot, Cfg::kTmem);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  auto tile_origin = [&](int j, int* img, int* x0, int* y0) {
    uint32_t t = blockIdx.x + (uint32_t)j * gridDim.x;         // (tiles < 2^31)
    const uint32_t u = t / (uint32_t)a.tiles_x;
    *x0 = (int)(t - u * (uint32_t)a.tiles_x) * a.bx;
    *img = (int)(u / (uint32_t)a.tiles_y);
    *y0 = (int)(u - (uint32_t)*img * (uint32_t)a.tiles_y) * a.by;
  };
  // (whole warps wait, so that addresses and descriptors stay in uniform registers)
  auto wait_warp = [&](uint64_t* bar, uint32_t ph) -> bool {
    return __all_sync(0xffffffffu, tc::mb_try(bar, ph)) || __all_sync(0xffffffffu, wait_live(bar, ph, abort_flag));
  };

  if (warp < 3) {
    const bool el = tc::elect_one();
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    auto next = [&]() { if (++s == Cfg::kStages) { s = 0; ph ^= 1u; } };
    if (warp < 2) {
      for (int j = 0; j < ntl && ok; ++j) {
        int img, x0, y0;
        tile_origin(j, &img, &x0, &y0);
        int tap = 0, cc = 0;
        for (int it = 0; it < nk && ok; it += Cfg::kSteps) {
          if (!(ok = wait_warp(&empty[s], ph ^ 1u))) break;
          const int m = min(Cfg::kSteps, nk - it);
          unsigned char* st = base + s * Cfg::kStage + (warp ? Cfg::kSteps * Cfg::kA : 0);
          if (el) {
            uses[warp * Cfg::kStages + s] += 1;
            tc::mb_expect_tx(&full[s], (uint32_t)(m * (warp ? Cfg::kB : Cfg::kA)));
          }
          for (int i = 0; i < m; ++i) {
            int dx = 0, dy = 0;
            if (a.taps == 9) { dx = (tap % 3 - 1) * a.sign; dy = (tap / 3 - 1) * a.sign; }
            if (el) {
              if (warp == 0) tc::tma_load_4d(st + i * Cfg::kA, &mX, cc * 32, x0 + dx, y0 + dy, img, &full[s]);
              else tc::tma_load_2d(st + i * Cfg::kB, &mW, tap * a.cin + cc * 32, co0, &full[s]);
            }
            if (++cc == cchunks) { cc = 0; ++tap; }
          }
          next();
        }
      }
    } else {
      constexpr uint32_t idesc = tc::idesc_bf16(128, BN, 0, 0);
      if (a.stall_flag) ok = __all_sync(0xffffffffu, stall_on_unset_flag(a.stall_flag, a.stall_cycles));
      const uint32_t sbase = tc::su32(base);
      for (int j = 0; j < ntl && ok; ++j) {
        const int b = j & 1;
        if (!(ok = wait_warp(&tempty[b], (uint32_t)(((j >> 1) & 1) ^ 1)))) break;
        tc::fence_after();
        const uint32_t acc = tmem + (uint32_t)(b * Cfg::kTmemBuf);
        for (int it = 0; it < nk; it += Cfg::kSteps) {
          if (!(ok = wait_warp(&full[s], ph))) break;
          tc::fence_after();
          const uint32_t sa = sbase + (uint32_t)(s * Cfg::kStage);
          const uint64_t da = tc::desc_sw64(sa, 16, 512), db = tc::desc_sw64(sa + Cfg::kSteps * Cfg::kA, 16, 512);
#pragma unroll
          for (int i = 0; i < Cfg::kSteps; ++i)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)                      // 16 BF16 = 32 bytes along K
              if (el && it + i < nk)
                tc::umma_bf16(acc, da + (uint64_t)((i * Cfg::kA + kk * 32) >> 4),
                              db + (uint64_t)((i * Cfg::kB + kk * 32) >> 4), idesc, (it | i | kk) ? 1u : 0u);
          if (el) tc::umma_commit(&empty[s]);
          next();
        }
        if (ok && el) tc::umma_commit(&tfull[b]);
      }
      if (el) tc::umma_commit(done);                       // arrives when every MMA issued above has completed
    }
    if (!ok && lane == 0) atomicExch(abort_flag, 1);
  } else {
    // epilogue warps: TMEM lane quarter (warp % 4) = pixels 32 (warp % 4) .. + 31 of the tile
    const int q = warp & 3;
    const int m = q * 32 + lane;
    for (int j = 0; j < ntl; ++j) {
      const int b = j & 1;
      bool ok = true;
      if (lane == 0) ok = wait_live(&tfull[b], (uint32_t)((j >> 1) & 1), abort_flag);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      tc::fence_after();
      int img, x0, y0;
      tile_origin(j, &img, &x0, &y0);
      const int px = x0 + (m % a.bx), py = y0 + (m / a.bx);
      const bool inside = px < a.w && py < a.h;
      const size_t pix = ((size_t)img * a.h + py) * a.w + px;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tc::tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * Cfg::kTmemBuf + c * 32), r);
        const int cb = co0 + c * 32;
        if (!inside || cb >= a.cout) continue;
        conv_store32(a, r, sbias + c * 32, pix, cb);
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::su32(&tempty[b])) : "memory");
    }
  }
  __syncwarp();
  // every MMA issued has completed before TMEM is freed; copies issued but
  // not consumed land before the CTA exits
  if (threadIdx.x == 0) tc::mb_wait(done, 0, kWaitCycles);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (*((volatile int*)abort_flag)) {
      atomicOr(a.err, 2);
      land_pairs(full, uses, Cfg::kStages);
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 2) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, Cfg::kTmem);
  }
}

// 3x3 over whole 128-pixel rows: a tile is 128 pixels of `rows` consecutive output
// rows (an accumulator each).  The weights of a (dy, 32 channels) step are loaded
// once for the tile's rows; a row's 136-pixel box of input row y + dy (from x - 1)
// serves the three dx taps (A operands that start 0, 1 and 2 pixels into it).  An
// output sums over dy, then channels, then dx, whatever the tile.
//
// What bounds it: an MMA of N channels takes max(N / 2, 32 + N / 4) clocks (the
// tensor rate; its operands from shared memory at 128 bytes a clock), but one warp
// that waits for a box, issues six and commits needs about 90 to 120 for each, and
// one that waits for a slot and loads a box about 500.  So up to four warps load
// boxes, a fifth the weights (three taps in one load), and up to four issue, each
// for its own output rows.  4 x 512 x 512 pixels, 192 -> 64 channels: 188 us (470
// with one warp each), where the MMAs take 150 to 180 at the clocks of such a load.
//
// A barrier's parity tells its last two phases apart only to a warp that waits for
// every one of them: loader w fills issuer w's own slots, and every issuer waits
// for every weight step.
//
// Warps 0-4 TMA, warps 5-8 MMA, warps 9-16 epilogue; one CTA per SM takes tiles
// blockIdx.x, + gridDim.x, ... of channel tile blockIdx.y.
struct RowsCfg {
  int rows, nbuf;                      // output rows per tile (1, 2 or a multiple of 4), accumulator sets (2: MMAs
                                       // and epilogue overlap)
  int na, nb;                          // slots: boxes (a multiple of the issuers), weight steps
  uint32_t tmem_cols;
};
constexpr int kRowsA = 136 * 64, kRowsAStride = (kRowsA + 1023) / 1024 * 1024;
constexpr int kRowsLoaders = 4, kRowsIssuers = 4, kRowsEpiWarps = 8;
constexpr int kRowsIssue0 = kRowsLoaders + 1, kRowsEpi0 = kRowsIssue0 + kRowsIssuers;       // first warp of each role
constexpr int kRowsThreads = 32 * (kRowsEpi0 + kRowsEpiWarps);
constexpr int kRowsA_Slots = 32, kRowsB_Slots = 16;     // at most
constexpr int kRowsSmem = 226 * 1024;                   // at most (1 KB for the biases)
constexpr int kRowsFixed = 1024 + kRowsEpiWarps * 2048 + (2 * kRowsA_Slots + 2 * kRowsB_Slots + 8) * 8 +
                           (kRowsA_Slots + kRowsB_Slots) * 4 + 64;

template <int BN>
__global__ void __launch_bounds__(kRowsThreads, 1) conv_fwd_rows(const __grid_constant__ CUtensorMap mX,
                                                                 const __grid_constant__ CUtensorMap mW, ConvArgs a,
                                                                 RowsCfg rc) {
  constexpr int kTap = BN * 64, kB = 3 * kTap;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = tc::su32(smem_raw);
  unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  unsigned char* sB = base + (size_t)rc.na * kRowsAStride;
  unsigned char* sE = sB + (size_t)rc.nb * kB;           // 2 KB per epilogue warp
  uint64_t* fullA = reinterpret_cast<uint64_t*>(sE + kRowsEpiWarps * 2048);
  uint64_t* emptyA = fullA + kRowsA_Slots;
  uint64_t* fullB = emptyA + kRowsA_Slots;
  uint64_t* emptyB = fullB + kRowsB_Slots;
  uint64_t* tfull = emptyB + kRowsB_Slots;             // [2] accumulators ready (MMA commit)
  uint64_t* tempty = tfull + 2;                        // [2] accumulators drained (epilogue warps)
  uint64_t* done = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* usesA = abort_flag + 1;                         // loads issued per slot
  int* usesB = usesA + kRowsA_Slots;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int tiles_r = (a.h + rc.rows - 1) / rc.rows;
  const long long tiles = (long long)a.n * tiles_r * a.tiles_x;
  const int ntl = blockIdx.x < tiles ? (int)((tiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  const int co0 = blockIdx.y * BN;
  const int cchunks = a.cin >> 5;
  const int ni = min(rc.rows, kRowsIssuers);           // issuing warps (1, 2 or 4): row r belongs to the r % ni-th
  const int own = rc.na / ni;                          // box slots per issuer

  {
    // (one barrier per thread: in turn they took 1.3 us)
    const int i = threadIdx.x;
    if (i < rc.na) { tc::mb_init(&fullA[i], 1); tc::mb_init(&emptyA[i], 1); usesA[i] = 0; }
    if (i < rc.nb) { tc::mb_init(&fullB[i], 1); tc::mb_init(&emptyB[i], ni); usesB[i] = 0; }
    if (i < 2) { tc::mb_init(&tfull[i], ni); tc::mb_init(&tempty[i], kRowsEpiWarps); }
    if (i == 0) { tc::mb_init(done, ni); *abort_flag = 0; }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __shared__ float sbias[BN];
  for (int c = threadIdx.x; c < BN; c += blockDim.x)
    sbias[c] = (a.bias && co0 + c < a.cout) ? a.bias[co0 + c] : 0.f;
  if (warp == kRowsIssue0) tc::tmem_alloc(tmem_slot, rc.tmem_cols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  // tile j of this CTA: image, first pixel, first row, rows inside the image
  auto tile_origin = [&](int j, int* img, int* x0, int* y0) -> int {
    uint32_t t = blockIdx.x + (uint32_t)j * gridDim.x;         // (tiles < 2^31)
    const uint32_t u = t / (uint32_t)a.tiles_x;
    *x0 = (int)(t - u * (uint32_t)a.tiles_x) * 128;
    *img = (int)(u / (uint32_t)tiles_r);
    *y0 = (int)(u - (uint32_t)*img * (uint32_t)tiles_r) * rc.rows;
    return min(rc.rows, a.h - *y0);
  };
  // a ring position: slot and the parity of its current use
  struct Ring {
    int s, n;
    uint32_t ph;
    __device__ __forceinline__ void next() { if (++s == n) { s = 0; ph ^= 1u; } }
  };

  // waits with the whole warp (converged control flow: a ring's addresses and the
  // descriptors stay in uniform registers)
  auto wait_warp = [&](uint64_t* bar, uint32_t ph) -> bool {
    return __all_sync(0xffffffffu, tc::mb_try(bar, ph)) || __all_sync(0xffffffffu, wait_live(bar, ph, abort_flag));
  };

  if (warp <= kRowsLoaders) {
    const bool el = tc::elect_one();
    Ring ra{0, own, 0}, rb{0, rc.nb, 0};
    auto load_b = [&](int dyi, int cc) -> bool {
      if (!wait_warp(&emptyB[rb.s], rb.ph ^ 1u)) return false;
      if (el) {
        unsigned char* st = sB + (size_t)rb.s * kB;
        usesB[rb.s] += 1;
        tc::mb_expect_tx(&fullB[rb.s], (uint32_t)kB);
        // the three taps of input row dy = dyi - 1 (mirrored for the input gradient)
        tc::tma_load_3d(st, &mW, cc * 32, co0, 3 * (1 + a.sign * (dyi - 1)), &fullB[rb.s]);
      }
      return true;
    };
    auto load_a = [&](int slot, int cc, int x0, int y, int img) -> bool {
      if (!wait_warp(&emptyA[slot], ra.ph ^ 1u)) return false;
      if (el) {
        usesA[slot] += 1;
        tc::mb_expect_tx(&fullA[slot], (uint32_t)kRowsA);
        tc::tma_load_4d(base + (size_t)slot * kRowsAStride, &mX, cc * 32, x0 - 1, y, img, &fullA[slot]);
      }
      return true;
    };
    bool ok = true;
    for (int j = 0; j < ntl && ok; ++j) {
      int img, x0, y0;
      const int nr = tile_origin(j, &img, &x0, &y0);
      for (int dyi = 0; dyi < 3 && ok; ++dyi)
        for (int cc = 0; cc < cchunks && ok; ++cc) {
          if (warp == kRowsLoaders) {
            ok = load_b(dyi, cc);
            rb.next();
          } else if (warp < ni) {
            for (int r = warp; r < nr && ok; r += ni) {
              ok = load_a(warp * own + ra.s, cc, x0, y0 + r + dyi - 1, img);
              ra.next();
            }
          }
        }
    }
    if (!ok && lane == 0) atomicExch(abort_flag, 1);
  } else if (warp < kRowsIssue0 + ni) {
    constexpr uint32_t idesc = tc::idesc_bf16(128, BN, 0, 0);
    const int w = warp - kRowsIssue0;
    const bool el = tc::elect_one();
    Ring ra{0, own, 0}, rb{0, rc.nb, 0};
    bool ok = true;
    if (a.stall_flag) ok = __all_sync(0xffffffffu, stall_on_unset_flag(a.stall_flag, a.stall_cycles));
    // the three dx taps of one box into one output row's accumulator; the swizzle
    // follows the absolute shared-memory address, which the TMA write and the MMA
    // read share, so a tap's start address simply moves by whole pixels
    auto taps = [&](uint32_t acc, uint32_t sa, uint32_t sb, bool first) {
      const uint64_t da = tc::desc_sw64(sa, 16, 512), db = tc::desc_sw64(sb, 16, 512);
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int kk = 0; kk < 2; ++kk)                          // 16 BF16 = 32 bytes along K
          if (el)
            tc::umma_bf16(acc, da + (uint64_t)((j * 64 + kk * 32) >> 4),
                          db + (uint64_t)(((a.sign > 0 ? j : 2 - j) * kTap + kk * 32) >> 4), idesc,
                          (j | kk) ? 1u : first ? 0u : 1u);
    };
    auto commit = [&](uint64_t* bar) {
      if (el) tc::umma_commit(bar);
    };
    auto wait_full = [&](uint64_t* bar, uint32_t ph) -> bool {
      if (!wait_warp(bar, ph)) return false;
      tc::fence_after();
      return true;
    };
    const uint32_t sA = tc::su32(base), sBb = tc::su32(sB);
    for (int j = 0; j < ntl && ok; ++j) {
      const int b = rc.nbuf == 2 ? j & 1 : 0;
      const int use = rc.nbuf == 2 ? j >> 1 : j;
      if (!(ok = wait_full(&tempty[b], (uint32_t)((use & 1) ^ 1)))) break;
      const uint32_t acc = tmem + (uint32_t)(b * rc.rows * BN);
      int img, x0, y0;
      const int nr = tile_origin(j, &img, &x0, &y0);
      for (int dyi = 0; dyi < 3 && ok; ++dyi)
        for (int cc = 0; cc < cchunks && ok; ++cc) {
          if (!(ok = wait_full(&fullB[rb.s], rb.ph))) break;
          for (int r = w; r < nr; r += ni) {
            const int slot = w * own + ra.s;
            if (!(ok = wait_full(&fullA[slot], ra.ph))) break;
            taps(acc + (uint32_t)(r * BN), sA + (uint32_t)slot * kRowsAStride, sBb + (uint32_t)rb.s * kB,
                 dyi == 0 && cc == 0);
            commit(&emptyA[slot]);
            ra.next();
          }
          commit(&emptyB[rb.s]);
          rb.next();
        }
      if (ok) commit(&tfull[b]);
    }
    if (!ok && lane == 0) atomicExch(abort_flag, 1);
    commit(done);                                        // arrives when every MMA issued above has completed
  } else if (warp >= kRowsEpi0) {
    // epilogue: TMEM lane quarter (warp % 4) = pixels 32 (warp % 4) .. + 31 of each
    // row; two warps per quarter share the rows' 32-channel blocks.  A block goes by
    // way of shared memory (64 bytes a pixel, chunks swizzled), so that four lanes
    // store a pixel's 64 bytes and read its mask; the mask's loads run a block ahead.
    const int q = warp & 3, half = (warp - kRowsEpi0) >> 2;
    unsigned char* stage = sE + (warp - kRowsEpi0) * 2048;
    const int pc = lane & 3, pr = lane >> 2;
    for (int j = 0; j < ntl; ++j) {
      const int b = rc.nbuf == 2 ? j & 1 : 0;
      const int use = rc.nbuf == 2 ? j >> 1 : j;
      int img, x0, y0;
      const int nr = tile_origin(j, &img, &x0, &y0);
      const int nblk = nr * (BN / 32), xq = x0 + 32 * q + pr;
      const size_t row0 = ((size_t)img * a.h + y0) * a.w;
      auto load_mask = [&](int k, uint4* mv) {
        if (!a.mask || k >= nblk) return;
        const __nv_bfloat16* mp = a.mask + (row0 + (size_t)(k / (BN / 32)) * a.w + xq) * a.mask_cs + co0 +
                                  k % (BN / 32) * 32 + 8 * pc;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (xq + 8 * i < a.w) mv[i] = __ldg(reinterpret_cast<const uint4*>(mp + (size_t)(8 * i) * a.mask_cs));
      };
      if (a.mask && j + 1 < ntl) {                       // the next tile's mask into L2
        int img1, x1, y1;
        const int nblk1 = tile_origin(j + 1, &img1, &x1, &y1) * (BN / 32);
        const int xp = x1 + 32 * q + pr;
        const __nv_bfloat16* mp = a.mask + (((size_t)img1 * a.h + y1) * a.w + xp) * a.mask_cs + co0 + 8 * pc;
        for (int k = half; k < nblk1; k += 2)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (!(pc & 1) && xp + 8 * i < a.w)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(
                  mp + ((size_t)(k / (BN / 32)) * a.w + 8 * i) * a.mask_cs + k % (BN / 32) * 32));
      }
      uint4 mv[4], mn[4];
      load_mask(half, mv);
      bool ok = true;
      if (lane == 0) ok = wait_live(&tfull[b], (uint32_t)(use & 1), abort_flag);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      tc::fence_after();
#pragma unroll 1
      for (int k = half; k < nblk; k += 2) {
        const int r = k / (BN / 32), c = k % (BN / 32);
        load_mask(k + 2, mn);
        uint32_t v[32];
        tc::tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((b * rc.rows + r) * BN + c * 32), v);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 o;
          __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int n = g * 8 + 2 * e;
            float f0 = __uint_as_float(v[n]) + sbias[c * 32 + n], f1 = __uint_as_float(v[n + 1]) + sbias[c * 32 + n + 1];
            if (a.relu) { f0 = fmaxf(f0, 0.f); f1 = fmaxf(f1, 0.f); }
            ob[e] = __floats2bfloat162_rn(f0, f1);
          }
          *reinterpret_cast<uint4*>(stage + lane * 64 + ((g ^ ((lane >> 1) & 3)) << 4)) = o;
        }
        __syncwarp();
        __nv_bfloat16* op = a.out + (row0 + (size_t)r * a.w + xq) * a.out_cs + co0 + c * 32 + 8 * pc;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int p = 8 * i + pr;
          uint4 o = *reinterpret_cast<const uint4*>(stage + p * 64 + ((pc ^ ((p >> 1) & 3)) << 4));
          if (a.mask) {
            const __nv_bfloat162 z = __float2bfloat162_rn(0.f);
            const __nv_bfloat162* m2 = reinterpret_cast<const __nv_bfloat162*>(&mv[i]);
            uint32_t* o2 = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e) o2[e] &= __hgt2_mask(m2[e], z);
            mv[i] = mn[i];
          }
          if (xq + 8 * i < a.w) *reinterpret_cast<uint4*>(op + (size_t)(8 * i) * a.out_cs) = o;
        }
        __syncwarp();
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::su32(&tempty[b])) : "memory");
    }
  }
  __syncwarp();
  // every MMA issued has completed before TMEM is freed; copies issued but
  // not consumed land before the CTA exits
  if (threadIdx.x == 0) tc::mb_wait(done, 0, kWaitCycles);
  __syncthreads();
  if (threadIdx.x == 0 && *((volatile int*)abort_flag)) {
    atomicOr(a.err, 2);
    // (each slot's last use; the earlier ones were consumed)
    for (int i = 0; i < rc.na; ++i)
      if (usesA[i]) tc::mb_wait(&fullA[i], (uint32_t)((usesA[i] - 1) & 1), kWaitCycles);
    for (int i = 0; i < rc.nb; ++i)
      if (usesB[i]) tc::mb_wait(&fullB[i], (uint32_t)((usesB[i] - 1) & 1), kWaitCycles);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == kRowsIssue0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, rc.tmem_cols);
  }
}

template <int BN> struct WgCfg {
  static constexpr int kKp = 64;                       // pixels per K step
  static constexpr int kBox = kKp * 64;                // one 32-channel group of kKp pixels
  static constexpr int kA = 4 * kBox;                  // four (tap, 32-channel) groups
  static constexpr int kB = (BN / 32) * kBox;
  static constexpr int kStage = kA + kB;
  static constexpr int kStages = BN >= 256 ? 4 : 5;
  static constexpr int kTmem = BN < 32 ? 32 : BN;
  static constexpr int kSmem = kStages * kStage + 1024 + 256;
};

template <int BN>
__global__ void __launch_bounds__(kConvThreads) conv_wgrad_tc(const __grid_constant__ CUtensorMap mX,
                                                              const __grid_constant__ CUtensorMap mD, WgArgs a) {
  typedef WgCfg<BN> Cfg;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = tc::su32(smem_raw);
  unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + Cfg::kStages * Cfg::kStage);
  uint64_t* empty = full + Cfg::kStages;
  uint64_t* done = empty + Cfg::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* issued = abort_flag + 1;
  int* consumed = abort_flag + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int cchunks = a.cin >> 5;
  const int groups = a.taps * cchunks;
  const int g0 = blockIdx.x * 4;
  const long long kb_total = (long long)a.n * a.tiles_y * a.tiles_x;
  const int kb0 = (int)(kb_total * blockIdx.y / gridDim.y);
  const int kb1 = (int)(kb_total * (blockIdx.y + 1) / gridDim.y);
  const int nk = kb1 - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) { tc::mb_init(&full[s], 1); tc::mb_init(&empty[s], 1); }
    tc::mb_init(done, 1);
    *abort_flag = 0; *issued = 0; *consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, Cfg::kTmem);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  if (threadIdx.x == 0) {
    int it = 0;
    for (; it < nk; ++it) {
      const int s = it % Cfg::kStages;
      const uint32_t ph = (uint32_t)((it / Cfg::kStages) & 1);
      if (!wait_live(&empty[s], ph ^ 1u, abort_flag) || *((volatile int*)abort_flag)) {
        atomicExch(abort_flag, 1);
        break;
      }
      int kb = kb0 + it;
      const int tx = kb % a.tiles_x; kb /= a.tiles_x;
      const int ty = kb % a.tiles_y;
      const int img = kb / a.tiles_y;
      const int x0 = tx * a.bx, y0 = ty * a.by;
      unsigned char* st = base + s * Cfg::kStage;
      tc::mb_expect_tx(&full[s], (uint32_t)Cfg::kStage);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int gg = min(g0 + g, groups - 1);     // rows past the last group: loaded, never stored
        const int tap = gg / cchunks, cc = gg - tap * cchunks;
        int dx = 0, dy = 0;
        if (a.taps == 9) { dx = tap % 3 - 1; dy = tap / 3 - 1; }
        tc::tma_load_4d(st + g * Cfg::kBox, &mX, cc * 32, x0 + dx, y0 + dy, img, &full[s]);
      }
#pragma unroll
      for (int j = 0; j < BN / 32; ++j)
        tc::tma_load_4d(st + Cfg::kA + j * Cfg::kBox, &mD, j * 32, x0, y0, img, &full[s]);
    }
    *issued = it;
  } else if (threadIdx.x == 32) {
    constexpr uint32_t idesc = tc::idesc_bf16(128, BN, 1, 1);
    int it = 0;
    bool stalled = false;
    if (a.stall_flag && !stall_on_unset_flag(a.stall_flag, a.stall_cycles)) {
      atomicExch(abort_flag, 1);
      stalled = true;
    }
    for (; it < nk && !stalled; ++it) {
      const int s = it % Cfg::kStages;
      const uint32_t ph = (uint32_t)((it / Cfg::kStages) & 1);
      if (!wait_live(&full[s], ph, abort_flag) || *((volatile int*)abort_flag)) {
        atomicExch(abort_flag, 1);
        break;
      }
      tc::fence_after();
      const uint32_t sa = tc::su32(base + s * Cfg::kStage);
#pragma unroll
      for (int kk = 0; kk < Cfg::kKp / 16; ++kk) {
        // 16 pixels = two 8-line K groups, 1024 bytes
        const uint64_t da = tc::desc_sw64(sa + kk * 1024, Cfg::kBox, 512);
        const uint64_t db = tc::desc_sw64(sa + Cfg::kA + kk * 1024, Cfg::kBox, 512);
        tc::umma_bf16(tmem, da, db, idesc, (it | kk) ? 1u : 0u);
      }
      tc::umma_commit(&empty[s]);
    }
    *consumed = it;
    tc::umma_commit(done);
  }
  __syncwarp();
  const bool ok_done = tc::mb_wait(done, 0, kWaitCycles);
  tc::fence_after();
  const bool good = __syncthreads_and(ok_done && !*((volatile int*)abort_flag));
  if (good && nk > 0) {
    const int m = warp * 32 + lane;
    const int row = g0 * 32 + m;                      // (tap, ci) row of dW^T
    const bool live = row < groups * 32;
#pragma unroll 1
    for (int c = 0; c < BN / 32; ++c) {
      uint32_t r[32];
      tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 32), r);
      if (!live) continue;
      float* dst = a.dwt + (size_t)row * a.cout + c * 32;
#pragma unroll
      for (int q = 0; q < 32; q += 4)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + q), "f"(__uint_as_float(r[q])),
                     "f"(__uint_as_float(r[q + 1])), "f"(__uint_as_float(r[q + 2])), "f"(__uint_as_float(r[q + 3]))
                     : "memory");
    }
  } else if (!good && threadIdx.x == 0) {
    atomicOr(a.err, 2);
  }
  if (threadIdx.x == 0) {
    for (int it = *consumed; it < *issued; ++it)
      tc::mb_wait(&full[it % Cfg::kStages], (uint32_t)((it / Cfg::kStages) & 1), kWaitCycles);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, Cfg::kTmem);
  }
}

// Weight gradient over whole 64-pixel rows (3x3, w >= 64): one CTA per
// (32-channel input chunk cc, group of dy rows) and K range.  Per K step
// (64 pixels of one row) it loads, for each of its dy, one 72-pixel row box
// of X starting at x - 1, and the dZ tile once.  The A operand of dy reads
// that box with a leading-dimension offset of one pixel row (64 bytes):
// M group g (rows 32 g .. 32 g + 31) is the box shifted by g pixels, i.e.
// the taps dx = g - 1 for g < 3 (group 3 is computed and dropped).  One
// accumulator per dy shares the dZ tile.
//
// What bounds it: an MMA takes 48 clocks at 64 channels, one warp that waits and
// issues about 120, so a warp issues for each dy (1-3); warps 0 and 4 load the X
// boxes and the dZ tile.
constexpr int kWgHThreads = 160;

template <int BN> struct WgHCfg {
  static constexpr int kABox = 72 * 64;
  static constexpr int kAStride = (kABox + 1023) / 1024 * 1024;
  static constexpr int kTmemBuf = pow2_at_least(BN);
  static constexpr int kNdy = (512 / kTmemBuf) >= 3 ? 3 : 2;   // dy rows per CTA (accumulators)
  static constexpr int kTmem = pow2_at_least(kNdy * kTmemBuf) > 512 ? 512 : pow2_at_least(kNdy * kTmemBuf);
  static constexpr int kBBox = 64 * 64;                // 64 pixels x 32 channels of dZ
  static constexpr int kA = kNdy * kAStride;
  static constexpr int kB = (BN / 32) * kBBox;
  static constexpr int kStage = kA + kB;
  static constexpr int kStagesRaw = 200 * 1024 / kStage;
  static constexpr int kStages = kStagesRaw > 6 ? 6 : kStagesRaw;
  static constexpr int kSmem = kStages * kStage + 1024 + 256;
};

template <int BN>
__global__ void __launch_bounds__(kWgHThreads) conv_wgrad_halo(const __grid_constant__ CUtensorMap mX,
                                                                const __grid_constant__ CUtensorMap mD, WgArgs a) {
  typedef WgHCfg<BN> Cfg;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = tc::su32(smem_raw);
  unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + Cfg::kStages * Cfg::kStage);
  uint64_t* empty = full + Cfg::kStages;
  uint64_t* done = empty + Cfg::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* uses = abort_flag + 1;                           // [2][kStages] loads issued per stage: X, dZ
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int cchunks = a.cin >> 5;
  const int cc = blockIdx.x % cchunks;
  const int dy0 = (blockIdx.x / cchunks) * Cfg::kNdy;           // first dy index (0..2) of this CTA
  const int ndy = min(Cfg::kNdy, 3 - dy0);
  const long long kb_total = (long long)a.n * a.tiles_y * a.tiles_x;
  const int kb0 = (int)(kb_total * blockIdx.y / gridDim.y);
  const int kb1 = (int)(kb_total * (blockIdx.y + 1) / gridDim.y);
  const int nk = kb1 - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      tc::mb_init(&full[s], 2); tc::mb_init(&empty[s], ndy);
      uses[s] = uses[Cfg::kStages + s] = 0;
    }
    tc::mb_init(done, ndy);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, Cfg::kTmem);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  auto wait_warp = [&](uint64_t* bar, uint32_t ph) -> bool {
    return __all_sync(0xffffffffu, tc::mb_try(bar, ph)) || __all_sync(0xffffffffu, wait_live(bar, ph, abort_flag));
  };
  const bool el = tc::elect_one();
  bool ok = true;
  int s = 0;
  uint32_t ph = 0;
  if (warp == 0 || warp == 4) {
    int kb = kb0;
    int tx = kb % a.tiles_x; kb /= a.tiles_x;
    int ty = kb % a.tiles_y, img = kb / a.tiles_y;
    for (int it = 0; it < nk; ++it) {
      if (!(ok = wait_warp(&empty[s], ph ^ 1u))) break;
      unsigned char* st = base + s * Cfg::kStage;
      if (el) {
        uses[(warp >> 2) * Cfg::kStages + s] += 1;
        if (warp == 0) {
          tc::mb_expect_tx(&full[s], (uint32_t)(ndy * Cfg::kABox));
          for (int d = 0; d < ndy; ++d)
            tc::tma_load_4d(st + d * Cfg::kAStride, &mX, cc * 32, tx * 64 - 1, ty + (dy0 + d - 1), img, &full[s]);
        } else {
          tc::mb_expect_tx(&full[s], (uint32_t)Cfg::kB);
#pragma unroll
          for (int j = 0; j < BN / 32; ++j)
            tc::tma_load_4d(st + Cfg::kA + j * Cfg::kBBox, &mD, j * 32, tx * 64, ty, img, &full[s]);
        }
      }
      if (++tx == a.tiles_x) { tx = 0; if (++ty == a.tiles_y) { ty = 0; ++img; } }
      if (++s == Cfg::kStages) { s = 0; ph ^= 1u; }
    }
  } else if (warp <= ndy) {
    constexpr uint32_t idesc = tc::idesc_bf16(128, BN, 1, 1);
    const int d = warp - 1;
    if (a.stall_flag) ok = __all_sync(0xffffffffu, stall_on_unset_flag(a.stall_flag, a.stall_cycles));
    const uint32_t sbase = tc::su32(base);
    for (int it = 0; it < nk && ok; ++it) {
      if (!(ok = wait_warp(&full[s], ph))) break;
      tc::fence_after();
      const uint32_t sa = sbase + (uint32_t)(s * Cfg::kStage);
      // 16 pixels = two 8-row K groups, 1024 bytes; M groups one pixel row apart
      const uint64_t da = tc::desc_sw64(sa + d * Cfg::kAStride, 64, 512);
      const uint64_t db = tc::desc_sw64(sa + Cfg::kA, Cfg::kBBox, 512);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        if (el)
          tc::umma_bf16(tmem + (uint32_t)(d * Cfg::kTmemBuf), da + (uint64_t)(kk * 64), db + (uint64_t)(kk * 64), idesc,
                        (it | kk) ? 1u : 0u);
      if (el) tc::umma_commit(&empty[s]);
      if (++s == Cfg::kStages) { s = 0; ph ^= 1u; }
    }
    if (el) tc::umma_commit(done);
  }
  if (!ok && lane == 0) atomicExch(abort_flag, 1);
  __syncwarp();
  const bool ok_done = tc::mb_wait(done, 0, kWaitCycles);
  tc::fence_after();
  const bool good = __syncthreads_and(ok_done && !*((volatile int*)abort_flag));
  if (good && nk > 0 && warp < 3) {
    // warp g = tap dx = g - 1 of each dy: dW^T row (3 dy + g) cin + cc 32 + lane
    for (int d = 0; d < ndy; ++d) {
      const int tap = 3 * (dy0 + d) + warp;
      const int row = tap * a.cin + cc * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(d * Cfg::kTmemBuf + c * 32), r);
        float* dst = a.dwt + (size_t)row * a.cout + c * 32;
#pragma unroll
        for (int q = 0; q < 32; q += 4)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + q), "f"(__uint_as_float(r[q])),
                       "f"(__uint_as_float(r[q + 1])), "f"(__uint_as_float(r[q + 2])), "f"(__uint_as_float(r[q + 3]))
                       : "memory");
      }
    }
  } else if (!good && threadIdx.x == 0) {
    atomicOr(a.err, 2);
  }
  if (threadIdx.x == 0) {
    if (*((volatile int*)abort_flag)) land_pairs(full, uses, Cfg::kStages);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, Cfg::kTmem);
  }
}

template <int BN>
oh_status launch_wgrad_halo(const CUtensorMap& mX, const CUtensorMap& mD, const WgArgs& a, long long kb_total,
                            cudaStream_t st) {
  typedef WgHCfg<BN> Cfg;
  OH_CUDA_TRY(cudaFuncSetAttribute(conv_wgrad_halo<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
  const int gx = (a.cin / 32) * ((3 + Cfg::kNdy - 1) / Cfg::kNdy);
  long long splits = std::max(1LL, (4LL * sm_count() + gx - 1) / gx);
  splits = std::min(splits, std::max(1LL, kb_total / 16));
  splits = std::min(splits, 65535LL);
  conv_wgrad_halo<BN><<<dim3(gx, (int)splits), kWgHThreads, Cfg::kSmem, st>>>(mX, mD, a);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

// Patch of `pixels` pixels for an image row of width w: bx = min(w, pixels),
// by = pixels / bx; widths below `pixels` must divide it.
bool patch_shape(int w, int pixels, int* bx, int* by) {
  if (w >= pixels) { *bx = pixels; *by = 1; return true; }
  if (pixels % w) return false;
  *bx = w; *by = pixels / w;
  return true;
}

template <int BN>
oh_status launch_fwd(const CUtensorMap& mX, const CUtensorMap& mW, const ConvArgs& a, long long tiles, cudaStream_t st) {
  typedef FwdCfg<BN> Cfg;
  OH_CUDA_TRY(cudaFuncSetAttribute(conv_fwd_tc<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
  // persistent grid: the CTAs that fit on an SM by shared memory and tensor
  // memory (512 columns), at most four, times the SMs, spread over the
  // output-channel tiles
  const int by_smem = (int)((228 * 1024) / (Cfg::kSmem + 1024));
  const int per_sm = std::max(1, std::min(4, std::min(by_smem, 512 / Cfg::kTmem)));
  const int ctiles = (a.cout + BN - 1) / BN;
  const long long want = std::max(1LL, (long long)sm_count() * per_sm / ctiles);
  const int gx = (int)std::min(tiles, want);
  conv_fwd_tc<BN><<<dim3(gx, ctiles), Cfg::kThreads, Cfg::kSmem, st>>>(mX, mW, a);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

// The row kernel's channel tile and rows per tile for a layer: the least estimated
// clocks of a CTA, from the MMAs' clocks (see conv_fwd_rows; 120 from one issuer), 40
// bytes a clock of loads, 2000 clocks of latency over the steps in flight, and 1000
// clocks per warp and block of the epilogue.
// Measured, 4 x 512 x 512 pixels, 192 -> 64 channels: 188 us with tiles of 4 rows and
// two accumulator sets, 211 with 8 rows and one, 288 with 2 rows; 64 -> 192: 242 us
// with channel tiles of 96 and 2 rows, 257 with 64 and 4, 284 with 192 and 2.
struct RowsPlan {
  RowsCfg c;
  int bn, smem;
};
RowsPlan rows_plan(const ConvArgs& a, int sms) {
  RowsPlan best{};
  float best_t = 0.f;
  const float cchunks = (float)(a.cin / 32);
  const int budget = kRowsSmem - kRowsFixed;
  for (int bn : {32, 64, 96, 128, 192, 256}) {
    if (a.cout % bn) continue;
    const int step = 3 * bn * 64;                        // weights of one (dy, 32 channels)
    const int gx = std::max(1, sms / (a.cout / bn));
    for (int rows = 1; rows <= 16 && rows * bn <= 512; rows *= 2) {
      const int ni = std::min(rows, kRowsIssuers), nbuf = 2 * rows * bn <= 512 ? 2 : 1;
      // as many steps in flight of both kinds as fit
      const int nb = std::min(kRowsB_Slots, std::max(3, budget / (rows * kRowsAStride + step)));
      const int na = std::min(kRowsA_Slots, (budget - nb * step) / kRowsAStride) / ni * ni;
      if (na < std::max(ni, 4)) continue;
      const uint32_t tiles = (uint32_t)a.n * a.tiles_x * ((uint32_t)(a.h + rows - 1) / rows);       // (< 2^31)
      const float waves = (float)((tiles + gx - 1) / gx);
      const float mma = std::max({bn / 2.f, 32.f + bn / 4.f, 120.f / ni});
      const float epi = (rows * (bn / 32) + 1) / 2 * 1000.f;
      const float calc = 3.f * cchunks * std::max({rows * 6.f * mma, (rows * kRowsA + step) / 40.f, 2000.f / nb,
                                                   2000.f * rows / na});
      const float t = waves * ((nbuf == 2 ? std::max(calc, epi) : calc + epi) + 300.f) + (nbuf == 2 ? epi : 0.f);
      if (best.bn == 0 || t < best_t) {
        best_t = t;
        best.bn = bn;
        best.smem = na * kRowsAStride + nb * step + kRowsFixed;
        best.c = RowsCfg{rows, nbuf, na, nb, (uint32_t)pow2_at_least(nbuf * rows * bn)};
      }
    }
  }
  return best;
}

template <int BN>
oh_status launch_rows(const CUtensorMap& mX, const CUtensorMap& mW, const ConvArgs& a, const RowsPlan& p,
                      int sms, cudaStream_t st) {
  // (the same limit whatever the plan: another thread may set it between here and the launch)
  OH_CUDA_TRY(cudaFuncSetAttribute(conv_fwd_rows<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem));
  const int ctiles = a.cout / BN;
  const long long tiles = (long long)a.n * ((a.h + p.c.rows - 1) / p.c.rows) * a.tiles_x;
  const int gx = (int)std::min(tiles, (long long)std::max(1, sms / ctiles));
  conv_fwd_rows<BN><<<dim3(gx, ctiles), kRowsThreads, p.smem, st>>>(mX, mW, a, p.c);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

template <int BN>
oh_status launch_wgrad(const CUtensorMap& mX, const CUtensorMap& mD, const WgArgs& a, int mtiles, int splits,
                       cudaStream_t st) {
  typedef WgCfg<BN> Cfg;
  OH_CUDA_TRY(cudaFuncSetAttribute(conv_wgrad_tc<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
  conv_wgrad_tc<BN><<<dim3(mtiles, splits), kConvThreads, Cfg::kSmem, st>>>(mX, mD, a);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

}  // namespace

oh_status tc_arch_check() {
  int dev = 0, major = 0, minor = 0;
  OH_CUDA_TRY(cudaGetDevice(&dev));
  OH_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  OH_CUDA_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev));
  if (major != 10 || minor != 3) return fail(OH_ERR_UNSUPPORTED_SIZE, "the tensor-core convolutions are built for sm_103a");
  return OH_OK;
}

oh_status conv_enqueue(oh_ctx* ctx, const ConvDesc& d, cudaStream_t st, const char* timer_name) {
  if (d.cin % 32 || d.cin <= 0 || d.cout <= 0 || d.cout % 32 || d.cout > 1024 || (d.taps != 9 && d.taps != 1))
    return fail(OH_ERR_INVALID_ARG, "convolution: cin and cout must be positive multiples of 32 (cout <= 1024), taps 1 or 9");
  if (d.x_cs % 8 || d.out_cs % 8 || (d.mask && (d.mask_cs % 8 || d.mask_cs < d.cout)) || d.x_cs < d.cin ||
      d.out_cs < d.cout)
    return fail(OH_ERR_INVALID_ARG, "convolution: channel strides must be multiples of 8 and cover the channels");
  if (!d.x || !d.w_mat || !d.out) return fail(OH_ERR_INVALID_ARG, "convolution: null tensor");
  if ((reinterpret_cast<uintptr_t>(d.x) | reinterpret_cast<uintptr_t>(d.w_mat) | reinterpret_cast<uintptr_t>(d.out) |
       reinterpret_cast<uintptr_t>(d.mask)) & 15)
    return fail(OH_ERR_INVALID_ARG, "convolution: tensors must be 16-byte aligned");
  OH_TRY(tc_arch_check());
  ConvArgs a{};
  if (!patch_shape(d.w, 128, &a.bx, &a.by)) return fail(OH_ERR_UNSUPPORTED_SIZE, "convolution: widths below 128 must divide 128");
  a.taps = d.taps; a.cin = d.cin; a.cout = d.cout; a.w = d.w; a.h = d.h; a.n = d.n;
  a.tiles_x = (d.w + a.bx - 1) / a.bx; a.tiles_y = (d.h + a.by - 1) / a.by;
  a.sign = d.sign;
  a.bias = d.bias; a.relu = d.relu;
  a.mask = reinterpret_cast<const __nv_bfloat16*>(d.mask); a.mask_cs = d.mask_cs;
  a.out = reinterpret_cast<__nv_bfloat16*>(d.out); a.out_cs = d.out_cs;
  a.err = ctx->dev_err;
  if (ctx->stall_mask & kStallConvolution) { a.stall_flag = ctx->dev_err + 1; a.stall_cycles = ctx->stall_cycles; }
  const long long tiles = (long long)a.tiles_x * a.tiles_y * d.n;
  if (tiles > 0x7fffffffLL) return fail(OH_ERR_UNSUPPORTED_SIZE, "convolution: too many pixel tiles");
  CUtensorMap mX, mW;
  // 3x3 over whole 128-pixel rows
  const char* hv = std::getenv("OH_CONV_HALO");
  if (d.taps == 9 && a.by == 1 && a.bx == 128 && !(hv && std::atoi(hv) == 0)) {
    const int sms = sm_count();
    const RowsPlan p = rows_plan(a, sms);
    OH_TRY(tc::map_act4d(&mX, d.x, d.cin, d.x_cs, d.w, d.h, d.n, 136, 1));
    OH_TRY(tc::map_taps3d(&mW, d.w_mat, d.cin, d.cout, d.taps, p.bn, 3));
    KernelTimer kt(ctx, timer_name, st);
    switch (p.bn) {
      case 32: return launch_rows<32>(mX, mW, a, p, sms, st);
      case 64: return launch_rows<64>(mX, mW, a, p, sms, st);
      case 96: return launch_rows<96>(mX, mW, a, p, sms, st);
      case 128: return launch_rows<128>(mX, mW, a, p, sms, st);
      case 192: return launch_rows<192>(mX, mW, a, p, sms, st);
      default: return launch_rows<256>(mX, mW, a, p, sms, st);
    }
  }
  // output-channel tile: all of cout up to 256 (384 as two halves), else the
  // largest of 256, 192, 128, 96, 64, 32 that divides it; halved while the
  // pixel tiles alone cannot fill two CTAs per SM
  int bn = 32;
  for (int c : {256, 192, 128, 96, 64})
    if (d.cout % c == 0) { bn = c; break; }
  while ((bn == 256 || bn == 128 || bn == 64 || bn == 192) && tiles * ((d.cout + bn - 1) / bn) < 2LL * sm_count())
    bn /= 2;
  OH_TRY(tc::map_act4d(&mX, d.x, d.cin, d.x_cs, d.w, d.h, d.n, a.bx, a.by));
  OH_TRY(tc::map_mat2d(&mW, d.w_mat, d.taps * d.cin, d.cout, bn));
  KernelTimer kt(ctx, timer_name, st);
  switch (bn) {
    case 32: return launch_fwd<32>(mX, mW, a, tiles, st);
    case 64: return launch_fwd<64>(mX, mW, a, tiles, st);
    case 96: return launch_fwd<96>(mX, mW, a, tiles, st);
    case 128: return launch_fwd<128>(mX, mW, a, tiles, st);
    case 192: return launch_fwd<192>(mX, mW, a, tiles, st);
    default: return launch_fwd<256>(mX, mW, a, tiles, st);
  }
}

oh_status wgrad_enqueue(oh_ctx* ctx, const WgradDesc& d, cudaStream_t st, const char* timer_name) {
  if (d.cin % 32 || d.cin <= 0 || (d.cout != 32 && d.cout != 64 && d.cout != 128 && d.cout != 256) ||
      (d.taps != 9 && d.taps != 1))
    return fail(OH_ERR_INVALID_ARG, "weight gradient: cin a positive multiple of 32, cout 32, 64, 128 or 256, taps 1 or 9");
  if (d.x_cs % 8 || d.dz_cs % 8 || d.x_cs < d.cin || d.dz_cs < d.cout)
    return fail(OH_ERR_INVALID_ARG, "weight gradient: channel strides must be multiples of 8 and cover the channels");
  if (!d.x || !d.dz || !d.dwt) return fail(OH_ERR_INVALID_ARG, "weight gradient: null tensor");
  if ((reinterpret_cast<uintptr_t>(d.x) | reinterpret_cast<uintptr_t>(d.dz) | reinterpret_cast<uintptr_t>(d.dwt)) & 15)
    return fail(OH_ERR_INVALID_ARG, "weight gradient: tensors must be 16-byte aligned");
  OH_TRY(tc_arch_check());
  WgArgs a{};
  if (!patch_shape(d.w, 64, &a.bx, &a.by)) return fail(OH_ERR_UNSUPPORTED_SIZE, "weight gradient: widths below 64 must divide 64");
  a.taps = d.taps; a.cin = d.cin; a.cout = d.cout; a.w = d.w; a.h = d.h; a.n = d.n;
  a.tiles_x = (d.w + a.bx - 1) / a.bx; a.tiles_y = (d.h + a.by - 1) / a.by;
  a.dwt = d.dwt;
  a.err = ctx->dev_err;
  if (ctx->stall_mask & kStallConvolution) { a.stall_flag = ctx->dev_err + 1; a.stall_cycles = ctx->stall_cycles; }
  const int groups = d.taps * (d.cin / 32);
  const int mtiles = (groups + 3) / 4;
  const long long kb_total = (long long)a.tiles_x * a.tiles_y * d.n;
  // 3x3 over whole 64-pixel rows: one row box per (dy, 32 channels) feeds the three dx taps
  const char* hv = std::getenv("OH_CONV_HALO");
  if (d.taps == 9 && a.by == 1 && a.bx == 64 && d.cout <= 128 && !(hv && std::atoi(hv) == 0)) {
    CUtensorMap mX, mD;
    OH_TRY(tc::map_act4d(&mX, d.x, d.cin, d.x_cs, d.w, d.h, d.n, 72, 1));
    OH_TRY(tc::map_act4d(&mD, d.dz, d.cout, d.dz_cs, d.w, d.h, d.n, 64, 1));
    KernelTimer kt(ctx, timer_name, st);
    switch (d.cout) {
      case 32: return launch_wgrad_halo<32>(mX, mD, a, kb_total, st);
      case 64: return launch_wgrad_halo<64>(mX, mD, a, kb_total, st);
      default: return launch_wgrad_halo<128>(mX, mD, a, kb_total, st);
    }
  }
  // K splits: about four CTAs per SM over all M tiles, each with at least 16 K steps
  long long splits = std::max(1LL, (4LL * sm_count() + mtiles - 1) / mtiles);
  splits = std::min(splits, std::max(1LL, kb_total / 16));
  splits = std::min(splits, 65535LL);
  CUtensorMap mX, mD;
  OH_TRY(tc::map_act4d(&mX, d.x, d.cin, d.x_cs, d.w, d.h, d.n, a.bx, a.by));
  OH_TRY(tc::map_act4d(&mD, d.dz, d.cout, d.dz_cs, d.w, d.h, d.n, a.bx, a.by));
  KernelTimer kt(ctx, timer_name, st);
  switch (d.cout) {
    case 32: return launch_wgrad<32>(mX, mD, a, mtiles, (int)splits, st);
    case 64: return launch_wgrad<64>(mX, mD, a, mtiles, (int)splits, st);
    case 128: return launch_wgrad<128>(mX, mD, a, mtiles, (int)splits, st);
    default: return launch_wgrad<256>(mX, mD, a, mtiles, (int)splits, st);
  }
}

}  // namespace oh

using namespace oh;

extern "C" {

oh_status oh_conv2d_bf16(oh_ctx* ctx, int taps, int sign, int n, int h, int w, int cin, int cout, const void* x,
                         int x_cs, const void* wmat, const float* bias, int relu, const void* mask, int mask_cs,
                         void* out, int out_cs, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CallScope cs(ctx, st);
  OH_TRY(cs.status());
  if (n < 1 || h < 1 || w < 1 || (sign != 1 && sign != -1)) return fail(OH_ERR_INVALID_ARG, "convolution: bad sizes or sign");
  ConvDesc d{};
  d.taps = taps; d.sign = sign; d.n = n; d.h = h; d.w = w; d.cin = cin; d.cout = cout;
  d.x = x; d.x_cs = x_cs; d.w_mat = wmat; d.bias = bias; d.relu = relu; d.mask = mask; d.mask_cs = mask_cs;
  d.out = out; d.out_cs = out_cs;
  return conv_enqueue(ctx, d, st, "conv_fwd_tc");
}

oh_status oh_conv2d_wgrad_bf16(oh_ctx* ctx, int taps, int n, int h, int w, int cin, int cout, const void* x, int x_cs,
                               const void* dz, int dz_cs, float* dwt, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CallScope cs(ctx, st);
  OH_TRY(cs.status());
  if (n < 1 || h < 1 || w < 1) return fail(OH_ERR_INVALID_ARG, "weight gradient: bad sizes");
  WgradDesc d{};
  d.taps = taps; d.n = n; d.h = h; d.w = w; d.cin = cin; d.cout = cout;
  d.x = x; d.x_cs = x_cs; d.dz = dz; d.dz_cs = dz_cs; d.dwt = dwt;
  return wgrad_enqueue(ctx, d, st, "conv_wgrad_tc");
}

}  // extern "C"
