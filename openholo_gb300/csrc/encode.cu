// Hologram encoders (OpenHolo_Encoding/fn_encoding.m:29-98), the phase-only
// uint8 encoding of Hologram_WRP.m:57-60 and the uint8 normalisations of
// Write_Result_image (HologramGenerator.cpp:528-565) and ophNormalize
// (oph_common.cpp:92-115).  Global maxima/minima use a two-level reduction
// (block partials, then one block), so results are deterministic.
#include <algorithm>
#include <cmath>
#include "context.h"
#include "fft_kernels.cuh"

namespace oh {

template <typename R> __device__ __forceinline__ R ratan2(R y, R x);
template <> __device__ __forceinline__ float ratan2<float>(float y, float x) { return atan2f(y, x); }
template <> __device__ __forceinline__ double ratan2<double>(double y, double x) { return atan2(y, x); }

enum RedOp { RED_MAX_ABS = 0, RED_MINMAX_REAL = 1, RED_MAX_NI = 2 };

// Block partial reductions: out[2*b] = min, out[2*b+1] = max of the mapped value.
template <typename R>
__global__ void __launch_bounds__(256) reduce_partial(const void* __restrict__ in, size_t n, int op, const R* __restrict__ refp, R* __restrict__ part) {
  typedef typename cplx_of<R>::type C;
  __shared__ R smin[256], smax[256];
  R mn = (R)INFINITY, mx = -(R)INFINITY;
  const R ref = refp ? refp[1] : (R)0;
  auto take = [&](C c) {
    R v;
    if (op == RED_MAX_ABS) v = hypot(c.x, c.y);
    else { R re = c.x + ref; v = re * re + c.y * c.y; }   // RED_MAX_NI
    mn = v < mn ? v : mn;
    mx = v > mx ? v : mx;
  };
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (op == RED_MINMAX_REAL) {
    for (; i < n; i += stride) {
      const R v = static_cast<const R*>(in)[i];
      mn = v < mn ? v : mn;
      mx = v > mx ? v : mx;
    }
  } else {
    // four independent loads in flight per thread before the math
    const C* src = static_cast<const C*>(in);
    for (; i + 3 * stride < n; i += 4 * stride) {
      C c[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) c[q] = src[i + q * stride];
#pragma unroll
      for (int q = 0; q < 4; ++q) take(c[q]);
    }
    for (; i < n; i += stride) take(src[i]);
  }
  smin[threadIdx.x] = mn; smax[threadIdx.x] = mx;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      smin[threadIdx.x] = min(smin[threadIdx.x], smin[threadIdx.x + s]);
      smax[threadIdx.x] = max(smax[threadIdx.x], smax[threadIdx.x + s]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { part[2 * blockIdx.x] = smin[0]; part[2 * blockIdx.x + 1] = smax[0]; }
}

template <typename R>
__global__ void reduce_final(R* part, int nb) {
  __shared__ R smin[256], smax[256];
  R mn = (R)INFINITY, mx = -(R)INFINITY;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) { mn = min(mn, part[2 * i]); mx = max(mx, part[2 * i + 1]); }
  smin[threadIdx.x] = mn; smax[threadIdx.x] = mx;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      smin[threadIdx.x] = min(smin[threadIdx.x], smin[threadIdx.x + s]);
      smax[threadIdx.x] = max(smax[threadIdx.x], smax[threadIdx.x + s]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { part[0] = smin[0]; part[1] = smax[0]; }
}

// Enqueue a min/max reduction; result (min,max) lands in red[0], red[1] on the device.
template <typename R>
static oh_status reduce(oh_ctx* ctx, const void* in, size_t n, int op, const R* refp, R** red, cudaStream_t st, const char* slot) {
  // 16 blocks of 256 threads per SM: one load in flight per thread, so the
  // thread count sets how many bytes are in flight (512 blocks kept the read
  // of a 66 MB field near a quarter of the HBM bandwidth)
  const int nb = (int)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, oh::sm_count() * 16));
  void* ptr;
  OH_TRY(scratch(ctx, slot, sizeof(R) * 2 * nb, &ptr));
  *red = (R*)ptr;
  KernelTimer kt(ctx, "reduce", st);
  reduce_partial<R><<<nb, 256, 0, st>>>(in, n, op, refp, *red);
  OH_LAUNCH_CHECK();
  reduce_final<R><<<1, 256, 0, st>>>(*red, nb);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

// Reference value max|U| read on the device by the map kernels.
template <typename R>
__global__ void __launch_bounds__(256) encode_map(int kind, int nx, int ny, const typename cplx_of<R>::type* __restrict__ U,
                                                  const R* __restrict__ red1, const R* __restrict__ red2, void* __restrict__ out) {
  typedef typename cplx_of<R>::type C;
  const R pi = (R)3.14159265358979323846;
  const size_t n = (size_t)nx * ny;
  auto emit = [&](size_t i, C u) {
    R* o = static_cast<R*>(out);
    switch (kind) {
      case OH_ENC_REAL: o[i] = u.x; break;
      case OH_ENC_AMPLITUDE: o[i] = hypot(u.x, u.y); break;
      case OH_ENC_PHASE_TO_AMP: o[i] = ratan2<R>(u.y, u.x) + pi / ((R)2 * pi); break;   // fn_encoding.m:57 as written
      case OH_ENC_NUM_INTERFERENCE: {
        const R ref = red1[1];
        const R re = u.x + ref;
        o[i] = (re * re + u.y * u.y) / red2[1];
      } break;
      case OH_ENC_BURCKHARDT: {
        const R m = red1[1];
        const R cr = u.x / m, ci = u.y / m;
        const R ph = ratan2<R>(ci, cr) + pi;
        const R am = hypot(cr, ci);
        const R s3 = (R)1.7320508075688772935;
        R a1 = 0, a2 = 0, a3 = 0;
        if (ph >= 0 && ph < 2 * pi / 3) {
          a1 = am * (cos(ph) + sin(ph) / s3);
          a2 = 2 * sin(ph) / s3;
        } else if (ph >= 2 * pi / 3 && ph < 4 * pi / 3) {
          a2 = am * (cos(ph - 2 * pi / 3) + sin(ph - 2 * pi / 3) / s3);
          a3 = 2 * sin(ph - 2 * pi / 3) / s3;
        } else if (ph >= 4 * pi / 3 && ph < 2 * pi) {
          a3 = am * (cos(ph - 4 * pi / 3) + sin(ph - 4 * pi / 3) / s3);
          a1 = 2 * sin(ph - 4 * pi / 3) / s3;
        }
        const size_t r = i / nx, c = i - r * nx;
        R* row = o + r * (size_t)(3 * nx);
        row[3 * c] = a1; row[3 * c + 1] = a2; row[3 * c + 2] = a3;
      } break;
      case OH_ENC_TWO_PHASE: {
        const R m = red1[1];
        const R cr = u.x / m, ci = u.y / m;
        const R am = hypot(cr, ci);
        const R ph = ratan2<R>(ci, cr) + pi;
        // MATLAB's acos of a rounding-level 1+eps is complex; its real part is 0
        const R del = acos(am < (R)1 ? am : (R)1);
        const size_t r = i / nx, c = i - r * nx;
        R* row = o + r * (size_t)(2 * nx);
        row[2 * c] = ph + del; row[2 * c + 1] = ph - del;
      } break;
      default: break;
    }
  };
  // four independent loads in flight per thread before the math
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    C u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] = U[i + q * stride];
#pragma unroll
    for (int q = 0; q < 4; ++q) emit(i + q * stride, u[q]);
  }
  for (; i < n; i += stride) emit(i, U[i]);
}

// ---- SSB (fn_encoding.m:33-41) ----------------------------------------------
// Real part of the inverse transform of the centred spectrum with one half
// zeroed, scaled to min..max.  The mask depends on one axis only, so the
// transforms along the other axis undo each other and are left out: one kernel
// per row (LEFT, RIGHT) or column strip (TOP, BOTTOM) does the forward
// transform, the mask and the inverse (the adjoint network, from storage order),
// and the block's minimum and maximum; the scaling kernel finishes the
// reduction.  Both transforms shift by floor(n/2) on both sides, as the 2-D
// transform does: over an odd length n the round trip moves the samples by
// one and multiplies sample m of the inverse by exp(-2 pi i m / n), the same
// along the axis left out.
//
// 1920x1080 FP32: two 2-D transforms, mask, reduction and scaling took 118 us;
// bound now by latency (one wave of blocks, 17 MB in, 8 MB out).
template <typename R> __device__ __forceinline__ bool is_nan(R v) { return v != v; }

// minimum and maximum of the block's values; a NaN among them makes both NaN
// (the whole image was NaN when a transform along either axis met one).  red: 2 values
// per warp of shared memory.
constexpr int kSsbThreads = 256, kSsbRed = 2 * kSsbThreads / 32;
template <typename R>
__device__ __forceinline__ void block_minmax(R mn, R mx, R* red, R* out) {
  auto lo = [](R a, R b) { return a < b || is_nan(a) ? a : b; };
  auto hi = [](R a, R b) { return a > b || is_nan(a) ? a : b; };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = lo(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = hi(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 4] = mn; red[(threadIdx.x >> 4) + 1] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 2; i < kSsbRed; i += 2) { mn = lo(mn, red[i]); mx = hi(mx, red[i + 1]); }
    out[0] = mn;
    out[1] = mx;
  }
}

// The masked axis has length n, the other length m: COLS ? strips of 1 << lw
// columns : 1 << lw rows per block.
template <typename R, bool COLS>
__global__ void __launch_bounds__(kSsbThreads, sizeof(R) == 8 ? 2 : 3) ssb_lines(int kind, const typename cplx_of<R>::type* __restrict__ in,
                                                 R* __restrict__ out, R* __restrict__ part, int n, int m, int lw,
                                                 FFTPlan pl, const void* __restrict__ tw_other) {
  typedef typename cplx_of<R>::type C;
  extern __shared__ unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int L = 1 << lw, l0 = blockIdx.x << lw, nl = min(L, m - l0);
  const int h = n / 2, ho = m / 2, lens = pl.lens;
  const bool odd = n & 1, odd_o = m & 1;
  // element i of line l: rows contiguous in shared memory, strips interleaved
  auto at = [&](int l, int p) { return COLS ? (p << lw) + l : l * lens + p; };
  auto line = [&](int l) { int s = l0 + l - 2 * ho; if (s < 0) s += m; return s; };   // the line read for line l
  if constexpr (COLS) {
    for (int idx = threadIdx.x; idx < n << lw; idx += blockDim.x) {
      const int l = idx & (L - 1), i = idx >> lw;
      int src = i - h; if (src < 0) src += n;
      buf[at(l, pl_at(pl, i))] = l < nl ? in[(size_t)src * m + line(l)] : mk((R)0, (R)0);
    }
  } else {
    for (int l = 0; l < nl; ++l) {
      const C* row = in + (size_t)line(l) * n;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int src = i - h; if (src < 0) src += n;
        buf[at(l, pl_at(pl, i))] = row[src];
      }
    }
  }
  block_fft<GFWD, C>(0, COLS ? 1 : nl, lens, COLS ? lw : 0, pl);
  // centred index c of the frequency at position p; MATLAB's floor(n/2), 1-based
  const bool upper = kind == OH_ENC_SSB_LEFT || kind == OH_ENC_SSB_TOP;
  for (int p = threadIdx.x; p < n; p += blockDim.x) {
    int c = pl.iperm[p] + h; if (c >= n) c -= n;
    if (upper ? c >= h - 1 : c <= h - 1)
      for (int l = 0; l < nl; ++l) buf[at(l, pl_at(pl, p))] = mk((R)0, (R)0);
  }
  block_fft<GADJ, C>(0, COLS ? 1 : nl, lens, COLS ? lw : 0, pl);
  const C* tw = static_cast<const C*>(pl.tw);
  const C* two = static_cast<const C*>(tw_other);
  const R scale = (R)(1.0 / (double)n);
  R mn = (R)INFINITY, mx = -(R)INFINITY;
  auto emit = [&](int l, int k) {
    int i = k - h; if (i < 0) i += n;
    C v = buf[at(l, pl_at(pl, i))];
    if (odd) v = cmul(v, tw[i]);
    if (odd_o) { int o = l0 + l - ho; if (o < 0) o += m; v = cmul(v, two[o]); }
    const R r = v.x * scale;
    out[COLS ? (size_t)k * m + l0 + l : (size_t)(l0 + l) * n + k] = r;
    // an infinity among one or two samples does not meet its opposite in the transform, as it
    // does in longer lines (nor its imaginary part the real ones without a third line)
    const R e = n < 3 ? r + (R)0 * (m < 3 ? r : v.x + v.y) : r;
    mn = e < mn || is_nan(e) ? e : mn;
    mx = e > mx || is_nan(e) ? e : mx;
  };
  if constexpr (COLS) {
    for (int idx = threadIdx.x; idx < n << lw; idx += blockDim.x)
      if ((idx & (L - 1)) < nl) emit(idx & (L - 1), idx >> lw);
  } else {
    for (int l = 0; l < nl; ++l)
      for (int k = threadIdx.x; k < n; k += blockDim.x) emit(l, k);
  }
  // (in the lines' memory: the longest lines leave none beside them)
  __syncthreads();
  block_minmax(mn, mx, reinterpret_cast<R*>(smem_raw), part + 2 * blockIdx.x);
}

// out = (out - min) / (max - min), the extremes of np block partials
template <typename R>
__global__ void __launch_bounds__(kSsbThreads) ssb_finish(size_t n, const R* __restrict__ part, int np, const R* in, R* out) {
  __shared__ R red[kSsbRed], ext[2];
  R mn = (R)INFINITY, mx = -(R)INFINITY;
  for (int i = threadIdx.x; i < np; i += blockDim.x) {
    const R a = part[2 * i], b = part[2 * i + 1];
    mn = a < mn || is_nan(a) ? a : mn;
    mx = b > mx || is_nan(b) ? b : mx;
  }
  block_minmax(mn, mx, red, ext);
  __syncthreads();
  const R lo = ext[0], rng = ext[1] - ext[0];
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    R v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = in[i + q * stride];
#pragma unroll
    for (int q = 0; q < 4; ++q) out[i + q * stride] = (v[q] - lo) / rng;
  }
  for (; i < n; i += stride) out[i] = (in[i] - lo) / rng;
}

template <typename R>
static oh_status run_ssb(oh_ctx* ctx, int kind, int nx, int ny, const void* field, void* out, cudaStream_t st) {
  typedef typename cplx_of<R>::type C;
  const int prec = sizeof(R) == 8 ? 1 : 0;
  FFTPlan px, py;
  OH_TRY(get_plan(ctx, nx, prec, &px));
  OH_TRY(get_plan(ctx, ny, prec, &py));
  const size_t smax = max_smem_per_block();
  if ((size_t)px.lens * sizeof(C) > smax || (size_t)py.lens * sizeof(C) > smax)
    return fail(OH_ERR_UNSUPPORTED_SIZE, "SSB: a side's line exceeds shared memory");
  const bool cols = kind == OH_ENC_SSB_TOP || kind == OH_ENC_SSB_BOTTOM;
  const FFTPlan& pl = cols ? py : px;
  const int n = cols ? ny : nx, m = cols ? nx : ny;
  // lines per block: up to 8 (columns: whole sectors) within 48 KB while the
  // SMs still get two blocks each
  int lw = 0;
  while (lw < 3 && ((size_t)pl.lens * sizeof(C) << (lw + 1)) <= 48 * 1024 && (m >> (lw + 1)) >= 2 * oh::sm_count()) ++lw;
  const int blocks = (m + (1 << lw) - 1) >> lw;
  const size_t smem = std::max((size_t)pl.lens * sizeof(C) << lw, kSsbRed * sizeof(R));
  const size_t total = (size_t)nx * ny;
  void* ptr;
  OH_TRY(scratch(ctx, "enc.red1", sizeof(R) * 2 * blocks, &ptr));
  // an output over the field itself waits in scratch until every line is read
  R* real = (R*)out;
  const char *f0 = (const char*)field, *o0 = (const char*)out;
  if (o0 < f0 + total * sizeof(C) && f0 < o0 + total * sizeof(R)) {
    void* tmp;
    OH_TRY(scratch(ctx, "enc.ssb", total * sizeof(R), &tmp));
    real = (R*)tmp;
  }
  auto kern = cols ? ssb_lines<R, true> : ssb_lines<R, false>;
  // (the same limit at every length: another thread may set it between here and the launch)
  OH_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax));
  {
    KernelTimer kt(ctx, "ssb_lines", st);
    kern<<<blocks, kSsbThreads, smem, st>>>(kind, (const C*)field, real, (R*)ptr, n, m, lw, pl, cols ? px.tw : py.tw);
    OH_LAUNCH_CHECK();
  }
  KernelTimer kt(ctx, "ssb_finish", st);
  ssb_finish<R><<<(int)std::min<size_t>((total + 1023) / 1024, oh::sm_count() * 16), kSsbThreads, 0, st>>>(total, (const R*)ptr, blocks, real, (R*)out);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

// ---- phase-only uint8 (Hologram_WRP.m:57-60) -----------------------------------
// Pass 1 writes angle + pi to scratch and every block's maximum, pass 2
// finishes the maximum and scales to bytes: one arc tangent per pixel (two
// before, one per pass) and two launches instead of three.
template <typename R>
__global__ void __launch_bounds__(256) phase_pass(const typename cplx_of<R>::type* __restrict__ U, size_t n,
                                                  R* __restrict__ ph, R* __restrict__ part) {
  typedef typename cplx_of<R>::type C;
  __shared__ R smx[8];
  R mx = -(R)INFINITY;
  auto take = [&](size_t i, C c) {
    const R v = ratan2<R>(c.y, c.x) + (R)3.14159265358979323846;
    ph[i] = v;
    mx = v > mx ? v : mx;
  };
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    C c[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) c[q] = U[i + q * stride];
#pragma unroll
    for (int q = 0; q < 4; ++q) take(i + q * stride, c[q]);
  }
  for (; i < n; i += stride) take(i, U[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) smx[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < 8; ++q) mx = max(mx, smx[q]);
    part[blockIdx.x] = mx;
  }
}

template <typename R>
__global__ void __launch_bounds__(256) phase_u8(const R* __restrict__ ph, size_t n, const R* __restrict__ part, int np,
                                                uint8_t* __restrict__ out) {
  __shared__ R smx[8];
  R mx = -(R)INFINITY;
  for (int i = threadIdx.x; i < np; i += blockDim.x) mx = max(mx, part[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) smx[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = smx[0];
#pragma unroll
  for (int q = 1; q < 8; ++q) mx = max(mx, smx[q]);
  auto byte = [&](R p) {
    R v = (R)255 * p / mx;
    // MATLAB uint8(): round half away from zero, saturate
    v = v < 0 ? 0 : (v > 255 ? 255 : v);
    return (uint8_t)floor(v + (R)0.5);
  };
  // four pixels per thread and store where the output is aligned
  const size_t stride = (size_t)gridDim.x * blockDim.x, first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t n4 = reinterpret_cast<uintptr_t>(out) % 4 == 0 ? n / 4 : 0;
  for (size_t i = first; i < n4; i += stride) {
    R p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) p[q] = ph[4 * i + q];
    reinterpret_cast<uchar4*>(out)[i] = make_uchar4(byte(p[0]), byte(p[1]), byte(p[2]), byte(p[3]));
  }
  for (size_t i = 4 * n4 + first; i < n; i += stride) out[i] = byte(ph[i]);
}

template <typename R>
static oh_status run_phase_u8(oh_ctx* ctx, size_t n, const void* field, void* out, cudaStream_t st) {
  typedef typename cplx_of<R>::type C;
  const int np = (int)std::min<size_t>((n + 255) / 256, oh::sm_count() * 6);
  void* ptr;
  OH_TRY(scratch(ctx, "enc.phase", n * sizeof(R) + sizeof(R) * np, &ptr));
  R* ph = (R*)ptr;
  R* part = ph + n;
  {
    KernelTimer kt(ctx, "phase_pass", st);
    phase_pass<R><<<np, 256, 0, st>>>((const C*)field, n, ph, part);
    OH_LAUNCH_CHECK();
  }
  KernelTimer kt(ctx, "phase_u8", st);
  phase_u8<R><<<(int)std::min<size_t>((n + 1023) / 1024, oh::sm_count() * 16), 256, 0, st>>>(ph, n, part, np, (uint8_t*)out);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

template <typename R>
__global__ void normalize_u8_kernel(int nx, int ny, const R* __restrict__ in, const R* __restrict__ red, uint8_t* __restrict__ out, int round_half) {
  const size_t n = (size_t)nx * ny;
  const R mn = red[0], mx = red[1];
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (round_half) {
      // ophNormalize: float math, +0.5, vertical flip
      const int r = (int)(i / nx), c = (int)(i - (size_t)r * nx);
      float v = (((float)in[i] - (float)mn) / ((float)mx - (float)mn)) * 255.f + 0.5f;
      out[(size_t)(ny - r - 1) * nx + c] = (uint8_t)(unsigned)v;
    } else {
      // Write_Result_image: (uint)((v - min)/(max - min)*255) in double
      double v = ((double)in[i] - (double)mn) / ((double)mx - (double)mn) * 255.0;
      out[i] = (uint8_t)(unsigned)v;
    }
  }
}

template <typename R>
static oh_status run_encode(oh_ctx* ctx, int kind, int nx, int ny, const void* field, void* out, cudaStream_t st) {
  typedef typename cplx_of<R>::type C;
  const size_t n = (size_t)nx * ny;
  const int grid = (int)std::min<size_t>((n + 255) / 256, oh::sm_count() * 16);
  R* red1 = nullptr;
  R* red2 = nullptr;
  if (kind >= OH_ENC_SSB_LEFT && kind <= OH_ENC_SSB_BOTTOM) return run_ssb<R>(ctx, kind, nx, ny, field, out, st);
  if (kind == OH_ENC_PHASE_ONLY_U8) return run_phase_u8<R>(ctx, n, field, out, st);
  if (kind == OH_ENC_NUM_INTERFERENCE || kind == OH_ENC_BURCKHARDT || kind == OH_ENC_TWO_PHASE)
    OH_TRY(reduce<R>(ctx, field, n, RED_MAX_ABS, (const R*)nullptr, &red1, st, "enc.red1"));
  if (kind == OH_ENC_NUM_INTERFERENCE) {
    // max |U + max|U||^2, the reference value read on the device
    OH_TRY(reduce<R>(ctx, field, n, RED_MAX_NI, red1, &red2, st, "enc.red2"));
  }
  KernelTimer kt(ctx, "encode_map", st);
  encode_map<R><<<grid, 256, 0, st>>>(kind, nx, ny, (const C*)field, red1, red2, out);
  OH_LAUNCH_CHECK();
  return OH_OK;
}

}  // namespace oh

using namespace oh;

extern "C" {

oh_status oh_encode(oh_ctx* ctx, oh_precision prec, int kind, int nx, int ny, const void* field, void* out, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CallScope cs(ctx, st);
  OH_TRY(cs.status());
  if (nx < 1 || ny < 1 || !field || !out) return fail(OH_ERR_INVALID_ARG, "oh_encode: bad size or null buffer");
  if (kind < OH_ENC_REAL || kind > OH_ENC_AMPLITUDE) return fail(OH_ERR_INVALID_ARG, "oh_encode: unknown encoding");
  if (prec == OH_FP64) return run_encode<double>(ctx, kind, nx, ny, field, out, st);
  return run_encode<float>(ctx, kind, nx, ny, field, out, st);
}

oh_status oh_normalize_u8(oh_ctx* ctx, oh_precision prec, int nx, int ny, const void* in, uint8_t* out, int round_half,
                          void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CallScope cs(ctx, st);
  OH_TRY(cs.status());
  if (nx < 1 || ny < 1 || !in || !out) return fail(OH_ERR_INVALID_ARG, "oh_normalize_u8: bad size or null buffer");
  const size_t n = (size_t)nx * ny;
  const int grid = (int)std::min<size_t>((n + 255) / 256, oh::sm_count() * 16);
  if (prec == OH_FP64) {
    double* red;
    OH_TRY(reduce<double>(ctx, in, n, RED_MINMAX_REAL, (const double*)nullptr, &red, st, "norm.red"));
    normalize_u8_kernel<double><<<grid, 256, 0, st>>>(nx, ny, (const double*)in, red, out, round_half);
  } else {
    float* red;
    OH_TRY(reduce<float>(ctx, in, n, RED_MINMAX_REAL, (const float*)nullptr, &red, st, "norm.red"));
    normalize_u8_kernel<float><<<grid, 256, 0, st>>>(nx, ny, (const float*)in, red, out, round_half);
  }
  OH_LAUNCH_CHECK();
  return OH_OK;
}

}  // extern "C"
