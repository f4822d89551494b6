// Depth-map passes on the plan-driven FFT engine: FP64 frames (computed in
// two-float arithmetic, or in FP64 where a frame's range asks for it), and FP32
// frames whose padded row or column length has no compile-time schedule.  The same
// frame pipeline as dm_kernels.cuh / dm_col_fast.cuh (row strips, layer flags,
// spectrum columns in the row FFT's storage order, inverses as the adjoint of
// the forward network), with run-time lengths.
#pragma once
#include "dm_kernels.cuh"

namespace oh {

// Amplitude of an image byte and exp(i phase) of a pixel per compute type; tab: the
// two-float directions (see ff_cis).
__device__ __forceinline__ void amp_of(uint8_t g, float* v) { *v = (float)g / 255.f; }
__device__ __forceinline__ void amp_of(uint8_t g, double* v) { *v = (double)g / 255.0; }
__device__ __forceinline__ void amp_of(uint8_t g, ff* v) { *v = ff((double)g / 255.0); }
template <typename R>
__device__ __forceinline__ typename cplx_of<R>::type phase_of(float radians, float turns, bool seeded, const float4* tab) {
  if constexpr (std::is_same<R, ff>::value) {
    if (!seeded && !(fabsf(radians) <= 16.f)) {           // turns to 2^-47 of a few
      double sn, cs;
      sincos((double)radians, &sn, &cs);
      return mk(ff(cs), ff(sn));
    }
    return ff_cis(seeded ? ff(turns) : ff_mulf(ff(0.15915494309189533576888376337251), radians), tab);
  } else {
    const R ph = seeded ? (R)turns * (R)6.283185307179586476925 : (R)radians;
    R sn, cs;
    sincos_r<R>(ph, &sn, &cs);
    return mk(cs, sn);
  }
}

// Row pass: nr (1 or 2) image rows per block.  The layers present in them are
// taken G at a time (short lines alone leave most threads idle): stage 0
// straight from the source pixels, the other stages in place, then the lines go
// to the strips in storage order (two columns per strip in FP32: two rows fill
// a 32-byte sector).
template <typename R>
__global__ void __launch_bounds__(256, 2) dm_row_gen(DMArgs<R> a, int nr, int G) {
  typedef typename cplx_of<R>::type C;
  extern __shared__ unsigned char smem_raw[];
  const int Px = a.Px, pnx = a.pnx, T = blockDim.x;
  const int lip = (pnx + 7) & ~7, lens = a.plx.lens;
  __shared__ int16_t present[kMaxEntries];
  __shared__ int s_np;
  C* buf = reinterpret_cast<C*>(smem_raw);              // [G][nr][lens]
  C* v = buf + G * nr * lens;                           // [nr][pnx] source values
  int16_t* li = reinterpret_cast<int16_t*>(v + nr * pnx);        // [nr][lip] layer slot per pixel
  uint32_t* mask = reinterpret_cast<uint32_t*>(li + nr * lip);   // [2][8] layers present per row
  const int r0 = blockIdx.x * nr;
  const int nrows = min(nr, a.pny - r0);
  int16_t* const slut = dm_row_slut();
  const float4* tab = nullptr;
  if constexpr (std::is_same<R, ff>::value) {
    __shared__ float4 dirs[256];
    if (a.phase_mode != OH_PHASE_REFERENCE) ff_directions(dirs, threadIdx.x, T);
    tab = dirs;
  }
  for (int i = threadIdx.x; i < 16; i += T) mask[i] = 0u;
  for (int i = threadIdx.x; i < 256; i += T) slut[i] = a.lut[i];
  __syncthreads();
  for (int l = 0; l < nrows; ++l)
    for (int c = threadIdx.x; c < pnx; c += T) {
      const size_t off = (size_t)(r0 + l) * pnx + c;
      int u = -1;
      C val = mk((R)0, (R)0);
      if (a.src) {                                      // a complex source field: one layer slot
        u = 0;
        val = a.src[off];
      } else {
        const uint8_t g = a.img[off];
        u = g > 0 ? (int)slut[a.depth[off]] : -1;
        if (u >= 0) {
          R amp;
          amp_of(g, &amp);
          if (a.phase_mode == OH_PHASE_REFERENCE) {
            val = mk(amp, (R)0);
          } else {
            const bool seeded = a.phase_mode == OH_PHASE_SEEDED;
            const C e = phase_of<R>(seeded ? 0.f : a.phase[off], seeded ? u24_at(a.seed, off) : 0.f, seeded, tab);
            val = mk(amp * e.x, amp * e.y);
          }
        }
      }
      if (u >= 0) {
        // neighbours mostly share a layer: one atomic per distinct slot of the active lanes
        const unsigned same = __match_any_sync(__activemask(), u);
        if ((threadIdx.x & 31) == __ffs(same) - 1) atomicOr(&mask[l * 8 + (u >> 5)], 1u << (u & 31));
      }
      li[l * lip + c] = (int16_t)u;
      v[l * pnx + c] = val;
    }
  __syncthreads();
  // the slots present in the block's rows, their flags per row
  auto has = [&](int l, int u) { return (mask[l * 8 + (u >> 5)] >> (u & 31)) & 1u; };
  if (threadIdx.x < 32) {
    int n = 0;
    for (int base = a.slot0; base < a.slot1; base += 32) {
      const int u = base + threadIdx.x;
      const bool p = u < a.slot1 && (has(0, u) || has(1, u));
      const unsigned m = __ballot_sync(0xffffffffu, p);
      if (p) {
        present[n + __popc(m & ((1u << threadIdx.x) - 1u))] = (int16_t)u;
        a.slot_any[u] = 1;
      }
      n += __popc(m);
    }
    if (threadIdx.x == 0) s_np = n;
  }
  for (int i = threadIdx.x; i < nrows * (a.slot1 - a.slot0); i += T) {
    const int l = nrows == 2 ? i & 1 : 0, ur = nrows == 2 ? i >> 1 : i;
    a.occ[(size_t)ur * a.occ_stride + r0 + l] = has(l, a.slot0 + ur) ? 1 : 0;
  }
  __syncthreads();
  const GStage g0 = gstage_of(a.plx, 0, sizeof(C));
  const int np = s_np, W = a.W, lw = a.lw;
  for (int q = 0; q < np; q += G) {
    const int nq = min(G, np - q), ng = nq * nrows;      // line k: slot q + k / nrows, row k % nrows
    auto slot_of = [&](int k) { return (int)present[q + (nrows == 2 ? k >> 1 : k)]; };
    // input i of the x-shifted, zero-padded line a[i] = u[(i - hx) mod Px]
    auto pixel = [&](int l, int u, int i) -> C {
      int x = i - a.hx;
      if (x < 0) x += Px;
      const int c = x - a.ox;
      return (unsigned)c < (unsigned)pnx && li[l * lip + c] == u ? v[l * pnx + c] : mk((R)0, (R)0);
    };
    if (a.plx.nst == 0) {
      if (threadIdx.x < ng) buf[threadIdx.x * lens] = pixel(nrows == 2 ? threadIdx.x & 1 : 0, slot_of(threadIdx.x), 0);
    } else {
      with_radix<false>(g0.r, [&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        const int total = g0.nb * ng;
        for (int idx = threadIdx.x; idx < total; idx += T) {
          int off, b, j;
          const int k = gsplit(g0, idx, ng, lens, 0, &off, &b);
          const int l = nrows == 2 ? k & 1 : 0, u = slot_of(k);
          C* p = buf + off + gbase(g0, b, &j);
          if constexpr (RR > 0) {
            C x[RR];
#pragma unroll
            for (int t = 0; t < RR; ++t) x[t] = pixel(l, u, j + t * g0.q);
            gbutterfly<RR, GFWD>(g0, j, x);
#pragma unroll
            for (int t = 0; t < RR; ++t) p[t * g0.qs] = x[t];
          } else {
            gbutterfly_any<GFWD, C>(g0, j, [&](int t) { return pixel(l, u, j + t * g0.q); },
                                    [&](int f, C y) { p[f * g0.qs] = y; });
          }
        }
      });
    }
    for (int s = 1; s < a.plx.nst; ++s) {
      __syncthreads();
      gstage_call<GFWD, C, false>(gstage_of(a.plx, s, sizeof(C)), 0, ng, lens, 0);
    }
    __syncthreads();
    for (int k = 0; k < nq; ++k) {
      C* dst = a.Rbuf + (size_t)(present[q + k] - a.slot0) * a.nstrips * a.pny * W;
      const C* line = buf + k * nrows * lens;
      for (int idx = threadIdx.x; idx < nrows * Px; idx += T) {
        const int w = idx & (W - 1), t = idx >> lw;
        const int l = nrows == 2 ? (t & 1) : 0, s = nrows == 2 ? (t >> 1) : t;
        dst[((size_t)s * a.pny + r0 + l) * W + w] = line[l * lens + pl_at(a.plx, (s << lw) + w)];
      }
    }
    __syncthreads();
  }
}

// exp(2 pi i t): table of 128 directions and a short polynomial on the rest
// (|x| <= pi / 128: the dropped terms are below 2e-15).  An FP64 sine and
// cosine by the general routine takes three to four times as many FP64
// instructions, of which this part issues one per 64 FP32 ones.
__device__ __forceinline__ double2 cis_turns(double t, const double2* tab) {
  const double big = 6755399441055744.0;                // 1.5 2^52: adding it rounds to an integer
  const double v = t * 128.0;
  const double n = v + big;
  const double x = (v - (n - big)) * 0.049087385212340519350978802863742;      // 2 pi / 128
  const double2 d = tab[__double2loint(n) & 127];
  const double x2 = x * x;
  const double s = fma(x * x2, fma(x2, 1.0 / 120.0, -1.0 / 6.0), x);
  const double c = fma(x2, fma(x2, fma(x2, -1.0 / 720.0, 1.0 / 24.0), -0.5), 1.0);
  return make_double2(fma(d.x, c, -d.y * s), fma(d.x, s, d.y * c));
}

// Directions of the column pass's sine/cosine table (FP64 cis_turns, two-float
// ff_cis).
template <typename R> constexpr int kDirs = sizeof(R) == 4 ? 0 : std::is_same<R, ff>::value ? 256 : 128;

// Two-float accumulators are renormalised at every layer step: left alone their low
// parts grow with the steps, and the errors of the products with them (216 layers: 3.4e-11
// of the frame; 6e-13 renormalised, for 2 % of the frame at 1920 x 1080).
__device__ __forceinline__ float2 normal(float2 v) { return v; }
__device__ __forceinline__ double2 normal(double2 v) { return v; }
__device__ __forceinline__ ffc normal(ffc v) { return mk(ff_quick(v.x.h, v.x.l), ff_quick(v.y.h, v.y.l)); }

// Shared memory of the column pass after the lines: kept rows' positions,
// active entries and their count, and in FP64 the direction table and (evenly
// spaced layers) the step factors.  All that the kernel uses: columns near the limit
// of a block's memory have no room for static variables beside it.
template <typename R>
inline size_t dm_col_gen_smem(int lens, int lwb, int G, int nrow, int n_entries, bool horner) {
  size_t o = (size_t)G * lens << lwb;
  if (sizeof(R) == 8) o += kDirs<R> + (horner ? (size_t)nrow << lwb : 0);
  o *= 2 * sizeof(R);
  return o + (((size_t)nrow * 2 + 15) & ~(size_t)15) + (size_t)n_entries * 2 + 16;
}

// Column pass: 1 << lwb spectrum columns (storage positions) per block for the
// whole frame.  The active layers are taken G at a time (short columns alone
// leave most threads idle): stage 0 straight from the strips (absent and padded
// rows are zeros), the other stages in place, then every thread adds H(e) times
// its samples into registers.  Only the spectrum rows [row0, row0 +
// nrow) that reach the crop are kept.  Transfer function: the entry's separable
// tables times exp(i k z' g), g = s^2 / (2 (1 + sqrt(1 - s))^2) held per sample;
// FP64 and two-float frames with evenly spaced layers accumulate acc = acc D + x
// instead (see dm_col_fast.cuh), D in shared memory.
//
// What bounds it: instruction issue in FP32 (FFT butterflies plus about 20
// instructions per kept sample and layer) and two-float (about 300 a sample in
// the FFT), the FP64 pipe in FP64.
template <typename R, int KMAX, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) dm_col_gen(DMArgs<R> a, int lwb, int G, int row0, int nrow) {
  typedef typename cplx_of<R>::type C;
  constexpr bool F64 = sizeof(R) == 8;
  constexpr bool KEEPG = KMAX <= 16;                    // g per sample in registers
  extern __shared__ unsigned char smem_raw[];
  const int W = 1 << lwb, Py = a.Py, pny = a.pny, lens = a.ply.lens, tid = threadIdx.x;
  const bool step = F64 && a.horner;
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int gs = lens << lwb;                           // a layer's lines
  C* tab = buf + (size_t)G * gs;
  C* dst = tab + kDirs<R>;
  uint16_t* pos = reinterpret_cast<uint16_t*>(dst + (step ? (size_t)nrow << lwb : 0));
  int16_t* list = reinterpret_cast<int16_t*>(pos + ((nrow + 7) & ~7));
  int* s_nact = reinterpret_cast<int*>(list + ((a.n_entries + 1) & ~1));      // (not static: see dm_col_gen_smem)
  const int w = tid & (W - 1), p = (blockIdx.x << lwb) + w;
  const bool valid = p < a.Px;
  int kx = 0;
  if (valid) { kx = a.plx.iperm[p] + a.hx; if (kx >= a.Px) kx -= a.Px; }
  const int nk = nrow << lwb;
  for (int i = tid; i < nrow; i += T) {
    int k = row0 + i - a.hy;                            // S[ky] = B[(ky - hy) mod Py]
    if (k < 0) k += Py;
    pos[i] = (uint16_t)a.ply.permp[k];
  }
  if (tid < 32) {
    int n = 0;
    for (int base = 0; base < a.n_entries; base += 32) {
      const int e = base + tid;
      const bool act = e < a.n_entries && a.slot_any[a.uslot_of_entry[e]] != 0;
      const unsigned m = __ballot_sync(0xffffffffu, act);
      if (act) list[n + __popc(m & ((1u << tid) - 1u))] = (int16_t)e;
      n += __popc(m);
    }
    if (tid == 0) *s_nact = n;
  }
  if constexpr (std::is_same<R, ff>::value) {
    ff_directions(reinterpret_cast<float4*>(tab), tid, T);
  } else if constexpr (F64) {
    for (int i = tid; i < 128; i += T) { double s, c; sincospi(i * (1.0 / 64.0), &s, &c); tab[i] = mk(c, s); }
  }
  auto resid = [&](int k) -> R {
    const int i = (tid + k * T) >> lwb;
    if constexpr (F64) {                                // g / 2 pi
      const double sv = (double)a.lfx[kx] + (double)a.lfy[row0 + i];
      const double den = 1.0 + sqrt(1.0 - sv);
      return (R)(sv * sv / (12.566370614359172953850573533118 * den * den));
    } else {
      const R sv = a.lfx[kx] + a.lfy[row0 + i];
      const R den = (R)1 + sqrt((R)1 - sv);
      return sv * sv / ((R)2 * den * den);
    }
  };
  C acc[KMAX];
  R g[KEEPG ? KMAX : 1];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    acc[k] = mk((R)0, (R)0);
    if constexpr (KEEPG) g[k] = tid + k * T < nk ? resid(k) : (R)0;
  }
  __syncthreads();
  const int nact = *s_nact;
  auto gof = [&](int k) -> R { if constexpr (KEEPG) return g[k]; else return resid(k); };
  // exp(i kz g) of sample k
  auto residual = [&](R kz, int k) -> C {
    if constexpr (std::is_same<R, ff>::value) return ff_cis(kz * gof(k), reinterpret_cast<const float4*>(tab));
    else if constexpr (F64) return cis_turns(kz * gof(k), tab);
    else { float sn, cs; __sincosf(kz * gof(k), &sn, &cs); return mk(cs, sn); }
  };
  if constexpr (F64) {
    if (step) {
      // D = H(z' - dz) / H(z') per kept sample
      const R kdz = (R)(-a.k * a.dz);
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
        const int idx = tid + k * T;
        if (idx < nk) {
          int ky = row0 + (idx >> lwb) - a.hy;
          if (ky < 0) ky += Py;
          dst[idx] = cmul(cmul(a.dxh[kx], a.dyh[a.ply.perm[ky]]), residual(kdz, k));
        }
      }
    }
  }
  const GStage g0 = gstage_of(a.ply, 0, sizeof(C));
  for (int q = 0; q < nact; q += G) {
    const int ng = min(G, nact - q);
    // input i of the y-shifted, zero-padded column of entry list[q + k]
    auto sample = [&](const C* src, const uint8_t* occ, int i) -> C {
      int y = i - a.hy;
      if (y < 0) y += Py;
      y -= a.oy;
      return valid && (unsigned)y < (unsigned)pny && __ldg(occ + y) ? src[y << a.lw] : mk((R)0, (R)0);
    };
    auto column = [&](int u) { return a.Rbuf + ((size_t)u * a.nstrips + (p >> a.lw)) * pny * a.W + (p & (a.W - 1)); };
    if (a.ply.nst == 0) {
      for (int k = tid >> lwb; k < ng; k += T >> lwb) {
        const int u = a.uslot_of_entry[list[q + k]];
        buf[k * gs + w] = sample(column(u), a.occ + (size_t)u * a.occ_stride, 0);
      }
    } else {
      with_radix<false>(g0.r, [&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        const int total = (g0.nb * ng) << lwb, st = g0.qs << lwb;
        for (int idx = tid; idx < total; idx += T) {
          int off, b, j;
          const int k = gsplit(g0, idx, ng, gs, lwb, &off, &b);
          const int u = a.uslot_of_entry[list[q + k]];
          const uint8_t* occ = a.occ + (size_t)u * a.occ_stride;
          const C* src = column(u);
          C* d = buf + off + (gbase(g0, b, &j) << lwb);
          if constexpr (RR > 0) {
            C x[RR];
#pragma unroll
            for (int t = 0; t < RR; ++t) x[t] = sample(src, occ, j + t * g0.q);
            gbutterfly<RR, GFWD>(g0, j, x);
#pragma unroll
            for (int t = 0; t < RR; ++t) d[t * st] = x[t];
          } else {
            gbutterfly_any<GFWD, C>(g0, j, [&](int t) { return sample(src, occ, j + t * g0.q); },
                                    [&](int f, C y) { d[f * st] = y; });
          }
        }
      });
    }
    for (int s = 1; s < a.ply.nst; ++s) {
      __syncthreads();
      const GStage gs1 = gstage_of(a.ply, s, sizeof(C));
      with_radix<false>(gs1.r, [&](auto rc) {
        gstage_loop<decltype(rc)::value, GFWD, C>(gs1, buf, ng, gs, lwb);
      });
    }
    __syncthreads();
    for (int k0 = 0; k0 < ng; ++k0) {
      const int e = list[q + k0];
      const C* line = buf + k0 * gs + w;
      if (F64 && step) {
        const int gap = q + k0 > 0 ? e - list[q + k0 - 1] : 0;      // levels without pixels: one more factor each
#pragma unroll
        for (int k = 0; k < KMAX; ++k) {
          const int idx = tid + k * T;
          if (idx < nk) {
            const C x = line[(int)pos[idx >> lwb] << lwb];
            if (gap) {
              const C d = dst[idx];
              for (int r = 1; r < gap; ++r) acc[k] = normal(cmul(acc[k], d));
              acc[k] = normal(mk(fma(acc[k].x, d.x, fma(-acc[k].y, d.y, x.x)), fma(acc[k].x, d.y, fma(acc[k].y, d.x, x.y))));
            } else {
              acc[k] = x;
            }
          }
        }
      } else if (valid) {
        const R kz = a.kzp[e];
        const C ex = a.exc[(size_t)e * a.Px + kx];
        const C* ey = a.ey + (size_t)e * Py + row0;
#pragma unroll
        for (int k = 0; k < KMAX; ++k) {
          const int idx = tid + k * T;
          if (idx < nk) {
            const C h = cmul(cmul(ex, ldg_c(ey + (idx >> lwb))), residual(kz, k));
            const C x = line[(int)pos[idx >> lwb] << lwb];
            if constexpr (F64) {
              acc[k].x = fma(h.x, x.x, fma(-h.y, x.y, acc[k].x));
              acc[k].y = fma(h.x, x.y, fma(h.y, x.x, acc[k].y));
            } else {
              acc[k] = cadd(acc[k], cmul(h, x));        // (one rounding of the sum per layer)
            }
          }
        }
      }
    }
    __syncthreads();
  }
  if (F64 && step && nact > 0 && valid) {
    // the recurrence ends with the last active entry's transfer function
    const int e = list[nact - 1];
    const R kz = a.kzp[e];
    const C ex = a.exc[(size_t)e * a.Px + kx];
    const C* ey = a.ey + (size_t)e * Py + row0;
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      const int idx = tid + k * T;
      if (idx < nk) acc[k] = cmul(acc[k], cmul(cmul(ex, ldg_c(ey + (idx >> lwb))), residual(kz, k)));
    }
  }

  // SSB crop, inverse y-FFT as the adjoint network, output rows.  The inverse
  // line b[i] = Uc[(i - hy) mod Py] wants spectrum row ky at i = (ky + hy) mod Py,
  // i.e. in storage order at permp[i].
  for (int i = tid; i < lens << lwb; i += T) buf[i] = mk((R)0, (R)0);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    const int idx = tid + k * T;
    if (idx < nk && valid) {
      const int ky = row0 + (idx >> lwb);
      if (a.spectrum) a.spectrum[(size_t)ky * a.Px + kx] = mk(to_out(acc[k].x), to_out(acc[k].y));
      if (kx >= a.cx1 && kx <= a.cx2 && ky >= a.cy1 && ky <= a.cy2) {
        int i = ky + a.hy;
        if (i >= Py) i -= Py;
        buf[(a.ply.permp[i] << lwb) + w] = acc[k];
      }
    }
  }
  block_fft<GADJ, C, false>(0, 1, 0, lwb, a.ply);
  for (int idx = tid; idx < pny << lwb; idx += T) {
    const int yl = idx >> lwb;
    int m = a.oy + yl - a.hy;
    if (m < 0) m += Py;
    if (valid) a.V[(size_t)yl * a.Px + p] = cmul(buf[(pl_at(a.ply, m) << lwb) + w], a.shy[yl]);
  }
}

// Output pass: one row per block.  V column p holds spectrum column kx =
// (iperm[p] + hx) mod Px, which the inverse line wants at j = (kx + hx) mod Px
// (the same storage position for even Px).
template <typename R>
__global__ void __launch_bounds__(256) dm_out_gen(DMArgs<R> a) {
  typedef typename cplx_of<R>::type C;
  extern __shared__ unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  const int yl = blockIdx.x, Px = a.Px;
  const C* row = a.V + (size_t)yl * Px;
  const bool even = 2 * a.hx == Px;
  for (int p = threadIdx.x; p < Px; p += blockDim.x) {
    int at;
    if (even) {
      at = pl_at(a.plx, p);
    } else {
      int j = a.plx.iperm[p] + 2 * a.hx;
      if (j >= Px) j -= Px;
      at = a.plx.permp[j];
    }
    buf[at] = row[p];
  }
  block_fft<GADJ, C, false>(0, 1, 0, 0, a.plx);
  for (int c = threadIdx.x; c < a.pnx; c += blockDim.x) {
    int m = a.ox + c - a.hx;
    if (m < 0) m += Px;
    C h = buf[pl_at(a.plx, m)];
    if (a.sig_x != 0) h = cmul(h, a.shx[c]);
    a.fringe[(size_t)yl * a.pnx + c] = to_out(h.x);
    if (a.field) a.field[(size_t)yl * a.pnx + c] = mk(to_out(h.x), to_out(h.y));
  }
}

// How a frame runs these passes (dm_generic.cuh's launches).
struct DMGenPlan {
  int nr, gr;             // image rows per row-pass block, layers taken at a time
  int lwb, gc;            // log2 columns per column-pass block, layers taken at a time
  int row0, nrow;         // spectrum rows kept
  bool wide;              // the column pass's many-samples variant
  size_t smem_row, smem_col, smem_out;
};
template <typename R> DMGenPlan dm_gen_plan(const DMArgs<R>& a, size_t smax);
template <typename R> cudaError_t dm_gen_row(const DMArgs<R>& a, const DMGenPlan& g, cudaStream_t st);
template <typename R> cudaError_t dm_gen_col(const DMArgs<R>& a, const DMGenPlan& g, cudaStream_t st);
template <typename R> cudaError_t dm_gen_out(const DMArgs<R>& a, const DMGenPlan& g, cudaStream_t st);

}  // namespace oh
