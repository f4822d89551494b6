// Plan-driven block FFT for lengths without a compile-time schedule (and for
// FP64): the stage radices are run-time values, each stage's butterfly a
// compile-time radix chosen by one switch per stage.  Radices 2..16, 18 and 30
// are straight-line code (odd primes 7, 11, 13 by the symmetric sum/difference
// form, composites by Cooley-Tukey or Good-Thomas); other primes up to 61 run
// an O(r^2) loop.  Index divisions use host-computed multipliers, twiddles
// come from per-stage tables laid out [output][offset] (coalesced over
// consecutive butterflies, exact values).
//
// What bounds it: instruction issue.  The run-time engine before this one took
// radices 2, 3, 4, 5, 8 and ran every other radix (7, 9, 15, 16 too) through
// the O(r^2) loop over local memory.
#pragma once
#include <type_traits>
#include "fft_fast.cuh"
#include "two_float.cuh"

namespace oh {

template <int P> struct PrimeTab;
template <> struct PrimeTab<7> {
  __device__ __forceinline__ static double c(int k) { constexpr double v[] = {1.0, 0.623489801858733530525, -0.222520933956314404289, -0.900968867902419126236, -0.900968867902419126236, -0.222520933956314404289, 0.623489801858733530525}; return v[k]; }
  __device__ __forceinline__ static double s(int k) { constexpr double v[] = {0.0, 0.781831482468029808708, 0.974927912181823607018, 0.433883739117558120476, -0.433883739117558120476, -0.974927912181823607018, -0.781831482468029808708}; return v[k]; }
};
template <> struct PrimeTab<11> {
  __device__ __forceinline__ static double c(int k) { constexpr double v[] = {1.0, 0.841253532831181168862, 0.415415013001886425529, -0.142314838273285140444, -0.654860733945285064057, -0.95949297361449738989, -0.95949297361449738989, -0.654860733945285064057, -0.142314838273285140444, 0.415415013001886425529, 0.841253532831181168862}; return v[k]; }
  __device__ __forceinline__ static double s(int k) { constexpr double v[] = {0.0, 0.540640817455597582108, 0.909631995354518371412, 0.989821441880932732376, 0.755749574354258283774, 0.281732556841429697711, -0.281732556841429697711, -0.755749574354258283774, -0.989821441880932732376, -0.909631995354518371412, -0.540640817455597582108}; return v[k]; }
};
template <> struct PrimeTab<13> {
  __device__ __forceinline__ static double c(int k) { constexpr double v[] = {1.0, 0.8854560256532098959, 0.568064746731155802512, 0.120536680255323053349, -0.35460488704253562597, -0.748510748171101098635, -0.970941817426052027157, -0.970941817426052027157, -0.748510748171101098635, -0.35460488704253562597, 0.120536680255323053349, 0.568064746731155802512, 0.8854560256532098959}; return v[k]; }
  __device__ __forceinline__ static double s(int k) { constexpr double v[] = {0.0, 0.464723172043768545656, 0.82298386589365639458, 0.992708874098053992801, 0.93501624268541482344, 0.663122658240795202377, 0.239315664287557767149, -0.239315664287557767149, -0.663122658240795202377, -0.93501624268541482344, -0.992708874098053992801, -0.82298386589365639458, -0.464723172043768545656}; return v[k]; }
};

// Odd prime DFT: a_k = x_k + x_{P-k}, b_k = x_k - x_{P-k}, k = 1..(P-1)/2;
// y_f, y_{P-f} = x_0 + sum_k cos(2 pi k f / P) a_k -/+ i sum_k sin(2 pi k f / P) b_k.
template <int P, int SGN, typename C>
__device__ __forceinline__ void dft_prime(C* x) {
  typedef decltype(x[0].x) R;
  constexpr int H = (P - 1) / 2;
  C a[H], b[H];
#pragma unroll
  for (int k = 0; k < H; ++k) { a[k] = cadd(x[k + 1], x[P - 1 - k]); b[k] = csub(x[k + 1], x[P - 1 - k]); }
  const C x0 = x[0];
  C y0 = x0;
#pragma unroll
  for (int k = 0; k < H; ++k) y0 = cadd(y0, a[k]);
  x[0] = y0;
#pragma unroll
  for (int f = 1; f <= H; ++f) {
    C m = x0, q = cscale(b[0], (R)PrimeTab<P>::s(f));
#pragma unroll
    for (int k = 0; k < H; ++k) m = caxpy((R)PrimeTab<P>::c((k + 1) * f % P), a[k], m);
#pragma unroll
    for (int k = 1; k < H; ++k) q = caxpy((R)PrimeTab<P>::s((k + 1) * f % P), b[k], q);
    x[f] = cadd_i<SGN>(m, q);                 // forward: m - i q
    x[P - f] = cadd_i<-SGN>(m, q);
  }
}

template <int SGN, typename C> struct DFT<7, SGN, C> {
  __device__ __forceinline__ static void run(C* x) { dft_prime<7, SGN>(x); }
};
template <int SGN, typename C> struct DFT<11, SGN, C> {
  __device__ __forceinline__ static void run(C* x) { dft_prime<11, SGN>(x); }
};
template <int SGN, typename C> struct DFT<13, SGN, C> {
  __device__ __forceinline__ static void run(C* x) { dft_prime<13, SGN>(x); }
};
template <int SGN, typename C> struct DFT<14, SGN, C> {
  __device__ __forceinline__ static void run(C* x) { dft_pfa<2, 7, SGN>(x); }
};

template <typename C> __device__ __forceinline__ C ldg_c(const C* p) { return __ldg(p); }
__device__ __forceinline__ ffc ldg_c(const ffc* p) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(p));
  return mk(ff(v.x, v.y), ff(v.z, v.w));
}

// Calls f(std::integral_constant<int, r>) for the straight-line radices and
// f(std::integral_constant<int, 0>) for any other.
// (18 and 30 occur in FP32's compile-time schedules only: WIDE takes them too.  The depth-map
// passes do without it, as its registers would cost every other length; columns of
// 4320 or 7680 that the fast pass refuses run those two stages through the loop.)
template <bool WIDE, class F>
__device__ __forceinline__ void with_radix(int r, F&& f) {
  switch (r) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 11: f(std::integral_constant<int, 11>{}); break;
    case 12: f(std::integral_constant<int, 12>{}); break;
    case 13: f(std::integral_constant<int, 13>{}); break;
    case 14: f(std::integral_constant<int, 14>{}); break;
    case 15: f(std::integral_constant<int, 15>{}); break;
    case 16: f(std::integral_constant<int, 16>{}); break;
    default:
      if constexpr (WIDE) {
        if (r == 18) { f(std::integral_constant<int, 18>{}); break; }
        if (r == 30) { f(std::integral_constant<int, 30>{}); break; }
      }
      f(std::integral_constant<int, 0>{});
      break;
  }
}

// The stages' directions: GFWD forward DIF, GINV inverse DIF (natural order
// in), GADJ the adjoint of the forward stage (storage order in, stages in
// reverse order, natural order out; see fstage_adj).
enum { GFWD = 0, GINV = 1, GADJ = 2 };

// One stage's numbers, by value (a reference to a kernel parameter would be
// copied to local memory at a call that is not inlined).
struct GStage {
  int n, r, q, qs, nb, padr, tws;
  uint32_t mq, mnb, mpad;
  const void* tw;        // this stage's table (null when q == 1)
  const void* full;      // W_n^e
};
__device__ __forceinline__ GStage gstage_of(const FFTPlan& pl, int s, size_t esz) {
  GStage g;
  g.n = pl.n; g.r = pl.radix[s]; g.q = pl.q[s]; g.qs = pl.qs[s]; g.padr = pl.padr;
  g.nb = g.n / g.r;
  g.mq = pl.mq[s]; g.mnb = pl.mnb[s]; g.mpad = pl.mpad;
  g.tws = g.n / (g.r * g.q);
  g.tw = g.q > 1 ? static_cast<const char*>(pl.stw) + (size_t)pl.two[s] * esz : nullptr;
  g.full = pl.tw;
  return g;
}

// Lines come as ng groups of 1 << lw interleaved lines, group k's element at
// stored position p of line w at k * ls + (p << lw) + w (lw = 0: contiguous
// lines ls apart).  Butterfly index idx -> offset of its line, butterfly b:
// line within the group fastest, then the butterfly, then the group.
__device__ __forceinline__ int gsplit(const GStage& g, int idx, int ng, int ls, int lw, int* off, int* b) {
  const int r = idx >> lw;
  const int k = ng > 1 ? fdiv(r, g.mnb) : 0;
  *b = r - k * g.nb;
  *off = k * ls + (idx & ((1 << lw) - 1));
  return k;
}

// Stored position of input 0 of butterfly b and its offset j.
__device__ __forceinline__ int gbase(const GStage& g, int b, int* j) {
  const int blk = g.q > 1 ? fdiv(b, g.mq) : b;
  *j = b - blk * g.q;
  const int p = blk * g.r * g.q + *j;
  return g.padr ? p + fdiv(p, g.mpad) : p;
}

// DFT and twiddles of one butterfly in registers (radix R > 0).
template <int R, int MODE, typename C>
__device__ __forceinline__ void gbutterfly(const GStage& g, int j, C* x) {
  constexpr int SGN = MODE == GFWD ? -1 : 1;
  const C* tw = static_cast<const C*>(g.tw) + j;
  if constexpr (MODE == GADJ) {
    if (j) {
#pragma unroll
      for (int f = 1; f < R; ++f) x[f] = cmulc(x[f], ldg_c(tw + (f - 1) * g.q));
    }
    DFT<R, 1, C>::run(x);
  } else {
    DFT<R, SGN, C>::run(x);
    if (j) {
#pragma unroll
      for (int f = 1; f < R; ++f) {
        const C w = ldg_c(tw + (f - 1) * g.q);
        x[f] = MODE == GFWD ? cmul(x[f], w) : cmulc(x[f], w);
      }
    }
  }
}

// One butterfly of any other radix, through get(t) and put(f, v).
template <int MODE, typename C, class G, class P>
__device__ __forceinline__ void gbutterfly_any(const GStage& g, int j, G get, P put) {
  C x[kMaxGenericRadix];
  const C* full = static_cast<const C*>(g.full);
  auto w = [&](int e) { C v = full[e]; if (MODE != GFWD) v.y = -v.y; return v; };
  for (int t = 0; t < g.r; ++t) {
    C v = get(t);
    if (MODE == GADJ && j && t) v = cmul(v, w(j * t * g.tws));
    x[t] = v;
  }
  const int step = g.n / g.r;
  for (int f = 0; f < g.r; ++f) {
    C acc = x[0];
    int m = 0;
    for (int t = 1; t < g.r; ++t) {
      m += f; if (m >= g.r) m -= g.r;
      acc = cadd(acc, cmul(x[t], w(m * step)));
    }
    if (MODE != GADJ && j && f) acc = cmul(acc, w(f * j * g.tws));
    put(f, acc);
  }
}

// One in-place stage.
template <int R, int MODE, typename C>
__device__ __forceinline__ void gstage_loop(const GStage& g, C* buf, int ng, int ls, int lw) {
  const int total = (g.nb * ng) << lw, st = g.qs << lw;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    int off, b, j;
    gsplit(g, idx, ng, ls, lw, &off, &b);
    C* p = buf + off + (gbase(g, b, &j) << lw);
    if constexpr (R > 0) {
      C x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = p[t * st];
      gbutterfly<R, MODE>(g, j, x);
#pragma unroll
      for (int t = 0; t < R; ++t) p[t * st] = x[t];
    } else {
      gbutterfly_any<MODE, C>(g, j, [&](int t) { return p[t * st]; }, [&](int f, C v) { p[f * st] = v; });
    }
  }
}

// The same as a call: one copy of the radices per kernel.  off is the lines'
// byte offset in the kernel's dynamic shared memory (so that the accesses stay
// shared-memory ones).
template <int MODE, typename C, bool WIDE>
__device__ __noinline__ void gstage_call(GStage g, int off, int ng, int ls, int lw) {
  extern __shared__ unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw + off);
  with_radix<WIDE>(g.r, [&](auto rc) { gstage_loop<decltype(rc)::value, MODE, C>(g, buf, ng, ls, lw); });
}

// Full in-place transform of the lines at byte offset off of the dynamic shared
// memory; a barrier before every stage and after the last.  WIDE: see
// with_radix (lengths with a compile-time schedule may pass through here).
template <int MODE, typename C, bool WIDE = sizeof(C) == 8>
__device__ __forceinline__ void block_fft(int off, int ng, int ls, int lw, const FFTPlan& pl) {
  for (int i = 0; i < pl.nst; ++i) {
    __syncthreads();
    gstage_call<MODE, C, WIDE>(gstage_of(pl, MODE == GADJ ? pl.nst - 1 - i : i, sizeof(C)), off, ng, ls, lw);
  }
  __syncthreads();
}

}  // namespace oh
