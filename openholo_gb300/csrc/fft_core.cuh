// Block-level mixed-radix FFT on data resident in shared memory.
//
// A length-n line (n = r0*r1*...*r_{S-1}) is transformed in place with the
// decimation-in-frequency (Sande-Tukey) recursion:
//   stage s works on blocks of m_s = r_s*q_s elements; for j < q_s it takes
//   x[j + t*q_s], t < r_s, forms the r_s-point DFT y_f, multiplies y_f by
//   W_{m_s}^{j f} and stores it back at j + f*q_s.
// After the last stage the spectrum value X[k] sits at position perm[k]
// (mixed-radix digit reversal); callers read outputs through that table, so
// no reordering pass is needed.  Twiddles W_n^e = exp(-2 pi i e/n) come from
// a table of n entries built on the host in double precision; SGN = -1 runs
// the forward transform, SGN = +1 the inverse (conjugate twiddles).
//
// Lines are addressed as buf[line*ls + i*es], so the same code serves a
// contiguous row (ls = n, es = 1) and a strip of W interleaved columns
// (ls = 1, es = W).
#pragma once
#include "oh_common.cuh"

namespace oh {

// (a line in shared memory needs at most six: 5^6; the batch kernel keeps two plans
// per frame in shared memory)
constexpr int kMaxStages = 8;
constexpr int kMaxGenericRadix = 64;

// A plan's line is stored with one pad element after every padr elements when
// its last radix is even (padr = that radix; the last stage would otherwise
// crowd its reads onto few shared-memory banks), else without pads (padr = 0).
// padr divides every stage's block and stride, so all stages keep fixed
// strides.  The compile-time engine (fft_fast.cuh) has layouts of its own.
struct FFTPlan {
  int n;
  int nst;
  int lens;               // stored length of a line: n, or n + n / padr
  int padr;
  uint32_t mpad;          // divider of padr (see fdiv)
  int radix[kMaxStages];
  int q[kMaxStages];      // stride inside a block at stage s
  int qs[kMaxStages];     // the stored stride
  int two[kMaxStages];    // first entry of stage s in stw
  uint32_t mq[kMaxStages];    // dividers of q and of n / radix
  uint32_t mnb[kMaxStages];
  const void* tw;         // n complex twiddles W_n^e (precision of the kernel)
  const void* stw;        // per stage with q > 1: W_{m_s}^{j f} at [f - 1][j], 1 <= f < radix, j < q
  const int* perm;        // perm[k]: position of X[k] after the last stage
  const int* iperm;       // iperm[pos]: frequency k stored at pos
  const int* permp;       // perm in stored positions
};

// i / d with m = ceil(2^32 / d) (0 stands for d = 1), exact while i d <= 2^32: here i is at
// most the elements of the lines that a block holds, below 2^15 like d
__device__ __forceinline__ int fdiv(int i, uint32_t m) { return m ? (int)__umulhi((uint32_t)i, m) : i; }

// stored position of line element p
__device__ __forceinline__ int pl_at(const FFTPlan& pl, int p) { return pl.padr ? p + fdiv(p, pl.mpad) : p; }

// ---- small DFT kernels (forward SGN=-1, inverse SGN=+1) -------------------

template <int SGN, typename C>
__device__ __forceinline__ void dft2(C& a, C& b) {
  C t = a; a = cadd(t, b); b = csub(t, b);
}

template <int SGN, typename C>
__device__ __forceinline__ void dft4(C& x0, C& x1, C& x2, C& x3) {
  C t0 = cadd(x0, x2), t1 = csub(x0, x2), t2 = cadd(x1, x3), t3 = csub(x1, x3);
  x0 = cadd(t0, t2); x2 = csub(t0, t2);
  x1 = cadd_i<SGN>(t1, t3); x3 = cadd_i<-SGN>(t1, t3);   // forward: t1 -/+ i t3
}

template <int SGN, typename C>
__device__ __forceinline__ void dft3(C& x0, C& x1, C& x2) {
  typedef decltype(x0.x) R;
  const R c = (R)0.86602540378443864676;   // sqrt(3)/2
  C t = cadd(x1, x2), d = csub(x1, x2);
  C y0 = cadd(x0, t);
  C m = caxpy((R)-0.5, t, x0);
  // forward y1 = m - i c d, y2 = m + i c d
  x0 = y0; x1 = caxpy_i<SGN>(c, d, m); x2 = caxpy_i<-SGN>(c, d, m);
}

template <int SGN, typename C>
__device__ __forceinline__ void dft5(C& x0, C& x1, C& x2, C& x3, C& x4) {
  typedef decltype(x0.x) R;
  const R c1 = (R)0.30901699437494742410;   // cos(2pi/5)
  const R c2 = (R)-0.80901699437494742410;  // cos(4pi/5)
  const R s1 = (R)0.95105651629515357212;   // sin(2pi/5)
  const R s2 = (R)0.58778525229247312917;   // sin(4pi/5)
  C a1 = cadd(x1, x4), b1 = csub(x1, x4), a2 = cadd(x2, x3), b2 = csub(x2, x3);
  C y0 = cadd(x0, cadd(a1, a2));
  const C p1 = caxpy(c2, a2, caxpy(c1, a1, x0));
  const C p2 = caxpy(c1, a2, caxpy(c2, a1, x0));
  const C q1 = caxpy(s2, b2, cscale(b1, s1));
  const C q2 = caxpy(-s1, b2, cscale(b1, s2));
  x0 = y0;
  // forward: p -/+ i q
  x1 = cadd_i<SGN>(p1, q1); x4 = cadd_i<-SGN>(p1, q1);
  x2 = cadd_i<SGN>(p2, q2); x3 = cadd_i<-SGN>(p2, q2);
}

template <int SGN, typename C>
__device__ __forceinline__ void dft8(C* x) {
  typedef decltype(x[0].x) R;
  const R h = (R)0.70710678118654752440;
  C e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6];
  C o0 = x[1], o1 = x[3], o2 = x[5], o3 = x[7];
  dft4<SGN>(e0, e1, e2, e3);
  dft4<SGN>(o0, o1, o2, o3);
  // w8^k for k = 1,2,3 (forward e^{-i pi k/4})
  C w1, w3;
  w1.x = h; w1.y = SGN < 0 ? -h : h;
  w3.x = -h; w3.y = SGN < 0 ? -h : h;
  o1 = cmul(o1, w1);
  o3 = cmul(o3, w3);
  x[0] = cadd(e0, o0); x[4] = csub(e0, o0);
  x[1] = cadd(e1, o1); x[5] = csub(e1, o1);
  x[2] = cadd_i<SGN>(e2, o2); x[6] = cadd_i<-SGN>(e2, o2);
  x[3] = cadd(e3, o3); x[7] = csub(e3, o3);
}

template <int SGN, typename C>
__device__ __forceinline__ C twiddle(const C* tw, int e) {
  C w = tw[e];
  if (SGN > 0) w.y = -w.y;
  return w;
}

}  // namespace oh
