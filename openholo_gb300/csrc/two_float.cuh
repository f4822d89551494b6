// Two-float arithmetic: a value as the unevaluated sum h + l of two FP32 numbers,
// about 47 bits.  FP64 runs at 1/64 of the FP32 rate on this part, so error-free
// FP32 transforms (Dekker, Knuth; products by FMA) are several times faster:
// 8 instructions for a sum, 4 for a product, against 64.
//
// Results are not renormalised: l may reach a few units in h's last place (after
// a cancellation of the h parts, any size); errors stay near 2^-47 of the
// operands.  Everything is written with explicitly rounded operations: a
// contraction to FMA would break the error terms.
#pragma once
#include <cstdint>
#include "oh_common.cuh"

namespace oh {

#define OH_FADD(a, b) __fadd_rn(a, b)
#define OH_FSUB(a, b) __fsub_rn(a, b)
#define OH_FMUL(a, b) __fmul_rn(a, b)
#define OH_FFMA(a, b, c) __fmaf_rn(a, b, c)
#define OH_FF __device__ __forceinline__

struct ff;
OH_FF ff operator+(ff a, ff b);
OH_FF ff operator*(ff a, ff b);
struct ff {
  float h, l;
  ff() = default;
  __host__ __device__ ff(float h_, float l_) : h(h_), l(l_) {}
  __host__ __device__ explicit ff(double v) : h((float)v), l((float)(v - (double)(float)v)) {}
  OH_FF explicit ff(float v) : h(v), l(0.f) {}
  OH_FF explicit ff(int v) : ff((double)v) {}
  friend OH_FF ff fma(ff a, ff b, ff c) { return a * b + c; }
  OH_FF explicit operator double() const { return (double)h + (double)l; }
};
struct alignas(16) ffc { ff x, y; };
template <> struct cplx_of<ff> { typedef ffc type; };
__host__ __device__ __forceinline__ ffc mk(ff x, ff y) { ffc r; r.x = x; r.y = y; return r; }

OH_FF ff ff_quick(float a, float b) {            // |a| >= |b| or a = 0
  const float s = OH_FADD(a, b);
  return {s, OH_FSUB(b, OH_FSUB(s, a))};
}
OH_FF ff ff_sum(float a, float b) {
  const float s = OH_FADD(a, b), t = OH_FSUB(s, a);
  return {s, OH_FADD(OH_FSUB(a, OH_FSUB(s, t)), OH_FSUB(b, t))};
}
OH_FF ff operator-(ff a) { return {-a.h, -a.l}; }
OH_FF ff operator+(ff a, ff b) {
  const ff s = ff_sum(a.h, b.h);
  return {s.h, OH_FADD(s.l, OH_FADD(a.l, b.l))};
}
OH_FF ff operator-(ff a, ff b) { return a + (-b); }
OH_FF ff operator*(ff a, ff b) {
  const float p = OH_FMUL(a.h, b.h);
  return {p, OH_FFMA(a.l, b.h, OH_FFMA(a.h, b.l, OH_FFMA(a.h, b.h, -p)))};
}
OH_FF ff ff_mulf(ff a, float b) {
  const float p = OH_FMUL(a.h, b);
  return {p, OH_FFMA(a.l, b, OH_FFMA(a.h, b, -p))};
}

// exp(i x) T for |x| <= pi / 256 (x.l any rounding error of it), T = (cos h, cos
// l, sin h, sin l) of a direction.
OH_FF ffc ff_rotate(ff x, float4 T) {
  const float x2 = OH_FMUL(x.h, x.h);
  const float x2l = OH_FFMA(OH_FMUL(2.f, x.h), x.l, OH_FFMA(x.h, x.h, -x2));
  // sin x = x - x^3 (1 / 6 - x^2 / 120), cos x - 1 = -x^2 / 2 + x^4 (1 / 24 - x^2 / 720)
  const ff s(x.h, OH_FFMA(OH_FMUL(-x.h, x2), OH_FFMA(x2, -0.0083333333f, 0.16666667f), x.l));
  const float ch = -0.5f * x2;
  const float cl = OH_FFMA(-0.5f, x2l, OH_FMUL(OH_FMUL(x2, x2), OH_FFMA(x2, -0.0013888889f, 0.041666668f)));
  ffc o;
  {
    const float p1 = OH_FMUL(T.x, ch), p2 = OH_FMUL(T.z, s.h);
    const float e1 = OH_FFMA(T.y, ch, OH_FFMA(T.x, cl, OH_FFMA(T.x, ch, -p1)));
    const float e2 = OH_FFMA(T.w, s.h, OH_FFMA(T.z, s.l, OH_FFMA(T.z, s.h, -p2)));
    const ff d = ff_sum(p1, -p2);
    const ff g = ff_sum(T.x, d.h);
    o.x = ff_quick(g.h, OH_FADD(g.l, OH_FADD(T.y, OH_FADD(d.l, OH_FSUB(e1, e2)))));
  }
  {
    const float p1 = OH_FMUL(T.z, ch), p2 = OH_FMUL(T.x, s.h);
    const float e1 = OH_FFMA(T.w, ch, OH_FFMA(T.z, cl, OH_FFMA(T.z, ch, -p1)));
    const float e2 = OH_FFMA(T.y, s.h, OH_FFMA(T.x, s.l, OH_FFMA(T.x, s.h, -p2)));
    const ff d = ff_sum(p1, p2);
    const ff g = ff_sum(T.z, d.h);
    o.y = ff_quick(g.h, OH_FADD(g.l, OH_FADD(T.w, OH_FADD(d.l, OH_FADD(e1, e2)))));
  }
  return o;
}

// exp(2 pi i t), |t| < 2^14; tab[i]: direction 2 pi i / 256 (see ff_rotate)
OH_FF ffc ff_cis(ff t, const float4* tab) {
  const float big = 12582912.f;                  // 1.5 2^23: adding it rounds to an integer
  const float v = OH_FADD(OH_FMUL(t.h, 256.f), big);
  const int idx = __float_as_int(v);
  const float r = OH_FSUB(t.h, OH_FMUL(OH_FSUB(v, big), 0.00390625f));     // exact
  const float c = 6.28318530717958647692f;                       // 2 pi = c + cl
  const float cl = (float)(6.28318530717958647692 - (double)6.28318530717958647692f);
  const float p = OH_FMUL(r, c);
  // (t.l is a rounding error of t, not of what is left of it: joined to the high part first,
  // as ff_rotate leaves out its products with x^2)
  return ff_rotate(ff_quick(p, OH_FFMA(t.l, c, OH_FFMA(r, cl, OH_FFMA(r, c, -p)))), tab[idx & 255]);
}

// Fills tab[i] with direction 2 pi i / 256; thread tid of nthr.
__device__ __forceinline__ void ff_directions(float4* tab, int tid, int nthr) {
  for (int i = tid; i < 256; i += nthr) {
    double s, c;
    sincospi(i * (1.0 / 128.0), &s, &c);
    const ff a(c), b(s);
    tab[i] = make_float4(a.h, a.l, b.h, b.l);
  }
}

}  // namespace oh
