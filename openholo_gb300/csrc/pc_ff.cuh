// The per-axis factors of the FP64 point-cloud sum in two-float arithmetic.
#pragma once
#include <cuda_bf16.h>
#include "two_float.cuh"

namespace oh {

// One axis of a point as a plane region sees it: the phase in turns at offset m
// from the region's centre is t0 + m (c1 + m (c2 + m (c3 + m c4))) mod 1 in 64-bit
// fractions of a turn plus m^5 (c5 + c6 m), the coefficients those of
// (r0 / lambda) (sqrt(1 + 2 s t + t^2) - 1), t = m pitch / r0; the reduced
// argument w / Qs = m (a + m b) of the cross term (see pc_tc.cu).
struct AxisRec {
  uint64_t t0, c1, c2, c3, c4;
  float c5, c6;
  ff a, b;
};

// exp(2 pi i t / 2^64); extra: a further phase in turns, below 1e-6; tab: see
// ff_rotate.
OH_FF ffc ff_cis64(uint64_t t, float extra, const float4* tab) {
  const uint64_t r = t + (1ull << 55);
  const int idx = (int)(r >> 56);
  const int64_t f = (int64_t)(t - ((uint64_t)idx << 56));         // [-2^55, 2^55)
  const int hi = (int)(f >> 24);
  const float A = (float)(hi >> 8);                              // 24 bits, units of 2^-32 turns
  const float B = (float)((((uint32_t)hi & 0xffu) << 24) | (uint32_t)(f & 0xffffff));   // units of 2^-64
  const float ch = 1.46291807926715968105e-9f;                   // 2 pi 2^-32 = ch + cl
  const float cl = (float)(1.4629180792671596810513378043098e-9 - (double)1.46291807926715968105e-9f);
  const float cb = 3.4061215800304e-19f;                         // 2 pi 2^-64
  const float p = OH_FMUL(A, ch);
  const float q = OH_FFMA(A, cl, OH_FFMA(A, ch, -p));
  return ff_rotate({p, OH_FFMA(6.28318530717958647692f, extra, OH_FFMA(B, cb, q))}, tab[idx & 255]);
}

OH_FF ffc axis_cis(const AxisRec& r, int m, const float4* tab) {
  const uint64_t um = (uint64_t)(int64_t)m;
  const uint64_t t = r.t0 + um * (r.c1 + um * (r.c2 + um * (r.c3 + um * r.c4)));
  const float mf = (float)m, m2 = mf * mf;
  return ff_cis64(t, OH_FMUL(OH_FMUL(m2, OH_FMUL(m2, mf)), OH_FFMA(r.c6, mf, r.c5)), tab);
}

// w (1 - 3/4 w + 5/8 w^2 - 35/64 w^3) / Qs, w / Qs = m (a + b m)
OH_FF ff axis_cross(const AxisRec& r, int m, float qs) {
  const float mf = (float)m, m2 = OH_FMUL(mf, mf);
  const float p1 = OH_FMUL(r.a.h, mf), p2 = OH_FMUL(r.b.h, m2);
  const float e1 = OH_FFMA(r.a.l, mf, OH_FFMA(r.a.h, mf, -p1)), e2 = OH_FFMA(r.b.l, m2, OH_FFMA(r.b.h, m2, -p2));
  const ff g = ff_sum(p1, p2);
  const float w = OH_FMUL(g.h, qs);
  const float corr = OH_FMUL(OH_FMUL(g.h, w), OH_FFMA(w, OH_FFMA(w, 0.546875f, -0.625f), 0.75f));
  const ff h = ff_sum(g.h, -corr);
  return {h.h, OH_FADD(h.l, OH_FADD(g.l, OH_FADD(e1, e2)))};
}

// v rounded to BF16, as a float
OH_FF float bf16_round(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}

// v, |v| <= 1, as multiples of 2^-8 (unless !UNIT: |v| <= 2^-8), of 2^-16 and of
// 2^-24, each at most 256 steps and so exact in BF16, then two BF16 rests (the
// last below 2^-42): s[0] + ... + s[4].
template <bool UNIT>
OH_FF void ff_slices(ff v, float* s) {
  float h = v.h;
  s[0] = 0.f;
  if (UNIT) { s[0] = OH_FSUB(OH_FADD(h, 49152.f), 49152.f); h = OH_FSUB(h, s[0]); }
  s[1] = OH_FSUB(OH_FADD(h, 192.f), 192.f);
  h = OH_FADD(OH_FSUB(h, s[1]), v.l);
  s[2] = OH_FSUB(OH_FADD(h, 0.75f), 0.75f);
  h = OH_FSUB(h, s[2]);
  s[3] = bf16_round(h);
  s[4] = OH_FSUB(h, s[3]);
}

}  // namespace oh
