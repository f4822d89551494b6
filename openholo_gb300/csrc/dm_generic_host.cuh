// Host side of dm_generic.cuh, instantiated once per precision
// (dm_generic_f32.cu, dm_generic_f64.cu, dm_generic_tf.cu).
#pragma once
#include <algorithm>
#include "dm_generic.cuh"

namespace oh {

// Samples per thread, threads per block and blocks per SM of the column pass: few
// enough samples that the accumulators (and g) stay in registers; the wide variant
// takes what is longer.  Two-float frames measured (1920 x 1080, 32 layers) 2.00 ms
// with four blocks of 128 threads, 2.29 with two of 256, 2.42 with three of 128.
template <typename R> struct DMGenCfg {
  static constexpr bool TF = std::is_same<R, ff>::value;
  static constexpr int K = sizeof(R) == 8 ? 10 : 8, T = sizeof(R) == 8 ? 128 : 256, MINB = TF ? 4 : 3;
  static constexpr int KW = 40, TW = sizeof(R) == 8 ? 256 : 512;
};

template <typename R>
DMGenPlan dm_gen_plan(const DMArgs<R>& a, size_t smax) {
  typedef DMGenCfg<R> CF;
  const size_t esz = 2 * sizeof(R);
  DMGenPlan g{};
  const size_t budget = (size_t)216 * 1024 / CF::MINB;  // column blocks of an SM
  const size_t rbudget = (size_t)(CF::TF ? 108 : 72) * 1024;            // two (three) row blocks
  const int sms = sm_count();
  // layers taken at a time: enough lines for two butterflies per thread in the
  // first stage, while they fit
  auto groups = [&](const FFTPlan& pl, int lines, int threads, int most) {
    const int per = std::max(1, pl.nst ? pl.n / pl.radix[0] : 1) * lines;
    return std::max(1, std::min({16, most, 2 * threads / per}));
  };
  auto row = [&](int nr, int G) {
    return (size_t)nr * ((size_t)G * a.plx.lens * esz + (size_t)a.pnx * esz + (size_t)((a.pnx + 7) & ~7) * 2) + 64;
  };
  // two rows per block fill whole sectors of the strips; one where two would
  // leave fewer blocks per SM than the budget's or the SMs short of blocks
  g.nr = row(2, 1) <= rbudget && a.pny >= 4 * sms ? 2 : 1;
  g.gr = groups(a.plx, g.nr, 256, a.slot1 - a.slot0);
  while (g.gr > 1 && row(g.nr, g.gr) > rbudget) --g.gr;
  g.smem_row = row(g.nr, g.gr);
  // spectrum rows that reach the crop (all of them when the spectrum is asked for)
  g.row0 = a.spectrum ? 0 : a.cy1;
  g.nrow = a.spectrum ? a.Py : a.cy2 - a.cy1 + 1;
  const bool horner = a.horner != 0;
  // the most columns per block (their loads and stores share sectors) that keep
  // the narrow variant, MINB blocks of shared memory per SM and four blocks
  // per SM of work
  g.lwb = -1;
  for (int lw = 1; lw >= 0; --lw) {
    const size_t sm = dm_col_gen_smem<R>(a.ply.lens, lw, 1, g.nrow, a.n_entries, horner);
    if ((g.nrow << lw) <= CF::K * CF::T && sm <= (lw ? budget : smax) &&
        (lw == 0 || (a.Px >> lw) >= 4 * sms)) {
      g.lwb = lw;
      break;
    }
  }
  g.wide = g.lwb < 0;
  if (g.wide) g.lwb = 0;
  g.gc = groups(a.ply, 1 << g.lwb, g.wide ? CF::TW : CF::T, a.n_entries);
  while (g.gc > 1 && dm_col_gen_smem<R>(a.ply.lens, g.lwb, g.gc, g.nrow, a.n_entries, horner) > budget) --g.gc;
  g.smem_col = dm_col_gen_smem<R>(a.ply.lens, g.lwb, g.gc, g.nrow, a.n_entries, horner);
  g.smem_out = (size_t)a.plx.lens * esz;
  return g;
}

// The same limit at every size: another thread may set it between here and the launch.
template <typename K>
static cudaError_t dm_gen_allow(K kern, size_t static_bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(max_smem_per_block() - static_bytes));
}

template <typename R>
cudaError_t dm_gen_row(const DMArgs<R>& a, const DMGenPlan& g, cudaStream_t st) {
  cudaError_t e = dm_gen_allow(dm_row_gen<R>, 8192);         // (its layer tables, the two-float directions)
  if (e != cudaSuccess) return e;
  dm_row_gen<R><<<(a.pny + g.nr - 1) / g.nr, 256, g.smem_row, st>>>(a, g.nr, g.gr);
  return cudaGetLastError();
}

template <typename R>
cudaError_t dm_gen_col(const DMArgs<R>& a, const DMGenPlan& g, cudaStream_t st) {
  typedef DMGenCfg<R> CF;
  const int blocks = (a.Px + (1 << g.lwb) - 1) >> g.lwb;
  auto launch = [&](auto kern, int threads) {
    cudaError_t e = dm_gen_allow(kern, 0);
    if (e != cudaSuccess) return e;
    kern<<<blocks, threads, g.smem_col, st>>>(a, g.lwb, g.gc, g.row0, g.nrow);
    return cudaGetLastError();
  };
  return g.wide ? launch(dm_col_gen<R, CF::KW, CF::TW, 1>, CF::TW) : launch(dm_col_gen<R, CF::K, CF::T, CF::MINB>, CF::T);
}

template <typename R>
cudaError_t dm_gen_out(const DMArgs<R>& a, const DMGenPlan& g, cudaStream_t st) {
  cudaError_t e = dm_gen_allow(dm_out_gen<R>, 0);
  if (e != cudaSuccess) return e;
  dm_out_gen<R><<<a.pny, 256, g.smem_out, st>>>(a);
  return cudaGetLastError();
}

#define OH_DM_GENERIC(R)                                                               \
  template DMGenPlan dm_gen_plan<R>(const DMArgs<R>&, size_t);                          \
  template cudaError_t dm_gen_row<R>(const DMArgs<R>&, const DMGenPlan&, cudaStream_t); \
  template cudaError_t dm_gen_col<R>(const DMArgs<R>&, const DMGenPlan&, cudaStream_t); \
  template cudaError_t dm_gen_out<R>(const DMArgs<R>&, const DMGenPlan&, cudaStream_t);

}  // namespace oh
