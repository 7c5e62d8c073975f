// Operator contractions along lines of points, with the products on the
// integer pipes (spd_soft.cuh).
#pragma once
#include "spd_device.cuh"

namespace spd {

// L values along one line of points, prepared once for the several operator
// rows that are applied to them.
template <int L>
struct Line {
#ifdef SPD_FUSED
  static constexpr int PREPARED = L < 2 ? L : 2;  // a sum's first product, or two
#else
  static constexpr int PREPARED = L;
#endif
  double v[L];
  Opnd o[PREPARED];
  bool soft;
  uint32_t eoff;
};
// ``use``: the operator's entries are all within coef_in_range.  A line is
// multiplied on the integer pipes when every value is a zero or within
// opnd_of's window (no subnormal, infinity or NaN, and with entries in range
// no product outside the normal range).  ``eoff``: the operator is the
// stored one times 2^k (exact), given as k << 20 with |k| <= 64.
template <int L>
SPD_FN void line_ready(Line<L>& ln, int use, uint32_t eoff = 0u) {
  uint32_t ok = use ? 0x40000000u : 0u;
#pragma unroll
  for (int s = 0; s < Line<L>::PREPARED; ++s) {
    ln.o[s] = opnd_of(ln.v[s], ok);
    ln.o[s].e += eoff;
  }
  ln.soft = ok != 0u;
  ln.eoff = eoff;
}

// Sum orders of a contraction: left to right, or even and odd terms
// separately and then added (dot_seq, dot_lanes2).  The order is a template
// argument: chosen at run time, both sums were executed.
template <int L, bool LANES2>
SPD_FN double sum_terms(const double* p) {
  if (!LANES2 || L == 1) {
    double acc = p[0];
#pragma unroll
    for (int s = 1; s < L; ++s) acc = acc + p[s];
    return acc;
  }
  double e = p[0], o = p[L > 1 ? 1 : 0];
#pragma unroll
  for (int s = 2; s < L; ++s) {
    if (s % 2 == 0) e = e + p[s];
    else o = o + p[s];
  }
  return e + o;
}

// out[r] = sum_s C[(r0 + r*step)*L + s] * line[s] for R rows of an operator:
// LANES2, the order of the x direction, or left to right.
//
// The fused build adds a product and the sum so far in one FP64 instruction;
// the first product of a sum (of each of the two, LANES2) runs on the integer
// pipes (k_interior at 512^2,
// p = 3: 24,320 -> 18,952 FP64 instructions per cell, 12.2 -> 9.6 ms a step).
template <int L, int R, bool LANES2>
SPD_FN void line_apply(const Coef* C, int r0, int step, const Line<L>& ln, double* out) {
  const uint32_t eoff = ln.eoff;
  if (ln.soft) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const Coef* A = C + (r0 + r * step) * L;
#ifdef SPD_FUSED
      // (odd terms: a single one is added to the even sum by itself)
      constexpr bool ODD = LANES2 && L > 3;
      double e = soft_prod(A[0], ln.o[0]), o = ODD ? soft_prod(A[ODD ? 1 : 0], ln.o[ODD ? 1 : 0]) : 0.0;
#pragma unroll
      for (int s = LANES2 ? 2 : 1; s < L; ++s) {
        double& acc = (ODD && s % 2) ? o : e;
        acc = fma(coef_value(A[s], eoff), ln.v[s], acc);
      }
      if (LANES2 && L > 1) e = ODD ? e + o : fma(coef_value(A[L > 1 ? 1 : 0], eoff), ln.v[L > 1 ? 1 : 0], e);
      out[r] = e;
#else
      double p[L];
#pragma unroll
      for (int s = 0; s < L; ++s) p[s] = soft_prod(A[s], ln.o[s]);
      out[r] = sum_terms<L, LANES2>(p);
#endif
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    double A[L];
#pragma unroll
    for (int s = 0; s < L; ++s) A[s] = coef_value(C[(r0 + r * step) * L + s], eoff);
    out[r] = LANES2 ? dot_lanes2<L>(A, ln.v) : dot_seq<L>(A, ln.v);
  }
}

}  // namespace spd
