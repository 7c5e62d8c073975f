// Operator contractions along lines of points, with the products on the
// integer pipes (spd_soft.cuh).
#pragma once
#include "spd_device.cuh"

namespace spd {

// L values along one line of points, prepared once for the several operator
// rows that are applied to them.
template <int L>
struct Line {
  double v[L];
#ifndef SPD_FUSED
  Opnd o[L];
  bool soft;
  uint32_t eoff;
#endif
};
// ``use``: the operator's entries are all within coef_in_range.  A line is
// multiplied on the integer pipes when every value is a zero or within
// opnd_of's window (no subnormal, infinity or NaN, and with entries in range
// no product outside the normal range).  ``eoff``: the operator is the
// stored one times 2^k (exact), given as k << 20 with |k| <= 64.
template <int L>
SPD_FN void line_ready(Line<L>& ln, int use, uint32_t eoff = 0u) {
#ifndef SPD_FUSED
  uint32_t ok = use ? 0x40000000u : 0u;
#pragma unroll
  for (int s = 0; s < L; ++s) {
    ln.o[s] = opnd_of(ln.v[s], ok);
    ln.o[s].e += eoff;
  }
  ln.soft = ok != 0u;
  ln.eoff = eoff;
#endif
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
template <int L, int R, bool LANES2>
SPD_FN void line_apply(const Coef* C, int r0, int step, const Line<L>& ln, double* out) {
#ifndef SPD_FUSED
  if (ln.soft) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double p[L];
#pragma unroll
      for (int s = 0; s < L; ++s) p[s] = soft_prod(C[(r0 + r * step) * L + s], ln.o[s]);
      out[r] = sum_terms<L, LANES2>(p);
    }
    return;
  }
  const uint32_t eoff = ln.eoff;
#else
  const uint32_t eoff = 0u;
#endif
#pragma unroll
  for (int r = 0; r < R; ++r) {
    double A[L];
#pragma unroll
    for (int s = 0; s < L; ++s) A[s] = coef_value(C[(r0 + r * step) * L + s], eoff);
    out[r] = LANES2 ? dot_lanes2<L>(A, ln.v) : dot_seq<L>(A, ln.v);
  }
}

}  // namespace spd
