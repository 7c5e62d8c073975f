// Device-side building blocks of the SD-ADER step: Euler thermodynamics,
// the LLF / HLLC / low-Mach HLLC Riemann solvers and the fixed-order
// contractions.  Every routine reproduces the operation order of the
// reference's NumPy expressions (file:line cited per function) so that the
// FP64 results are bit-identical to it; this file must be compiled with
// --fmad=false so that no a*b+c is fused.
#pragma once
#include <cstdint>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "spd_soft.cuh"

namespace spd {


constexpr int MAXN = 5;   // p <= 4
constexpr int MAXNF = 6;
constexpr int MAXT = 6;   // m <= 5
constexpr int NGH = 2;    // subcell ghost layers (Nghc)

// Block index a kernel body works on and the number of blocks of its grid.
// A plain launch passes the hardware indices; a batched launch over many
// instances passes the block's index within its own instance's share of the
// grid and the size of that share.
struct Blk {
  unsigned id, n;
};
#ifdef __CUDACC__
// Start of a kernel of the step.  The step's kernels are launched with
// programmatic stream serialization (launch_step): a kernel may become
// resident while the one before it drains, waits here until that one's writes
// are visible, and then lets the next one be brought up.  A step of a 32^2
// grid is about 56 dependent kernels of 2-5 us, so what lies between them
// counts.  In a plain launch both instructions do nothing.
__device__ __forceinline__ void step_kernel_begin() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}
__device__ __forceinline__ Blk hw_blk() {
  step_kernel_begin();
  return Blk{blockIdx.x, gridDim.x};
}
#endif

enum Riemann : int { RS_LLF = 0, RS_HLLC = 1, RS_LHLLC = 2 };
enum Limiter : int { LIM_MINMOD = 0, LIM_MONCEN = 1 };
enum BcKind : int { BC_PERIODIC = 0, BC_REFLECTIVE = 1, BC_GRADFREE = 2, BC_IC = 3, BC_EQ = 4, BC_PRESSURE = 5 };

// ---------------------------------------------------------------------------
// Scalars: the physics below is written for a generic scalar S, instantiated
// with double (the step itself, same arithmetic as written) and with the
// forward-mode dual number Dual<N> (value plus N tangents), which the
// adjoint kernels use for the Jacobian-transpose products of local maps.
// ---------------------------------------------------------------------------
template <int N>
struct Dual {
  double v;
  double d[N];
  SPD_FN Dual() {}
  SPD_FN Dual(double x) : v(x) {
#pragma unroll
    for (int i = 0; i < N; ++i) d[i] = 0.0;
  }
};
template <int N>
SPD_FN Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v + b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] + b.d[i];
  return r;
}
template <int N>
SPD_FN Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v - b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] - b.d[i];
  return r;
}
template <int N>
SPD_FN Dual<N> operator-(const Dual<N>& a) {
  Dual<N> r; r.v = -a.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = -a.d[i];
  return r;
}
template <int N>
SPD_FN Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v * b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
  return r;
}
template <int N>
SPD_FN Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v / b.v;
  const double ib = 1.0 / b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
  return r;
}
template <int N> SPD_FN Dual<N> operator+(const Dual<N>& a, double b) { return a + Dual<N>(b); }
template <int N> SPD_FN Dual<N> operator+(double a, const Dual<N>& b) { return Dual<N>(a) + b; }
template <int N> SPD_FN Dual<N> operator-(const Dual<N>& a, double b) { return a - Dual<N>(b); }
template <int N> SPD_FN Dual<N> operator-(double a, const Dual<N>& b) { return Dual<N>(a) - b; }
template <int N>
SPD_FN Dual<N> operator*(const Dual<N>& a, double b) {
  Dual<N> r; r.v = a.v * b;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b;
  return r;
}
template <int N> SPD_FN Dual<N> operator*(double a, const Dual<N>& b) { return b * a; }
template <int N> SPD_FN Dual<N> operator/(const Dual<N>& a, double b) { return a / Dual<N>(b); }
template <int N> SPD_FN Dual<N> operator/(double a, const Dual<N>& b) { return Dual<N>(a) / b; }
template <int N> SPD_FN bool operator<(const Dual<N>& a, const Dual<N>& b) { return a.v < b.v; }
template <int N> SPD_FN bool operator>(const Dual<N>& a, const Dual<N>& b) { return a.v > b.v; }
template <int N> SPD_FN bool operator<=(const Dual<N>& a, const Dual<N>& b) { return a.v <= b.v; }
template <int N> SPD_FN bool operator>=(const Dual<N>& a, const Dual<N>& b) { return a.v >= b.v; }
template <int N> SPD_FN bool operator!=(const Dual<N>& a, const Dual<N>& b) { return a.v != b.v; }
template <int N> SPD_FN bool operator<(const Dual<N>& a, double b) { return a.v < b; }
template <int N> SPD_FN bool operator>(const Dual<N>& a, double b) { return a.v > b; }

// Correctly rounded a / b from a correctly rounded reciprocal rb = RN(1/b)
// by Markstein's correction (P. Markstein, IBM J. Res. Dev. 34(1), 1990;
// Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed., Thm. 5.3):
// q = RN(a*rb) is within one ulp of a/b, the residual a - b*q is exact in
// one fused multiply-add, and RN(q + r*rb) is RN(a/b).  The theorem needs
// every quantity away from underflow and overflow, so the corrected quotient
// is used only when the biased exponents of b lie in [23, 2023] and those of
// a and q in [63, 2023] (then rb and q are normal, and the exact residual, a
// multiple of ulp(b)*ulp(q) >= 2^-1074, is representable).  Outside that
// window: a zero, infinite or NaN numerator or divisor makes q itself the
// IEEE quotient (value and sign) and q is returned; any other operand pair
// (subnormal or huge b, a or q near underflow or overflow) is divided by
// IEEE division.  Three FP64 operations instead of a full division where
// one divisor serves several quotients.
SPD_FN double div_rcp(double a, double b, double rb) {
  const double q = a * rb;
  const double r = fma(-q, b, a);
  const double q2 = fma(r, rb, q);
  // the window tests on the high words (|x|'s exponent is bits 30..20 of
  // the high word; |x| is zero when both words of |x| are, infinite or NaN
  // when the high word of |x| is >= that of infinity): integer pipes, where
  // the same tests on the 64-bit patterns cost about one FP64 instruction
  // per quotient (measured with ncu)
  const unsigned ha = hi_word(a) & 0x7fffffffu, hb = hi_word(b) & 0x7fffffffu, hq = hi_word(q) & 0x7fffffffu;
  const unsigned ea = ha >> 20, eb = hb >> 20, eq = hq >> 20;
  if (eb >= 23u && eb <= 2023u) {
    if ((ha | lo_word(a)) == 0u || ha >= 0x7ff00000u) return q;
    if (ea >= 63u && ea <= 2023u && eq >= 63u && eq <= 2023u) return q2;
  } else if ((hb | lo_word(b)) == 0u || hb >= 0x7ff00000u) {
    return q;
  }
  return div_ieee_slow(a, b);
}

// c ? a : b by value
template <class S>
SPD_FN S sel(bool c, const S& a, const S& b) { return c ? a : b; }
// A Num out of range may have any value, so a choice made by comparing two of
// them stands only if both are in range; a bound (always exact) counts only
// where it is taken.
SPD_FN Num sel(bool c, const Num& a, const Num& b) { return Num(c ? a.v : b.v, a.ok & b.ok); }
template <class S>
SPD_FN S bounded(bool c, const S& a, double bound) { return c ? a : S(bound); }
SPD_FN Num bounded(bool c, const Num& a, double bound) { return Num(c ? a.v : bound, a.ok); }
SPD_FN double half(double x) { return 0.5 * x; }
template <int N> SPD_FN Dual<N> half(const Dual<N>& x) { return 0.5 * x; }
SPD_FN double sval(double x) { return x; }
template <int N> SPD_FN double sval(const Dual<N>& x) { return x.v; }
SPD_FN double ad_sqrt(double x) { return sqrt_soft(x); }
template <int N>
SPD_FN Dual<N> ad_sqrt(const Dual<N>& x) {
  Dual<N> r; r.v = sqrt(x.v);
  const double k = 0.5 / r.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = x.d[i] * k;
  return r;
}
// |x| by clearing the sign bit (integer pipe; the same bits as fabs)
SPD_FN double abs_bits(double x) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
#else
  return fabs(x);
#endif
}
SPD_FN double ad_abs(double x) { return abs_bits(x); }
template <int N>
SPD_FN Dual<N> ad_abs(const Dual<N>& x) {
  if (x.v > 0) return x;
  if (x.v < 0) return -x;
  return Dual<N>(fabs(x.v));
}

// a / b with b's reciprocal prepared by recip_of (double: div_soft; dual
// numbers: plain division, the reciprocal unused)
template <class S>
struct RecipOf {
  using T = S;
};
template <>
struct RecipOf<double> {
  using T = Recip;
};
template <>
struct RecipOf<Num> {
  using T = Recip;
};
SPD_FN double div_by(double a, double b, const Recip& rb) { return div_soft(a, b, rb); }
SPD_FN Recip recip_of(double b) { return recip_soft(b); }
// a prepared reciprocal of a double
using Rcp = typename RecipOf<double>::T;
// a / b
SPD_FN double quot(double a, double b) { return div_by(a, b, recip_of(b)); }
template <int N>
SPD_FN Dual<N> div_by(const Dual<N>& a, const Dual<N>& b, const Dual<N>&) { return a / b; }
template <int N, class R>
SPD_FN Dual<N> div_by(const Dual<N>& a, double b, const R&) { return a / b; }
template <int N>
SPD_FN Dual<N> recip_of(const Dual<N>&) { return Dual<N>(0.0); }

// NumPy's maximum / minimum: NaN in either argument propagates.
template <class S>
SPD_FN S np_max(const S& a, const S& b) { return (a >= b || a != a) ? a : b; }
template <class S>
SPD_FN S np_min(const S& a, const S& b) { return (a <= b || a != a) ? a : b; }
// Order-preserving int64 key of a double's bit pattern b: negatives
// reflected and moved up by one, so that -0 and +0 share the key 0 and every
// other pair of non-NaN values compares as in IEEE (shifts, xor and a
// subtraction on the integer pipes).
SPD_FN long long ieee_key(long long b) {
  const long long s = b >> 63;  // 0 or -1
  return (b ^ (s & 0x7fffffffffffffffLL)) - s;
}
// its inverse (the key 0 gives +0)
SPD_FN long long ieee_key_inverse(long long k) {
  const long long s = k >> 63;
  return (k + s) ^ (s & 0x7fffffffffffffffLL);
}
// The same two functions for doubles on the device, evaluated on the
// integer keys (NaN first): identical results, no FP64-pipe comparison.
#ifdef __CUDA_ARCH__
template <>
__device__ __forceinline__ double np_max<double>(const double& a, const double& b) {
  const long long ba = __double_as_longlong(a), bb = __double_as_longlong(b);
  return (nan_w(a) || (!nan_w(b) && ieee_key(ba) >= ieee_key(bb))) ? a : b;
}
template <>
__device__ __forceinline__ double np_min<double>(const double& a, const double& b) {
  const long long ba = __double_as_longlong(a), bb = __double_as_longlong(b);
  return (nan_w(a) || (!nan_w(b) && ieee_key(ba) <= ieee_key(bb))) ? a : b;
}
#endif
// a > b with IEEE semantics (false when either is NaN; -0 equals +0).  For
// doubles on the device it is evaluated on the integer keys: an FP64
// comparison issues on the FP64 pipe, which bounds the Riemann solvers.
SPD_FN bool fgt(double a, double b) {
#ifdef __CUDA_ARCH__
  return !nan_w(a) && !nan_w(b) && ieee_key(__double_as_longlong(a)) > ieee_key(__double_as_longlong(b));
#else
  return a > b;
#endif
}
// a >= b with IEEE semantics, the same way
SPD_FN bool fge(double a, double b) {
#ifdef __CUDA_ARCH__
  return !nan_w(a) && !nan_w(b) && ieee_key(__double_as_longlong(a)) >= ieee_key(__double_as_longlong(b));
#else
  return a >= b;
#endif
}
SPD_FN bool fgt(const Num& a, const Num& b) { return fgt(a.v, b.v); }
SPD_FN bool fgt(const Num& a, double b) { return fgt(a.v, b); }
SPD_FN bool fgt(double a, const Num& b) { return fgt(a, b.v); }
SPD_FN Num np_max(const Num& a, const Num& b) { return Num(np_max(a.v, b.v), a.ok & b.ok); }
SPD_FN Num np_min(const Num& a, const Num& b) { return Num(np_min(a.v, b.v), a.ok & b.ok); }
template <int N> SPD_FN bool fgt(const Dual<N>& a, const Dual<N>& b) { return a.v > b.v; }
template <int N> SPD_FN bool fgt(const Dual<N>& a, double b) { return a.v > b; }
template <int N> SPD_FN bool fgt(double a, const Dual<N>& b) { return a > b.v; }

// Dual forms: same value; at a tie the derivative is the mean of the two
// arguments' derivatives (the subgradient torch.maximum / torch.minimum
// propagate).
template <int N>
SPD_FN Dual<N> tie_mean(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = 0.5 * (a.d[i] + b.d[i]);
  return r;
}
template <int N>
SPD_FN Dual<N> np_max(const Dual<N>& a, const Dual<N>& b) {
  if (a.v == b.v) return tie_mean(a, b);
  return (a.v >= b.v || a.v != a.v) ? a : b;
}
template <int N>
SPD_FN Dual<N> np_min(const Dual<N>& a, const Dual<N>& b) {
  if (a.v == b.v) return tie_mean(a, b);
  return (a.v <= b.v || a.v != a.v) ? a : b;
}

// Branch control of the piecewise-smooth maps (Riemann solvers, slope
// limiters).  BM = 0: live comparisons (the step); BM = 1: live, and each
// comparison's outcome is appended to ``w`` (a decision tape word);
// BM = 2: the outcomes are read back from ``w`` instead of compared, which
// evaluates the same smooth branch at a perturbed state (the frozen-branch
// map that the adjoint differentiates).
template <int BM>
struct Br {
  unsigned w = 0;
  int k = 0;
};
template <int BM>
SPD_FN bool pick(Br<BM>* br, bool live) {
  if (BM == 0) return live;
  if (BM == 1) {
    if (live) br->w |= (1u << br->k);
    ++br->k;
    return live;
  }
  const bool b = (br->w >> br->k) & 1u;
  ++br->k;
  return b;
}
// |x| whose sign is a recorded decision under BM != 0
template <int BM, class S>
SPD_FN S abs_br(const S& x, Br<BM>* br) {
  if (BM == 0) return ad_abs(x);
  return pick(br, sval(x) >= 0.0) ? x : -x;
}

// Velocity index k (0-based) of the rotated frame used for direction idim:
// np.roll(vels, -idim) (src/sdader_simulator.py:219).
template <int D>
SPD_FN int rvel(int idim, int k) { return 1 + (idim + k) % D; }

// U -> W (src/hydro.py:48-86); the kinetic term sums in the order of the
// velocity list, which is the rotated list inside the Riemann wrapper
// (src/riemann_solver.py:10-29) and the plain list elsewhere.
// ``r0_out`` (optional) receives 1/rho for later quotients by rho.
// ``iso``: the isothermal system (src/hydro.py:84,123,169): the kinetic term
// of the energy is multiplied by 0 and the energy flux by 0.
template <int D, class S>
SPD_FN void prim(const S* U, S* W, double gamma, int idim_order, typename RecipOf<S>::T* r0_out = nullptr,
                 bool iso = false) {
  constexpr int P_ = D + 1;
  W[0] = U[0];
  S K = 0.0;
  const auto r0 = recip_of(U[0]);
  if (r0_out) *r0_out = r0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const int v = rvel<D>(idim_order, k);
    W[v] = div_by(U[v], U[0], r0);
    const S w2 = W[v] * W[v];
    K = (k == 0) ? w2 : K + w2;
  }
  K = K * half(U[0]);
  if (iso) K = K * 0.0;
  W[P_] = (gamma - 1.0) * (U[P_] - K);
}

// W -> U (src/hydro.py:88-125).
template <int D, class S>
SPD_FN void cons(const S* W, S* U, double gamma, int idim_order, bool iso = false, const Rcp* rg = nullptr) {
  constexpr int P_ = D + 1;
  U[0] = W[0];
  S K = 0.0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const int v = rvel<D>(idim_order, k);
    U[v] = W[v] * W[0];
    const S w2 = W[v] * W[v];
    K = (k == 0) ? w2 : K + w2;
  }
  K = K * half(W[0]);
  if (iso) K = K * 0.0;
  U[P_] = div_by(W[P_], gamma - 1.0, rg ? *rg : recip_of(gamma - 1.0)) + K;
}

// Euler flux in the rotated frame of direction idim (src/hydro.py:127-170).
template <int D, class S>
SPD_FN void flux(const S* W, S* F, double gamma, int idim, bool iso = false, const Rcp* rg = nullptr) {
  constexpr int P_ = D + 1;
  const int v1 = rvel<D>(idim, 0);
  S K = 0.0, m = 0.0;
#pragma unroll
  for (int k = D - 1; k >= 0; --k) {
    const int v = rvel<D>(idim, k);
    m = W[0] * W[v];
    const S mv = m * W[v];
    K = (k == D - 1) ? mv : K + mv;
    F[v] = m * W[v1];
  }
  const S E = div_by(W[P_], gamma - 1.0, rg ? *rg : recip_of(gamma - 1.0)) + half(K);
  F[0] = m;
  F[v1] = m * W[v1] + W[P_];
  F[P_] = W[v1] * (E + W[P_]);
  if (iso) F[P_] = F[P_] * 0.0;
}

// Sound speed with floor (src/hydro.py:3-46).
template <class S, int BM = 0>
SPD_FN S sound_speed(const S& P, const S& rho, double gamma, double min_c2,
                                         Br<BM>* br = nullptr,
                                         const typename RecipOf<S>::T* rrho = nullptr) {
  S c2 = div_by(gamma * P, rho, rrho ? *rrho : recip_of(rho));
  c2 = bounded(pick(br, fgt(c2, min_c2)), c2, min_c2);
  return ad_sqrt(c2);
}

// LLF (src/riemann_solver.py:31-65).
template <int D, class S, int BM = 0>
SPD_FN void llf(const S* WL, const S* WR, const S* UL, const S* UR, S* F, double gamma,
                                    double min_c2, int idim, Br<BM>* br = nullptr, const typename RecipOf<S>::T* rL = nullptr,
                                    const typename RecipOf<S>::T* rR = nullptr, bool iso = false,
                                    const Rcp* rg = nullptr) {
  constexpr int V = D + 2, P_ = D + 1;
  const int v1 = rvel<D>(idim, 0);
  S FL[V], FR[V];
  flux<D>(WL, FL, gamma, idim, iso, rg);
  flux<D>(WR, FR, gamma, idim, iso, rg);
  const S cL = sound_speed(WL[P_], WL[0], gamma, min_c2, br, rL) + abs_br(WL[v1], br);
  const S cR = sound_speed(WR[P_], WR[0], gamma, min_c2, br, rR) + abs_br(WR[v1], br);
  const S cmax = sel(pick(br, fgt(cL, cR)), cL, cR);
  const S hc = half(cmax);
#pragma unroll
  for (int v = 0; v < V; ++v) F[v] = half(FR[v] + FL[v]) - hc * (UR[v] - UL[v]);
}

// HLLC (src/riemann_solver.py:67-145) and its low-Mach variant (:147-212).
// Only the branch the reference's np.where chain selects is evaluated.
template <int D, class S, int BM = 0>
SPD_FN void hllc(const S* WL, const S* WR, const S* UL, const S* UR, S* F, double gamma,
                                     double min_c2, int idim, bool low_mach, Br<BM>* br = nullptr,
                                     const typename RecipOf<S>::T* rL = nullptr, const typename RecipOf<S>::T* rR = nullptr, bool iso = false) {
  // vstar and sR decide between states that do not hang on them, and their
  // range flags would be lost there
  static_assert(!std::is_same<S, Num>::value, "HLLC's choices carry no range flag");
  constexpr int P_ = D + 1;
  const int v1 = rvel<D>(idim, 0);
  const S cL = sound_speed(WL[P_], WL[0], gamma, min_c2, br, rL) + abs_br(WL[v1], br);
  const S cR = sound_speed(WR[P_], WR[0], gamma, min_c2, br, rR) + abs_br(WR[v1], br);
  const S cmax = sel(pick(br, fgt(cL, cR)), cL, cR);
  const S vL = WL[v1], vR = WR[v1];
  const S sL = sel(pick(br, fgt(vR, vL)), vL, vR) - cmax;
  const S sR = sel(pick(br, fgt(vL, vR)), vL, vR) + cmax;
  const S rcL = WL[0] * (vL - sL);
  const S rcR = WR[0] * (sR - vR);
  const S den = rcR + rcL;
  const auto rden = recip_of(den);
  const S vstar = div_by(rcR * vR + rcL * vL + (WL[P_] - WR[P_]), den, rden);
  S Pstar;
  if (low_mach) {
    S mx, Mach;
    if constexpr (BM == 0) {
      mx = np_max(ad_abs(vL), ad_abs(vR)) / cmax;
      Mach = np_min(S(1.0), mx);
    } else {
      const S aL = abs_br(vL, br), aR = abs_br(vR, br);
      mx = (pick(br, aL >= aR || aL != aL) ? aL : aR) / cmax;
      Mach = pick(br, S(1.0) <= mx) ? S(1.0) : mx;
    }
    const S phi = Mach * (2.0 - Mach);
    Pstar = div_by(rcR * WL[P_] + rcL * WR[P_] + phi * rcL * rcR * (vL - vR), den, rden);
  } else {
    Pstar = div_by(rcR * WL[P_] + rcL * WR[P_] + rcL * rcR * (vL - vR), den, rden);
  }
  S r, vg, Pg, e;
  if constexpr (BM == 0) {
    // the left and right star states are the same formulas with the sides
    // swapped: one path with per-lane operands, so a warp whose lanes take
    // both sides (an FP64 warp instruction costs the same with any number of
    // active lanes) evaluates the reciprocal and quotients once
    if (fgt(sL, 0.0)) {
      r = WL[0]; vg = vL; Pg = WL[P_]; e = UL[P_];
    } else if (fgt(vstar, 0.0) || fgt(sR, 0.0)) {
      const bool lft = fgt(vstar, 0.0);
      const S s = sel(lft, sL, sR), v = sel(lft, vL, vR);
      const S w0 = sel(lft, WL[0], WR[0]), wP = sel(lft, WL[P_], WR[P_]), uP = sel(lft, UL[P_], UR[P_]);
      const S d = s - vstar;
      const auto rd = recip_of(d);
      r = div_by(w0 * (s - v), d, rd);
      e = div_by((s - v) * uP - wP * v + Pstar * vstar, d, rd);
      vg = vstar; Pg = Pstar;
    } else {
      r = WR[0]; vg = vR; Pg = WR[P_]; e = UR[P_];
    }
  } else if (pick(br, fgt(sL, 0.0))) {
    r = WL[0]; vg = vL; Pg = WL[P_]; e = UL[P_];
  } else if (pick(br, fgt(vstar, 0.0))) {
    const S d = sL - vstar;
    const auto rd = recip_of(d);
    r = div_by(WL[0] * (sL - vL), d, rd);
    e = div_by((sL - vL) * UL[P_] - WL[P_] * vL + Pstar * vstar, d, rd);
    vg = vstar; Pg = Pstar;
  } else if (pick(br, fgt(sR, 0.0))) {
    const S d = sR - vstar;
    const auto rd = recip_of(d);
    r = div_by(WR[0] * (sR - vR), d, rd);
    e = div_by((sR - vR) * UR[P_] - WR[P_] * vR + Pstar * vstar, d, rd);
    vg = vstar; Pg = Pstar;
  } else {
    r = WR[0]; vg = vR; Pg = WR[P_]; e = UR[P_];
  }
  F[0] = r * vg;
  F[v1] = F[0] * vg + Pg;
  F[P_] = vg * (e + Pg);
  if (D > 1) {
    const bool left = pick(br, fgt(vstar, 0.0));
#pragma unroll
    for (int k = 1; k < D; ++k) {
      const int v = rvel<D>(idim, k);
      F[v] = F[0] * sel(left, WL[v], WR[v]);
    }
  }
  if (iso) F[P_] = F[P_] * 0.0;
}

// U -> W (plain velocity order) and the Euler flux along direction d in the
// rotated frame, in 1D and 2D with their products on the integer pipes as
// above: k_interior 11.2 -> 10.6 ms and k_fv_candidate 1.22 -> 1.14 ms at
// 512^2, p=3.  In 3D the integer pipes are the busier ones already (48^3,
// p=2: 7.45 -> 7.87 and 1.2 -> 1.31 ms), so their products stay FP64.
template <int D>
struct NumEuler {
#if defined(__CUDA_ARCH__) && !defined(SPD_FUSED)
  static constexpr bool value = D <= 2;
#else
  static constexpr bool value = false;
#endif
};
#if defined(__CUDA_ARCH__)
template <int D>
__device__ __noinline__ void prim_slow(const double* U, double* W, double gamma, int idim_order, bool iso) {
  prim<D>(U, W, gamma, idim_order, nullptr, iso);
}
#endif
template <int D>
SPD_FN void prim_num(const double* U, double* W, double gamma, int idim_order, Recip* r0, bool iso) {
  constexpr int V = D + 2;
  Num u[V], w[V];
  uint32_t ok = 0x40000000u;
#pragma unroll
  for (int v = 0; v < V; ++v) u[v] = Num(U[v]);
  prim<D>(u, w, gamma, idim_order, r0, iso);
#pragma unroll
  for (int v = 0; v < V; ++v) {
    ok &= w[v].ok;
    W[v] = w[v].v;
  }
#if defined(__CUDA_ARCH__)
  if (ok != 0u) return;
  double us[V], ws[V];
#pragma unroll
  for (int v = 0; v < V; ++v) us[v] = U[v];
  prim_slow<D>(us, ws, gamma, idim_order, iso);
#pragma unroll
  for (int v = 0; v < V; ++v) W[v] = ws[v];
#endif
}
template <int D>
SPD_FN void prims(const double* U, double* W, double gamma, bool iso) {
  if constexpr (NumEuler<D>::value) prim_num<D>(U, W, gamma, 0, nullptr, iso);
  else prim<D>(U, W, gamma, 0, nullptr, iso);
}
// the solver of a kernel instantiated for SV
template <int SV>
SPD_FN int solver_of(int solver) {
  if (SV == RS_LLF) return RS_LLF;
  if (SV == RS_HLLC) return solver == RS_LHLLC ? RS_LHLLC : RS_HLLC;
  return solver;
}
#ifndef SPD_FUSED
// LLF in plain FP64 arithmetic, out of line
template <int D>
#ifdef __CUDA_ARCH__
__device__ __noinline__
#else
inline
#endif
    void
    llf_plain(const double* WL, const double* WR, const double* UL, const double* UR, double* F, double gamma,
              double min_c2, int idim, bool iso) {
  llf<D, double>(WL, WR, UL, UR, F, gamma, min_c2, idim, (Br<0>*)nullptr, nullptr, nullptr, iso);
}
#endif
// Riemann wrapper (src/riemann_solver.py:10-29): inputs conservative
// (prims=false) or primitive (prims=true); rotated velocity order.
template <int D, class S, int BM = 0>
SPD_FN void riemann(int solver, const S* ML, const S* MR, S* F, double gamma, double min_c2, int idim, bool prims,
                       Br<BM>* br = nullptr, bool iso = false, const Rcp* rg = nullptr) {
  constexpr int V = D + 2;
  S WL[V], WR[V], UL[V], UR[V];
  typename RecipOf<S>::T rL, rR;  // 1/rho of the two states when the conversion computed it
  const typename RecipOf<S>::T* prL = nullptr;
  const typename RecipOf<S>::T* prR = nullptr;
  if (prims) {
#pragma unroll
    for (int v = 0; v < V; ++v) { WL[v] = ML[v]; WR[v] = MR[v]; }
    cons<D>(WL, UL, gamma, idim, iso, rg);
    cons<D>(WR, UR, gamma, idim, iso, rg);
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) { UL[v] = ML[v]; UR[v] = MR[v]; }
    bool done = false;
    if constexpr (BM == 0 && std::is_same<S, double>::value && NumEuler<D>::value) {
      if (solver != RS_LLF) {
        // the conversions' products on the integer pipes, HLLC's own not
        prim_num<D>(UL, WL, gamma, idim, &rL, iso);
        prim_num<D>(UR, WR, gamma, idim, &rR, iso);
        done = true;
      }
    }
    if (!done) {
      prim<D>(UL, WL, gamma, idim, &rL, iso);
      prim<D>(UR, WR, gamma, idim, &rR, iso);
    }
    prL = &rL;
    prR = &rR;
  }
#ifndef SPD_FUSED
  if constexpr (BM == 0 && D <= 2 && std::is_same<S, double>::value) {
    // (1D, 2D) LLF's products on the integer pipes, the conversions' on the FP64 pipe:
    // an even split of the two (251x190, p=3: 1.40 -> 1.15 ms; all on the
    // integer pipes 1.19).  HLLC, whose products hang on one another, keeps
    // the FP64 pipe (512^2: 2.81 ms, 3.14 with integer products, 3.32 with
    // those of the conversions too).  A problem with a value out of their
    // range is solved again in plain FP64 arithmetic.
    if (solver == RS_LLF) {
      Num wl[V], wr[V], ul[V], ur[V], f[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        wl[v] = Num(WL[v]);
        wr[v] = Num(WR[v]);
        ul[v] = Num(UL[v]);
        ur[v] = Num(UR[v]);
      }
      llf<D, Num>(wl, wr, ul, ur, f, gamma, min_c2, idim, (Br<0>*)nullptr, prL, prR, iso, rg);
      uint32_t ok = 0x40000000u;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        ok &= f[v].ok;
        F[v] = f[v].v;
      }
      if (ok != 0u) return;
      double a[V], b[V], c[V], e[V], o[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        a[v] = WL[v];
        b[v] = WR[v];
        c[v] = UL[v];
        e[v] = UR[v];
      }
      llf_plain<D>(a, b, c, e, o, gamma, min_c2, idim, iso);
#pragma unroll
      for (int v = 0; v < V; ++v) F[v] = o[v];
      return;
    }
  }
#endif
  if (solver == RS_LLF) llf<D, S, BM>(WL, WR, UL, UR, F, gamma, min_c2, idim, br, prL, prR, iso, rg);
  else hllc<D, S, BM>(WL, WR, UL, UR, F, gamma, min_c2, idim, solver == RS_LHLLC, br, prL, prR, iso);
}

#if defined(__CUDA_ARCH__)
template <int D>
__device__ __noinline__ void euler_slow(const double* U, double* W, double* F, double gamma, int d, bool iso) {
  prim<D>(U, W, gamma, 0, nullptr, iso);
  if (F == nullptr) return;
  double Wr[D + 2], Fr[D + 2];
  Wr[0] = W[0];
  Wr[D + 1] = W[D + 1];
#pragma unroll
  for (int q = 0; q < D; ++q) Wr[1 + q] = W[rvel<D>(d, q)];
  flux<D>(Wr, Fr, gamma, 0, iso);
  F[0] = Fr[0];
  F[D + 1] = Fr[D + 1];
#pragma unroll
  for (int q = 0; q < D; ++q) F[rvel<D>(d, q)] = Fr[1 + q];
}
#endif
// flux of the conservative state U; store(v, F_v) takes its components
template <int D, class Store>
SPD_FN void euler_flux(const double* U, double gamma, int d, bool iso, const Rcp* rg, Store store) {
  constexpr int V = D + 2;
  using S = typename std::conditional<NumEuler<D>::value, Num, double>::type;
  // the velocities in the rotated order of direction d, as flux's own order
  // for direction 0
  S u[V], w[V], wr[V], f[V];
#pragma unroll
  for (int v = 0; v < V; ++v) u[v] = S(U[v]);
  prim<D>(u, w, gamma, 0, nullptr, iso);
  wr[0] = w[0];
  wr[D + 1] = w[D + 1];
#pragma unroll
  for (int q = 0; q < D; ++q) {
    S x = w[1 + q];
    if (D > 1) x = sel(d == 1, w[1 + (q + 1) % D], x);
    if (D > 2) x = sel(d == 2, w[1 + (q + 2) % D], x);
    wr[1 + q] = x;
  }
  flux<D>(wr, f, gamma, 0, iso, rg);
#if defined(__CUDA_ARCH__)
  if constexpr (NumEuler<D>::value) {
    uint32_t ok = 0x40000000u;
#pragma unroll
    for (int v = 0; v < V; ++v) ok &= f[v].ok;
    double fs[V];
    if (ok != 0u) {
#pragma unroll
      for (int v = 0; v < V; ++v) fs[v] = f[v].v;
    } else {
      double us[V], ws[V], fl[V];
#pragma unroll
      for (int v = 0; v < V; ++v) us[v] = U[v];
      euler_slow<D>(us, ws, fl, gamma, d, iso);
      fs[0] = fl[0];
      fs[D + 1] = fl[D + 1];
#pragma unroll
      for (int q = 0; q < D; ++q) fs[1 + q] = fl[rvel<D>(d, q)];
    }
    store(0, fs[0]);
    store(D + 1, fs[D + 1]);
#pragma unroll
    for (int q = 0; q < D; ++q) store(rvel<D>(d, q), fs[1 + q]);
    return;
  }
#endif
  store(0, sval(f[0]));
  store(D + 1, sval(f[D + 1]));
#pragma unroll
  for (int q = 0; q < D; ++q) store(rvel<D>(d, q), sval(f[1 + q]));
}

// One output of a 1D operator contraction: sum_s A[s] * x[s], left to right,
// or (dot_lanes2) in the order of an einsum over the contiguous x axis, even
// and odd terms accumulated separately and then added (src/transforms.py:3-25).
template <int L>
SPD_FN double dot_seq(const double* A, const double* x) {
  double acc = A[0] * x[0];
#pragma unroll
  for (int s = 1; s < L; ++s) acc = acc + A[s] * x[s];
  return acc;
}
template <int L>
SPD_FN double dot_lanes2(const double* A, const double* x) {
  double e = A[0] * x[0];
  if (L == 1) return e;
  double o = A[1] * x[1];
#pragma unroll
  for (int s = 2; s < L; ++s) {
    if (s % 2 == 0) e = e + A[s] * x[s];
    else o = o + A[s] * x[s];
  }
  return e + o;
}

// Limiters (src/muscl.py:12-59); NaN semantics follow the np.where forms.
// (comparisons through fgt / fge: integer keys on the device)
SPD_FN double minmod(double SL, double SR) {
  double r = quot(SR, SL);
  r = fgt(1.0, r) ? r : 1.0;
  return (fgt(r, 0.0) ? r : 0.0) * SL;
}
SPD_FN double np_sign(double x) {
  return fgt(x, 0.0) ? 1.0 : (fgt(0.0, x) ? -1.0 : ((fge(x, 0.0) && fge(0.0, x)) ? 0.0 : x));
}
SPD_FN double moncen(double dUL, double dUR, double dxL, double dxR, double dxM) {
  const double dUC = quot(dxL * dUL + dxR * dUR, dxL + dxR);
  const Rcp rM = recip_of(dxM);
  double slope = np_min(abs_bits(div_by(2.0 * dUL * dxL, dxM, rM)), abs_bits(div_by(2.0 * dUR * dxR, dxM, rM)));
  slope = np_sign(dUC) * np_min(slope, abs_bits(dUC));
  return fge(dUL * dUR, 0.0) ? slope : 0.0;
}

// Limited slope with its branch as a decision code (BM as in Br): minmod
// code = 0 (0*SL), 1 (ratio*SL), 2 (SL); moncen code = bit 0 zero slope,
// bits 1-2 sign of the centred slope (0, +, -), bits 3-4 the minimum taken
// (1: left, 2: right, 3: centred), bits 5-6 the sign inside its |.|.
SPD_FN int sign_code(double x) { return (x > 0.0) ? 1 : ((x < 0.0) ? 2 : 0); }
SPD_FN double code_sign(int c) { return c == 1 ? 1.0 : (c == 2 ? -1.0 : 0.0); }
template <int BM>
SPD_FN double limiter_br(int limiter, double SL, double SR, double hl, double hr, double hm,
                                             unsigned char* code) {
  if (limiter == LIM_MINMOD) {
    if (BM == 2) {
      const int c = *code;
      if (c == 1) return (SR / SL) * SL;
      return (c == 2 ? 1.0 : 0.0) * SL;
    }
    const double v = minmod(SL, SR);
    if (BM == 1) {
      const double r = SR / SL;
      *code = (unsigned char)((r < 1.0) ? ((r > 0.0) ? 1 : 0) : 2);
    }
    return v;
  }
  const double dUC = (hl * SL + hr * SR) / (hl + hr);
  const double q1 = 2.0 * SL * hl / hm, q2 = 2.0 * SR * hr / hm;
  if (BM == 2) {
    const int c = *code;
    if (c & 1) return 0.0;
    const int sel = (c >> 3) & 3;
    const double q = sel == 1 ? q1 : (sel == 2 ? q2 : dUC);
    return code_sign((c >> 1) & 3) * (code_sign((c >> 5) & 3) * q);
  }
  const double v = moncen(SL, SR, hl, hr, hm);
  if (BM == 1) {
    const double c1 = fabs(q1), c2 = fabs(q2), c3 = fabs(dUC);
    const double m12 = np_min(c1, c2);
    const int sel12 = (c1 <= c2 || c1 != c1) ? 1 : 2;
    const int sel = (m12 <= c3 || m12 != m12) ? sel12 : 3;
    const double q = sel == 1 ? q1 : (sel == 2 ? q2 : dUC);
    const int zero = (SL * SR >= 0.0) ? 0 : 1;
    *code = (unsigned char)(zero | (sign_code(dUC) << 1) | (sel << 3) | (sign_code(q) << 5));
  }
  return v;
}

}  // namespace spd
