// Reverse-mode vector-Jacobian products of the pointwise Euler maps of the
// step (primitive/conservative conversion, Euler flux, LLF and HLLC /
// low-Mach HLLC Riemann solvers, src/hydro.py and src/riemann_solver.py).
// Each routine recomputes the forward values with the forward's own
// arithmetic (so every branch is taken as in the forward step) and then
// accumulates the adjoints of its inputs.  Derivative conventions at kinks
// follow the dual-number forms in spd_device.cuh: |x| has derivative 0 at
// 0, a tie of numpy-style maximum/minimum gives each argument half, and a
// select (a > b ? a : b) differentiates the selected argument.
#pragma once
#include "spd_device.cuh"

namespace spd {

SPD_FN double sgn0(double x) { return (x > 0.0) ? 1.0 : ((x < 0.0) ? -1.0 : 0.0); }

// W = prim(U): Ua += (dW/dU)^T Wa
// (Adjoint-only arithmetic below uses reciprocals freely: its values need
// no bitwise match; values that decide a branch are recomputed exactly.)
template <int D>
SPD_FN void prim_vjp_add(const double* U, const double* Wa, double* Ua, double gamma) {
  constexpr int P_ = D + 1;
  const double r = U[0];
  const double rr = quot(1.0, r);
  double w[D + 2], ks = 0.0;
#pragma unroll
  for (int v = 1; v <= D; ++v) {
    w[v] = U[v] * rr;
    ks = fma(w[v], w[v], ks);
  }
  const double Pa = Wa[P_];
  const double Ka = -(gamma - 1.0) * Pa;
  Ua[P_] -= Ka;
  const double ksa = 0.5 * Ka * r;
  double ra = fma(0.5 * Ka, ks, Wa[0]);
#pragma unroll
  for (int v = 1; v <= D; ++v) {
    const double wa = fma(2.0 * w[v], ksa, Wa[v]) * rr;
    Ua[v] += wa;
    ra = fma(-wa, w[v], ra);
  }
  Ua[0] += ra;
}

// U = cons(W): Wa += (dU/dW)^T Ua
template <int D>
SPD_FN void cons_vjp_add(const double* W, const double* Ua, double* Wa, double gamma) {
  constexpr int P_ = D + 1;
  const double r = W[0];
  double ks = 0.0;
#pragma unroll
  for (int v = 1; v <= D; ++v) ks = fma(W[v], W[v], ks);
  Wa[P_] = fma(Ua[P_], quot(1.0, gamma - 1.0), Wa[P_]);
  const double ha = 0.5 * Ua[P_];
  const double ksa = ha * r;
  double ra = fma(ha, ks, Ua[0]);
#pragma unroll
  for (int v = 1; v <= D; ++v) {
    Wa[v] += fma(2.0 * W[v], ksa, Ua[v] * r);
    ra = fma(Ua[v], W[v], ra);
  }
  Wa[0] += ra;
}

// F = flux(W) in direction idim: Wa += (dF/dW)^T Fa
template <int D>
SPD_FN void flux_vjp_add(const double* W, const double* Fa, double* Wa, double gamma, int idim) {
  constexpr int P_ = D + 1;
  const int v1 = rvel<D>(idim, 0);
  const double r = W[0], u = W[v1], P = W[P_];
  double ks = 0.0;
#pragma unroll
  for (int v = 1; v <= D; ++v) ks = fma(W[v], W[v], ks);
  const double rg = quot(1.0, gamma - 1.0);
  const double hk = 0.5 * ks;
  const double E = fma(P, rg, r * hk);
  const double Ea = Fa[P_] * u;
  const double m1 = Fa[v1] * u;
  double ra = fma(Ea, hk, fma(m1, u, Fa[0] * u));
  double ua = fma(Fa[P_], E + P, fma(2.0 * r, m1, Fa[0] * r));
  const double Ear = Ea * r;
#pragma unroll
  for (int k = 1; k < D; ++k) {
    const int vt = rvel<D>(idim, k);
    const double a = Fa[vt] * W[vt], b = Fa[vt] * r;
    ra = fma(a, u, ra);
    ua = fma(a, r, ua);
    Wa[vt] = fma(b, u, Wa[vt]);
  }
#pragma unroll
  for (int v = 1; v <= D; ++v) Wa[v] = fma(Ear, W[v], Wa[v]);
  Wa[0] += ra;
  Wa[v1] += ua;
  Wa[P_] += fma(Ea, rg, fma(Fa[P_], u, Fa[v1]));
}

// c = sound_speed(P, rho) (floored): adds dc/dP * ca, dc/drho * ca
SPD_FN void sound_speed_vjp_add(double P, double rho, double gamma, double min_c2, double ca, double& Pa,
                                double& ra) {
  const Rcp q = recip_of(rho);
  const double c2 = div_by(gamma * P, rho, q);  // the forward's quotient (decides the floor)
  if (!fgt(c2, min_c2)) return;
  const double x = ca * quot(0.5, ad_sqrt(c2)) * div_by(1.0, rho, q);
  Pa = fma(x, gamma, Pa);
  ra = fma(-x, c2, ra);
}

// LLF / HLLC flux F(ML, MR): (MLa, MRa) = J^T Fa (written).  prims: the
// inputs are primitive states (else conservative), as in riemann().
template <int D>
SPD_FN void riemann_vjp_rev(int solver, const double* ML, const double* MR, const double* Fa, double* MLa,
                            double* MRa, double gamma, double min_c2, int idim, bool prims) {
  constexpr int V = D + 2, P_ = D + 1;
  const int v1 = rvel<D>(idim, 0);
  double WL[V], WR[V], UL[V], UR[V];
  if (prims) {
#pragma unroll
    for (int v = 0; v < V; ++v) { WL[v] = ML[v]; WR[v] = MR[v]; }
    cons<D>(WL, UL, gamma, idim);
    cons<D>(WR, UR, gamma, idim);
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) { UL[v] = ML[v]; UR[v] = MR[v]; }
    prim<D>(UL, WL, gamma, idim);
    prim<D>(UR, WR, gamma, idim);
  }
  double WLa[V], WRa[V], ULa[V], URa[V];
#pragma unroll
  for (int v = 0; v < V; ++v) { WLa[v] = 0.0; WRa[v] = 0.0; ULa[v] = 0.0; URa[v] = 0.0; }
  const double cL = sound_speed(WL[P_], WL[0], gamma, min_c2) + fabs(WL[v1]);
  const double cR = sound_speed(WR[P_], WR[0], gamma, min_c2) + fabs(WR[v1]);
  const bool Lmax = fgt(cL, cR);
  const double cmax = Lmax ? cL : cR;
  double cmax_a = 0.0;
  if (solver == RS_LLF) {
    const double hc = 0.5 * cmax;
    double FLa[V], FRa[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      FLa[v] = 0.5 * Fa[v];
      FRa[v] = 0.5 * Fa[v];
      URa[v] -= hc * Fa[v];
      ULa[v] += hc * Fa[v];
      cmax_a -= 0.5 * Fa[v] * (UR[v] - UL[v]);
    }
    flux_vjp_add<D>(WL, FLa, WLa, gamma, idim);
    flux_vjp_add<D>(WR, FRa, WRa, gamma, idim);
  } else {
    const bool low_mach = solver == RS_LHLLC;
    const double vL = WL[v1], vR = WR[v1];
    const bool minL = fgt(vR, vL), maxL = fgt(vL, vR);
    const double sL = (minL ? vL : vR) - cmax;
    const double sR = (maxL ? vL : vR) + cmax;
    const double rcL = WL[0] * (vL - sL);
    const double rcR = WR[0] * (sR - vR);
    const double den = rcR + rcL;
    const Rcp qden = recip_of(den);
    const double rden = div_by(1.0, den, qden);
    const double vstar = div_by(rcR * vR + rcL * vL + (WL[P_] - WR[P_]), den, qden);
    double phi = 1.0, Mach = 0.0, mx = 0.0;
    if (low_mach) {
      mx = quot(np_max(fabs(vL), fabs(vR)), cmax);
      Mach = np_min(1.0, mx);
      phi = Mach * (2.0 - Mach);
    }
    const double Pstar = low_mach ? div_by(rcR * WL[P_] + rcL * WR[P_] + phi * rcL * rcR * (vL - vR), den, qden)
                                  : div_by(rcR * WL[P_] + rcL * WR[P_] + rcL * rcR * (vL - vR), den, qden);
    int region;
    double r, vg, Pg, e, dd = 1.0, rdd = 1.0;
    if (fgt(sL, 0.0)) {
      region = 0; r = WL[0]; vg = vL; Pg = WL[P_]; e = UL[P_];
    } else if (fgt(vstar, 0.0) || fgt(sR, 0.0)) {
      // left (region 1) and right (region 2) star states: one path with
      // per-lane operands (both sides of a warp evaluate it once)
      const bool lft = fgt(vstar, 0.0);
      region = lft ? 1 : 2;
      const double s = lft ? sL : sR, v = lft ? vL : vR;
      const double w0 = lft ? WL[0] : WR[0], wP = lft ? WL[P_] : WR[P_], uP = lft ? UL[P_] : UR[P_];
      dd = s - vstar;
      const Rcp qd = recip_of(dd);
      rdd = div_by(1.0, dd, qd);
      r = div_by(w0 * (s - v), dd, qd);
      e = div_by((s - v) * uP - wP * v + Pstar * vstar, dd, qd);
      vg = vstar; Pg = Pstar;
    } else {
      region = 3; r = WR[0]; vg = vR; Pg = WR[P_]; e = UR[P_];
    }
    const double F0 = r * vg;
    const bool left = fgt(vstar, 0.0);
    // reverse of the flux assembly
    double F0a = Fa[0] + Fa[v1] * vg;
#pragma unroll
    for (int k = 1; k < D; ++k) {
      const int vt = rvel<D>(idim, k);
      const double wv = left ? WL[vt] : WR[vt];
      F0a = fma(Fa[vt], wv, F0a);
      if (left) WLa[vt] = fma(Fa[vt], F0, WLa[vt]);
      else WRa[vt] = fma(Fa[vt], F0, WRa[vt]);
    }
    const double ra = F0a * vg;
    const double vga = F0a * r + Fa[v1] * F0 + Fa[P_] * (e + Pg);
    const double Pga = Fa[v1] + Fa[P_] * vg;
    const double ea = Fa[P_] * vg;
    double vstar_a = 0.0, Pstar_a = 0.0, sL_a = 0.0, sR_a = 0.0, vL_a = 0.0, vR_a = 0.0;
    if (region == 0) {
      WLa[0] += ra; vL_a += vga; WLa[P_] += Pga; ULa[P_] += ea;
    } else if (region == 3) {
      WRa[0] += ra; vR_a += vga; WRa[P_] += Pga; URa[P_] += ea;
    } else {
      vstar_a += vga;
      Pstar_a += Pga;
      const bool isL = region == 1;
      const double rho = isL ? WL[0] : WR[0];
      const double vK = isL ? vL : vR;
      const double sK = isL ? sL : sR;
      const double EK = isL ? UL[P_] : UR[P_];
      const double PK = isL ? WL[P_] : WR[P_];
      // r = rho (sK - vK) / dd, dd = sK - vstar (rdd = 1 / dd from above)
      double rho_a = ra * (sK - vK) * rdd;
      double sK_a = (ra * rho - ra * r) * rdd;
      double vK_a = -ra * rho * rdd;
      vstar_a += ra * r * rdd;
      // e = ((sK - vK) EK - PK vK + Pstar vstar) / dd
      const double na = ea * rdd;
      sK_a += -na * e + na * EK;
      vstar_a += na * e + na * Pstar;
      vK_a += -na * EK - na * PK;
      const double EK_a = na * (sK - vK);
      const double PK_a = -na * vK;
      Pstar_a = fma(na, vstar, Pstar_a);
      if (isL) {
        WLa[0] += rho_a; vL_a += vK_a; sL_a += sK_a; ULa[P_] += EK_a; WLa[P_] += PK_a;
      } else {
        WRa[0] += rho_a; vR_a += vK_a; sR_a += sK_a; URa[P_] += EK_a; WRa[P_] += PK_a;
      }
    }
    // Pstar = (rcR PL + rcL PR + phi rcL rcR (vL - vR)) / den
    double rcL_a = 0.0, rcR_a = 0.0, den_a = 0.0;
    {
      const double na = Pstar_a * rden;
      den_a = fma(-na, Pstar, den_a);
      rcR_a += na * WL[P_] + na * phi * rcL * (vL - vR);
      rcL_a += na * WR[P_] + na * phi * rcR * (vL - vR);
      WLa[P_] = fma(na, rcR, WLa[P_]);
      WRa[P_] = fma(na, rcL, WRa[P_]);
      vL_a += na * phi * rcL * rcR;
      vR_a -= na * phi * rcL * rcR;
      if (low_mach) {
        const double phi_a = na * rcL * rcR * (vL - vR);
        const double Mach_a = phi_a * (2.0 - 2.0 * Mach);
        // Mach = np_min(1, mx)
        const double wmx = (mx == 1.0) ? 0.5 : ((1.0 <= mx || mx != mx) ? 0.0 : 1.0);
        const double mx_a = Mach_a * wmx;
        // mx = np_max(|vL|, |vR|) / cmax
        cmax_a -= quot(mx_a * mx, cmax);
        const double aL = fabs(vL), aR = fabs(vR);
        const double m_a = quot(mx_a, cmax);
        double wL, wR;
        if (aL == aR) { wL = 0.5; wR = 0.5; }
        else if (aL >= aR || aL != aL) { wL = 1.0; wR = 0.0; }
        else { wL = 0.0; wR = 1.0; }
        vL_a += m_a * wL * sgn0(vL);
        vR_a += m_a * wR * sgn0(vR);
      }
    }
    // vstar = (rcR vR + rcL vL + (PL - PR)) / den
    {
      const double na = vstar_a * rden;
      den_a = fma(-na, vstar, den_a);
      rcR_a = fma(na, vR, rcR_a);
      rcL_a = fma(na, vL, rcL_a);
      vR_a = fma(na, rcR, vR_a);
      vL_a = fma(na, rcL, vL_a);
      WLa[P_] += na;
      WRa[P_] -= na;
    }
    rcR_a += den_a;
    rcL_a += den_a;
    // rcL = rhoL (vL - sL); rcR = rhoR (sR - vR)
    WLa[0] += rcL_a * (vL - sL);
    vL_a = fma(rcL_a, WL[0], vL_a);
    sL_a = fma(-rcL_a, WL[0], sL_a);
    WRa[0] += rcR_a * (sR - vR);
    sR_a = fma(rcR_a, WR[0], sR_a);
    vR_a = fma(-rcR_a, WR[0], vR_a);
    // sL = min-select(vL, vR) - cmax; sR = max-select(vL, vR) + cmax
    if (minL) vL_a += sL_a; else vR_a += sL_a;
    cmax_a -= sL_a;
    if (maxL) vL_a += sR_a; else vR_a += sR_a;
    cmax_a += sR_a;
    WLa[v1] += vL_a;
    WRa[v1] += vR_a;
  }
  // cmax = select(cL, cR); c = sound_speed(P, rho) + |v|
  {
    const double cLa = Lmax ? cmax_a : 0.0, cRa = Lmax ? 0.0 : cmax_a;
    sound_speed_vjp_add(WL[P_], WL[0], gamma, min_c2, cLa, WLa[P_], WLa[0]);
    sound_speed_vjp_add(WR[P_], WR[0], gamma, min_c2, cRa, WRa[P_], WRa[0]);
    WLa[v1] += cLa * sgn0(WL[v1]);
    WRa[v1] += cRa * sgn0(WR[v1]);
  }
  // back to the inputs
#pragma unroll
  for (int v = 0; v < V; ++v) { MLa[v] = 0.0; MRa[v] = 0.0; }
  if (prims) {
#pragma unroll
    for (int v = 0; v < V; ++v) { MLa[v] = WLa[v]; MRa[v] = WRa[v]; }
    cons_vjp_add<D>(WL, ULa, MLa, gamma);
    cons_vjp_add<D>(WR, URa, MRa, gamma);
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v) { MLa[v] = ULa[v]; MRa[v] = URa[v]; }
    prim_vjp_add<D>(UL, WLa, MLa, gamma);
    prim_vjp_add<D>(UR, WRa, MRa, gamma);
  }
}

}  // namespace spd
