// Viscous fluxes of the SD-ADER predictor (src/sdader_simulator.py:245-268,
// src/hydro.py:172-241), added after the element-interface Riemann solves of
// every Picard iteration and subtracted from the flux at every flux point by
// the interior kernel.  Bit-identical to the reference's NumPy path:
//
//  * ViscGrad: density and velocities at the nf flux points of every
//    direction d (interpolation of the iterate, then the quotients of
//    U -> W), with both edge points replaced by the LEFT state of their
//    element interface (ML: the right-edge state of the cell on the left,
//    or the domain-boundary state of src/sd_boundary.py:32-68), stored as
//    Wfp[d]; the velocities' derivative along d at the solution points,
//    divided by h_d, stored as dWsp[d].  The viscous flux reads no other
//    variable, so neither the energy's line nor the pressure is formed
//    (128^2, p = 3, 8 launches: 1.15 -> 0.66 ms);
//  * ViscFlux: for every flux direction d and gradient direction e, the
//    velocities' dWsp[e] that the flux reads (all for e = d, those along d
//    and e otherwise: 7 of 15 derivatives in 3D; 1.66 -> 1.07 ms)
//    interpolated to the flux points of d, with both edge points replaced by
//    the RIGHT state of their interface (MR: the left-edge value of the cell
//    on the right, or the boundary state); the viscous flux from Wfp[d] and
//    these gradients, times rho and nu, stored as G[d] (layout of the
//    flux-point fluxes, [v][t][j][f][cell]).
//
// Boundary states (store_BC / apply_BC of src/sd_boundary.py, applied to the
// primitive and gradient arrays as the reference does): periodic -> the
// opposite edge; reflective -> the cell's own edge with the normal-velocity
// component negated; gradfree -> the cell's own edge; ic, eq -> the stored
// initial conservative edge traces, unchanged; pressure -> the same stored
// values, which also overwrite the domain-edge point of the array itself.
#pragma once
#include <type_traits>

#include "spd_kernels.cuh"

namespace spd {

// threads per block: the flux points of a line, 432 bytes a thread in 3D at
// degree 4, in 48 KB of shared memory
constexpr int VISC_THREADS = 64;

template <int D, int P>
struct ViscGrad {
  static __device__ __forceinline__ void run(Blk B, const Ops& op, const Geo& g, int Teff,
                                             const double* __restrict__ Uin, int Tu, const double* tr0,
                                             const double* tr1, const double* tr2, const double* bf0,
                                             const double* bf1, const double* bf2, double* W0, double* W1,
                                             double* W2, double* __restrict__ dWsp, const double* mq0,
                                             const double* mq1, const double* mq2) {
    using k = K<D, P>;
    // density and velocities, the variables 0..D
    constexpr int NV = D + 1;
    // their values at the flux points of the thread's line (shared memory, so
    // that the loops over variables can stay rolled)
    __shared__ double scr[NV * k::nf * VISC_THREADS];
    auto velocities = [](const double* M, double* W) {
      const Rcp r0 = recip_of(M[0]);
      W[0] = M[0];
#pragma unroll
      for (int v = 1; v < NV; ++v) W[v] = div_by(M[v], M[0], r0);
    };
    auto Wf = [&](int v, int f) -> double& { return scr[(v * k::nf + f) * VISC_THREADS + threadIdx.x]; };
    // well-balanced mode: the conservative equilibrium at the flux points is
    // part of the state whose primitives are taken (src/sdader_simulator.py:221-223)
    const double* meq[3] = {mq0, mq1, mq2};
    const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
    // one thread per (cell, direction, node, line)
    if (tid >= g.Nc * (D * k::NJ) * Teff) return;
    const long long c = tid % g.Nc;
    const int r = (int)(tid / g.Nc);
    const int dir = r / (Teff * k::NJ), t = r / k::NJ % Teff, j = r % k::NJ;
    const int tu = (Tu == 1) ? 0 : t;
    const double* trace[3] = {tr0, tr1, tr2};
    const double* bcfix[3] = {bf0, bf1, bf2};
    double* Wfp[3] = {W0, W1, W2};
    int cx, cy, cz;
    cell_coords(g, c, cx, cy, cz);
    auto line = [&](auto dc) {
      constexpr int d = decltype(dc)::value;
      const int cd = (d == 0) ? cx : (d == 1 ? cy : cz);
      const int Nd = g.N[d];
      const int b0 = g.bc[d][0], b1 = g.bc[d][1];
      const long long step = (d == 0) ? 1 : (d == 1 ? g.N[0] : (long long)g.N[0] * g.N[1]);
      const long long ntrans = g.Nc / Nd;
      const long long ct = (d == 0) ? (cy + (long long)g.N[1] * cz) : (d == 1 ? (cx + (long long)g.N[0] * cz)
                                                                              : (cx + (long long)g.N[0] * cy));
      {
        auto tr = [&](int side, int v, long long cell) -> double {
          double val = trace[d][(((long long)(side * k::V + v) * g.T + t) * k::NJ + j) * g.Nc + cell];
          if (meq[0]) val = val + meq[d][(((long long)v * k::NJ + j) * k::nf + (side ? k::nf - 1 : 0)) * g.Nc + cell];
          return val;
        };
        auto fix = [&](int side, int v) -> double {
          return bcfix[d][(((long long)side * k::V + v) * k::NJ + j) * ntrans + ct];
        };
#pragma unroll 1
        for (int v = 0; v < NV; ++v) {
          Line<k::n> ln;
#pragma unroll
          for (int s = 0; s < k::n; ++s)
            ln.v[s] = Uin[(((long long)v * Tu + tu) * k::NS + sp_index<D, P>(d, j, s)) * g.Nc + c];
          line_ready<k::n>(ln, op.soft);
          double m[k::nf - 2];
          line_apply<k::n, k::nf - 2, d == 0>(op.c_sp_to_fp, 1, 1, ln, m);
#pragma unroll
          for (int f = 1; f < k::nf - 1; ++f) Wf(v, f) = m[f - 1];
        }
#pragma unroll
        for (int f = 1; f < k::nf - 1; ++f) {
          double M[NV], W[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            M[v] = Wf(v, f);
            if (meq[0]) M[v] = M[v] + meq[d][(((long long)v * k::NJ + j) * k::nf + f) * g.Nc + c];
          }
          velocities(M, W);
#pragma unroll
          for (int v = 0; v < NV; ++v) Wf(v, f) = W[v];
        }
        // right edge: the cell's own right-edge state (its trace), or the
        // stored state on a "pressure" side
        {
          double M[NV], W[NV];
          if (cd == Nd - 1 && b1 == BC_PRESSURE) {
#pragma unroll
            for (int v = 0; v < NV; ++v) W[v] = fix(1, v);
          } else {
#pragma unroll
            for (int v = 0; v < NV; ++v) M[v] = tr(1, v, c);
            velocities(M, W);
          }
#pragma unroll
          for (int v = 0; v < NV; ++v) Wf(v, k::nf - 1) = W[v];
        }
        // left edge: the right-edge state of the cell on the left, or the
        // boundary state
        {
          double M[NV], W[NV];
          if (cd > 0 || b0 == BC_PERIODIC || b0 == BC_REFLECTIVE || b0 == BC_GRADFREE) {
            const long long src = (cd > 0) ? c - step : (b0 == BC_PERIODIC ? c + (Nd - 1) * step : c);
            const int side = (cd > 0 || b0 == BC_PERIODIC) ? 1 : 0;
#pragma unroll
            for (int v = 0; v < NV; ++v) M[v] = tr(side, v, src);
            velocities(M, W);
            if (cd == 0 && b0 == BC_REFLECTIVE) W[d + 1] = W[d + 1] * -1.0;
          } else {
#pragma unroll
            for (int v = 0; v < NV; ++v) W[v] = fix(0, v);
          }
#pragma unroll
          for (int v = 0; v < NV; ++v) Wf(v, 0) = W[v];
        }
        const bool pow2 = g.h_pow2[d] != 0;
#pragma unroll 1
        for (int v = 0; v < NV; ++v) {
          Line<k::nf> lf;
#pragma unroll
          for (int f = 0; f < k::nf; ++f) {
            lf.v[f] = Wf(v, f);
            Wfp[d][((((long long)v * g.T + t) * k::NJ + j) * k::nf + f) * g.Nc + c] = lf.v[f];
          }
          if (v == 0) continue;
          line_ready<k::nf>(lf, op.soft, op.dfp_eoff[d]);
          double dv[k::n];
          line_apply<k::nf, k::n, d == 0>(op.c_dfp, 0, 1, lf, dv);
#pragma unroll
          for (int so = 0; so < k::n; ++so) {
            const double val = pow2 ? dv[so] : div_by(dv[so], g.h[d], g.rh[d]);
            dWsp[((((long long)d * D + v - 1) * g.T + t) * k::NS + sp_index<D, P>(d, j, so)) * g.Nc + c] = val;
          }
        }
      }
    };
    if (dir == 0) line(std::integral_constant<int, 0>());
    if (D > 1 && dir == 1) line(std::integral_constant<int, (D > 1 ? 1 : 0)>());
    if (D > 2 && dir == 2) line(std::integral_constant<int, (D > 2 ? 2 : 0)>());
  }
};
template <int D, int P>
__global__ void k_visc_grad(Ops op, Geo g, int Teff, const double* __restrict__ Uin, int Tu, const double* tr0,
                            const double* tr1, const double* tr2, const double* bf0, const double* bf1,
                            const double* bf2, double* W0, double* W1, double* W2, double* __restrict__ dWsp,
                            const double* mq0, const double* mq1, const double* mq2) {
  ViscGrad<D, P>::run(hw_blk(), op, g, Teff, Uin, Tu, tr0, tr1, tr2, bf0, bf1, bf2, W0, W1, W2, dWsp, mq0, mq1, mq2);
}

template <int D, int P>
struct ViscFlux {
  static __device__ __forceinline__ void run(Blk B, const Ops& op, const Geo& g, int Teff,
                                             const double* __restrict__ dWsp, const double* W0, const double* W1,
                                             const double* W2, const double* bf0, const double* bf1,
                                             const double* bf2, double nu, double beta, double* G0, double* G1,
                                             double* G2) {
    using k = K<D, P>;
    constexpr int P_ = D + 1;
    // velocity gradients at the flux points of the thread's line
    __shared__ double scr[D * D * k::nf * VISC_THREADS];
    auto gf = [&](int e, int v, int f) -> double& {
      return scr[((e * D + v - 1) * k::nf + f) * VISC_THREADS + threadIdx.x];
    };
    const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
    // one thread per (cell, direction, node, line)
    if (tid >= g.Nc * (D * k::NJ) * Teff) return;
    const long long c = tid % g.Nc;
    const int r = (int)(tid / g.Nc);
    const int dir = r / (Teff * k::NJ), t = r / k::NJ % Teff, j = r % k::NJ;
    const double* bcfix[3] = {bf0, bf1, bf2};
    const double* Wfp[3] = {W0, W1, W2};
    double* G[3] = {G0, G1, G2};
    int cx, cy, cz;
    cell_coords(g, c, cx, cy, cz);
    auto line = [&](auto dc) {
      constexpr int d = decltype(dc)::value;
      const int cd = (d == 0) ? cx : (d == 1 ? cy : cz);
      const int Nd = g.N[d];
      const int b0 = g.bc[d][0], b1 = g.bc[d][1];
      const long long step = (d == 0) ? 1 : (d == 1 ? g.N[0] : (long long)g.N[0] * g.N[1]);
      const long long ntrans = g.Nc / Nd;
      const long long ct = (d == 0) ? (cy + (long long)g.N[1] * cz) : (d == 1 ? (cx + (long long)g.N[0] * cz)
                                                                              : (cx + (long long)g.N[0] * cy));
      const int v1 = rvel<D>(d, 0);
      {
        auto fix = [&](int side, int v) -> double {
          return bcfix[d][(((long long)side * k::V + v) * k::NJ + j) * ntrans + ct];
        };
        auto sp_val = [&](int e, int v, int s, long long cell) -> double {
          return dWsp[((((long long)e * D + v - 1) * g.T + t) * k::NS + sp_index<D, P>(d, j, s)) * g.Nc + cell];
        };
        // gradients along every direction e at the flux points of d
        {
#pragma unroll 1
          for (int ev = 0; ev < D * D; ++ev) {
            const int e = ev / D, v = ev % D + 1;
            if (e != d && v != e + 1 && v != d + 1) continue;
            Line<k::n> ln;
#pragma unroll
            for (int s = 0; s < k::n; ++s) ln.v[s] = sp_val(e, v, s, c);
            line_ready<k::n>(ln, op.soft);
            double gl[k::nf];
            line_apply<k::n, k::nf - 1, d == 0>(op.c_sp_to_fp, 0, 1, ln, gl);
            // left edge: the cell's own left-edge value (MR of its left
            // interface) unless a "pressure" side overwrote it
            if (cd == 0 && b0 == BC_PRESSURE) gl[0] = fix(0, v);
            // right edge: the left-edge value of the cell on the right, or
            // the boundary state (from the cell's own right-edge value)
            const bool inner = cd < Nd - 1 || b1 == BC_PERIODIC;
            const long long nb = !inner ? c : ((cd < Nd - 1) ? c + step : c - (Nd - 1) * step);
#pragma unroll
            for (int s = 0; s < k::n; ++s) ln.v[s] = sp_val(e, v, s, nb);
            line_ready<k::n>(ln, op.soft);
            double r;
            line_apply<k::n, 1, d == 0>(op.c_sp_to_fp, inner ? 0 : k::nf - 1, 1, ln, &r);
            if (!inner) {
              if (b1 == BC_REFLECTIVE) {
                if (v == d + 1) r = r * -1.0;
              } else if (b1 != BC_GRADFREE) {
                r = fix(1, v);
              }
            }
            gl[k::nf - 1] = r;
#pragma unroll
            for (int f = 0; f < k::nf; ++f) gf(e, v, f) = gl[f];
          }
        }
#pragma unroll
        for (int f = 0; f < k::nf; ++f) {
          double W[D + 1];  // density and velocities, all that Wfp holds
#pragma unroll
          for (int v = 0; v <= D; ++v)
            W[v] = Wfp[d][((((long long)v * g.T + t) * k::NJ + j) * k::nf + f) * g.Nc + c];
          double F[k::V];
          F[v1] = 2.0 * gf(d, v1, f) - beta * gf(d, v1, f);
          F[P_] = W[v1] * F[v1];
#pragma unroll
          for (int kk = 1; kk < D; ++kk) {
            const int vel = rvel<D>(d, kk);
            F[v1] = F[v1] - beta * gf(vel - 1, vel, f);
            F[vel] = gf(d, vel, f) + gf(vel - 1, v1, f);
            F[P_] = F[P_] + W[vel] * F[vel];
          }
          F[0] = 0.0;
#pragma unroll
          for (int v = 0; v < k::V; ++v)
            G[d][((((long long)v * g.T + t) * k::NJ + j) * k::nf + f) * g.Nc + c] = F[v] * W[0] * nu;
        }
      }
    };
    if (dir == 0) line(std::integral_constant<int, 0>());
    if (D > 1 && dir == 1) line(std::integral_constant<int, (D > 1 ? 1 : 0)>());
    if (D > 2 && dir == 2) line(std::integral_constant<int, (D > 2 ? 2 : 0)>());
  }
};
template <int D, int P>
__global__ void k_visc_flux(Ops op, Geo g, int Teff, const double* __restrict__ dWsp, const double* W0,
                            const double* W1, const double* W2, const double* bf0, const double* bf1,
                            const double* bf2, double nu, double beta, double* G0, double* G1, double* G2) {
  ViscFlux<D, P>::run(hw_blk(), op, g, Teff, dWsp, W0, W1, W2, bf0, bf1, bf2, nu, beta, G0, G1, G2);
}

}  // namespace spd
