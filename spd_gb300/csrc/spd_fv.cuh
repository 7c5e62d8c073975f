// Subcell finite-volume update with a-posteriori limiting for sm_103a:
// high-order flux application, ghost fills, NAD/SED/PAD trouble detection,
// blending, MUSCL-Hancock fallback fluxes on the affected faces only, and
// the CFL reduction.  Bit-identical to src/sdader_simulator.py:333-349,
// src/fv_simulator.py, src/trouble_detection.py and src/muscl.py.
#pragma once
#include "spd_kernels.cuh"

namespace spd {

struct FvGeo {
  const double* dx[3];       // active subcell widths, X_d values
  const double* hfp[3];      // extended subcell widths, Xe_d values
  const double* hcv[3];      // extended centre distances, Xe_d - 1 values
  const Rcp* rdx[3];      // reciprocals of dx
  const Rcp* rhcv[3];     // reciprocals of hcv
  const double* ihcv[3];  // 1 / hcv (the adjoint's products)
  const double* c2[3];       // centres[j+1] - centres[j-1], Xe_d values (ends unused)
  const Rcp* rc2[3];      // reciprocals of c2
};

__device__ __forceinline__ void q_coords(const Geo& g, long long q, int& ix, int& iy, int& iz) {
  ix = (int)(q % g.X[0]);
  long long r = q / g.X[0];
  iy = (int)(r % g.X[1]);
  iz = (int)(r / g.X[1]);
}

template <int D>
__device__ __forceinline__ long long ext_of(const Geo& g, int ix, int iy, int iz) {
  const int xe = ix + NGH, ye = (D >= 2) ? iy + NGH : 0, ze = (D >= 3) ? iz + NGH : 0;
  return xe + (long long)g.Xe[0] * (ye + (long long)g.Xe[1] * ze);
}

__device__ __forceinline__ long long ext_stride(const Geo& g, int d) {
  return d == 0 ? 1LL : (d == 1 ? (long long)g.Xe[0] : (long long)g.Xe[0] * g.Xe[1]);
}

__device__ __forceinline__ long long face_id(const Geo& g, int d, int fx, int fy, int fz) {
  const int FX = g.X[0] + (d == 0), FY = g.X[1] + (d == 1);
  return fx + (long long)FX * (fy + (long long)FY * fz);
}

__host__ __device__ __forceinline__ long long n_faces(const Geo& g, int d) {
  return (long long)(g.X[0] + (d == 0)) * (g.X[1] + (d == 1)) * (g.X[2] + (d == 2));
}

// Order-preserving int64 key of a double (ieee_key of its bits: the two
// zeros share a key, as they compare equal in IEEE) and its inverse (the
// key of either zero gives +0); NaN test on the bits.
__device__ __forceinline__ long long order_key(double x) { return ieee_key(__double_as_longlong(x)); }
__device__ __forceinline__ double from_order_key(long long k) { return __longlong_as_double(ieee_key_inverse(k)); }
__device__ __forceinline__ bool is_nan_bits(double x) { return nan_w(x); }
// NumPy maximum (a if a >= b or a is NaN, else b) on the integer pipes
__device__ __forceinline__ double np_max_key(double a, double b) {
  if (is_nan_bits(a)) return a;
  if (is_nan_bits(b)) return b;
  return order_key(a) >= order_key(b) ? a : b;
}
// x != 0.0 on the bits (true for NaN, false for both zeros)
__device__ __forceinline__ bool nonzero_bits(double x) { return nonzero_w(x); }
// x > 0 on the bits (false for zeros, negatives and NaN)
__device__ __forceinline__ bool gt0_key(double x) { return gt0_w(x); }

// gravity source of one subcell (src/fv_simulator.py:200-203 with
// src/simulator.py:197-203): dUdt[vel] += rho * dphi_vel, dUdt[P] +=
// m_vel * dphi_vel, direction by direction; gphi [d][subcell]
template <int D>
__device__ __forceinline__ void potential_source(const Geo& g, const double* __restrict__ gphi, long long q,
                                                 const double* u, double* dudt) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const double gp = gphi[(long long)d * g.Nq + q];
    dudt[d + 1] = dudt[d + 1] + u[0] * gp;
    if (!g.iso) dudt[D + 1] = dudt[D + 1] + u[d + 1] * gp;
  }
}

// Primitives of one subcell's state (src/sdader_simulator.py:351-356): in
// the well-balanced mode (Ueq non-null) the perturbation
// prim(U + U_eq) - prim(U_eq), with prim(U_eq) given as Weq; [v][subcell]
template <int D>
__device__ __forceinline__ void prims_cv(const Geo& g, const double* u, double* W, const double* __restrict__ Ueq,
                                         const double* __restrict__ Weq, long long q) {
  constexpr int V = D + 2;
  if (Ueq == nullptr) {
    prims<D>(u, W, g.gamma, g.iso != 0);
    return;
  }
  double uf[V];
#pragma unroll
  for (int v = 0; v < V; ++v) uf[v] = u[v] + Ueq[(long long)v * g.Nq + q];
  prims<D>(uf, W, g.gamma, g.iso != 0);
#pragma unroll
  for (int v = 0; v < V; ++v) W[v] = W[v] - Weq[(long long)v * g.Nq + q];
}

// dUdt of one subcell from the face fluxes (src/fv_simulator.py:189-205)
template <int D>
__device__ __forceinline__ void flux_divergence(const Geo& g, const FvGeo& fg, int ix, int iy, int iz,
                                                const double* const* F, int v, double& out) {
  const int ii[3] = {ix, iy, iz};
  double acc = 0.0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const long long nf = n_faces(g, d);
    const long long fl = face_id(g, d, ix, iy, iz);
    const long long fr = face_id(g, d, ix + (d == 0), iy + (d == 1), iz + (d == 2));
    const double part = div_by(F[d][(long long)v * nf + fr] - F[d][(long long)v * nf + fl], fg.dx[d][ii[d]],
                                fg.rdx[d][ii[d]]);
    acc = (d == 0) ? part : acc + part;
  }
  out = acc;
}

// Ghost layers.  The reference fills them direction by direction
// (src/fv_simulator.py:224-273), each fill reading the ghosts of the
// directions before it, so a ghost subcell's value follows from one active
// subcell: along every ghost direction the periodic or the nearest-edge image
// (whose layers are not mirrored), the normal velocity negated at a
// reflective side, and at a side with a fixed state the stored layer.  They
// are gathered so, all directions at once, by blocks of the kernels that run
// before their readers (six fills of 4 us each per substep at 32^2; written
// by the subcells they mirror instead, the few ghost owners in every warp
// slowed k_fv_candidate from 1.2 to 2.2 ms at 48^3).
struct GhostPos {
  int e[3];       // extended coordinates
  int a[3];       // extended coordinates of the active subcell it mirrors
  int side[3];    // side along d, or -1: not a ghost along d
};
template <int D>
__host__ __device__ __forceinline__ long long n_ghosts(const Geo& g) { return g.Nqe - g.Nq; }
// the idx-th ghost position: per direction d the layers along d over all
// positions of the directions before and the active ones of those after
template <int D>
__device__ __forceinline__ GhostPos ghost_pos(const Geo& g, long long idx) {
  GhostPos p;
  int d = 0;
#pragma unroll
  for (int q = D - 1; q > 0; --q) {
    long long n = 2 * NGH;
    for (int r = 0; r < D; ++r) n *= (r < q) ? g.Xe[r] : (r > q ? g.X[r] : 1);
    if (d == 0) {
      if (idx < n) d = q;
      else idx -= n;
    }
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    p.e[r] = p.a[r] = 0;
    p.side[r] = -1;
    if (r >= D) continue;
    const int n = (r < d) ? g.Xe[r] : (r > d ? g.X[r] : 2 * NGH);
    const int k = (int)(idx % n);
    idx /= n;
    p.e[r] = (r < d) ? k : (r > d ? k + NGH : (k < NGH ? k : g.X[r] + k));
    const int X = g.X[r];
    p.side[r] = p.e[r] < NGH ? 0 : (p.e[r] >= X + NGH ? 1 : -1);
    p.a[r] = p.e[r];
    if (p.side[r] == 0) p.a[r] = p.e[r] + (g.bc[r][0] == BC_PERIODIC ? X : NGH);
    if (p.side[r] == 1) p.a[r] = p.e[r] - (g.bc[r][1] == BC_PERIODIC ? X : NGH);
  }
  return p;
}
__device__ __forceinline__ long long ext_at(const Geo& g, const int* e) {
  return e[0] + (long long)g.Xe[0] * (e[1] + (long long)g.Xe[1] * e[2]);
}
// entry of direction d's boundary buffer [side][v][layer][other] for the ghost
// position e
__device__ __forceinline__ long long bc_entry(const Geo& g, int d, int side, int nv, int v, const int* e) {
  const int o0 = (d == 0) ? 1 : 0, o1 = (d == 2) ? 1 : 2;
  const long long nother = (long long)g.Xe[o0] * g.Xe[o1];
  const int layer = (side == 0) ? e[d] : e[d] - (g.X[d] + NGH);
  return (((long long)side * nv + v) * NGH + layer) * nother + e[o0] + (long long)g.Xe[o0] * e[o1];
}
struct BcBufs {
  double* b[3];
};
__device__ __forceinline__ bool fixed_bc(int kind) { return kind == BC_IC || kind == BC_PRESSURE; }
// variable v of the ghost position p from the active values of ext
template <int D>
__device__ __forceinline__ double ghost_value(const Geo& g, const BcBufs& bc, const GhostPos& p, int v,
                                              const double* __restrict__ ext) {
  double w = ext[(long long)v * g.Nqe + ext_at(g, p.a)];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    if (p.side[d] < 0) continue;
    const int kind = g.bc[d][p.side[d]];
    if (kind == BC_REFLECTIVE) {
      if (v == d + 1) w = w * -1.0;
    } else if (kind == BC_EQ) {
      w = 0.0;
    } else if (fixed_bc(kind)) {
      // the stored layer, at this ghost along the directions before d and at
      // the mirrored subcell along those after
      int at[3] = {0, 0, 0};
#pragma unroll
      for (int q = 0; q < D; ++q) at[q] = (q <= d) ? p.e[q] : p.a[q];
      w = bc.b[d][bc_entry(g, d, p.side[d], D + 2, v, at)];
    }
  }
  return w;
}

// counters that a substep accumulates, zeroed by its first kernel
struct Counters {
  int* flags;                  // [0] any possible trouble
  unsigned long long* counts;  // [0..1], [3] and [4..4+D) of spd_ctx::counts
};

// candidate update with the high-order fluxes of time node i, W_old and
// W_new into the extended arrays (src/sdader_simulator.py:336-340,
// src/trouble_detection.py:10-13)
template <int D>
struct FvCandidate {
// write_ext: 0 = no primitives (no limiting); 1 = W_old = prim(U_cv) and
// W_new = prim(U_new) into ext_old / ext_new; 2 = as 1 with W_old read from
// ext_new, which holds prim(U_cv) at this point (the previous substep's
// W_new, refreshed by k_fv_correct where the fallback changed U_cv): the
// same values without a second primitive conversion.  W_cv (the step's last
// substep, else null): the primitives of the new state in the subcell layout,
// which k_fv_correct refreshes likewise (src/sdader_simulator.py:351-359).
static __device__ __forceinline__ void run(Blk B, const Geo& g, const FvGeo& fg, const double* __restrict__ dt_ptr,
                                           double w_i, const double* F0, const double* F1, const double* F2,
                                           const double* __restrict__ U_cv, double* __restrict__ U_new,
                                           double* ext_old, double* ext_new, int write_ext, const Counters& ct, double* __restrict__ W_cv,
                                           const double* __restrict__ gphi, const double* __restrict__ Ueq,
                                           const double* __restrict__ Weq) {
  constexpr int V = D + 2;
  const long long q = B.id * (long long)blockDim.x + threadIdx.x;
  if (q == 0 && write_ext) {
    ct.flags[0] = 0;
    ct.counts[0] = ct.counts[1] = ct.counts[3] = 0;
    for (int d = 0; d < D; ++d) ct.counts[4 + d] = 0;
  }
  if (q >= g.Nq) return;
  int ix, iy, iz;
  q_coords(g, q, ix, iy, iz);
  const double* F[3] = {F0, F1, F2};
  const double dti = *dt_ptr * w_i;
  double u[V], un[V], dudt[V];
#pragma unroll
  for (int v = 0; v < V; ++v) u[v] = U_cv[(long long)v * g.Nq + q];
#pragma unroll
  for (int v = 0; v < V; ++v) flux_divergence<D>(g, fg, ix, iy, iz, F, v, dudt[v]);
  if (gphi != nullptr) potential_source<D>(g, gphi, q, u, dudt);
#pragma unroll
  for (int v = 0; v < V; ++v) {
    un[v] = u[v] - dudt[v] * dti;
    U_new[(long long)v * g.Nq + q] = un[v];
  }
  if (write_ext) {
    const long long e = ext_of<D>(g, ix, iy, iz);
    double W[V];
    if (write_ext == 2) {
#pragma unroll
      for (int v = 0; v < V; ++v) W[v] = ext_new[(long long)v * g.Nqe + e];
    } else {
      prims_cv<D>(g, u, W, Ueq, Weq, q);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) ext_old[(long long)v * g.Nqe + e] = W[v];
    prims_cv<D>(g, un, W, Ueq, Weq, q);
#pragma unroll
    for (int v = 0; v < V; ++v) ext_new[(long long)v * g.Nqe + e] = W[v];
    if (W_cv != nullptr) {
#pragma unroll
      for (int v = 0; v < V; ++v) W_cv[(long long)v * g.Nq + q] = W[v];
    }
  }
}
};
template <int D>
__global__ void k_fv_candidate(Geo g, FvGeo fg, const double* __restrict__ dt_ptr, double w_i,
                               const double* F0, const double* F1, const double* F2,
                               const double* __restrict__ U_cv, double* __restrict__ U_new, double* ext_old,
                               double* ext_new, int write_ext, Counters ct,
                               double* __restrict__ W_cv, const double* __restrict__ gphi, const double* __restrict__ Ueq,
                               const double* __restrict__ Weq) {
  FvCandidate<D>::run(hw_blk(), g, fg, dt_ptr, w_i, F0, F1, F2, U_cv, U_new, ext_old, ext_new, write_ext, ct, W_cv,
                      gphi, Ueq, Weq);
}

// ghost fill of one direction (src/fv_simulator.py:224-273): store the
// boundary buffer when the reference does, then copy it into the ghost
// layers.  bcbuf layout [side][v][g][other], other = the extended index of
// the remaining directions (lower direction fastest).  The adjoint rebuilds a
// substep's primitives with it; the step gathers its ghosts (ghost_value).
template <int D>
struct Ghost {
static __device__ __forceinline__ void run(Blk B, const Geo& g, int d, int nv, double* ext, double* bcbuf) {
  const int o0 = (d == 0) ? 1 : 0;
  const int o1 = (d == 2) ? 1 : 2;
  const long long nother = (long long)g.Xe[o0] * g.Xe[o1];
  const long long total = 2LL * nv * NGH * nother;
  const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
  if (tid >= total) return;
  const long long other = tid % nother;
  long long r = tid / nother;
  const int gi = (int)(r % NGH);
  r /= NGH;
  const int v = (int)(r % nv);
  const int side = (int)(r / nv);
  const int a = (int)(other % g.Xe[o0]);
  const int b = (int)(other / g.Xe[o0]);
  const int Xd = g.X[d];
  const int kind = g.bc[d][side];
  auto ext_index = [&](int e) -> long long {
    int c[3];
    c[d] = e;
    c[o0] = a;
    c[o1] = b;
    return c[0] + (long long)g.Xe[0] * (c[1] + (long long)g.Xe[1] * c[2]);
  };
  const long long bidx = (((long long)side * nv + v) * NGH + gi) * nother + other;
  double val;
  bool store = false;
  int src = 0;
  if (kind == BC_PERIODIC) { store = true; src = (side == 0) ? Xd + gi : NGH + gi; }
  else if (kind == BC_REFLECTIVE || kind == BC_GRADFREE) { store = true; src = (side == 0) ? NGH + gi : Xd + gi; }
  if (store) {
    val = ext[(long long)v * g.Nqe + ext_index(src)];
    if (kind == BC_REFLECTIVE && v == d + 1) val = val * -1.0;
    bcbuf[bidx] = val;
  } else if (kind == BC_EQ) {
    val = 0.0;
    bcbuf[bidx] = val;
  } else {
    val = bcbuf[bidx];
  }
  const int dst = (side == 0) ? gi : Xd + NGH + gi;
  ext[(long long)v * g.Nqe + ext_index(dst)] = val;
}
};
template <int D>
__global__ void k_ghost(Geo g, int d, int nv, double* ext, double* bcbuf) {
  Ghost<D>::run(hw_blk(), g, d, nv, ext, bcbuf);
}

// NAD: relaxed discrete maximum principle over the cross stencil
// (src/trouble_detection.py:14-38).  mask bit v = possible trouble of var v.
//
// Bound by the integer pipes.  A variable is first tried on the upper words
// of the values' order-preserving keys: one unit there is at least 2^-21 of
// the value and at most 2^-20 (of the larger value, where a power of two lies
// between), so a new value within ``slack`` units of the stencil's extrema
// lies within a relative distance of (slack + 1) 2^-20 of them, and only the
// others take the exact bounds.  slack < 0: no such test (a zero or
// differential tolerance).  512^2: 0.70 -> 0.55 ms a step; none in 3D, where a
// fluid at rest makes it fail more often than it saves (48^3: 0.59 -> 0.97).
//
// The grid's blocks after the first ``nb_main`` fill the ghosts of ext_old and
// ext_new; the stencil reads its own images of active subcells instead.
__device__ __forceinline__ int key_hi(double x) {
  const int h = (int)hi_word(x);
  return h ^ ((h >> 31) & 0x7fffffff);
}
template <int D>
struct Nad {
// the stencil neighbour of an active subcell at a domain side
static __device__ __forceinline__ double outside(const Geo& g, const BcBufs& bc, const double* __restrict__ ext_old,
                                                 int v, const int* c, int d, int step) {
  GhostPos p;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    p.e[r] = p.a[r] = (r < D) ? c[r] + NGH + (r == d ? step : 0) : 0;
    p.side[r] = (r != d) ? -1 : (step < 0 ? 0 : 1);
    if (r == d) p.a[r] = p.e[r] - step * (g.bc[d][p.side[r]] == BC_PERIODIC ? g.X[d] : NGH);
  }
  return ghost_value<D>(g, bc, p, v, ext_old);
}
// the flags of one subcell, SIDE: with a neighbour outside the domain
template <bool SIDE>
static __device__ __forceinline__ unsigned flags_of(const Geo& g, const BcBufs& bc, const int* ii, long long e,
                                                    double tol, int slack, int delta, int relax,
                                                    const double* __restrict__ ext_old,
                                                    const double* __restrict__ ext_new) {
  constexpr int V = D + 2;
  unsigned m = 0;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const double* W = ext_old + (long long)v * g.Nqe;
    const double c0 = W[e];
    double nb[2 * D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const long long st = ext_stride(g, d);
      nb[2 * d] = (!SIDE || ii[d] > 0) ? W[e - st] : outside(g, bc, ext_old, v, ii, d, -1);
      nb[2 * d + 1] = (!SIDE || ii[d] < g.X[d] - 1) ? W[e + st] : outside(g, bc, ext_old, v, ii, d, 1);
    }
    const double wn = ext_new[(long long)v * g.Nqe + e];
    if constexpr (D <= 2) {
      int hmx = key_hi(c0), hmn = hmx;
#pragma unroll
      for (int k = 0; k < 2 * D; ++k) {
        const int h = key_hi(nb[k]);
        hmx = max(hmx, h);
        hmn = min(hmn, h);
      }
      const int hw = key_hi(wn);
      // all finite, infinities' and NaN's keys out of reach, and both extrema
      // normal numbers
      const bool normal = hmx < 0x7fe00000 && hmn > (int)0x801fffff && (hmx >= 0x00100000 || hmx <= (int)0xffefffff) &&
                          (hmn >= 0x00100000 || hmn <= (int)0xffefffff);
      if (slack >= 0 && normal && hw >= hmn - slack && hw <= hmx + slack) continue;
    }
    // maximum / minimum of the cross stencil on order-preserving integer
    // keys (integer pipes; the FP64 pipe is the step's bottleneck).  A NaN
    // anywhere makes NumPy's maximum/minimum NaN and the point troubled.
    bool nan = is_nan_bits(c0);
    long long kmx = order_key(c0), kmn = kmx;
#pragma unroll
    for (int k = 0; k < 2 * D; ++k) {
      nan = nan || is_nan_bits(nb[k]);
      const long long kk = order_key(nb[k]);
      kmx = max(kmx, kk);
      kmn = min(kmn, kk);
    }
    double mx = from_order_key(kmx), mn = from_order_key(kmn);
    if (relax) {
      if (delta) {
        const double eps = tol * (mx - mn);
        mn = mn - eps;
        mx = mx + eps;
      } else {
        mn = mn - abs_bits(mn) * tol;
        mx = mx + abs_bits(mx) * tol;
      }
    }
    // !(wn >= mn) || !(wn <= mx) on the integer keys: true when any of the
    // three is NaN, else the ordered comparison (the keys equate -0, +0)
    const long long kw = order_key(wn);
    const bool pt = nan || is_nan_bits(wn) || is_nan_bits(mn) || is_nan_bits(mx) || kw < order_key(mn) ||
                    kw > order_key(mx);
    m |= (pt ? 1u : 0u) << v;
  }
  return m;
}
// With sed_list non-null, the flagged (subcell, density / pressure) pairs
// are also appended to sed_list (item 2*q + is_pressure) for k_sed.
static __device__ __forceinline__ void run(Blk B, const Geo& g, unsigned nb_main, const BcBufs& bc, double tol,
                                           int slack, int delta, int relax, double* __restrict__ ext_old,
                                           double* __restrict__ ext_new, unsigned char* __restrict__ mask,
                                           int* any_flag, long long* __restrict__ sed_list,
                                           unsigned long long* __restrict__ sed_count) {
  constexpr int V = D + 2;
  if (B.id >= nb_main) {
    const long long n = n_ghosts<D>(g);
    const long long i = (B.id - nb_main) * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GhostPos p = ghost_pos<D>(g, i);
    const long long e = ext_at(g, p.e);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      ext_old[(long long)v * g.Nqe + e] = ghost_value<D>(g, bc, p, v, ext_old);
      ext_new[(long long)v * g.Nqe + e] = ghost_value<D>(g, bc, p, v, ext_new);
    }
    return;
  }
  const long long q = B.id * (long long)blockDim.x + threadIdx.x;
  unsigned int m = 0;
  if (q < g.Nq) {
    int ii[3];
    q_coords(g, q, ii[0], ii[1], ii[2]);
    bool side = false;
#pragma unroll
    for (int d = 0; d < D; ++d) side = side || ii[d] == 0 || ii[d] == g.X[d] - 1;
    const long long e = ext_of<D>(g, ii[0], ii[1], ii[2]);
    m = side ? flags_of<true>(g, bc, ii, e, tol, slack, delta, relax, ext_old, ext_new)
             : flags_of<false>(g, bc, ii, e, tol, slack, delta, relax, ext_old, ext_new);
    mask[q] = (unsigned char)m;
  }
  const unsigned ballot = __ballot_sync(0xffffffffu, m != 0);
  if (ballot != 0 && (threadIdx.x & 31) == 0) atomicOr(any_flag, 1);
  if (sed_list != nullptr && ballot != 0) {
    constexpr int P_ = D + 1;
    const bool f0 = m & 1u, fP = (m >> P_) & 1u;
    const unsigned b0 = __ballot_sync(0xffffffffu, f0), bP = __ballot_sync(0xffffffffu, fP);
    if (b0 | bP) {
      const int lane = threadIdx.x & 31;
      const unsigned lt = (1u << lane) - 1u;
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(sed_count, (unsigned long long)(__popc(b0) + __popc(bP)));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (f0) sed_list[base + __popc(b0 & lt)] = 2 * q;
      if (fP) sed_list[base + __popc(b0) + __popc(bP & lt)] = 2 * q + 1;
    }
  }
}
};
template <int D>
__global__ void k_nad(const __grid_constant__ Geo g, unsigned nb_main, const __grid_constant__ BcBufs bc, double tol,
                      int slack, int delta, int relax, double* __restrict__ ext_old, double* __restrict__ ext_new,
                      unsigned char* __restrict__ mask, int* any_flag, long long* __restrict__ sed_list,
                      unsigned long long* __restrict__ sed_count) {
  Nad<D>::run(hw_blk(), g, nb_main, bc, tol, slack, delta, relax, ext_old, ext_new, mask, any_flag, sed_list, sed_count);
}

// smooth-extrema relaxation factor of one variable along direction d at
// active subcell i (src/trouble_detection.py:104-137, including its
// one-sided minimum at the first and last active subcell).
__device__ __forceinline__ double sed_alpha_dir(const double* W, long long e0, long long st, int i, int Xd,
                                                const double* c2, const Rcp* rc2, const double* hfp) {
  // line accessors in extended coordinates j along d; c2[j] = cen[j+1] -
  // cen[j-1] and rc2[j] its correctly rounded reciprocal (the quotients
  // below are the IEEE ones, div_soft)
  auto U = [&](int j) { return W[e0 + (long long)j * st]; };
  const int k = i + NGH;
  const int lo = (i == 0) ? k - 1 : k - 2;
  const int hi = (i == Xd - 1) ? k + 1 : k + 2;
  double dUs[5];
#pragma unroll
  for (int o = 0; o < 5; ++o) {
    const int j = k - 2 + o;
    if (j >= lo && j <= hi) dUs[o] = div_by(U(j + 1) - U(j - 1), c2[j], rc2[j]);
  }
  auto dU = [&](int j) { return dUs[j - (k - 2)]; };
  auto aLR = [&](int kk, double& aL, double& aR) {
    const double dUm = dU(kk - 1), dU0 = dU(kk), dUp = dU(kk + 1);
    const double d2U = div_by(dUp - dUm, c2[kk], rc2[kk]);
    const double dv = 0.5 * hfp[kk] * d2U;
    const Rcp rdv = recip_of(dv);
    const double vL = dUm - dU0;
    const double vR = dUp - dU0;
    // comparisons on the integer keys / words (IEEE semantics)
    const double selL = fgt(0.0, dv) ? (fgt(vL, 0.0) ? vL : 0.0) : (fgt(0.0, vL) ? vL : 0.0);
    aL = div_by(-selL, dv, rdv);
    if (!nonzero_w(dv)) aL = 1.0;  // |dv| <= 0
    aL = fgt(1.0, aL) ? aL : 1.0;
    const double selR = fgt(dv, 0.0) ? (fgt(vR, 0.0) ? vR : 0.0) : (fgt(0.0, vR) ? vR : 0.0);
    aR = div_by(selR, dv, rdv);
    if (!nonzero_w(dv)) aR = 1.0;
    aR = fgt(1.0, aR) ? aR : 1.0;
  };
  auto A = [&](int kk) {
    double aL, aR;
    aLR(kk, aL, aR);
    return fgt(aL, aR) ? aR : aL;
  };
  if (i == 0) return np_min(A(k), A(k + 1));
  if (i == Xd - 1) {
    double aL, aR;
    aLR(k, aL, aR);
    return np_min(A(k - 1), aL);
  }
  return np_min(A(k - 1), np_min(A(k), A(k + 1)));
}

// SED (k_sed) and the trouble flags with PAD (k_troubles),
// src/trouble_detection.py:40-70.
template <int D>
struct Sed {
// smooth-extrema relaxation of the NAD flags of density and pressure: one
// list item per flagged (subcell, variable) pair, item = 2*q + (variable is
// pressure), compacted by k_nad so that this FP64 work runs on full warps.
// A pair whose smoothness indicator alpha is not < 1 clears its bit of the
// NAD mask (bytes of one 32-bit word may belong to other items, hence the
// atomic AND).
static __device__ __forceinline__ void run(Blk B, const Geo& g, const FvGeo& fg, const long long* __restrict__ list,
                                           const unsigned long long* __restrict__ count,
                                           const double* __restrict__ ext_new, unsigned char* mask) {
  constexpr int P_ = D + 1;
  const unsigned long long cnt = *count;
  for (unsigned long long idx = B.id * (unsigned long long)blockDim.x + threadIdx.x; idx < cnt;
       idx += (unsigned long long)B.n * blockDim.x) {
    const long long item = list[idx];
    const long long q = item >> 1;
    const int var = (item & 1) ? P_ : 0;
    int ix, iy, iz;
    q_coords(g, q, ix, iy, iz);
    const long long e = ext_of<D>(g, ix, iy, iz);
    const int ii[3] = {ix, iy, iz};
    const double* W = ext_new + (long long)var * g.Nqe;
    double alpha = W[e] * 0.0 + 1.0;
    for (int d = 0; d < D; ++d) {
      const long long st = ext_stride(g, d);
      const long long e0 = e - (long long)(ii[d] + NGH) * st;
      const double an = sed_alpha_dir(W, e0, st, ii[d], g.X[d], fg.c2[d], fg.rc2[d], fg.hfp[d]);
      alpha = (an < alpha) ? an : alpha;
    }
    if (!(alpha < 1.0))
      atomicAnd(reinterpret_cast<unsigned*>(mask) + (q >> 2), ~(1u << (8 * (unsigned)(q & 3) + var)));
  }
}
};
template <int D>
__global__ void k_sed(Geo g, FvGeo fg, const long long* __restrict__ list, const unsigned long long* __restrict__ count,
                      const double* __restrict__ ext_new, unsigned char* mask) {
  Sed<D>::run(hw_blk(), g, fg, list, count, ext_new, mask);
}

// trouble flags (NAD flags of density or pressure after the smooth-extrema
// relaxation) and PAD; writes the troubles into var 0 of the theta-source
// extended array and the troubles array.
//
// The troubles' ghosts: at periodic sides the image's trouble; elsewhere the
// reference leaves its boundary buffer as the last fill of the primitives
// left it, whose variable 0 is the density of W_new where any subcell was
// flagged (and the smoothness relaxation ran), else of W_old
// (src/fv_simulator.py:224-273, src/trouble_detection.py:40-72).  The buffers
// themselves are kept as the fills leave them.
// The grid's blocks after the first ``nb_main`` do the ghosts, a periodic
// image's flag computed again from its subcell's.
template <int D>
struct Troubles {
static __device__ __forceinline__ double flag(const Geo& g, int pad, double min_rho, double max_rho, double min_P,
                                              const unsigned char* __restrict__ mask,
                                              const double* __restrict__ ext_new, const double* __restrict__ Weq,
                                              long long q, long long e) {
  constexpr int P_ = D + 1;
  const unsigned m = mask[q];
  const int pt0 = m & 1u, ptP = (m >> P_) & 1u;
  // max(pt0, ptP) as a double: constants, no conversion on the FP64 pipe
  double t = (pt0 | ptP) ? 1.0 : 0.0;
  if (pad) {
    double r = ext_new[e];
    double P = ext_new[(long long)P_ * g.Nqe + e];
    if (Weq) {
      // the full state's primitives (src/trouble_detection.py:59-60)
      r = r + Weq[q];
      P = P + Weq[(long long)P_ * g.Nq + q];
    }
    // comparisons on the integer keys (IEEE semantics: NaN fails them)
    t = fge(r, min_rho) ? t : 1.0;
    t = fge(max_rho, r) ? t : 1.0;
    t = fge(P, min_P) ? t : 1.0;
  }
  return t;
}
static __device__ __forceinline__ void run(Blk B, const Geo& g, unsigned nb_main, int pad, double min_rho,
                                           double max_rho, double min_P, const unsigned char* __restrict__ mask,
                                           const int* __restrict__ flags, int sed, const double* __restrict__ ext_old,
                                           const double* __restrict__ ext_new, const BcBufs& bc,
                                           double* __restrict__ theta_src, double* __restrict__ troubles,
                                           const double* __restrict__ Weq) {
  constexpr int V = D + 2;
  if (B.id >= nb_main) {
    const long long i = (B.id - nb_main) * (long long)blockDim.x + threadIdx.x;
    if (i >= n_ghosts<D>(g)) return;
    const GhostPos p = ghost_pos<D>(g, i);
    const double* W = (sed && *flags != 0) ? ext_new : ext_old;
    const long long xe = ext_at(g, p.e);
    bool image = true;
    int last = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (p.side[d] < 0) continue;
      image = image && g.bc[d][p.side[d]] == BC_PERIODIC;
      last = d;
    }
    double th;
    if (image) {
      const long long q = (p.a[0] - NGH) + (long long)g.X[0] * ((D > 1 ? p.a[1] - NGH : 0) +
                                                              (long long)g.X[1] * (D > 2 ? p.a[2] - NGH : 0));
      th = flag(g, pad, min_rho, max_rho, min_P, mask, ext_new, Weq, q, ext_at(g, p.a));
    } else {
      th = W[xe];
    }
    theta_src[xe] = th;
    const int side = p.side[last], kind = g.bc[last][side];
    if (fixed_bc(kind)) return;
    double* b = last == 0 ? bc.b[0] : (last == 1 ? bc.b[1] : bc.b[2]);
#pragma unroll
    for (int v = 0; v < V; ++v)
      b[bc_entry(g, last, side, V, v, p.e)] = (v == 0 && kind == BC_PERIODIC) ? th : W[(long long)v * g.Nqe + xe];
    return;
  }
  const long long q = B.id * (long long)blockDim.x + threadIdx.x;
  if (q >= g.Nq) return;
  int ix, iy, iz;
  q_coords(g, q, ix, iy, iz);
  const long long e = ext_of<D>(g, ix, iy, iz);
  const double t = flag(g, pad, min_rho, max_rho, min_P, mask, ext_new, Weq, q, e);
  theta_src[e] = t;
  troubles[q] = t;
}
};
template <int D>
__global__ void k_troubles(Geo g, unsigned nb_main, int pad, double min_rho, double max_rho, double min_P,
                           const unsigned char* __restrict__ mask, const int* __restrict__ flags, int sed,
                           const double* __restrict__ ext_old, const double* __restrict__ ext_new, BcBufs bc,
                           double* __restrict__ theta_src, double* __restrict__ troubles,
                           const double* __restrict__ Weq) {
  Troubles<D>::run(hw_blk(), g, nb_main, pad, min_rho, max_rho, min_P, mask, flags, sed, ext_old, ext_new, bc,
                   theta_src, troubles, Weq);
}

// extended-grid coordinates
__device__ __forceinline__ void e_coords(const Geo& g, long long e, int& xe, int& ye, int& ze) {
  xe = (int)(e % g.Xe[0]);
  long long r = e / g.Xe[0];
  ye = (int)(r % g.Xe[1]);
  ze = (int)(r / g.Xe[1]);
}

// first / second (/ third) neighbour blending (src/trouble_detection.py:
// 139-164); the 3D neighbour pairs are those the reference's index tuples
// select.
template <int D>
struct BlendNeighbours {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const double* __restrict__ src,
                                           double* __restrict__ out) {
  const long long e = B.id * (long long)blockDim.x + threadIdx.x;
  if (e >= g.Nqe) return;
  int c[3];
  e_coords(g, e, c[0], c[1], c[2]);
  auto at = [&](int x, int y, int z) { return src[x + (long long)g.Xe[0] * (y + (long long)g.Xe[1] * z)]; };
  auto inb = [&](int d, int v) { return v >= 0 && v < g.Xe[d]; };
  double th = src[e];
  for (int d = 0; d < D; ++d) {
    for (int s = -1; s <= 1; s += 2) {
      int cc[3] = {c[0], c[1], c[2]};
      cc[d] += s;
      if (inb(d, cc[d])) th = np_max_key(0.75 * at(cc[0], cc[1], cc[2]), th);
    }
  }
  if (D == 2) {
    for (int sy = -1; sy <= 1; sy += 2)
      for (int sx = -1; sx <= 1; sx += 2)
        if (inb(0, c[0] + sx) && inb(1, c[1] + sy)) th = np_max_key(0.5 * at(c[0] + sx, c[1] + sy, 0), th);
  } else if (D == 3) {
    // (axis pair, offsets) per (i, idim); axes listed as (first, second)
    // cut axis; offset 0 with range e < last (cut a) or e >= 1 (cut b)
    const int axes[3][2] = {{1, 0}, {2, 1}, {0, 2}};  // idim 0: (y,x); 1: (z,y); 2: (x,z)
    // per i: (offset, cutkind) for the first and the second cut axis;
    // cutkind 0 = a (target e < last), 1 = b (target e >= 1)
    const int offs[4][2] = {{+1, +1}, {0, -1}, {-1, +1}, {0, -1}};
    const int kinds[4][2] = {{0, 0}, {0, 1}, {1, 0}, {1, 1}};
    for (int i = 0; i < 4; ++i) {
      for (int idim = 0; idim < 3; ++idim) {
        bool ok = true;
        int cc[3] = {c[0], c[1], c[2]};
        for (int k2 = 0; k2 < 2; ++k2) {
          const int ax = axes[idim][k2];
          const int last = g.Xe[ax] - 1;
          if (kinds[i][k2] == 0 && c[ax] >= last) ok = false;
          if (kinds[i][k2] == 1 && c[ax] < 1) ok = false;
          cc[ax] += offs[i][k2];
        }
        if (ok) th = np_max_key(0.5 * at(cc[0], cc[1], cc[2]), th);
      }
    }
    // third neighbours: offsets on (z, y, x)
    const int t3[4][3] = {{+1, +1, +1}, {+1, +1, -1}, {+1, -1, +1}, {+1, -1, -1}};
    for (int i = 0; i < 4; ++i) {
      const int oz = t3[i][0], oy = t3[i][1], ox = t3[i][2];
      const bool ok = (oz > 0 ? c[2] < g.Xe[2] - 1 : c[2] >= 1) && (oy > 0 ? c[1] < g.Xe[1] - 1 : c[1] >= 1) &&
                      (ox > 0 ? c[0] < g.Xe[0] - 1 : c[0] >= 1);
      if (ok) th = np_max_key(0.375 * at(c[0] + ox, c[1] + oy, c[2] + oz), th);
    }
  }
  out[e] = th;
}
};
template <int D>
__global__ void k_blend_neighbours(Geo g, const double* __restrict__ src, double* __restrict__ out) {
  BlendNeighbours<D>::run(hw_blk(), g, src, out);
}

// last blending layer (src/trouble_detection.py:167-169): per direction two
// sequential in-place sweeps, the directions one after the other.  The value
// after the sweeps of the directions below LEVEL, from the 3^LEVEL input
// values it depends on: one launch reading 9 (27) cached values instead of
// one per direction.
template <int LEVEL>
__device__ __forceinline__ double blended(const Geo& g, const int* c, long long e, const double* __restrict__ in) {
  if constexpr (LEVEL == 0) {
    return in[e];
  } else {
    constexpr int d = LEVEL - 1;
    const long long st = ext_stride(g, d);
    const int k = c[d];
    const double t0 = blended<d>(g, c, e, in);
    // after the first sweep: here and at the cell before
    double a0 = t0;
    if (k < g.Xe[d] - 1) a0 = np_max_key(gt0_key(blended<d>(g, c, e + st, in)) ? 0.25 : 0.0, t0);
    if (k < 1) return a0;
    const double am = np_max_key(gt0_key(t0) ? 0.25 : 0.0, blended<d>(g, c, e - st, in));
    return np_max_key(gt0_key(am) ? 0.25 : 0.0, a0);
  }
}
template <int D>
struct BlendLast {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const double* __restrict__ in,
                                           double* __restrict__ out) {
  const long long e = B.id * (long long)blockDim.x + threadIdx.x;
  if (e >= g.Nqe) return;
  int c[3];
  e_coords(g, e, c[0], c[1], c[2]);
  out[e] = blended<D>(g, c, e, in);
}
};
template <int D>
__global__ void k_blend_last(Geo g, const double* __restrict__ in, double* __restrict__ out) {
  BlendLast<D>::run(hw_blk(), g, in, out);
}

// Appends ``value`` of every lane with ``keep`` to list (order within the
// list unspecified), one atomic per warp.  All 32 lanes of the warp must
// call it.
__device__ __forceinline__ void warp_append(bool keep, long long value, long long* __restrict__ list,
                                            unsigned long long* __restrict__ count) {
  const unsigned b = __ballot_sync(0xffffffffu, keep);
  if (b == 0) return;
  const int lane = threadIdx.x & 31;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(b));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (keep) list[base + __popc(b & ((1u << lane) - 1u))] = value;
}

// Affected faces of every direction (src/trouble_detection.py:81-87) and the
// lists of what the fallback needs, one thread per extended subcell, which
// looks at the faces on both of its sides: the faces that need a fallback
// flux, the extended subcells next to one (their slopes and predictions) and
// the active subcells next to one (the corrected update).  Compacted lists,
// because an FP64 warp instruction costs the same with 1 or 32 active lanes.
// With theta == nullptr the affected faces already in ``aff`` are used
// (replayed decisions).
struct AffectedOut {
  double* aff[3];
  long long* flist[3];
  long long *cells, *active;
  unsigned long long* counts;  // [0] cells, [1] active, [4 + d] faces
};
template <int D>
struct AffectedAll {
static __device__ __forceinline__ void run(Blk B, const Geo& g, int godunov, const double* __restrict__ theta,
                                           const AffectedOut& out) {
  const long long e = B.id * (long long)blockDim.x + threadIdx.x;
  bool mark = false, inside = e < g.Nqe;
  int c[3] = {0, 0, 0};
  if (inside) e_coords(g, e, c[0], c[1], c[2]);
  bool in_dir[3] = {true, true, true};
#pragma unroll
  for (int d = 0; d < D; ++d) in_dir[d] = inside && c[d] >= NGH && c[d] < NGH + g.X[d];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    // the other coordinates are active
    const bool row = inside && (D < 2 || in_dir[d == 0 ? 1 : 0]) && (D < 3 || in_dir[d == 2 ? 1 : 2]);
    const long long st = ext_stride(g, d);
    const int fr = c[d] - 1;  // the face above; fr - 1 is the one below
    int f[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) f[q] = (q < D) ? c[q] - NGH : 0;
    bool need = false;
    long long fid = 0;
    if (row && fr >= 0 && fr <= g.X[d]) {
      f[d] = fr;
      fid = face_id(g, d, f[0], f[1], f[2]);
      double a;
      if (theta) {
        a = np_max_key(theta[e], theta[e + st]);
        out.aff[d][fid] = a;
      } else {
        a = out.aff[d][fid];
      }
      need = godunov || nonzero_bits(a);
      mark = mark || need;
    }
    if (row && fr >= 1 && fr - 1 <= g.X[d]) {
      f[d] = fr - 1;
      const double a = theta ? np_max_key(theta[e - st], theta[e]) : out.aff[d][face_id(g, d, f[0], f[1], f[2])];
      mark = mark || godunov || nonzero_bits(a);
    }
    warp_append(need, fid, out.flist[d], out.counts + 4 + d);
  }
  warp_append(mark, e, out.cells, out.counts);
  const long long q = (c[0] - NGH) + (long long)g.X[0] * ((D > 1 ? c[1] - NGH : 0) +
                                                        (long long)g.X[1] * (D > 2 ? c[2] - NGH : 0));
  warp_append(mark && in_dir[0] && in_dir[1] && in_dir[2], q, out.active, out.counts + 1);
}
};
template <int D>
__global__ void k_affected_all(Geo g, int godunov, const double* __restrict__ theta, AffectedOut out) {
  AffectedAll<D>::run(hw_blk(), g, godunov, theta, out);
}

// x / 2 without the FP64 pipe (the quotient of a value near underflow, an
// infinity or NaN with it)
__device__ __forceinline__ double halved(double x) {
  const unsigned h = hi_word(x), e = h & 0x7ff00000u;
  if (e > 0x00100000u && e < 0x7ff00000u) return from_words(h - 0x100000u, lo_word(x));
  return nonzero_w(x) ? div_ieee_slow(x, 2.0) : x;
}

// subcells per block of the kernels over work lists whose threads are
// (subcell of the list, variable) pairs, one warp per variable
constexpr int LIST_CELLS = 32;

// MUSCL-Hancock: limited gradients, slopes and the half-step primitive
// predictor of the marked extended subcells (src/muscl.py:61-75,129-173,
// 175-216).  One thread per (subcell, variable): the gradients of a variable
// are its own, the predictor then reads the others' from shared memory.  The
// lists are short (a thread per subcell with all its variables was 114
// registers and a chain of 24 quotients: 44 us a launch at 96^2).
template <int D, int BM = 0>
struct MusclCells {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const FvGeo& fg, int limiter,
                                           const double* __restrict__ dt_ptr, double w_i,
                                           const long long* __restrict__ list,
                                           const unsigned long long* __restrict__ count,
                                           const double* __restrict__ W_ext, double* __restrict__ Mpred,
                                           double* __restrict__ S, unsigned char* ltape,
                                           const double* __restrict__ Meq, const double* __restrict__ gphi) {
  constexpr int V = D + 2, P_ = D + 1;
  // state (the full one in the well-balanced mode), its limited gradients and
  // the equilibrium's
  __shared__ double sW[V][LIST_CELLS], sg[D][V][LIST_CELLS], sq[D][V][LIST_CELLS];
  const unsigned long long cnt = *count;
  const double dti = *dt_ptr * w_i;
  const bool wb = Meq != nullptr;
  const int l = threadIdx.x, v = threadIdx.y;
  for (unsigned long long base = (unsigned long long)B.id * LIST_CELLS; base < cnt;
       base += (unsigned long long)B.n * LIST_CELLS) {
    const bool on = base + l < cnt;
    long long e = 0;
    int c[3] = {0, 0, 0};
    double W = 0.0;
    __syncthreads();  // the readers of the round before
    if (on) {
      e = list[base + l];
      e_coords(g, e, c[0], c[1], c[2]);
      const double* M = W_ext + (long long)v * g.Nqe;
      const double* Q = Meq + (long long)v * g.Nqe;
      W = M[e];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const long long st = ext_stride(g, d);
        const int k = c[d];
        const double hl = fg.hcv[d][k - 1], hr = fg.hcv[d][k], hm = fg.hfp[d][k];
        const Rcp rhl = fg.rhcv[d][k - 1], rhr = fg.rhcv[d][k];
        const double SL = div_by(W - M[e - st], hl, rhl);
        const double SR = div_by(M[e + st] - W, hr, rhr);
        double dm;
        if (BM == 0) dm = (limiter == LIM_MINMOD) ? minmod(SL, SR) : moncen(SL, SR, hl, hr, hm);
        else dm = limiter_br<BM>(limiter, SL, SR, hl, hr, hm, &ltape[((long long)d * V + v) * g.Nqe + e]);
        sg[d][v][l] = dm;
        S[((long long)d * V + v) * g.Nqe + e] = halved(dm) * hm;
        if (wb) {
          // the equilibrium's limited gradient (src/muscl.py:203-204)
          const double QL = div_by(Q[e] - Q[e - st], hl, rhl);
          const double QR = div_by(Q[e + st] - Q[e], hr, rhr);
          sq[d][v][l] = (limiter == LIM_MINMOD) ? minmod(QL, QR) : moncen(QL, QR, hl, hr, hm);
        }
      }
      // the prediction takes the full state in the well-balanced mode
      // (src/muscl.py:205-207); the state it is added to is (M + M_eq) - M_eq
      sW[v][l] = wb ? W + Q[e] : W;
    }
    __syncthreads();
    if (!on) continue;
    // the variable's time derivative, the terms in the reference's order
    double dtW = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int vel = d + 1;
      const double w = sW[vel][l];
      if (v == 0) {
        dtW = dtW - (w * sg[d][0][l] + sW[0][l] * sg[d][vel][l]);
        if (wb) dtW = dtW - w * sq[d][0][l];
      } else if (v == P_) {
        dtW = dtW - (w * sg[d][P_][l] + g.gamma * sW[P_][l] * sg[d][vel][l]);
        if (wb) dtW = dtW - w * sq[d][P_][l];
      } else {
        if (v == vel) dtW = dtW - (w * sg[d][vel][l] + quot(sg[d][P_][l], sW[0][l]));
        // src/muscl.py:167-173: the transverse terms use the equilibrium
        // gradient in the well-balanced mode, as the reference's reassigned
        // dW does
        if (v >= 2) dtW = dtW - w * (wb ? sq[d][v][l] : sg[d][v][l]);
      }
    }
    if (v == P_) dtW = dtW * 0.0;
    if (wb && gphi != nullptr && v >= 1 && v <= D) {
      // gravity in the prediction (src/muscl.py:208-212), active subcells only
      bool active = true;
#pragma unroll
      for (int d = 0; d < D; ++d) active = active && c[d] >= NGH && c[d] < NGH + g.X[d];
      if (active) {
        const double drho = quot(sW[0][l] - Meq[e], sW[0][l]);
        const long long q = (c[0] - NGH) + (long long)g.X[0] * ((D > 1 ? c[1] - NGH : 0) +
                                                              (long long)g.X[1] * (D > 2 ? c[2] - NGH : 0));
        dtW = dtW + drho * gphi[(long long)(v - 1) * g.Nq + q];
      }
    }
    const double at = wb ? sW[v][l] - Meq[(long long)v * g.Nqe + e] : W;
    Mpred[(long long)v * g.Nqe + e] = at + halved(dtW) * dti;
  }
}
};
template <int D, int BM = 0>
__global__ void k_muscl_cells(Geo g, FvGeo fg, int limiter, const double* __restrict__ dt_ptr, double w_i,
                              const long long* __restrict__ list, const unsigned long long* __restrict__ count,
                              const double* __restrict__ W_ext, double* __restrict__ Mpred, double* __restrict__ S,
                              unsigned char* ltape, const double* __restrict__ Meq, const double* __restrict__ gphi) {
  MusclCells<D, BM>::run(hw_blk(), g, fg, limiter, dt_ptr, w_i, list, count, W_ext, Mpred, S, ltape, Meq, gphi);
}

// DIR >= 0 fixes the direction at compile time (the rotated velocity indices
// become constants: with a runtime direction the states are indexed in local
// memory); DIR = -1 takes it from d_rt.  SV as in RiemannSd.
template <int D, int BM = 0, int DIR = -1, int SV = -1>
struct MusclFaces {
// direction d's affected faces from their compacted list (k_affected_all), a
// grid-stride loop over full warps
static __device__ __forceinline__ void run(Blk B, const Geo& g, int d_rt, int solver,
                                           const long long* __restrict__ flist,
                                           const unsigned long long* __restrict__ fcount,
                                           const double* __restrict__ Mpred, const double* __restrict__ S,
                                           double* __restrict__ F_FB, unsigned* ftape,
                                           const double* __restrict__ Mq, const double* __restrict__ Fq) {
  const unsigned long long cnt = *fcount;
  for (unsigned long long idx = B.id * (unsigned long long)blockDim.x + threadIdx.x; idx < cnt;
       idx += (unsigned long long)B.n * blockDim.x)
    face(g, DIR >= 0 ? DIR : d_rt, solver, flist[idx], Mpred, S, F_FB, ftape, Mq, Fq);
}
// Mq, Fq (well-balanced mode): the equilibrium's primitive state and flux
// at the faces, added to both states and subtracted from the flux
// (src/fv_simulator.py:150-165)
static __device__ __forceinline__ void face(const Geo& g, int d, int solver, long long fidx,
                                            const double* __restrict__ Mpred, const double* __restrict__ S,
                                            double* __restrict__ F_FB, unsigned* ftape,
                                            const double* __restrict__ Mq = nullptr,
                                            const double* __restrict__ Fq = nullptr) {
  constexpr int V = D + 2;
  const long long nf = n_faces(g, d);
  const int FX = g.X[0] + (d == 0), FY = g.X[1] + (d == 1);
  int f[3];
  f[0] = (int)(fidx % FX);
  long long r = fidx / FX;
  f[1] = (int)(r % FY);
  f[2] = (int)(r / FY);
  int e1[3];
  for (int k = 0; k < 3; ++k) e1[k] = (k < D) ? f[k] + NGH : 0;
  e1[d] = f[d] + 1;
  const long long i1 = e1[0] + (long long)g.Xe[0] * (e1[1] + (long long)g.Xe[1] * e1[2]);
  const long long i2 = i1 + ext_stride(g, d);
  double ML[V], MR[V], F[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    ML[v] = Mpred[(long long)v * g.Nqe + i1] + S[((long long)d * V + v) * g.Nqe + i1];
    MR[v] = Mpred[(long long)v * g.Nqe + i2] - S[((long long)d * V + v) * g.Nqe + i2];
    if (Mq) {
      MR[v] = MR[v] + Mq[(long long)v * nf + fidx];
      ML[v] = ML[v] + Mq[(long long)v * nf + fidx];
    }
  }
  Br<BM> br;
  if (BM == 2) br.w = ftape[fidx];
  riemann<D, double, BM>(solver_of<SV>(solver), ML, MR, F, g.gamma, g.min_c2, d, true, &br, g.iso != 0, &g.rgm1);
  if (BM == 1) ftape[fidx] = br.w;
#pragma unroll
  for (int v = 0; v < V; ++v) F_FB[(long long)v * nf + fidx] = Fq ? F[v] - Fq[(long long)v * nf + fidx] : F[v];
}
};
template <int D, int BM = 0, int DIR = -1, int SV = -1>
__global__ void k_muscl_faces(Geo g, int d, int solver, const long long* __restrict__ flist,
                              const unsigned long long* __restrict__ fcount, const double* __restrict__ Mpred,
                              const double* __restrict__ S, double* __restrict__ F_FB, unsigned* ftape,
                              const double* __restrict__ Mq, const double* __restrict__ Fq) {
  MusclFaces<D, BM, DIR, SV>::run(hw_blk(), g, d, solver, flist, fcount, Mpred, S, F_FB, ftape, Mq, Fq);
}

// the same over the lists of all directions in one launch, each list from the
// next whole warp on
struct FaceLists {
  const long long* list[3];
  const unsigned long long* count;  // [d]
  double* F[3];
  const double* Mq[3];
  const double* Fq[3];
};
template <int D, int SV>
struct MusclFacesAll {
static __device__ __forceinline__ void run(Blk B, const Geo& g, int solver, const FaceLists& fl,
                                           const double* __restrict__ Mpred, const double* __restrict__ S) {
  unsigned long long end[3] = {0, 0, 0}, cnt[3];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    cnt[d] = fl.count[d];
    end[d] = (d > 0 ? end[d - 1] : 0) + ((cnt[d] + 31) & ~31ULL);
  }
  for (unsigned long long idx = B.id * (unsigned long long)blockDim.x + threadIdx.x; idx < end[D - 1];
       idx += (unsigned long long)B.n * blockDim.x) {
    if (idx < end[0]) {
      if (idx < cnt[0])
        MusclFaces<D, 0, 0, SV>::face(g, 0, solver, fl.list[0][idx], Mpred, S, fl.F[0], nullptr, fl.Mq[0], fl.Fq[0]);
    } else if (D > 1 && idx < end[1]) {
      const unsigned long long k = idx - end[0];
      if (k < cnt[1])
        MusclFaces<D, 0, (D > 1 ? 1 : 0), SV>::face(g, 1, solver, fl.list[1][k], Mpred, S, fl.F[1], nullptr, fl.Mq[1],
                                                    fl.Fq[1]);
    } else if (D > 2) {
      const unsigned long long k = idx - end[1];
      if (k < cnt[2])
        MusclFaces<D, 0, (D > 2 ? 2 : 0), SV>::face(g, 2, solver, fl.list[2][k], Mpred, S, fl.F[2], nullptr, fl.Mq[2],
                                                    fl.Fq[2]);
    }
  }
}
};
template <int D, int SV>
__global__ void k_muscl_faces_all(Geo g, int solver, FaceLists fl, const double* __restrict__ Mpred,
                                  const double* __restrict__ S) {
  MusclFacesAll<D, SV>::run(hw_blk(), g, solver, fl, Mpred, S);
}

// corrected update of the subcells next to an affected face
// (src/sdader_simulator.py:325-331,346)
// One thread per (subcell, variable); the first variable's warp then takes
// the new primitives.
template <int D>
struct FvCorrect {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const FvGeo& fg, const double* __restrict__ dt_ptr,
                                           double w_i, int godunov, const long long* __restrict__ list,
                                           const unsigned long long* __restrict__ count, const double* F0,
                                           const double* F1, const double* F2, const double* B0, const double* B1,
                                           const double* B2, const double* A0, const double* A1, const double* A2,
                                           const double* __restrict__ U_cv, double* __restrict__ U_new,
                                           double* __restrict__ ext_new, double* __restrict__ W_cv,
                                           const double* __restrict__ gphi, const double* __restrict__ Ueq,
                                           const double* __restrict__ Weq) {
  constexpr int V = D + 2;
  __shared__ double sU[V][LIST_CELLS];
  const unsigned long long cnt = *count;
  const double* FH[3] = {F0, F1, F2};
  const double* FB[3] = {B0, B1, B2};
  const double* AF[3] = {A0, A1, A2};
  const double dti = *dt_ptr * w_i;
  const int l = threadIdx.x, v = threadIdx.y;
  for (unsigned long long base = (unsigned long long)B.id * LIST_CELLS; base < cnt;
       base += (unsigned long long)B.n * LIST_CELLS) {
    const bool on = base + l < cnt;
    long long q = 0;
    int ii[3] = {0, 0, 0};
    __syncthreads();  // the readers of the round before
    if (on) {
      q = list[base + l];
      q_coords(g, q, ii[0], ii[1], ii[2]);
      const double u = U_cv[(long long)v * g.Nq + q];
      double dudt = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const long long nf = n_faces(g, d);
        double Fv[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const long long f = face_id(g, d, ii[0] + (d == 0 ? s : 0), ii[1] + (d == 1 ? s : 0), ii[2] + (d == 2 ? s : 0));
          const double ho = FH[d][(long long)v * nf + f];
          const double a = AF[d][f];
          if (godunov) Fv[s] = 1.0 * FB[d][(long long)v * nf + f] + (1.0 - 1.0) * ho;
          else if (nonzero_w(a)) Fv[s] = a * FB[d][(long long)v * nf + f] + (1.0 - a) * ho;
          else Fv[s] = ho;
        }
        const double part = div_by(Fv[1] - Fv[0], fg.dx[d][ii[d]], fg.rdx[d][ii[d]]);
        dudt = (d == 0) ? part : dudt + part;
      }
      if (gphi != nullptr) {
        // the gravity source's terms of this variable (potential_source)
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const double gp = gphi[(long long)d * g.Nq + q];
          if (v == d + 1) dudt = dudt + U_cv[q] * gp;
          if (v == D + 1 && !g.iso) dudt = dudt + U_cv[(long long)(d + 1) * g.Nq + q] * gp;
        }
      }
      const double un = u - dudt * dti;
      U_new[(long long)v * g.Nq + q] = un;
      sU[v][l] = un;
    }
    __syncthreads();
    if (!on || v != 0) continue;
    // the primitives of the corrected state: the next substep's W_old
    // (k_fv_candidate with write_ext == 2) and, in the last substep, W_cv
    double un[V], W[V];
#pragma unroll
    for (int k = 0; k < V; ++k) un[k] = sU[k][l];
    prims_cv<D>(g, un, W, Ueq, Weq, q);
    const long long e = ext_of<D>(g, ii[0], ii[1], ii[2]);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      ext_new[(long long)k * g.Nqe + e] = W[k];
      if (W_cv != nullptr) W_cv[(long long)k * g.Nq + q] = W[k];
    }
  }
}
};
template <int D>
__global__ void k_fv_correct(Geo g, FvGeo fg, const double* __restrict__ dt_ptr, double w_i, int godunov,
                             const long long* __restrict__ list, const unsigned long long* __restrict__ count,
                             const double* F0, const double* F1, const double* F2, const double* B0,
                             const double* B1, const double* B2, const double* A0, const double* A1,
                             const double* A2, const double* __restrict__ U_cv, double* __restrict__ U_new,
                             double* __restrict__ ext_new, double* __restrict__ W_cv,
                             const double* __restrict__ gphi, const double* __restrict__ Ueq, const double* __restrict__ Weq) {
  FvCorrect<D>::run(hw_blk(), g, fg, dt_ptr, w_i, godunov, list, count, F0, F1, F2, B0, B1, B2, A0, A1, A2, U_cv,
                    U_new, ext_new, W_cv, gphi, Ueq, Weq);
}

// Well-balanced mode around the step (src/sdader_simulator.py:363-376):
// sign -1: U_sp -= U_eq_sp before the predictor; sign +1: U_sp += U_eq_sp
// after the update.  One thread per solution-point value.
struct WbShift {
  static __device__ __forceinline__ void run(Blk B, long long n, double sign, double* __restrict__ U_sp,
                                             const double* __restrict__ Ueq) {
    const long long i = B.id * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    U_sp[i] = (sign < 0.0) ? U_sp[i] - Ueq[i] : U_sp[i] + Ueq[i];
  }
};
static __global__ void k_wb_shift(long long n, double sign, double* __restrict__ U_sp, const double* __restrict__ Ueq) {
  WbShift::run(hw_blk(), n, sign, U_sp, Ueq);
}
// U_cv += U_eq_cv, then W_cv = prim(U_cv) (src/sdader_simulator.py:375-376)
template <int D>
struct WbEnd {
  static __device__ __forceinline__ void run(Blk B, const Geo& g, double* __restrict__ U_cv,
                                             const double* __restrict__ Ueq, double* __restrict__ W_cv) {
    constexpr int V = D + 2;
    const long long q = B.id * (long long)blockDim.x + threadIdx.x;
    if (q >= g.Nq) return;
    double u[V], W[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      u[v] = U_cv[(long long)v * g.Nq + q] + Ueq[(long long)v * g.Nq + q];
      U_cv[(long long)v * g.Nq + q] = u[v];
    }
    prims<D>(u, W, g.gamma, g.iso != 0);
#pragma unroll
    for (int v = 0; v < V; ++v) W_cv[(long long)v * g.Nq + q] = W[v];
  }
};
template <int D>
__global__ void k_wb_end(Geo g, double* __restrict__ U_cv, const double* __restrict__ Ueq, double* __restrict__ W_cv) {
  WbEnd<D>::run(hw_blk(), g, U_cv, Ueq, W_cv);
}

// dt = cfl * h / cmax from the reduced maximum of d*c_s + sum |v| (NaN when
// a NaN entered the reduction) (src/sd_simulator.py:214-227)
// dt = cfl * min(h / c_max, h^2 / nu / 4) (src/sd_simulator.py:214-227; the
// viscous limit only when dt_visc >= 0; Python's min keeps its first
// argument unless the second is smaller, so a NaN dt stays NaN)
struct DtFinal {
  static __device__ __forceinline__ void run(Blk, double h, double cfl, unsigned long long* cmax_bits, int* nan_flag,
                                             double* dt, double dt_visc) {
    if (threadIdx.x != 0) return;
    const double cmax = *nan_flag ? __longlong_as_double(0x7ff8000000000000LL)
                                  : __longlong_as_double((long long)*cmax_bits);
    double dtt = h / cmax;
    if (dt_visc >= 0.0 && dt_visc < dtt) dtt = dt_visc;
    *dt = cfl * dtt;
    // for the next reduction
    *cmax_bits = 0;
    *nan_flag = 0;
  }
};
static __global__ void k_dt_final(double h, double cfl, unsigned long long* cmax_bits, int* nan_flag, double* dt,
                                  double dt_visc) {
  DtFinal::run(hw_blk(), h, cfl, cmax_bits, nan_flag, dt, dt_visc);
}

}  // namespace spd
