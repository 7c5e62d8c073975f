// SD-ADER step kernels for sm_103a, templated on the space dimension D and
// the polynomial degree P.  FP64 on the CUDA cores; bit-identical to the
// reference's NumPy path (src/sdader_simulator.py and callees).
//
// Device layouts (cells and subcells x-fastest):
//   U_sp   [v][s][c]        s = kx + n*(ky + n*kz),  c = cx + Nx*(cy + Ny*cz)
//   U_ader [v][t][s][c]
//   trace  [d][side][v][t][j][c]   edge-point states of direction d,
//                                  j = transverse point of the cell face
//   Fi     [d][v][t][j][iface]     element-interface Riemann fluxes
//   Ffp    [d][v][t][j][f][c]      flux-point fluxes (FV update only)
//   FV     [v][iz][iy][ix]         subcell arrays (U_cv, W_cv, U_new)
//   ext    [v][ze][ye][xe]         subcell arrays with 2 ghost layers
#pragma once
#include "spd_lines.cuh"

namespace spd {

// threads per block of the interior kernel, and its blocks per SM: their
// barriers overlap
constexpr int INTERIOR_THREADS = 256;
constexpr int INTERIOR_BLOCKS = 3;
// the tile of 3D at degree 4 leaves room for two, and 128 registers
template <int D, int P>
constexpr int interior_blocks = (D == 3 && P == 4) ? 2 : INTERIOR_BLOCKS;

struct Ops {
  double sp_to_fp[MAXNF * MAXN];
  double dfp_to_sp[MAXN * MAXNF];
  double sp_to_cv[MAXN * MAXN];
  double invader[MAXT * MAXT];
  double w_tp[MAXT];
  // the same matrices as operands of the integer-pipe products; ``soft``:
  // every entry is in their range
  Coef c_sp_to_fp[MAXNF * MAXN];
  Coef c_dfp[MAXN * MAXNF];
  Coef c_sp_to_cv[MAXN * MAXN];
  Coef c_invader[MAXT * MAXT];
  Coef c_w_tp[MAXT];
  int soft;
  // 1/h_d as a power of two, k << 20, for directions whose h_d is one
  // (Geo::h_pow2), else 0: scaling every product and partial sum of the
  // derivative by 2^k is exact (away from underflow and overflow), so
  // sum(dfp*F)*(1/h) == sum((dfp/h)*F).  0 in the fused build.
  unsigned dfp_eoff[3];
};

struct Geo {
  int N[3];        // cells per direction (1 for absent directions)
  int X[3];        // subcells per direction (N*n, 1 for absent)
  int Xe[3];       // extended subcells per direction (X+4, 1 for absent)
  int T;           // ADER time nodes
  long long Nc;    // cells
  long long Nq;    // subcells
  long long Nqe;   // extended subcells
  double h[3];
  double inv_h[3];  // 1/h (the adjoint's products)
  Rcp rh[3];        // reciprocals of h and gamma - 1 for quotients
  Rcp rgm1;
  int h_pow2[3];
  double gamma, min_c2;
  int bc[3][2];
  int iso;  // isothermal (src/hydro.py:84,123,169)
};

template <int D, int P>
struct K {
  static constexpr int n = P + 1;
  static constexpr int nf = P + 2;
  static constexpr int V = D + 2;
  static constexpr int NS = (D == 1) ? n : (D == 2 ? n * n : n * n * n);
  static constexpr int NJ = NS / n;
};

// in-cell point index of point k along direction d on transverse line j
template <int D, int P>
__device__ __forceinline__ int sp_index(int d, int j, int k) {
  constexpr int n = P + 1;
  if (d == 0) return k + n * j;
  if (d == 1) return (j % n) + n * k + n * n * (j / n);
  return j + n * n * k;
}

__device__ __forceinline__ void cell_coords(const Geo& g, long long c, int& cx, int& cy, int& cz) {
  cx = (int)(c % g.N[0]);
  long long r = c / g.N[0];
  cy = (int)(r % g.N[1]);
  cz = (int)(r / g.N[1]);
}

// interface id along d for the cell with coordinates (cx,cy,cz), index i along d
__device__ __forceinline__ long long iface_id(const Geo& g, int d, int cx, int cy, int cz, int i) {
  if (d == 0) return (long long)i + (long long)(g.N[0] + 1) * (cy + (long long)g.N[1] * cz);
  if (d == 1) return (long long)cx + (long long)g.N[0] * (i + (long long)(g.N[1] + 1) * cz);
  return (long long)cx + (long long)g.N[0] * (cy + (long long)g.N[1] * i);
}

__host__ __device__ __forceinline__ long long n_iface(const Geo& g, int d) {
  return g.Nc / g.N[d] * (g.N[d] + 1);
}

// ---------------------------------------------------------------------------
// edge traces of one variable on one line along d: sp -> fp 0 and fp nf-1
// (src/sdader_simulator.py:220, src/transforms.py:3-25).  ``at(s)`` gives the
// variable at solution point s; LANES2: d is x.
// ---------------------------------------------------------------------------
template <int D, int P, bool LANES2, class At>
__device__ __forceinline__ void trace_line(const Ops& op, const Geo& g, At at, long long c, double* trace, int t_out,
                                           int d, int j, int v) {
  using k = K<D, P>;
  Line<k::n> ln;
#pragma unroll
  for (int s = 0; s < k::n; ++s) ln.v[s] = at(sp_index<D, P>(LANES2 ? 0 : d, j, s));
  line_ready<k::n>(ln, op.soft);
  double e[2];
  line_apply<k::n, 2, LANES2>(op.c_sp_to_fp, 0, k::nf - 1, ln, e);
  trace[(((long long)(0 * k::V + v) * g.T + t_out) * k::NJ + j) * g.Nc + c] = e[0];
  trace[(((long long)(1 * k::V + v) * g.T + t_out) * k::NJ + j) * g.Nc + c] = e[1];
}
// traces of item r = (d*NJ + j)*V + v of time node tu of an iterate U (Tu
// stored); D*NJ*V items
template <int D, int P>
__device__ __forceinline__ void write_trace(const Ops& op, const Geo& g, const double* __restrict__ U, int Tu, int tu,
                                            long long c, int r, double* t0, double* t1, double* t2, int t_out) {
  using k = K<D, P>;
  const int v = r % k::V, j = r / k::V % k::NJ, d = r / (k::V * k::NJ);
  auto at = [&](int s) { return U[(((long long)v * Tu + tu) * k::NS + s) * g.Nc + c]; };
  if (d == 0) trace_line<D, P, true>(op, g, at, c, t0, t_out, 0, j, v);
  else trace_line<D, P, false>(op, g, at, c, d == 1 ? t1 : t2, t_out, d, j, v);
}

// Every kernel of the step is a body ``run(Blk, args...)`` plus a plain
// ``__global__`` wrapper that passes the hardware block index; the batched
// ensemble launches the same bodies over many instances at once.
template <int D, int P>
struct TracesSp {
  static __device__ __forceinline__ void run(Blk B, const Ops& op, const Geo& g, const double* __restrict__ U_sp,
                                             double* t0, double* t1, double* t2) {
    // one thread per (cell, line, variable)
    const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
    if (tid >= g.Nc * (D * K<D, P>::NJ * K<D, P>::V)) return;
    write_trace<D, P>(op, g, U_sp, 1, 0, tid % g.Nc, (int)(tid / g.Nc), t0, t1, t2, 0);
  }
};
template <int D, int P>
__global__ void k_traces_sp(Ops op, Geo g, const double* __restrict__ U_sp, double* t0, double* t1, double* t2) {
  TracesSp<D, P>::run(hw_blk(), op, g, U_sp, t0, t1, t2);
}

// traces of every (cell, time node) of an iterate U (Tu time nodes stored)
template <int D, int P>
__global__ void k_traces_ader(Ops op, Geo g, const double* __restrict__ U, int Tu, int Teff, double* t0, double* t1,
                              double* t2) {
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  constexpr int lines = D * K<D, P>::NJ * K<D, P>::V;
  if (tid >= g.Nc * Teff * lines) return;
  const int r = (int)(tid / g.Nc);
  const int t = r / lines;
  write_trace<D, P>(op, g, U, Tu, (Tu == 1) ? 0 : t, tid % g.Nc, r % lines, t0, t1, t2, t);
}

// ---------------------------------------------------------------------------
// element-interface Riemann fluxes for direction d
// (src/sdader_simulator.py:225-234, src/sd_boundary.py:7-76)
// ---------------------------------------------------------------------------
// DIR >= 0 fixes the direction at compile time (the rotated velocity
// indices become constants); DIR = -1 takes it from d_rt.  SV: RS_LLF, RS_HLLC
// (either HLLC form, by ``solver``) or -1 (any): one solver per kernel keeps
// its registers its own.
template <int D, int P, int BM = 0, int DIR = -1, bool EQ = false, int SV = -1>
struct RiemannSd {
static __device__ __forceinline__ void run(Blk B, const Geo& g, int d_rt, int Teff, int solver,
                                           const double* __restrict__ trace, const double* __restrict__ bcfix,
                                           double* __restrict__ Fi, unsigned* tape,
                                           const double* __restrict__ meq) {
  using k = K<D, P>;
  const int d = (DIR >= 0) ? DIR : d_rt;
  const long long nI = n_iface(g, d);
  const long long total = (long long)Teff * k::NJ * nI;
  const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
  if (tid >= total) return;
  const long long iface = tid % nI;
  const long long r = tid / nI;
  const int j = (int)(r % k::NJ);
  const int t = (int)(r / k::NJ);
  // decode interface -> (i along d, transverse cell coords)
  int cx = 0, cy = 0, cz = 0, i = 0;
  if (d == 0) {
    i = (int)(iface % (g.N[0] + 1));
    long long q = iface / (g.N[0] + 1);
    cy = (int)(q % g.N[1]);
    cz = (int)(q / g.N[1]);
  } else if (d == 1) {
    cx = (int)(iface % g.N[0]);
    long long q = iface / g.N[0];
    i = (int)(q % (g.N[1] + 1));
    cz = (int)(q / (g.N[1] + 1));
  } else {
    cx = (int)(iface % g.N[0]);
    long long q = iface / g.N[0];
    cy = (int)(q % g.N[1]);
    i = (int)(q / g.N[1]);
  }
  const int Nd = g.N[d];
  auto cell_at = [&](int idx) -> long long {
    int x = cx, y = cy, z = cz;
    if (d == 0) x = idx; else if (d == 1) y = idx; else z = idx;
    return x + (long long)g.N[0] * (y + (long long)g.N[1] * z);
  };
  // transverse cell index of the face plane
  const long long ct = (d == 0) ? (cy + (long long)g.N[1] * cz) : (d == 1 ? (cx + (long long)g.N[0] * cz)
                                                                            : (cx + (long long)g.N[0] * cy));
  const long long ntrans = g.Nc / Nd;
  // the edge state: the trace of the iterate, plus (well-balanced mode,
  // src/sdader_simulator.py:221-223) the equilibrium at that flux point
  auto tr = [&](int side, int v, long long cell) -> double {
    double val = trace[(((long long)(side * k::V + v) * g.T + t) * k::NJ + j) * g.Nc + cell];
    if constexpr (EQ) {
      if (meq) val = val + meq[(((long long)v * k::NJ + j) * k::nf + (side ? k::nf - 1 : 0)) * g.Nc + cell];
    }
    return val;
  };
  auto fix = [&](int side, int v) -> double {
    return bcfix[(((long long)side * k::V + v) * k::NJ + j) * ntrans + ct];
  };
  double ML[k::V], MR[k::V];
  const int b0 = g.bc[d][0], b1 = g.bc[d][1];
  if (i == 0) {
    const long long c0 = cell_at(0);
#pragma unroll
    for (int v = 0; v < k::V; ++v) {
      double val;
      if (b0 == BC_PERIODIC) val = tr(1, v, cell_at(Nd - 1));
      else if (b0 == BC_REFLECTIVE) val = (v == d + 1) ? tr(0, v, c0) * -1.0 : tr(0, v, c0);
      else if (b0 == BC_GRADFREE) val = tr(0, v, c0);
      else val = fix(0, v);
      ML[v] = val;
      MR[v] = (b0 == BC_PRESSURE) ? fix(0, v) : tr(0, v, c0);
    }
    if (Nd == 1 && b1 == BC_PRESSURE) { /* right trace of the same cell is not used here */ }
  } else if (i == Nd) {
    const long long cl = cell_at(Nd - 1);
#pragma unroll
    for (int v = 0; v < k::V; ++v) {
      double val;
      if (b1 == BC_PERIODIC) val = (b0 == BC_PRESSURE) ? fix(0, v) : tr(0, v, cell_at(0));
      else if (b1 == BC_REFLECTIVE) val = (v == d + 1) ? tr(1, v, cl) * -1.0 : tr(1, v, cl);
      else if (b1 == BC_GRADFREE) val = tr(1, v, cl);
      else val = fix(1, v);
      MR[v] = val;
      ML[v] = (b1 == BC_PRESSURE) ? fix(1, v) : tr(1, v, cl);
    }
  } else {
    const long long cl = cell_at(i - 1), cr = cell_at(i);
#pragma unroll
    for (int v = 0; v < k::V; ++v) {
      ML[v] = tr(1, v, cl);
      MR[v] = tr(0, v, cr);
    }
  }
  double F[k::V];
  Br<BM> br;
  if (BM == 2) br.w = tape[tid];
  // the isothermal system only in the EQ form: a runtime flag costs the
  // plain form an FP64 multiply per flux (the compiler predicates it)
  riemann<D, double, BM>(solver_of<SV>(solver), ML, MR, F, g.gamma, g.min_c2, d, false, &br, EQ && g.iso != 0,
                         &g.rgm1);
  if (BM == 1) tape[tid] = br.w;
#pragma unroll
  for (int v = 0; v < k::V; ++v) Fi[(((long long)v * g.T + t) * k::NJ + j) * nI + iface] = F[v];
}
};
// all directions in one launch, each from the next block on (on small grids a
// launch costs more than its problems)
struct RiemannDirs {
  const double* trace[3];
  const double* bcfix[3];
  double* Fi[3];
  const double* meq[3];
  unsigned blocks[3];  // per direction
};
template <int D, int P, bool EQ, int SV>
struct RiemannAll {
  static __device__ __forceinline__ void run(Blk B, const Geo& g, int Teff, int solver, const RiemannDirs& r) {
    if (B.id < r.blocks[0]) {
      RiemannSd<D, P, 0, 0, EQ, SV>::run(B, g, 0, Teff, solver, r.trace[0], r.bcfix[0], r.Fi[0], nullptr, r.meq[0]);
      return;
    }
    if (D > 1 && B.id < r.blocks[0] + r.blocks[1]) {
      const Blk b{B.id - r.blocks[0], r.blocks[1]};
      RiemannSd<D, P, 0, (D > 1 ? 1 : 0), EQ, SV>::run(b, g, 1, Teff, solver, r.trace[1], r.bcfix[1], r.Fi[1], nullptr,
                                                       r.meq[1]);
      return;
    }
    if (D > 2) {
      const Blk b{B.id - r.blocks[0] - r.blocks[1], r.blocks[2]};
      RiemannSd<D, P, 0, (D > 2 ? 2 : 0), EQ, SV>::run(b, g, 2, Teff, solver, r.trace[2], r.bcfix[2], r.Fi[2], nullptr,
                                                       r.meq[2]);
    }
  }
};
template <int D, int P, bool EQ, int SV>
__global__ void __launch_bounds__(128, 4) k_riemann_all(Geo g, int Teff, int solver, RiemannDirs r) {
  RiemannAll<D, P, EQ, SV>::run(hw_blk(), g, Teff, solver, r);
}
// EQ: the form for the well-balanced mode (meq non-null: the equilibrium
// at the flux points added to every edge state) and the isothermal system;
// the plain form reads neither
template <int D, int P, int BM = 0, int DIR = -1, bool EQ = false, int SV = -1>
__global__ void k_riemann_sd(Geo g, int d_rt, int Teff, int solver, const double* __restrict__ trace,
                             const double* __restrict__ bcfix, double* __restrict__ Fi, unsigned* tape,
                             const double* __restrict__ meq) {
  RiemannSd<D, P, BM, DIR, EQ, SV>::run(hw_blk(), g, d_rt, Teff, solver, trace, bcfix, Fi, tape, meq);
}

// ---------------------------------------------------------------------------
// interior flux points, derivative, Picard update (src/sdader_simulator.py:
// 148-200) or the final SD update (:202-208) or the flux-point output for
// the FV update (:288-298).  mode: 0 = Picard (writes U_ader and the next
// traces), 1 = SD update of U_sp, 2 = write Ffp.
//
// Block = CPB cells x rows of threads.  Shared memory holds the flux
// derivative of the cells' nodes, [(v*NS + s)*Tn + t][cell], Tn nodes stored,
// and, for a chunk of (node, line) pairs, the states and then the fluxes at
// their interior flux points, [(line*V + v)*(nf-2) + f][cell].  Per direction
// and chunk the rows take (line, variable) pairs to interpolate, then (line,
// flux point) pairs for the fluxes, then (line, variable) pairs for the
// derivative.  In the end they take (variable, point) pairs: the T values of
// the derivative are read once, prepared once and contracted into the T new
// nodes, which replace them, and the lines of the new nodes give the next
// traces.
//
// Bound: the FP64 additions beside the integer pipes (spd_soft.cuh).  A row's
// work is one variable or one point, not a line of all variables, because
// small grids leave warps to spare (32^2, p=3: a thread per line was 512
// warps on 608 schedulers) and because with every product inlined the loop
// bodies have to be few and small.
// ---------------------------------------------------------------------------
// EXT: optional terms, each present when its pointer is not null -- the
// viscous fluxes G[d] (src/sdader_simulator.py:268, layout of Ffp),
// subtracted from the flux at every flux point, Riemann edges included,
// before the derivative (spd_visc.cuh); the gravity source of the
// potential gradient gphi [d][s][cell] added to the derivative
// (src/sdader_simulator.py:154-157, src/simulator.py:197-203).
template <int D, int P, bool EXT = false>
struct Interior {
using k = K<D, P>;
static constexpr int ni = k::nf - 2;
struct Args {
  int mode, Teff, Tu, Tn;
  const double* Uin;
  bool visc, wb, iso;
};
// the arrays of one direction
struct Dir {
  const double* Fi;
  double* Ffp;
  const double *Gv, *meq, *feq;
};

// states at the interior flux points of lines [l0, l1) along d
template <bool LANES2>
static __device__ __forceinline__ void interpolate(const Ops& op, const Geo& g, const Args& a, int d, int l0, int l1,
                                                   long long c, double* scr) {
  const int CPB = blockDim.x;
#pragma unroll 1
  for (int i = threadIdx.y; i < (l1 - l0) * k::V; i += (int)blockDim.y) {
    const int v = i % k::V, line = l0 + i / k::V;
    const int t = line / k::NJ, j = line % k::NJ;
    const double* u = a.Uin + (((long long)v * a.Tu + (a.Tu == 1 ? 0 : t)) * k::NS) * g.Nc + c;
    Line<k::n> ln;
#pragma unroll
    for (int s = 0; s < k::n; ++s) ln.v[s] = u[sp_index<D, P>(d, j, s) * g.Nc];
    line_ready<k::n>(ln, op.soft);
    double m[ni];
    line_apply<k::n, ni, LANES2>(op.c_sp_to_fp, 1, 1, ln, m);
#pragma unroll
    for (int f = 0; f < ni; ++f) scr[(i * ni + f) * CPB] = m[f];
  }
}

// their fluxes, in place
static __device__ __forceinline__ void fluxes(const Geo& g, const Args& a, int d, int l0, int l1, long long c,
                                              double* scr, const double* __restrict__ meq) {
  const int CPB = blockDim.x;
#pragma unroll 1
  for (int i = threadIdx.y; i < (l1 - l0) * ni; i += (int)blockDim.y) {
    const int f = i % ni, l = i / ni;
    double* at = scr + (l * k::V * ni + f) * CPB;
    double M[k::V];
#pragma unroll
    for (int v = 0; v < k::V; ++v) M[v] = at[v * ni * CPB];
    if (a.wb) {
      const int j = (l0 + l) % k::NJ;
#pragma unroll
      for (int v = 0; v < k::V; ++v) M[v] = M[v] + meq[(((long long)v * k::NJ + j) * k::nf + f + 1) * g.Nc + c];
    }
    euler_flux<D>(M, g.gamma, d, a.iso, &g.rgm1, [&](int v, double F) { at[v * ni * CPB] = F; });
  }
}

// the derivative of their fluxes into the tile (added to the lower
// directions'), or the flux-point output
template <bool LANES2>
static __device__ __forceinline__ void derive(const Ops& op, const Geo& g, const Args& a, int d, int l0, int l1,
                                              long long c, double* tile, const double* scr, const Dir& dir) {
  const int CPB = blockDim.x;
  int cx, cy, cz;
  cell_coords(g, c, cx, cy, cz);
  const long long nI = n_iface(g, d);
  const int cd = (d == 0) ? cx : (d == 1 ? cy : cz);
  const long long il = iface_id(g, d, cx, cy, cz, cd);
  const long long ir = iface_id(g, d, cx, cy, cz, cd + 1);
  const bool pow2 = g.h_pow2[d] != 0;
#pragma unroll 1
  for (int i = threadIdx.y; i < (l1 - l0) * k::V; i += (int)blockDim.y) {
    const int v = i % k::V, line = l0 + i / k::V;
    const int t = line / k::NJ, j = line % k::NJ;
    const long long vtj = ((long long)v * g.T + t) * k::NJ + j;
    Line<k::nf> lf;
    lf.v[0] = dir.Fi[vtj * nI + il];
    lf.v[k::nf - 1] = dir.Fi[vtj * nI + ir];
#pragma unroll
    for (int f = 0; f < ni; ++f) lf.v[f + 1] = scr[(i * ni + f) * CPB];
    if (a.wb) {
      // F -> F' (src/sdader_simulator.py:235-237), before the viscous flux
#pragma unroll
      for (int f = 0; f < k::nf; ++f)
        lf.v[f] = lf.v[f] - dir.feq[(((long long)v * k::NJ + j) * k::nf + f) * g.Nc + c];
    }
    if (a.visc) {
#pragma unroll
      for (int f = 0; f < k::nf; ++f) lf.v[f] = lf.v[f] - dir.Gv[(vtj * k::nf + f) * g.Nc + c];
    }
    if (a.mode == 2) {
#pragma unroll
      for (int f = 0; f < k::nf; ++f) dir.Ffp[(vtj * k::nf + f) * g.Nc + c] = lf.v[f];
      continue;
    }
    line_ready<k::nf>(lf, op.soft, op.dfp_eoff[d]);
    double val[k::n];
    line_apply<k::nf, k::n, LANES2>(op.c_dfp, 0, 1, lf, val);
#pragma unroll
    for (int so = 0; so < k::n; ++so) {
      const double x = pow2 ? val[so] : div_by(val[so], g.h[d], g.rh[d]);
      double* slot = &tile[((v * k::NS + sp_index<D, P>(d, j, so)) * a.Tn + t) * CPB];
      *slot = LANES2 ? x : *slot + x;
    }
  }
}

template <bool LANES2>
static __device__ __forceinline__ void direction(const Ops& op, const Geo& g, const Args& a, int dd, int chunk,
                                                 long long c, bool active, double* tile, double* scr, const Dir& dir) {
  const int d = LANES2 ? 0 : dd;
  const int lines = a.Teff * k::NJ;
#pragma unroll 1
  for (int l0 = 0; l0 < lines; l0 += chunk) {
    const int l1 = l0 + chunk < lines ? l0 + chunk : lines;
    // the tile's and the chunk's readers of before are done
    if (!LANES2 || l0 > 0) __syncthreads();
    if (active) interpolate<LANES2>(op, g, a, d, l0, l1, c, scr);
    __syncthreads();
    if (active) fluxes(g, a, d, l0, l1, c, scr, dir.meq);
    __syncthreads();
    if (active) derive<LANES2>(op, g, a, d, l0, l1, c, tile, scr, dir);
  }
}

// U_ader of one (variable, point) from the derivative of its TT nodes
template <int TT>
static __device__ __forceinline__ void picard(const Ops& op, const Geo& g, double* slot, int CPB, int Teff, double dt,
                                              double usp, double* __restrict__ out, long long stride) {
  double acc[TT];
  // Teff == 1: one derivative for all nodes
#ifndef SPD_FUSED
  if (Teff == 1) {
    // one operand, TT x TT products
    Line<1> one;
    one.v[0] = slot[0];
    line_ready<1>(one, op.soft);
    double p[TT * TT];
    line_apply<1, TT * TT, false>(op.c_invader, 0, 1, one, p);
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[t] = sum_terms<TT, false>(p + t * TT);
  } else
#endif
  {
    // (also the fused build's form for one value: its terms after the first
    // are one rounding each, not a product and a sum)
    Line<TT> ln;
#pragma unroll
    for (int p = 0; p < TT; ++p) ln.v[p] = slot[Teff == 1 ? 0 : p * CPB];
    line_ready<TT>(ln, op.soft);
    line_apply<TT, TT, false>(op.c_invader, 0, 1, ln, acc);
  }
#pragma unroll
  for (int t = 0; t < TT; ++t) {
    const double u = usp - acc[t] * dt;
    out[t * stride] = u;
    slot[t * CPB] = u;
  }
}

static __device__ __forceinline__ void run(Blk B, const Ops& op, const Geo& g, int mode, int Teff, int chunk,
                                           const double* __restrict__ Uin, int Tu, const double* __restrict__ dt_ptr,
                                           double* __restrict__ U_sp, double* __restrict__ U_ader, const double* Fi0,
                                           const double* Fi1, const double* Fi2, double* tr0, double* tr1,
                                           double* tr2, double* Ffp0, double* Ffp1, double* Ffp2,
                                           const double* G0 = nullptr, const double* G1 = nullptr,
                                           const double* G2 = nullptr, const double* gphi = nullptr,
                                           const double* M0 = nullptr, const double* M1 = nullptr,
                                           const double* M2 = nullptr, const double* E0 = nullptr,
                                           const double* E1 = nullptr, const double* E2 = nullptr) {
  const bool pot = EXT && gphi != nullptr;
  // the isothermal system runs in the EXT form only (a runtime flag would
  // cost the plain form a predicated FP64 multiply per flux point)
  const Args a{mode, Teff, Tu, (mode == 0) ? g.T : Teff, Uin, EXT && G0 != nullptr, EXT && M0 != nullptr,
               EXT && g.iso != 0};
  extern __shared__ double dudt_s[];
  const int CPB = blockDim.x, rows = blockDim.y;
  const int cl = threadIdx.x, row = threadIdx.y;
  const long long c = B.id * (long long)CPB + cl;
  const bool active = c < g.Nc;
  double* scr = dudt_s + (mode == 2 ? 0 : k::V * k::NS * a.Tn * CPB) + cl;
  direction<true>(op, g, a, 0, chunk, c, active, dudt_s + cl, scr, Dir{Fi0, Ffp0, G0, M0, E0});
#pragma unroll 1
  for (int d = 1; d < D; ++d)
    direction<false>(op, g, a, d, chunk, c, active, dudt_s + cl, scr,
                     d == 1 ? Dir{Fi1, Ffp1, G1, M1, E1} : Dir{Fi2, Ffp2, G2, M2, E2});
  if (mode == 2) return;
  if (pot) {
    __syncthreads();
    // dUdt[vel] += rho * dphi_vel, dUdt[P] += m_vel * dphi_vel, direction by
    // direction, with the iterate the fluxes came from
    for (int i = row; active && i < Teff * k::NS; i += rows) {
      const int s = i % k::NS, t = i / k::NS;
      const int tu = (Tu == 1) ? 0 : t;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double gp = gphi[((long long)d * k::NS + s) * g.Nc + c];
        const double u0 = Uin[(((long long)0 * Tu + tu) * k::NS + s) * g.Nc + c];
        const double uv = Uin[(((long long)(d + 1) * Tu + tu) * k::NS + s) * g.Nc + c];
        double* sv = &dudt_s[(((d + 1) * k::NS + s) * a.Tn + t) * CPB + cl];
        *sv = *sv + u0 * gp;
        if (!a.iso) {
          double* sp = &dudt_s[(((D + 1) * k::NS + s) * a.Tn + t) * CPB + cl];
          *sp = *sp + uv * gp;
        }
      }
    }
  }
  __syncthreads();
  const double dt = *dt_ptr;
  if (mode == 1) {
    for (int kk = row; active && kk < k::V * k::NS; kk += rows) {
      const double* slot = &dudt_s[kk * Teff * CPB + cl];
      double acc;
      if (Teff == k::n) {
        Line<k::n> ln;
#pragma unroll
        for (int t = 0; t < k::n; ++t) ln.v[t] = slot[t * CPB];
        line_ready<k::n>(ln, op.soft);
        line_apply<k::n, 1, false>(op.c_w_tp, 0, 1, ln, &acc);
      } else {
        // m != p (or T = 1): Teff counts the stored nodes
        acc = op.w_tp[0] * slot[0];
        for (int t = 1; t < g.T; ++t) acc = acc + op.w_tp[t] * slot[(Teff == 1 ? 0 : t) * CPB];
      }
      double* u = &U_sp[(long long)kk * g.Nc + c];
      *u = *u - acc * dt;
    }
    return;
  }
  for (int kk = row; active && kk < k::V * k::NS; kk += rows) {
    const int v = kk / k::NS, s = kk % k::NS;
    double* slot = &dudt_s[kk * a.Tn * CPB + cl];
    const double usp = U_sp[(long long)kk * g.Nc + c];
    double* out = &U_ader[(((long long)v * g.T) * k::NS + s) * g.Nc + c];
    const long long stride = (long long)k::NS * g.Nc;
    if (g.T == k::n) {
      picard<k::n>(op, g, slot, CPB, Teff, dt, usp, out, stride);
    } else {
      // m != p
      double x[MAXT];
      for (int p = 0; p < g.T; ++p) x[p] = slot[(Teff == 1 ? 0 : p) * CPB];
      for (int t = 0; t < g.T; ++t) {
        double acc = op.invader[t * g.T + 0] * x[0];
        for (int p = 1; p < g.T; ++p) acc = acc + op.invader[t * g.T + p] * x[p];
        const double u = usp - acc * dt;
        out[t * stride] = u;
        slot[t * CPB] = u;
      }
    }
  }
  __syncthreads();
  if (!active) return;
#pragma unroll 1
  for (int item = row; item < D * g.T * k::NJ * k::V; item += rows) {
    const int d = item / (g.T * k::NJ * k::V), r = item % (g.T * k::NJ * k::V);
    const int v = r % k::V, t = r / (k::V * k::NJ), j = r / k::V % k::NJ;
    auto at = [&](int s) { return dudt_s[((v * k::NS + s) * g.T + t) * CPB + cl]; };
    if (d == 0) trace_line<D, P, true>(op, g, at, c, tr0, t, 0, j, v);
    else trace_line<D, P, false>(op, g, at, c, d == 1 ? tr1 : tr2, t, d, j, v);
  }
}
};
template <int D, int P>
__global__ void __launch_bounds__(INTERIOR_THREADS, (interior_blocks<D, P>)) k_interior(Ops op, Geo g, int mode, int Teff, int chunk, const double* __restrict__ Uin, int Tu,
                           const double* __restrict__ dt_ptr, double* __restrict__ U_sp, double* __restrict__ U_ader,
                           const double* Fi0, const double* Fi1, const double* Fi2, double* tr0, double* tr1,
                           double* tr2, double* Ffp0, double* Ffp1, double* Ffp2) {
  Interior<D, P>::run(hw_blk(), op, g, mode, Teff, chunk, Uin, Tu, dt_ptr, U_sp, U_ader, Fi0, Fi1, Fi2, tr0, tr1, tr2, Ffp0,
                      Ffp1, Ffp2);
}
template <int D, int P>
struct InteriorExt {
  static __device__ __forceinline__ void run(Blk B, const Ops& op, const Geo& g, int mode, int Teff, int chunk,
                                             const double* __restrict__ Uin, int Tu, const double* __restrict__ dt_ptr,
                                             double* __restrict__ U_sp, double* __restrict__ U_ader,
                                             const double* Fi0, const double* Fi1, const double* Fi2, double* tr0,
                                             double* tr1, double* tr2, double* Ffp0, double* Ffp1, double* Ffp2,
                                             const double* G0, const double* G1, const double* G2,
                                             const double* gphi, const double* M0, const double* M1,
                                             const double* M2, const double* E0, const double* E1,
                                             const double* E2) {
    Interior<D, P, true>::run(B, op, g, mode, Teff, chunk, Uin, Tu, dt_ptr, U_sp, U_ader, Fi0, Fi1, Fi2, tr0, tr1, tr2, Ffp0,
                              Ffp1, Ffp2, G0, G1, G2, gphi, M0, M1, M2, E0, E1, E2);
  }
};
template <int D, int P>
__global__ void __launch_bounds__(INTERIOR_THREADS, (interior_blocks<D, P>)) k_interior_ext(Ops op, Geo g, int mode, int Teff, int chunk, const double* __restrict__ Uin, int Tu,
                               const double* __restrict__ dt_ptr, double* __restrict__ U_sp,
                               double* __restrict__ U_ader, const double* Fi0, const double* Fi1, const double* Fi2,
                               double* tr0, double* tr1, double* tr2, double* Ffp0, double* Ffp1, double* Ffp2,
                               const double* G0, const double* G1, const double* G2, const double* gphi,
                               const double* M0, const double* M1, const double* M2, const double* E0,
                               const double* E1, const double* E2) {
  InteriorExt<D, P>::run(hw_blk(), op, g, mode, Teff, chunk, Uin, Tu, dt_ptr, U_sp, U_ader, Fi0, Fi1, Fi2, tr0, tr1, tr2,
                         Ffp0, Ffp1, Ffp2, G0, G1, G2, gphi, M0, M1, M2, E0, E1, E2);
}

// ---------------------------------------------------------------------------
// transverse subcell averaging of the flux points and scatter to the FV face
// arrays of time node t (src/sd_simulator.py:208-212,
// src/sdader_simulator.py:310-323).  One thread per (direction, cell, t, fp).
// F_HO layout [t][v][face], faces x-fastest with X_d + 1 along d.
// ---------------------------------------------------------------------------
struct FaceArrays {
  const double* Ffp[3];
  double* F_HO[3];
};
template <int D, int P>
struct IntegrateFaces {
static __device__ __forceinline__ void run(Blk B, const Ops& op, const Geo& g, const FaceArrays& fa) {
  using k = K<D, P>;
  const long long total = g.Nc * g.T * k::nf;  // per direction
  const long long gid = B.id * (long long)blockDim.x + threadIdx.x;
  if (gid >= D * total) return;
  const int d = (int)(gid / total);
  const long long tid = gid - d * total;
  const double* __restrict__ Ffp = d == 0 ? fa.Ffp[0] : (d == 1 ? fa.Ffp[1] : fa.Ffp[2]);
  double* __restrict__ F_HO = d == 0 ? fa.F_HO[0] : (d == 1 ? fa.F_HO[1] : fa.F_HO[2]);
  const long long c = tid % g.Nc;
  const long long r = tid / g.Nc;
  const int f = (int)(r % k::nf);
  const int t = (int)(r / k::nf);
  int cx, cy, cz;
  cell_coords(g, c, cx, cy, cz);
  const int cd = (d == 0) ? cx : (d == 1 ? cy : cz);
  if (f == k::nf - 1 && cd != g.N[d] - 1) return;
  const int fd = (f == k::nf - 1) ? g.N[d] * k::n : cd * k::n + f;
  const int FX = g.X[0] + (d == 0), FY = g.X[1] + (d == 1);
  const long long nface = (long long)FX * FY * (g.X[2] + (d == 2));
  // the other directions in increasing order
  int o0 = -1, o1 = -1;
  for (int e = 0; e < D; ++e) {
    if (e == d) continue;
    if (o0 < 0) o0 = e; else o1 = e;
  }
#pragma unroll 1
  for (int v = 0; v < k::V; ++v) {
    double G[k::NJ];
#pragma unroll
    for (int j = 0; j < k::NJ; ++j)
      G[j] = Ffp[((((long long)v * g.T + t) * k::NJ + j) * k::nf + f) * g.Nc + c];
    // transverse index j = a + n*b where a is the lower other direction
    if (D >= 2) {
      double G1[k::NJ];
      // along o0 (index a)
#pragma unroll
      for (int b = 0; b < k::NJ / k::n; ++b) {
        Line<k::n> ln;
#pragma unroll
        for (int a = 0; a < k::n; ++a) ln.v[a] = G[a + k::n * b];
        line_ready<k::n>(ln, op.soft);
        if (o0 == 0) line_apply<k::n, k::n, true>(op.c_sp_to_cv, 0, 1, ln, &G1[k::n * b]);
        else line_apply<k::n, k::n, false>(op.c_sp_to_cv, 0, 1, ln, &G1[k::n * b]);
      }
      if (D == 3) {
#pragma unroll
        for (int a = 0; a < k::n; ++a) {
          Line<k::n> ln;
#pragma unroll
          for (int b = 0; b < k::n; ++b) ln.v[b] = G1[a + k::n * b];
          line_ready<k::n>(ln, op.soft);
          double o[k::n];
          line_apply<k::n, k::n, false>(op.c_sp_to_cv, 0, 1, ln, o);  // o1 is y or z
#pragma unroll
          for (int bo = 0; bo < k::n; ++bo) G[a + k::n * bo] = o[bo];
        }
      } else {
#pragma unroll
        for (int jj = 0; jj < k::NJ; ++jj) G[jj] = G1[jj];
      }
    }
    for (int j = 0; j < k::NJ; ++j) {
      const int a = j % k::n, b = j / k::n;
      int fc[3] = {0, 0, 0};
      fc[d] = fd;
      const int cc[3] = {cx, cy, cz};
      if (o0 >= 0) fc[o0] = cc[o0] * k::n + a;
      if (o1 >= 0) fc[o1] = cc[o1] * k::n + b;
      const long long fid = fc[0] + (long long)FX * (fc[1] + (long long)FY * fc[2]);
      F_HO[((long long)t * k::V + v) * nface + fid] = G[j];
    }
  }
}
};
template <int D, int P>
__global__ void k_integrate_faces(Ops op, Geo g, FaceArrays fa) {
  IntegrateFaces<D, P>::run(hw_blk(), op, g, fa);
}

// ---------------------------------------------------------------------------
// whole-cell transforms sp <-> subcell averages (src/transforms.py:27-45)
// Kt[i][o] holds the operator product ((A*A)*A) of input point i and output
// point o, formed exactly as the reference's einsum does.
// ROWS = false: one left-to-right sum over all input points (contiguous
//               input), 1D: two-lane sum, 2D with n = 2: row pairs;
// ROWS = true : per-row sums along x, then the row sums in order (strided
//               input, src/sdader_simulator.py:302-307).
//
// One thread per (cell, variable, tile of O output points); the input points
// are taken in the order of the sums, each prepared once for the tile's
// products (spd_soft.cuh).  The bound is the FP64 addition per term; a tile
// keeps the sums in registers, where all n^d inputs of a cell at once were
// 250 registers in 3D at degree 4.  A sum starts from -0, which leaves its
// first term as it is.
// ---------------------------------------------------------------------------
template <int D, int P>
struct Full {
  using k = K<D, P>;
  static constexpr int O = (k::NS <= 9) ? k::NS : (k::NS % 9 == 0 ? 9 : (k::NS % 8 == 0 ? 8 : 5));
  static constexpr int tiles = k::NS / O;
  static_assert(k::NS % O == 0, "tiles of outputs");
  // subcell index of point s of cell c
  static __device__ __forceinline__ long long subcell(const Geo& g, long long c, int s) {
    int cx, cy, cz;
    cell_coords(g, c, cx, cy, cz);
    const int kx = s % k::n, ky = (s / k::n) % k::n, kz = s / (k::n * k::n);
    return (cx * k::n + kx) + (long long)g.X[0] * ((D >= 2 ? cy * k::n + ky : 0) +
                                                  (long long)g.X[1] * (D >= 3 ? cz * k::n + kz : 0));
  }
  template <bool ROWS, class Get>
  static __device__ __forceinline__ void apply(const Coef* __restrict__ Kt, int soft, int o0, Get get, double* acc) {
    double part[O];  // the row's sum, or in 1D the sum of the odd terms
#pragma unroll
    for (int o = 0; o < O; ++o) acc[o] = part[o] = -0.0;
#pragma unroll 1
    for (int r = 0; r < k::NS / k::n; ++r) {
#pragma unroll
      for (int l = 0; l < k::n; ++l) {
        const int s = r * k::n + l;
        const Coef* K = Kt + (long long)s * k::NS + o0;
        const double x = get(s);
        double p[O];
#ifdef SPD_FUSED
#pragma unroll
        for (int o = 0; o < O; ++o) p[o] = coef_value(K[o], 0u) * x;
#else
        uint32_t ok = soft ? 0x40000000u : 0u;
        const Opnd xo = opnd_of(x, ok);
        if (ok != 0u) {
#pragma unroll
          for (int o = 0; o < O; ++o) p[o] = soft_prod(K[o], xo);
        } else {
#pragma unroll
          for (int o = 0; o < O; ++o) p[o] = coef_value(K[o], 0u) * x;
        }
#endif
#pragma unroll
        for (int o = 0; o < O; ++o) {
          if (D == 1 ? l % 2 == 1 : ROWS || (D == 2 && k::n == 2))
            part[o] = (D > 1 && l == 0) ? p[o] : part[o] + p[o];
          else
            acc[o] = acc[o] + p[o];
        }
      }
      if (D > 1 && (ROWS || (D == 2 && k::n == 2))) {
#pragma unroll
        for (int o = 0; o < O; ++o) acc[o] = acc[o] + part[o];
      }
    }
    if (D == 1) {
#pragma unroll
      for (int o = 0; o < O; ++o) acc[o] = acc[o] + part[o];
    }
  }
};

// U_cv (FV layout) = sp_to_cv(U_sp) for every cell and variable
template <int D, int P>
struct SpToCv {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const Coef* __restrict__ Kt, int soft,
                                           const double* __restrict__ U_sp, double* __restrict__ U_cv) {
  using k = K<D, P>;
  using F = Full<D, P>;
  const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
  if (tid >= g.Nc * (k::V * F::tiles)) return;
  const long long c = tid % g.Nc;
  const int r = (int)(tid / g.Nc);
  const int v = r / F::tiles, o0 = r % F::tiles * F::O;
  double acc[F::O];
  F::template apply<false>(Kt, soft, o0, [&](int s) { return U_sp[((long long)v * k::NS + s) * g.Nc + c]; }, acc);
#pragma unroll
  for (int o = 0; o < F::O; ++o) U_cv[(long long)v * g.Nq + F::subcell(g, c, o0 + o)] = acc[o];
}
};
template <int D, int P>
__global__ void k_sp_to_cv(Geo g, const Coef* __restrict__ Kt, int soft, const double* __restrict__ U_sp,
                           double* __restrict__ U_cv) {
  SpToCv<D, P>::run(hw_blk(), g, Kt, soft, U_sp, U_cv);
}

// U_sp = cv_to_sp(U_cv) (strided view order)
template <int D, int P>
struct CvToSp {
static __device__ __forceinline__ void run(Blk B, const Geo& g, const Coef* __restrict__ Kt, int soft,
                                           const double* __restrict__ U_cv, double* __restrict__ U_sp) {
  using k = K<D, P>;
  using F = Full<D, P>;
  const long long tid = B.id * (long long)blockDim.x + threadIdx.x;
  if (tid >= g.Nc * (k::V * F::tiles)) return;
  const long long c = tid % g.Nc;
  const int r = (int)(tid / g.Nc);
  const int v = r / F::tiles, o0 = r % F::tiles * F::O;
  double acc[F::O];
  F::template apply<true>(Kt, soft, o0, [&](int s) { return U_cv[(long long)v * g.Nq + F::subcell(g, c, s)]; }, acc);
#pragma unroll
  for (int o = 0; o < F::O; ++o) U_sp[((long long)v * k::NS + o0 + o) * g.Nc + c] = acc[o];
}
};
template <int D, int P>
__global__ void k_cv_to_sp(Geo g, const Coef* __restrict__ Kt, int soft, const double* __restrict__ U_cv,
                           double* __restrict__ U_sp) {
  CvToSp<D, P>::run(hw_blk(), g, Kt, soft, U_cv, U_sp);
}

}  // namespace spd
