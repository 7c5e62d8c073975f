// The viscous kernels' bodies run on the CPU, unoptimised, thread by thread,
// every device array ending at a page that may not be touched: an access
// beyond an array of the sizes that the context allocates ends the program.
#include <sys/mman.h>
#include <unistd.h>

#include <cmath>
#include <cstdio>
#include <initializer_list>

#include "cpu_device_shim.h"
#include "spd_visc.cuh"

using namespace spd;

static double* guarded(size_t count) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = count * sizeof(double);
  const size_t body = (bytes + page - 1) / page * page;
  char* m = (char*)mmap(nullptr, body + page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (m == MAP_FAILED || mprotect(m + body, page, PROT_NONE) != 0) return nullptr;
  return (double*)(m + body - bytes);
}

// the operators' values do not matter here: sp_to_fp picks a point, dfp_to_sp
// takes a difference
template <int D, int P>
int run(int bc) {
  using k = K<D, P>;
  static Ops op;
  Geo g{};
  g.T = 2;
  g.Nc = 1;
  for (int d = 0; d < 3; ++d) {
    g.N[d] = d < D ? 2 + d : 1;
    g.X[d] = d < D ? g.N[d] * k::n : 1;
    g.Xe[d] = d < D ? g.X[d] + 4 : 1;
    g.Nc *= g.N[d];
    g.h[d] = 1.0;
    g.rh[d] = recip_of(1.0);
    g.bc[d][0] = g.bc[d][1] = bc;
  }
  g.gamma = 1.4;
  for (int f = 0; f < k::nf; ++f)
    for (int s = 0; s < k::n; ++s) op.sp_to_fp[f * k::n + s] = (s == (f < k::n ? f : k::n - 1)) ? 1.0 : 0.0;
  for (int s = 0; s < k::n; ++s)
    for (int f = 0; f < k::nf; ++f) op.dfp_to_sp[s * k::nf + f] = f == s + 1 ? 1.0 : (f == s ? -1.0 : 0.0);
  for (int i = 0; i < k::nf * k::n; ++i) {
    op.c_sp_to_fp[i] = coef_of(op.sp_to_fp[i]);
    op.c_dfp[i] = coef_of(op.dfp_to_sp[i]);
  }
  op.soft = 0;
  const size_t lines = (size_t)g.T * k::NJ * k::nf * g.Nc;
  double* U = guarded((size_t)k::V * g.T * k::NS * g.Nc);
  for (size_t i = 0; i < (size_t)k::V * g.T * k::NS * g.Nc; ++i) U[i] = 1.0 + 0.01 * (double)(i % 7);
  double* dWsp = guarded((size_t)D * D * g.T * k::NS * g.Nc);
  double *tr[3] = {}, *bf[3] = {}, *W[3] = {}, *G[3] = {};
  for (int d = 0; d < D; ++d) {
    const size_t nt = (size_t)2 * k::V * g.T * k::NJ * g.Nc, nb = (size_t)2 * k::V * k::NJ * (g.Nc / g.N[d]);
    tr[d] = guarded(nt);
    for (size_t i = 0; i < nt; ++i) tr[d][i] = 1.0;
    bf[d] = guarded(nb);
    for (size_t i = 0; i < nb; ++i) bf[d][i] = 1.0;
    W[d] = guarded((size_t)(D + 1) * lines);  // density and velocities
    G[d] = guarded((size_t)k::V * lines);
  }
  const long long threads = g.Nc * (D * k::NJ) * g.T;
  blockDim.x = VISC_THREADS;
  const unsigned blocks = (unsigned)((threads + VISC_THREADS - 1) / VISC_THREADS);
  for (unsigned b = 0; b < blocks; ++b)
    for (threadIdx.x = 0; threadIdx.x < VISC_THREADS; ++threadIdx.x)
      ViscGrad<D, P>::run(Blk{b, blocks}, op, g, g.T, U, g.T, tr[0], tr[1], tr[2], bf[0], bf[1], bf[2], W[0], W[1],
                          W[2], dWsp, nullptr, nullptr, nullptr);
  for (unsigned b = 0; b < blocks; ++b)
    for (threadIdx.x = 0; threadIdx.x < VISC_THREADS; ++threadIdx.x)
      ViscFlux<D, P>::run(Blk{b, blocks}, op, g, g.T, dWsp, W[0], W[1], W[2], bf[0], bf[1], bf[2], 0.1, 2.0 / 3.0,
                          G[0], G[1], G[2]);
  // the mass flux is zero, every other component finite
  int bad = 0;
  for (int d = 0; d < D; ++d)
    for (size_t i = 0; i < (size_t)k::V * lines; ++i) bad += i < lines ? G[d][i] != 0.0 : !std::isfinite(G[d][i]);
  return bad;
}

int main() {
  int bad = 0;
  for (int bc : {BC_PERIODIC, BC_REFLECTIVE, BC_GRADFREE, BC_IC, BC_EQ, BC_PRESSURE})
    bad += run<1, 1>(bc) + run<1, 4>(bc) + run<2, 2>(bc) + run<2, 3>(bc) + run<3, 1>(bc);
  printf("%d values wrong\n", bad);
  return bad != 0;
}
