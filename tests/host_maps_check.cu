// The Euler maps and Riemann solvers of spd_device.cuh in the forms that the
// step's kernels call (products on the integer pipes where they run there,
// with their fallback) against the same maps in plain FP64 arithmetic, bit for
// bit (any NaN equals any other): fluid states with values put to zeros of
// either sign (the density included), the ends of the exponent window,
// subnormals, infinities or NaN.  Runs on the host; with the argument "gpu" on
// the device.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "spd_device.cuh"

using namespace spd;

static double bits(unsigned long long b) {
  double x;
  memcpy(&x, &b, sizeof(x));
  return x;
}
constexpr int W = 5;  // values of a state, as many as 3D has

struct Problem {
  double L[W], R[W], gamma, min_c2;
  int prims, iso;
};
static double special(std::mt19937_64& rng) {
  static const unsigned edges[] = {0, 0, 1, 510, 511, 512, 513, 700, 766, 767, 768, 1278, 1279, 1280, 1400, 1533, 1534, 1535, 1536, 2046, 2047};
  const unsigned long long r = rng(), sign = r & (1ULL << 63);
  const unsigned long long man = (r >> 8) % 4 == 0 ? 0ULL : rng() & 0xfffffffffffffULL;
  return bits(sign | (unsigned long long)edges[(r >> 24) % 21] << 52 | man);
}
static Problem draw(std::mt19937_64& rng, int i) {
  Problem p;
  std::uniform_real_distribution<double> u(0.1, 3.0);
  double* s[2] = {p.L, p.R};
  for (int k = 0; k < 2; ++k)
    for (int v = 0; v < W; ++v) s[k][v] = (v == 1 || v == 2) && rng() % 2 ? -u(rng) : u(rng);
  // up to three special values; every fourth problem a density of zero
  for (unsigned n = (unsigned)(rng() % 4); n > 0; --n) s[rng() % 2][rng() % W] = special(rng);
  if (i % 4 == 0) s[rng() % 2][0] = rng() % 2 ? 0.0 : -0.0;
  static const double floors[] = {1e-20, 1e-10, 0.0, 1e-300, 1.0};
  p.gamma = rng() % 2 ? 1.4 : 5.0 / 3.0;
  p.min_c2 = floors[rng() % 5];
  p.prims = (int)(rng() % 2);
  p.iso = rng() % 8 == 0;
  return p;
}

template <int N>
SPD_FN int differ(const double* a, const double* b) {
  int n = 0;
  for (int v = 0; v < N; ++v)
    n += !((a[v] != a[v] && b[v] != b[v]) || (hi_word(a[v]) == hi_word(b[v]) && lo_word(a[v]) == lo_word(b[v])));
  return n;
}
// mismatches: [0] LLF, [1] HLLC forms, [2] conversions, [3] fluxes
template <int D>
SPD_FN void check_dim(const Problem& p, int* bad) {
  constexpr int V = D + 2;
  const Rcp rg = recip_of(p.gamma - 1.0);
  const bool iso = p.iso != 0, prims_in = p.prims != 0;
  for (int d = 0; d < D; ++d) {
    for (int solver = RS_LLF; solver <= RS_LHLLC; ++solver) {
      double WL[V], WR[V], UL[V], UR[V], f[V], g[V];
      for (int v = 0; v < V; ++v) {
        WL[v] = UL[v] = p.L[v];
        WR[v] = UR[v] = p.R[v];
      }
      riemann<D, double>(solver, UL, UR, f, p.gamma, p.min_c2, d, prims_in, (Br<0>*)nullptr, iso, &rg);
      Rcp rL, rR;
      if (prims_in) {
        cons<D, double>(WL, UL, p.gamma, d, iso);
        cons<D, double>(WR, UR, p.gamma, d, iso);
        rL = recip_of(WL[0]);
        rR = recip_of(WR[0]);
      } else {
        prim<D, double>(UL, WL, p.gamma, d, &rL, iso);
        prim<D, double>(UR, WR, p.gamma, d, &rR, iso);
      }
      if (solver == RS_LLF)
        llf<D, double>(WL, WR, UL, UR, g, p.gamma, p.min_c2, d, (Br<0>*)nullptr, &rL, &rR, iso);
      else
        hllc<D, double>(WL, WR, UL, UR, g, p.gamma, p.min_c2, d, solver == RS_LHLLC, (Br<0>*)nullptr, &rL, &rR, iso);
      bad[solver == RS_LLF ? 0 : 1] += differ<V>(f, g);
    }
    double U[V], P[V], f[V], r[V], F[V];
    for (int v = 0; v < V; ++v) U[v] = p.L[v];
    euler_flux<D>(U, p.gamma, d, iso, &rg, [&](int v, double x) { f[v] = x; });
    prim<D, double>(U, P, p.gamma, 0, nullptr, iso);
    flux<D, double>(P, F, p.gamma, d, iso);
    bad[3] += differ<V>(f, F);
    prims<D>(U, r, p.gamma, iso);
    bad[2] += differ<V>(r, P);
  }
}
SPD_FN void check_one(const Problem& p, int* bad) {
  check_dim<1>(p, bad);
  check_dim<2>(p, bad);
  check_dim<3>(p, bad);
}
__global__ void k_check(const Problem* p, int n, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int b[4] = {0, 0, 0, 0};
  check_one(p[i], b);
  for (int k = 0; k < 4; ++k)
    if (b[k]) atomicAdd(bad + k, b[k]);
}

int main(int argc, char** argv) {
  const bool gpu = argc > 1 && !strcmp(argv[1], "gpu");
  std::mt19937_64 rng(1205);
  const int n = 1 << 16;
  std::vector<Problem> p;
  for (int i = 0; i < n; ++i) p.push_back(draw(rng, i));
  // a zero density with gamma P >= 2: its quotient's exponent wraps
  const double l[W] = {0.0, 0.3, 2.0, 2.0, 2.0}, r[W] = {1.0, 0.2, 1.0, 1.0, 1.0};
  memcpy(p[0].L, l, sizeof(l));
  memcpy(p[0].R, r, sizeof(r));
  p[0].gamma = 1.4;
  p[0].min_c2 = 1e-20;
  p[0].prims = 1;
  p[0].iso = 0;
  int bad[4] = {0, 0, 0, 0};
  if (!gpu) {
    for (const Problem& q : p) check_one(q, bad);
  } else {
    Problem* dp;
    int* db;
    cudaMalloc(&dp, p.size() * sizeof(Problem));
    cudaMalloc(&db, sizeof(bad));
    cudaMemcpy(dp, p.data(), p.size() * sizeof(Problem), cudaMemcpyHostToDevice);
    cudaMemset(db, 0, sizeof(bad));
    k_check<<<(n + 127) / 128, 128>>>(dp, n, db);
    const cudaError_t e = cudaMemcpy(bad, db, sizeof(bad), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      printf("%s\n", cudaGetErrorString(e));
      return 2;
    }
  }
  printf("mismatches: LLF %d, HLLC %d, conversions %d, fluxes %d\n", bad[0], bad[1], bad[2], bad[3]);
  return bad[0] + bad[1] + bad[2] + bad[3] ? 1 : 0;
}
