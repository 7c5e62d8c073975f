// The first Picard iteration's contraction in the fused build: one derivative
// value for all time nodes, whose terms after the first are added with fused
// multiply-adds, one rounding each, as in the later iterations.  The interior
// kernel's function runs on the CPU, on operators whose terms cancel.
#include <cmath>
#include <cstdio>
#include <random>

#include "cpu_device_shim.h"
#include "spd_kernels.cuh"

using namespace spd;

template <int T>
int check(std::mt19937_64& rng) {
  std::uniform_real_distribution<double> u(-2.0, 2.0);
  static Ops op;
  op.soft = 1;
  double A[T * T];
  for (int i = 0; i < T * T; ++i) {
    A[i] = u(rng);
    op.c_invader[i] = coef_of(A[i]);
  }
  Geo g{};
  g.T = T;
  const double x = u(rng);
  double slot[T], out[T];
  for (int t = 0; t < T; ++t) slot[t] = x;
  Interior<2, T - 1>::template picard<T>(op, g, slot, 1, 1, 1.0, 0.0, out, 1);
  int bad = 0;
  for (int t = 0; t < T; ++t) {
    double acc = A[t * T] * x;
    for (int s = 1; s < T; ++s) acc = std::fma(A[t * T + s], x, acc);
    bad += !(out[t] == 0.0 - acc * 1.0 && slot[t] == out[t]);
  }
  return bad;
}

int main() {
  std::mt19937_64 rng(5);
  int bad = 0;
  for (int i = 0; i < 10000; ++i) bad += check<2>(rng) + check<3>(rng) + check<4>(rng) + check<5>(rng);
  printf("%d sums differ from the fused ones\n", bad);
  return bad != 0;
}
