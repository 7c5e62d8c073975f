// The integer-pipe arithmetic of spd_soft.cuh and spd_lines.cuh against IEEE
// arithmetic, bit for bit (any NaN equals any other): quotients, square roots
// and operator contractions over significands and exponents at the edges of
// what the fast paths accept (short, all-ones and near-power-of-two
// significands, the exponent windows' ends, zeros, subnormals, infinities,
// NaN).  Runs on the host; with the argument "gpu" also on the device, whose
// reciprocal approximations and carry chains are others.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "spd_lines.cuh"

using namespace spd;

static double bits(unsigned long long b) {
  double x;
  memcpy(&x, &b, sizeof(x));
  return x;
}

static double draw(std::mt19937_64& rng) {
  const unsigned long long r = rng();
  unsigned long long man = rng() & 0xfffffffffffffULL;
  switch (r & 7) {
    case 0: man = (man >> ((r >> 8) % 53)) << ((r >> 8) % 53); break;       // trailing zeros
    case 1: man = 0xfffffffffffffULL & ~((1ULL << ((r >> 8) % 53)) - 1); break;  // leading ones
    case 2: man = (r >> 8) % 8; break;                                      // just above a power of two
    case 3: man = 0xfffffffffffffULL - (r >> 8) % 8; break;                 // just below
    default: break;
  }
  static const unsigned edges[] = {0, 1, 510, 511, 512, 513, 766, 767, 768, 1022, 1023, 1024, 1278, 1279, 1280,
                                   1534, 1535, 1536, 1537, 2045, 2046, 2047};
  const unsigned pick = (unsigned)((r >> 16) % 16);
  unsigned long long e;
  if (pick < 3) e = edges[(r >> 24) % (sizeof(edges) / sizeof(edges[0]))];
  else if (pick < 10) e = 1023 - 40 + (r >> 24) % 80;
  else e = 1023 - 480 + (r >> 24) % 960;
  if (pick == 15 && (r & 1)) return bits(r & (1ULL << 63));  // a zero
  return bits((r & (1ULL << 63)) | (e << 52) | man);
}

SPD_FN bool same(double a, double b) {
  return (a != a && b != b) || (hi_word(a) == hi_word(b) && lo_word(a) == lo_word(b));
}

template <int L, int R, bool LANES2>
SPD_FN int check_lines(const Coef* C, const double* A, int use, const double* x, int kk) {
  const int k = use ? kk : 0;  // an operator out of range is not scaled
  Line<L> ln;
  for (int s = 0; s < L; ++s) ln.v[s] = x[s];
  line_ready<L>(ln, use, (uint32_t)k << 20);
  double out[R];
  line_apply<L, R, LANES2>(C, 0, 1, ln, out);
  int bad = 0;
  for (int r = 0; r < R; ++r) {
    double As[L];
    for (int s = 0; s < L; ++s) As[s] = from_words(hi_word(A[r * L + s]) + ((uint32_t)k << 20), lo_word(A[r * L + s]));
    bad += !same(out[r], LANES2 ? dot_lanes2<L>(As, ln.v) : dot_seq<L>(As, ln.v));
  }
  return bad;
}

// counts of mismatches: quotients, roots, contractions
SPD_FN void check_one(const double* v, const Coef* C, const double* A, int use, int* bad) {
  bad[0] += !same(div_by(v[0], v[1], recip_of(v[1])), v[0] / v[1]);
  bad[0] += !same(quot(v[2] * v[3], v[3]), v[2] * v[3] / v[3]);
  bad[1] += !same(ad_sqrt(v[2]), sqrt(v[2]));
  const double s = fabs(v[4]) * fabs(v[4]);
  bad[1] += !same(ad_sqrt(s), sqrt(s));
  bad[2] += check_lines<2, 3, true>(C, A, use, v, 0) + check_lines<2, 2, false>(C, A, use, v, 4);
  bad[2] += check_lines<5, 4, true>(C, A, use, v, -3) + check_lines<4, 4, false>(C, A, use, v, 0);
  bad[2] += check_lines<6, 5, false>(C, A, use, v, 9) + check_lines<1, 6, false>(C, A, use, v, 0);
}

__global__ void k_check(const double* v, const Coef* C, const double* A, int use, int n, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int b[3] = {0, 0, 0};
  check_one(v + 6 * (long long)i, C, A, use, b);
  for (int k = 0; k < 3; ++k)
    if (b[k]) atomicAdd(bad + k, b[k]);
}

int main(int argc, char** argv) {
  const bool gpu = argc > 1 && !strcmp(argv[1], "gpu");
  std::mt19937_64 rng(20260728);
  const int n = gpu ? 1 << 20 : 1 << 18;
  int failed = 0;
  for (int round = 0; round < 4; ++round) {
    // operator entries: generic, short, at the ends of their range, and one
    // operator that is out of it
    std::vector<double> A(36), v(6 * (size_t)n);
    int use = 1;
    for (size_t i = 0; i < A.size(); ++i) {
      std::uniform_real_distribution<double> u(-4.0, 4.0);
      A[i] = round == 1 ? (double)((int)(rng() % 15) - 7) / 8 + 0x1p-30 : u(rng);
      if (round == 2 && i % 5 == 0) A[i] = (i & 1) ? 0x1p256 : -0x1p-256;
      if (round == 3 && i == 7) A[i] = 0.0;
      use = use && coef_in_range(A[i]);
    }
    std::vector<Coef> C(A.size());
    for (size_t i = 0; i < A.size(); ++i) C[i] = coef_of(A[i]);
    for (double& x : v) x = draw(rng);
    for (int i = 0; i + 8 < n; i += 8)
      for (int s = 0; s < 6; ++s) {
        v[6 * (size_t)i + s] = 0.0;                                     // a line at rest
        if (s != 2) v[6 * ((size_t)i + 1) + s] = bits(rng() & (1ULL << 63));  // zeros of either sign around a value
      }
    int bad[3] = {0, 0, 0};
    if (!gpu) {
      for (int i = 0; i < n; ++i) check_one(&v[6 * (size_t)i], C.data(), A.data(), use, bad);
    } else {
      double *dv, *dA;
      Coef* dC;
      int* db;
      cudaMalloc(&dv, v.size() * sizeof(double));
      cudaMalloc(&dA, A.size() * sizeof(double));
      cudaMalloc(&dC, C.size() * sizeof(Coef));
      cudaMalloc(&db, sizeof(bad));
      cudaMemcpy(dv, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice);
      cudaMemcpy(dA, A.data(), A.size() * sizeof(double), cudaMemcpyHostToDevice);
      cudaMemcpy(dC, C.data(), C.size() * sizeof(Coef), cudaMemcpyHostToDevice);
      cudaMemset(db, 0, sizeof(bad));
      k_check<<<(n + 127) / 128, 128>>>(dv, dC, dA, use, n, db);
      const cudaError_t e = cudaMemcpy(bad, db, sizeof(bad), cudaMemcpyDeviceToHost);
      if (e != cudaSuccess) {
        printf("%s\n", cudaGetErrorString(e));
        return 2;
      }
      cudaFree(dv);
      cudaFree(dA);
      cudaFree(dC);
      cudaFree(db);
    }
    printf("operator %d: mismatches: quotients %d, roots %d, contractions %d\n", round, bad[0], bad[1], bad[2]);
    failed += bad[0] + bad[1] + bad[2];
  }
  return failed ? 1 : 0;
}
