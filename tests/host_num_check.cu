// The expressions of spd_soft.cuh's Num (values whose products, quotients and
// roots run on the integer pipes, with a flag for their range) against IEEE
// arithmetic: a result whose flag is set has the IEEE bits, and the flag is
// set for operands well inside the range.  Operands: generic ones, the ends of
// the exponent window, zeros of either sign, subnormals, infinities, NaN, and
// pairs whose product rounds to 2^1025, just above the largest double.  Runs
// on the host; with the argument "gpu" on the device.
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
static double draw(std::mt19937_64& rng) {
  const unsigned long long r = rng(), sign = r & (1ULL << 63);
  unsigned long long man = rng() & 0xfffffffffffffULL;
  if ((r & 3) == 0) man = (man >> ((r >> 8) % 53)) << ((r >> 8) % 53);  // trailing zeros
  if ((r & 3) == 1) man = 0xfffffffffffffULL - (r >> 8) % 4;            // just below a power of two
  static const unsigned edges[] = {0, 1, 511, 512, 513, 766, 767, 1278, 1279, 1280, 1534, 1535, 1536, 2046, 2047};
  const unsigned pick = (unsigned)((r >> 16) % 16);
  if (pick == 15) return bits(sign);
  if (pick < 5) return bits(sign | (unsigned long long)edges[(r >> 24) % 15] << 52 | man);
  if (pick < 11) return bits(sign | (1023ULL - 30 + (r >> 24) % 60) << 52 | man);
  return bits(sign | (512ULL + (r >> 24) % 1024) << 52 | man);
}

SPD_FN int wrong(const Num& a, double b) {
  if (a.ok == 0u) return 0;
  return !(hi_word(a.v) == hi_word(b) && lo_word(a.v) == lo_word(b));
}
// mismatches of one pair; flagged counts its results in range
SPD_FN int check_pair(double x, double y, int* flagged) {
  const Num a(x), b(y);
  const Num r[8] = {a + b, a - b, a * b, a / b, half(a), -a, ad_abs(a), ad_sqrt(ad_abs(a))};
  const double e[8] = {x + y, x - y, x * y, x / y, 0.5 * x, -x, fabs(x), sqrt(fabs(x))};
  int bad = 0;
  for (int k = 0; k < 8; ++k) {
    bad += wrong(r[k], e[k]);
    *flagged += r[k].ok != 0u;
  }
  return bad;
}
__global__ void k_check(const double* v, int n, int* bad, int* flagged) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int f = 0;
  const int b = check_pair(v[2 * (long long)i], v[2 * (long long)i + 1], &f);
  if (b) atomicAdd(bad, b);
  atomicAdd(flagged, f);
}

int main(int argc, char** argv) {
  const bool gpu = argc > 1 && !strcmp(argv[1], "gpu");
  std::mt19937_64 rng(20261205);
  const int n = 1 << 18;
  std::vector<double> v(2 * (size_t)n);
  for (int i = 0; i < n; ++i) {
    double &x = v[2 * (size_t)i], &y = v[2 * (size_t)i + 1];
    x = draw(rng);
    y = draw(rng);
    if (i % 8 == 0) {
      // x in [2^512, 2^513), y next to 2^1025 / x
      x = bits((1535ULL << 52) | (rng() & 0xfffffffffffffULL));
      unsigned long long b;
      y = 0x1p513 / (x * 0x1p-512);
      memcpy(&b, &y, sizeof(b));
      y = bits(b + rng() % 3 - 1) * (rng() & 1 ? -1.0 : 1.0);
    }
  }
  v[0] = 1.5 * 0x1p512;
  v[1] = 0x1p514 / 3.0;
  v[2] = 0x1.4ccccea53f144p+512;
  v[3] = 0x1.89d89b5abcefbp+512;
  int bad = 0, flagged = 0;
  if (!gpu) {
    for (int i = 0; i < n; ++i) bad += check_pair(v[2 * (size_t)i], v[2 * (size_t)i + 1], &flagged);
  } else {
    double* dv;
    int* dr;
    int r[2] = {0, 0};
    cudaMalloc(&dv, v.size() * sizeof(double));
    cudaMalloc(&dr, sizeof(r));
    cudaMemcpy(dv, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemset(dr, 0, sizeof(r));
    k_check<<<(n + 127) / 128, 128>>>(dv, n, dr, dr + 1);
    const cudaError_t e = cudaMemcpy(r, dr, sizeof(r), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      printf("%s\n", cudaGetErrorString(e));
      return 2;
    }
    bad = r[0];
    flagged = r[1];
  }
  printf("mismatches %d, results in range %d of %d\n", bad, flagged, 8 * n);
  return bad != 0 || flagged < 2 * n;
}
