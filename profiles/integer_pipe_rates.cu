// Issue cost of FP64 operations and of the integer-pipe products, reciprocals
// and roots of spd_soft.cuh: eight warps per SM sub-partition, four
// independent chains per thread, CUDA events around one launch after one
// warm-up launch.  Cycles of an SM sub-partition per warp operation, at the
// clock given as the argument (MHz).
//
//   nvcc -std=c++17 -O3 --fmad=false -gencode arch=compute_103a,code=sm_103a
//        -I spd_gb300/csrc profiles/integer_pipe_rates.cu -o rates && ./rates 2070
#include <cstdio>
#include <cstdlib>

#include "spd_soft.cuh"

using namespace spd;

constexpr int BLOCKS = 152 * 8, THREADS = 128, ITERS = 1000, CHAINS = 4, UNROLL = 4;

enum Op { ADD, MUL, FMA, PRODUCT, PRODUCT_ADD, MUL_ADD, RECIP, RECIP_FP64, QUOTIENT, QUOTIENT_FP64, ROOT, ROOT_FP64 };

template <int OP>
__global__ void k_rate(double* out, const double* in, const __grid_constant__ Coef c, double a) {
  double x[CHAINS], acc[CHAINS];
  for (int i = 0; i < CHAINS; ++i) {
    x[i] = in[(threadIdx.x + 32 * i) & 1023];
    acc[i] = 1.0 + i;
  }
#pragma unroll 1
  for (int it = 0; it < ITERS; ++it) {
#pragma unroll
    for (int r = 0; r < UNROLL; ++r) {
#pragma unroll
      for (int i = 0; i < CHAINS; ++i) {
        uint32_t ok = 0x40000000u;
        if (OP == ADD) x[i] = x[i] + a;
        if (OP == MUL) x[i] = x[i] * a;
        if (OP == FMA) x[i] = fma(x[i], a, a);
        // the split of the operand included, as in a contraction of one term
        if (OP == PRODUCT) x[i] = soft_prod(c, opnd_of(x[i], ok));
        if (OP == PRODUCT_ADD) {
          acc[i] = acc[i] + soft_prod(c, opnd_of(x[i], ok));
          x[i] = from_words(hi_word(x[i]) ^ (unsigned)r, lo_word(x[i]) + it);
        }
        if (OP == MUL_ADD) {
          acc[i] = acc[i] + x[i] * a;
          x[i] = from_words(hi_word(x[i]) ^ (unsigned)r, lo_word(x[i]) + it);
        }
        if (OP == RECIP) {
          const Recip q = recip_soft(x[i]);
          x[i] = from_words((hi_word(x[i]) & 0xfff00000u) | (q.mh & 0xfffffu), q.ml);
        }
        if (OP == RECIP_FP64) x[i] = 1.0 / x[i];
        if (OP == QUOTIENT) x[i] = div_soft(a, x[i], recip_soft(x[i]));
        if (OP == QUOTIENT_FP64) x[i] = a / x[i];
        if (OP == ROOT) x[i] = sqrt_soft(x[i]);
        if (OP == ROOT_FP64) x[i] = sqrt(x[i]);
      }
    }
  }
  double s = 0.0;
  for (int i = 0; i < CHAINS; ++i) s += x[i] + acc[i];
  out[blockIdx.x * THREADS + threadIdx.x] = s;
}

template <int OP>
void run(const char* name, double* out, const double* in, double mhz) {
  const double a = 1.0000001;
  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  k_rate<OP><<<BLOCKS, THREADS>>>(out, in, coef_of(a), a);
  cudaEventRecord(t0);
  k_rate<OP><<<BLOCKS, THREADS>>>(out, in, coef_of(a), a);
  cudaEventRecord(t1);
  const cudaError_t e = cudaEventSynchronize(t1);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, t0, t1);
  const double warp_ops = (double)BLOCKS * (THREADS / 32) * ITERS * UNROLL * CHAINS / (152 * 4);
  printf("%-34s %8.3f ms  %6.1f cycles  %s\n", name, ms, ms * 1e-3 * mhz * 1e6 / warp_ops, cudaGetErrorString(e));
}

int main(int argc, char** argv) {
  const double mhz = argc > 1 ? atof(argv[1]) : 2070.0;
  double *out, *in, h[1024];
  cudaMalloc(&out, sizeof(double) * BLOCKS * THREADS);
  cudaMalloc(&in, sizeof(h));
  for (int i = 0; i < 1024; ++i) h[i] = 1.0 + i * 0.000123;
  cudaMemcpy(in, h, sizeof(h), cudaMemcpyHostToDevice);
  run<ADD>("FP64 add", out, in, mhz);
  run<MUL>("FP64 multiply", out, in, mhz);
  run<FMA>("FP64 fused multiply-add", out, in, mhz);
  run<PRODUCT>("integer product", out, in, mhz);
  run<PRODUCT_ADD>("integer product, FP64 add", out, in, mhz);
  run<MUL_ADD>("FP64 multiply, FP64 add", out, in, mhz);
  run<RECIP>("integer reciprocal (Recip)", out, in, mhz);
  run<RECIP_FP64>("FP64 1 / x", out, in, mhz);
  run<QUOTIENT>("integer quotient", out, in, mhz);
  run<QUOTIENT_FP64>("FP64 a / b", out, in, mhz);
  run<ROOT>("integer root", out, in, mhz);
  run<ROOT_FP64>("FP64 root", out, in, mhz);
  cudaFree(out);
  cudaFree(in);
  return 0;
}
