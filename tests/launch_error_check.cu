// A batched launch that CUDA refuses gives its error back and does not leave
// it behind for the next check of an unrelated call: a block of 2048 threads,
// which no device takes (the host refuses it, nothing is launched).
#include <cstdio>

#include "spd_kernels.cuh"
#include "spd_batch.cuh"

using namespace spd_batch;

struct Body {
  static __device__ void run(spd::Blk, int, double*) {}
};

int main() {
  BatchRec R;
  R.begin_instance(true);
  R.add<Body>("refused", dim3(1), dim3(2048), 0, PackBuild<int, double*>::make(1, (double*)nullptr));
  R.add_zero(nullptr, 0);
  if (!R.end_instance()) return 1;
  R.sites[1]->block = dim3(2048, 1, 1);
  for (auto& site : R.sites) {
    const cudaError_t e = site->launch(0);
    const cudaError_t left = cudaGetLastError();
    std::printf("%s: returned \"%s\", left \"%s\"\n", site->name, cudaGetErrorString(e), cudaGetErrorString(left));
    if (e == cudaSuccess || left != cudaSuccess) return 1;
  }
  return 0;
}
