// Smooth-length pass, FP32 arithmetic, r2c lines.
#include <cuda_runtime.h>

#include "pencilfft_gb300.h"
#include "pfgb_sm.cuh"

namespace pfgb {

int launch_sm_f32_r2c(int, const FastArgs& A, int64_t grid, int threads, size_t smem, cudaStream_t s) {
  return launch_sm_one<float, -1, OP_R2C>(A, grid, threads, smem, s);
}

}  // namespace pfgb
