// Smooth-length pass, FP32, R2R lines (complex, or two real lines as one).
#include <cuda_runtime.h>

#include "pencilfft_gb300.h"
#include "pfgb_sm.cuh"

namespace pfgb {

int launch_sm_f32_r2r(bool cplx, const FastArgs& A, int64_t grid, int threads, size_t smem, cudaStream_t s) {
  return cplx ? launch_sm_one<float, -1, OP_R2R_C>(A, grid, threads, smem, s) : launch_sm_one<float, -1, OP_R2R_R>(A, grid, threads, smem, s);
}

}  // namespace pfgb
