// FP64 rotation on the FP64 pipe (see mk_f64mm.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mk {
// R (nrow x ncol, ld ldr) = A (nrow x nrow) . X (nrow x ncol, ld ldx), row-major; R must not overlap X
int rot_f64(const double *A, const double *X, int64_t ldx, double *R, int64_t ldr, int64_t nrow, int64_t ncol,
            cudaStream_t st);
}  // namespace mk
