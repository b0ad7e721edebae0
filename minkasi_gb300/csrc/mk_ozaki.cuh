// FP64 detector rotation by exact integer slices on the bf16 tensor cores
// (see mk_ozaki.cu).  R (nrow x ncol, ld ldr) = A (nrow x nrow) . X (nrow x
// ncol, ld ldx), all row-major FP64.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace mk {
constexpr int64_t OZ_MAXROW = 1040;  // largest detector count (bounds the scratch)
bool ozaki_supported(int64_t nrow);
// scratch bytes of one call (256-byte aligned buffer; sample columns go in
// blocks, so it does not grow with ncol)
size_t ozaki_ws_bytes(int64_t nrow);
// stream-ordered on st; R must not overlap X.  `err` is a device int set to 1
// if a bounded wait inside the kernel timed out; what the kernel's block had to
// write is NaN then.
int ozaki_rotate_f64(const double *A, const double *X, int64_t ldx, double *R, int64_t ldr, int64_t nrow,
                     int64_t ncol, void *ws, size_t ws_bytes, int *err, cudaStream_t st);
}  // namespace mk
