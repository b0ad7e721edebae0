// FP64 detector rotation R = A . X (minkasi/mapmaking/noise.py:704,709) on
// GB300's FP64 pipe, which runs two fused multiply-adds per clock and SM: the
// kernel gives it nothing but those and keeps every SM equally loaded; loads,
// shared memory and everything else hide behind it.
#include "mk_common.cuh"
#include "mk_f64mm.cuh"

namespace mk {
namespace {

// A thread owns one sample and OB output detectors; per input detector it
// reads its sample (coalesced) and OB entries of A (shared memory, broadcast)
// for OB multiply-adds.  Two-warp CTAs over (samples / 64) x (detectors / OB)
// leave the SMs within a few per cent of each other where cuBLAS's 64 x 64
// tiles left a third of the last wave idle.  53 detectors x 20,001
// samples: 107 us for 228; 64 x 65,341: 448 for 523; 256 x 130,978: 13.7 ms for
// 15.7 (0.63 T multiply-adds per second, the pipe's rate); 2 x 100,000: 10 us for 113.
constexpr int RT = 64;    // threads per CTA
constexpr int RK = 256;   // input detectors per pass over shared memory

template <int OB>
__global__ void __launch_bounds__(RT) k_rot_f64(const double *__restrict__ A, const double *__restrict__ X, int64_t ldx,
                                                double *__restrict__ R, int64_t ldr, int nrow, int64_t ncol) {
  __shared__ __align__(16) double sa[RK][OB + (OB & 1)];
  const int64_t j = (int64_t)blockIdx.x * RT + threadIdx.x;
  const int i0 = blockIdx.y * OB;
  const double *x = X + (j < ncol ? j : ncol - 1);
  double acc[OB];
#pragma unroll
  for (int i = 0; i < OB; i++) acc[i] = 0.0;
  for (int k0 = 0; k0 < nrow; k0 += RK) {
    const int kn = min(RK, nrow - k0);
    if (k0) __syncthreads();
    for (int e = threadIdx.x; e < OB * kn; e += RT) {
      const int i = e / kn, k = e - i * kn;
      sa[k][i] = i0 + i < nrow ? A[(int64_t)(i0 + i) * nrow + k0 + k] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < kn; k++) {
      const double v = __ldg(x + (int64_t)(k0 + k) * ldx);
#pragma unroll
      for (int i = 0; i < OB; i++) acc[i] = fma(sa[k][i], v, acc[i]);
    }
  }
  if (j < ncol) {
#pragma unroll
    for (int i = 0; i < OB; i++)
      if (i0 + i < nrow) __stcs(R + (int64_t)(i0 + i) * ldr + j, acc[i]);
  }
}

template <int OB>
int rot_launch(const double *A, const double *X, int64_t ldx, double *R, int64_t ldr, int nrow, int64_t ncol,
               cudaStream_t st) {
  const dim3 g((unsigned)((ncol + RT - 1) / RT), (unsigned)((nrow + OB - 1) / OB));
  k_rot_f64<OB><<<g, RT, 0, st>>>(A, X, ldx, R, ldr, nrow, ncol);
  return launch_status("FP64 rotation");
}

}  // namespace

int rot_f64(const double *A, const double *X, int64_t ldx, double *R, int64_t ldr, int64_t nrow, int64_t ncol,
            cudaStream_t st) {
  if (ncol <= 0) return MK_OK;
  // detectors per thread: 8, or fewer where that pads less, or where it leaves the
  // SM with the most CTAs at least a tenth less to do (a few CTAs per SM and a
  // nearly empty last wave; a quarter of a multiply-add more for a thread's loads).
  // 96 x 1,000 with 8 and 6: 37.8 and 30.1 us, 128 x 1,000 with 8 and 7: 48.5 and
  // 45.7 (DGEMM 35.7 and 44.8), 300 x 1,000 with 6 and 8: 176 and 159; for less than
  // a tenth 200 x 3,000 lost (8 and 7: 213 and 223).
  const int nd = (int)nrow;
  const int64_t cols = (ncol + RT - 1) / RT, sms = sm_count();
  const auto cost = [&](int c) { return (cols * ((nd + c - 1) / c) + sms - 1) / sms * (4 * c + 1); };
  int ob = 8;
  for (int c = 7; c >= 5; c--)
    if ((nd + c - 1) / c * c < (nd + ob - 1) / ob * ob) ob = c;
  const int64_t enough = cost(ob) * 9 / 10;
  for (int c = 8, base = ob; c >= 5; c--)
    if (cost(c) <= enough && (ob == base || cost(c) < cost(ob))) ob = c;
  switch (ob) {
    case 5: return rot_launch<5>(A, X, ldx, R, ldr, nd, ncol, st);
    case 6: return rot_launch<6>(A, X, ldx, R, ldr, nd, ncol, st);
    case 7: return rot_launch<7>(A, X, ldx, R, ldr, nd, ncol, st);
    default: return rot_launch<8>(A, X, ldx, R, ldr, nd, ncol, st);
  }
}

}  // namespace mk
