// FP64 DCT-I by the four-step FFT through Bluestein's algorithm: the kernels of
// mk_fft4_kern.cuh in double precision (8 or 4 transforms per CTA, 256
// threads).  Lengths that need no Bluestein run in mk_fft4_i64.cu.
#define MK_FFT4_NS f4d
#define MK_FFT4_C double2
#define MK_FFT4_RT double
#define MK_FFT4_FBHI 8
#define MK_FFT4_FBLO 4
#define MK_FFT4_NTHI 256
#define MK_FFT4_NTLO 256
#define MK_FFT4_MINBLO 2
#define MK_FFT4_SMOOTH 0
#include "mk_fft4.cuh"
#undef MK_FFT4_RMAX
#define MK_FFT4_RMAX MK_FFT4_RMAX64
#include "mk_fft4_kern.cuh"

namespace mk {
namespace f4d {
// the whole four-step twiddle table from the two short ones (FP64 plans)
__global__ void k_fft4_tfull(C *__restrict__ out, const Fft4Dev p) {
  const int n = p.H1 * p.P;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int j1 = i / p.P, e = i - j1 * p.P;
    out[i] = (e >> 5) < p.nb32 ? cmul(tab(p.tblk)[j1 * p.nb32 + (e >> 5)], tab(p.tlane)[32 * j1 + (e & 31)])
                               : mkc((RT)0, (RT)0);
  }
}
}  // namespace f4d

int fft4_dct_f64(const Fft4Plan &p, const double *x, int64_t ldx, int64_t nrow, double2 *T, double *out,
                 int64_t ldo, int epi, const double *w, int64_t ldw, cudaStream_t st) {
  return f4d::dct_launch(p, x, ldx, nrow, T, out, ldo, epi, w, ldw, st);
}

int fft4_tfull_f64(const Fft4Dev &d, double2 *out) {
  f4d::k_fft4_tfull<<<mk_grid((int64_t)d.H1 * d.P, 256, 8), 256>>>(out, d);
  const int rc = launch_status("fft4 twiddle table");
  if (rc) return rc;
  MK_CUDA(cudaStreamSynchronize(0));
  return MK_OK;
}

}  // namespace mk
