// FP64 products on GB300's FP64 pipe, which runs two fused multiply-adds per
// clock and SM: the kernels below give it nothing but those and keep every SM
// equally loaded; loads, shared memory and everything else hide behind it.
//   R = A . X      detector rotations (minkasi/mapmaking/noise.py:704,709)
//   G = X . X^T    the Gram matrix of a timestream, whose eigenvectors are its
//                  left singular vectors (noise.py:627-640)
#include "mk_common.cuh"
#include "mk_f64mm.cuh"

namespace mk {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// ---- rotation ------------------------------------------------------------
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

// ---- Gram matrix -----------------------------------------------------------
// Detectors go in blocks of GB; a warp takes one pair of blocks (the upper
// triangle of pairs: G is symmetric) and one slice of the samples, lanes along
// the samples, GB^2 sums per lane.  The sums of the lanes are folded by
// recursive halving (each step adds half as many values), written per slice,
// and summed over the slices in order: the result does not depend on timing.
// 64 x 65,341: 302 us for 738 (cuBLAS, both triangles, through torch); 256 x
// 130,978: 7.3 ms for 15.8.
constexpr int GB = 8;
constexpr int GW = 4;  // warps per CTA

__device__ __forceinline__ void block_pair(int e, int nb, int &bi, int &bj) {  // e-th pair bi <= bj
  bi = 0;
  while (e >= nb - bi) {
    e -= nb - bi;
    bi++;
  }
  bj = bi + e;
}

__global__ void __launch_bounds__(GW * 32) k_gram(const double *__restrict__ X, int64_t ldx, int nrow, int64_t ncol,
                                                  int nb, int nslice, double *__restrict__ part) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * GW + (threadIdx.x >> 5);
  const int npair = nb * (nb + 1) / 2;
  if (w >= (int64_t)npair * nslice) return;
  const int e = (int)(w % npair), s = (int)(w / npair);
  int bi, bj;
  block_pair(e, nb, bi, bj);
  const int64_t t0 = ncol * s / nslice, t1 = ncol * (s + 1) / nslice;
  const double *pi[GB], *pj[GB];
#pragma unroll
  for (int i = 0; i < GB; i++) {
    pi[i] = X + (int64_t)min(bi * GB + i, nrow - 1) * ldx;
    pj[i] = X + (int64_t)min(bj * GB + i, nrow - 1) * ldx;
  }
  double acc[GB * GB];
#pragma unroll
  for (int i = 0; i < GB * GB; i++) acc[i] = 0.0;
  if (bi == bj) {
    for (int64_t t = t0 + lane; t < t1; t += 32) {
      double a[GB];
#pragma unroll
      for (int i = 0; i < GB; i++) a[i] = __ldg(pi[i] + t);
#pragma unroll
      for (int i = 0; i < GB; i++)
#pragma unroll
        for (int j = i; j < GB; j++) acc[i * GB + j] = fma(a[i], a[j], acc[i * GB + j]);
    }
  } else {
    for (int64_t t = t0 + lane; t < t1; t += 32) {
      double a[GB];
#pragma unroll
      for (int i = 0; i < GB; i++) a[i] = __ldg(pi[i] + t);
#pragma unroll
      for (int j = 0; j < GB; j++) {
        const double b = __ldg(pj[j] + t);
#pragma unroll
        for (int i = 0; i < GB; i++) acc[i * GB + j] = fma(a[i], b, acc[i * GB + j]);
      }
    }
  }
  // lane l ends with entries 2 l', 2 l' + 1 (l' the bit reversal the halving
  // leaves): at distance d a lane keeps the half its bit selects
#pragma unroll
  for (int d = 16, n = GB * GB / 2; d >= 1; d >>= 1, n >>= 1) {
    const bool up = (lane & d) != 0;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const double give = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
      acc[i] = keep + __shfl_xor_sync(FULL, give, d);
    }
  }
  double *out = part + ((int64_t)s * npair + e) * (GB * GB) + 2 * lane;
  out[0] = acc[0];
  out[1] = acc[1];
}

// G (nrow x nrow, both triangles) from the partial sums
__global__ void __launch_bounds__(GB *GB) k_gram_sum(const double *__restrict__ part, int nrow, int nb, int nslice,
                                                     double *__restrict__ G) {
  const int npair = nb * (nb + 1) / 2, e = blockIdx.x;
  int bi, bj;
  block_pair(e, nb, bi, bj);
  const int i = bi * GB + threadIdx.x / GB, j = bj * GB + threadIdx.x % GB;
  if (i >= nrow || j >= nrow || i > j) return;
  double s = 0.0;
#pragma unroll 8
  for (int k = 0; k < nslice; k++) s += part[((int64_t)k * npair + e) * (GB * GB) + threadIdx.x];
  G[(int64_t)i * nrow + j] = s;
  G[(int64_t)j * nrow + i] = s;
}

int gram_slices(int64_t nrow, int64_t ncol) {
  const int64_t nb = (nrow + GB - 1) / GB, npair = nb * (nb + 1) / 2;
  // up to 32 warps per SM (four waves of the 8 that fit), each with at least 512 samples
  int64_t s = (int64_t)sm_count() * 32 / npair;
  if (s > ncol / 512) s = ncol / 512;
  return (int)(s < 1 ? 1 : s);
}

}  // namespace

int rot_f64(const double *A, const double *X, int64_t ldx, double *R, int64_t ldr, int64_t nrow, int64_t ncol,
            cudaStream_t st) {
  if (ncol <= 0) return MK_OK;
  // detectors per thread: 8, or fewer where that pads less
  const int nd = (int)nrow;
  int ob = 8;
  for (int c = 7; c >= 5; c--)
    if ((nd + c - 1) / c * c < (nd + ob - 1) / ob * ob) ob = c;
  switch (ob) {
    case 5: return rot_launch<5>(A, X, ldx, R, ldr, nd, ncol, st);
    case 6: return rot_launch<6>(A, X, ldx, R, ldr, nd, ncol, st);
    case 7: return rot_launch<7>(A, X, ldx, R, ldr, nd, ncol, st);
    default: return rot_launch<8>(A, X, ldx, R, ldr, nd, ncol, st);
  }
}

}  // namespace mk

extern "C" size_t mk_gram_scratch_bytes(int64_t nrow, int64_t ncol) {
  if (nrow < 1 || ncol < 1) return 0;
  const int64_t nb = (nrow + mk::GB - 1) / mk::GB;
  return (size_t)mk::gram_slices(nrow, ncol) * (size_t)(nb * (nb + 1) / 2) * mk::GB * mk::GB * sizeof(double);
}

extern "C" int mk_gram(double *G, const double *X, int64_t ldx, int64_t nrow, int64_t ncol, void *scratch,
                       void *stream) {
  MK_CHECK_ARG(G && X && scratch, "mk_gram: null pointer");
  MK_CHECK_ARG(nrow >= 1 && nrow <= 46340 && ncol >= 1 && ldx >= ncol, "mk_gram: bad sizes");
  cudaStream_t st = mk::as_stream(stream);
  const int nb = (int)((nrow + mk::GB - 1) / mk::GB), ns = mk::gram_slices(nrow, ncol);
  const int64_t npair = (int64_t)nb * (nb + 1) / 2;
  mk::k_gram<<<(unsigned)((npair * ns + mk::GW - 1) / mk::GW), mk::GW * 32, 0, st>>>(X, ldx, (int)nrow, ncol, nb, ns,
                                                                                    (double *)scratch);
  mk::k_gram_sum<<<(unsigned)npair, mk::GB * mk::GB, 0, st>>>((const double *)scratch, (int)nrow, nb, ns, G);
  return mk::launch_status("mk_gram");
}
