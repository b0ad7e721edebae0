// DCT-I of detector rows by a four-step FFT in shared memory (FP32 and FP64).
//
// DCT-I of a row x (length n = m + 1) is the DFT of its even extension
// e_j = x_{min(j, 2m - j)} (length L = 2m), which is real.  Two rows r, r+1
// therefore share one complex transform: F = DFT(e_r + i e_{r+1}) gives
// DCT(x_r)_k = Re F_k and DCT(x_{r+1})_k = Im F_k, k = 0..m.
//
// With L = L1 L2 (both <= FFT4_LMAX, factors in {2,3,5,7,11}), j = j1 + L1 j2
// and k = k2 + L2 k1, a four-step FFT has
//   pass A: for each j1, A_j1[k2] = sum_j2 e_{j1 + L1 j2} W_L2^{j2 k2}
//   pass B: for each k2, F[k2 + L2 k1] = sum_j1 W_L^{j1 k2} A_j1[k2] W_L1^{j1 k1}
// e and F are even, which halves both passes and what goes between them:
//   * column L1 - j1 of e is column j1 reversed, so
//     A_{L1-j1}[k2] = W_L2^{-k2} A_j1[L2 - k2] and
//     W_L^{(L1-j1) k2} A_{L1-j1}[k2] = W_L^{-j1 k2} A_j1[L2 - k2]:
//     pass A runs the H1 = L1 / 2 + 1 columns j1 <= L1 / 2 only, and multiplies
//     A_j1[k2] by W_L^{j1 k2} for k2 <= L2 / 2 and by W_L^{j1 (k2 - L2)} beyond;
//     pass B's column k <= L2 / 2 reads entry k for row j1 and entry L2 - k for
//     row L1 - j1.  Entries above L2 / 2 sit `pad` further, so that they start
//     at a multiple of 32 (the twiddle blocks), with the other sign's value of
//     entry L2 / 2 (L2 even) before them at L2 / 2 + pad;
//   * F_{L-k} = F_k, and L - (k2 + L2 k1) lies in column L2 - k2, so pass B
//     runs the H2 = L2 / 2 + 1 columns k2 <= L2 / 2 only and writes each
//     output to k or L - k, whichever is <= m.
// In FP32 one DCT-I of 256 x 130,978 takes 0.171 ms against 0.307 with all
// columns (0.193 before the butterflies' operation counts and the index
// arithmetic were cut); Bluestein (below) on 256 x 144,278 0.727 ms against
// 0.953 (FP64 13.1 against 20.1).  FP64 without Bluestein: mk_fft4_i64.cu.
// Each CTA runs 8 or 16 (FP64: 4 or 8) transforms of one pass in shared memory (mixed-radix
// decimation in time, butterflies in place), interleaved over its threads.
// The first stage of each pass reads its inputs straight from global memory
// (pass A forms the even extension there); pass A's last stage twiddles its
// outputs and stores them to T; pass B's last stage writes k <= m
// straight to the rows with the epilogue (plain, times the inverse-spectrum
// weights, or with columns 0 and m halved).  Twiddles come from tables computed in
// double precision on the host.
//
// Lengths whose 2m has a prime factor above 11 (minkasi's truncate_tod leaves
// some) go through Bluestein's algorithm on the same passes.  With the chirp
// c_t = exp(-i pi t^2 / 2m) (even in t), W^{jk} = c_j c_k conj(c_{k-j}) for
// W = exp(-i pi / m), and the extension is periodic in j with period 2m, so
//   F_k = c_k sum_{j=-m}^{m} (e'_j c_j) conj(c_{k-j}),   e'_{-j} = e'_j = z_{|j|},
// with e' halved at the two ends j = +-m (the same point of the period, split
// between them so that e' c is even).  Only k = 0..m are needed, so the lags
// k - j cover [-m, 2m].  F is then a circular convolution a (*) b of a smooth
// length M > 3m, with a at positions j mod M and b_t = conj(c_t) at t mod M.
// (M = 3m never occurs: then 2m would be smooth.)  a and DFT(a) are even, so
// pass A and the first half of the middle pass run half of their columns as
// above; the middle pass finishes DFT(a) for the columns k2 and L2 - k2
// together, multiplies by B^ = DFT_M(b) / M, conjugates (U = conj(DFT(a) B^))
// and runs the first step of DFT(U) on both columns in shared memory; pass B
// on the transposed shape finishes DFT(U), which has no symmetry, and writes
// c_k conj(DFT(U)_k) for k <= m with the usual epilogue.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mk {

constexpr int FFT4_LMAX = 1536;  // longest transform of one pass
// largest radix the kernels hold in registers, FP32 and FP64
#ifndef MK_FFT4_RMAX
#define MK_FFT4_RMAX 16
#endif
#ifndef MK_FFT4_RMAX64
#define MK_FFT4_RMAX64 16
#endif
constexpr int FFT4_MAXR = 16;    // most radix stages of one pass

// device view of a plan (kernel argument)
struct Fft4Dev {
  int64_t n, m, L;  // row length, m = n - 1, transform length (2m, or M for Bluestein)
  int64_t Lx;       // even-extension length 2m
  bool blue;        // Bluestein: L = M, chirp and bhat set
  bool f64;         // FP64 plan: tables of double2, FP64 kernels
  int L1, L2;
  int H1, H2;        // L1 / 2 + 1, L2 / 2 + 1: the columns an even transform needs
  int pad, qh;       // T's upper entries are shifted by pad; qh = (L2 / 2) mod (last span of L2), or -1 (L2 odd)
  int P, PV;         // row pitch of T (L2 + pad) and of V (L1), rounded up to 16
  int64_t tsz, vsz;  // elements of T and of V per row pair
  int nb32;          // blocks of 32 covering a row of T
  // entry e of a row of T belongs to column e below up() and to e - pad - L2 from there on (a multiple of 32)
  __host__ __device__ int up() const { return (L2 + 1) / 2 + pad; }
  int fba, fbb;      // transforms per CTA of pass A (length L2) and pass B (length L1): 8 or 16
  int nr1, nr2;
  int r1[FFT4_MAXR], r2[FFT4_MAXR];
  // per stage: span Ns of the earlier stages, 1 / Ns, offset of its twiddles
  int ns1[FFT4_MAXR], ns2[FFT4_MAXR], to1[FFT4_MAXR], to2[FFT4_MAXR];
  float inv1[FFT4_MAXR], inv2[FFT4_MAXR];
  // complex tables: float2, double2, or (FP64 without Bluestein, i64()) 16-byte fixed-point entries
  // stage twiddles W_{Ns R}^{r k} at [to + (r - 1) Ns + k]
  const void *stw1, *stw2;
  const int *iperm1, *iperm2;  // natural index at each digit-reversed (DIT input) position
  const int *perm1;            // Bluestein: digit-reversed position of each natural index (length L1)
  // four-step twiddle of entry e of row j1 of T: tblk[j1 nb32 + e / 32] * tlane[32 j1 + e % 32]; FP64 plans
  // hold the products too, tfull[j1 P + e]
  const void *tlane, *tblk, *tfull;
  const void *chirp;  // Bluestein: c_t for t < m, c_m / 2 at m, c_m at m + 1
  const void *bhat;   // Bluestein: DFT_M(b) / M
  // Bluestein's middle pass: W_M^{k2 o1} = tblk2[k2 nb32b + o1 / 32] * tlane2[32 k2 + o1 % 32]
  const void *tlane2, *tblk2;
  int nb32b;  // ceil(L1 / 32)
  // the plan's passes run in fixed point (mk_fft4_i64.cu): stw1, stw2 and tfull hold its twiddles
  __host__ __device__ bool i64() const { return f64 && !blue; }
};

// epilogues of pass B
enum { FFT4_PLAIN = 0, FFT4_FILTER = 1, FFT4_HALVE = 2 };

struct Fft4Plan {
  Fft4Dev d{};
  void *tables = nullptr;  // device tables (plan-owned memory)
};

// The transform for rows of length n: L = 2(n-1) split into L1 x L2 with
// radix lists, or, when 2(n-1) has a prime factor above 11 and `bluestein`
// is set, the smallest splittable M >= 3(n-1); false when neither fits
// within FFT4_LMAX x FFT4_LMAX.
bool fft4_shape(int64_t n, Fft4Dev *d, bool bluestein = true, bool f64 = false);
// the rank of the L1 x L2 split new plans take (0: closest to sqrt(L))
void fft4_set_split_rank(int r);
int fft4_split_rank();
// bytes of the device tables for that shape
size_t fft4_table_bytes(const Fft4Dev &d);
// bytes of the scratch (T, and V for Bluestein) for nrow rows
size_t fft4_t_bytes(const Fft4Dev &d, int64_t nrow);
// computes the tables on the host (B^ with a double-precision cuFFT
// transform) and uploads them to `dev_tables`
int fft4_init(Fft4Plan *p, int64_t n, void *dev_tables, bool bluestein = true, bool f64 = false);
// out rows (ld ldo) = DCT-I of x rows (ld ldx) with the given epilogue;
// T is scratch of fft4_t_bytes; w (ld ldw) only for FFT4_FILTER.
int fft4_dct(const Fft4Plan &p, const float *x, int64_t ldx, int64_t nrow, float2 *T, float *out,
             int64_t ldo, int epi, const float *w, int64_t ldw, cudaStream_t st);
// the same for an FP64 plan (fft4_init with f64) that runs Bluestein
int fft4_dct_f64(const Fft4Plan &p, const double *x, int64_t ldx, int64_t nrow, double2 *T, double *out,
                 int64_t ldo, int epi, const double *w, int64_t ldw, cudaStream_t st);
// fills out[H1 P] with an FP64 plan's four-step twiddles (returns when done)
int fft4_tfull_f64(const Fft4Dev &d, double2 *out);

// FP64 plans without Bluestein (d.i64()): scratch bytes, the transform, and the
// fixed-point four-step twiddles.  chained: x is the output of this plan's
// last FFT4_FILTER transform of as many rows (whose largest values the scratch
// still holds).
size_t fft4_i64_bytes(const Fft4Dev &d, int64_t nrow);
int fft4_dct_i64(const Fft4Plan &p, const double *x, int64_t ldx, int64_t nrow, void *scratch, double *out,
                 int64_t ldo, int epi, const double *w, int64_t ldw, bool chained, cudaStream_t st);
int fft4_i64_tfull(const Fft4Dev &d, void *out);

}  // namespace mk
