// FP64 detector rotation R = A . X on the bf16 tensor cores, by exact
// integer slicing (the splitting scheme of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication and its applications", Numer. Algorithms
// 59, 2012):
//   * each row i of A is scaled by 2^-sa_i and each sample column j of X by
//     2^-sx_j (powers of two: exact), so every scaled entry is below 1;
//   * the scaled entries are rounded to fixed point, F 2^-55, and F is cut
//     into S = 7 signed digits of 8 bits, -128 .. 128, exact in bf16 (whose
//     significand holds 8 bits): A = 2^sa sum_p A_p 2^(1-8p), X likewise;
//   * A_p X_q is then an integer matrix; the products with the same t = p + q
//     add up to less than 7 * 128 * 2^14 < 2^24 over 128 detectors, so FP32
//     accumulation in tensor memory is exact in any order.  The 28 products
//     with t <= S + 1 are formed;
//   * per output the sums of each t are combined in integers (hi: t <= 4, lo:
//     t >= 5) and rounded to FP64 once: R = 2^(sa_i + sx_j - 62) (hi 2^32 + lo).
// The error is that of the dropped products, about 2^-57 per term relative to
// the row and column scales (signed digits: they add up like random numbers;
// 8 unsigned digits of 7 bits left about twice as much).
//
// One call is: k_oz_prep_a (operand image of A), then per block of sample
// columns k_oz_slice_x (operand images of X, 14 B per sample, which stay in
// L2) and k_oz_gemm.
//
// k_oz_gemm.  MMA tile: M = 128 samples x N = 7 x 32 columns, K = 16; the
// accumulator's column block t - 2 (32 detectors each) collects the products
// of that t.  For slice q of X the B operand is [0 x (q-1), A_1 .. A_{8-q}],
// so each MMA has the same shape and accumulator (MMAs on one accumulator are
// only ordered when their shapes agree); in shared memory the 7 slices of A
// follow 6 blocks of zero rows and slice q starts 7 - q blocks in.  21 of the
// 49 block products are with zeros.  One accumulation covers 128 detectors (4 chunks of
// 32); two accumulators of 224 columns let the epilogue drain one while the
// next fills.
// 256 x 130,978: 0.84 ms per rotation (slices 0.23, products 0.56), against
// 3.49 ms for 8 slices of 7 bits multiplied by 12 cuBLAS bf16 GEMMs whose FP32
// results (96 B per sample) a last kernel combined; DGEMM takes 15.7 ms.
// Roles: warps 0-7 drain (warp w: TMEM lanes 32 (w % 4), 16 of the block's 32
// detectors), warp 8 streams operand chunks with bulk copies (X: ring of 3 x
// 56 KB, A: ring of 2), warp 9 issues the MMAs.
#include <cuda_bf16.h>

#include "mk_async.cuh"
#include "mk_common.cuh"
#include "mk_ozaki.cuh"

namespace mk {
namespace {

constexpr int OZ_S = 7;               // slices per operand
constexpr int OZ_FRAC = 8 * OZ_S - 1; // fixed-point bits of a scaled entry (55)
constexpr int OZ_NOSCALE = -100000;   // a row / column holding a non-finite value
constexpr int OZ_M = 128;             // samples per tile
constexpr int OZ_ND = 32;             // detectors per tile
constexpr int OZ_KC = 32;             // K per chunk: one 64-byte swizzle row of bf16
constexpr int OZ_N = OZ_S * OZ_ND;    // accumulator columns (224)
constexpr int OZ_DRAIN = 4;           // chunks per accumulation (128 detectors)
constexpr uint32_t XS_BYTES = OZ_M * 64;                  // one slice of an X chunk
constexpr uint32_t X_BYTES = OZ_S * XS_BYTES;             // an X chunk (57,344)
constexpr uint32_t AS_BYTES = OZ_ND * 64;                 // one slice of an A chunk
constexpr uint32_t A_BYTES = OZ_S * AS_BYTES;             // an A chunk (14,336)
constexpr uint32_t Z_BYTES = (OZ_S - 1) * AS_BYTES;       // the zero rows before it
constexpr int XSTG = 3, ASTG = 2;
constexpr uint32_t OZ_SMEM = XSTG * X_BYTES + ASTG * (Z_BYTES + A_BYTES) + 1024;
constexpr int EPI_WARPS = 8, OZ_THREADS = (EPI_WARPS + 2) * 32;
constexpr int64_t OZ_IMG_BYTES = 72ll << 20;  // X images of one block: they should stay in L2 (129 MB)
constexpr int64_t OZ_TILES = 512;  // most tiles of one block (its launch is several waves long)
// F + OZ_BIAS has the digits + 128 as its bytes (the top one 0 .. 256)
constexpr unsigned long long OZ_BIAS = 0x0080808080808080ull;

// exponent e with |x| < 2^e for the largest |x| given as bits; OZ_NOSCALE if
// that value is not finite; 0 for an all-zero row or column
__device__ __forceinline__ int scale_of(unsigned long long maxbits) {
  const int ef = (int)((maxbits >> 52) & 0x7FF);
  if (ef == 0x7FF) return OZ_NOSCALE;
  if (maxbits == 0) return 0;
  return ef == 0 ? -1021 : ef - 1022;
}

__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

// round(x 2^(55 - sc)) + OZ_BIAS for |x| < 2^sc (half away from zero)
__device__ __forceinline__ unsigned long long fixed_biased(double x, int sc) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ef = (int)((b >> 52) & 0x7FF);
  unsigned long long m = b & 0x000FFFFFFFFFFFFFull;
  if (ef) m |= 0x0010000000000000ull;
  // |x| = m 2^(E), E = (ef ? ef : 1) - 1075; F = m 2^(E + 55 - sc), at most a shift by 2 to the left
  const int sh = (ef ? ef : 1) - 1075 + OZ_FRAC - sc;
  if (sh >= 0)
    m = sh > 2 ? 0ull : m << sh;
  else
    m = sh > -64 ? (m + (1ull << (-sh - 1))) >> (-sh) : 0ull;
  return (b >> 63 ? 0ull - m : m) + OZ_BIAS;
}

// digit p (0 .. 6) of a biased fixed-point value, as a float
__device__ __forceinline__ float digit(unsigned long long F, int p) {
  const uint32_t hi = (uint32_t)(F >> 32), lo = (uint32_t)F;
  // 2^23 + (digit + 128) built in the mantissa; the subtraction is exact
  const uint32_t u = p == 0   ? 0x4B000000u + (hi >> 16)
                     : p <= 2 ? __byte_perm(hi, 0x4B000000u, 0x7650 | (2 - p))
                              : __byte_perm(lo, 0x4B000000u, 0x7650 | (6 - p));
  return __uint_as_float(u) - 8388736.0f;
}

// two digits as a bf16 pair (exact: the low halves of the floats are zero)
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// byte offset of the 16-byte group c (8 values of k) of row r in a K-major
// tile of 64-byte rows with the 64-byte swizzle
__device__ __forceinline__ uint32_t sw64_off(uint32_t r, uint32_t c) { return r * 64u + ((c ^ ((r >> 1) & 3u)) << 4); }

// the operand image of A, one CTA per (padded) row: per detector block and
// K-chunk 7 slices of 32 rows x 32 k; sa[i] the row exponents
__global__ void __launch_bounds__(128) k_oz_prep_a(const double *__restrict__ A, int nrow, int nkc,
                                                   int *__restrict__ sa, char *__restrict__ img) {
  const int i = blockIdx.x;
  __shared__ unsigned long long sh[4];
  __shared__ int ssc;
  unsigned long long m = 0;
  if (i < nrow)
    for (int k = threadIdx.x; k < nrow; k += 128) {
      const unsigned long long a = abs_bits(A[(size_t)i * nrow + k]);
      m = a > m ? a : m;
    }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, m, off);
    m = o > m ? o : m;
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 0; w < 4; w++) m = sh[w] > m ? sh[w] : m;
    ssc = scale_of(m);
    sa[i] = ssc;
  }
  __syncthreads();
  const int sc = ssc, d = i % OZ_ND;
  char *base = img + (size_t)(i / OZ_ND) * nkc * A_BYTES;
  for (int k = threadIdx.x; k < nkc * OZ_KC; k += 128) {
    const bool in = i < nrow && k < nrow && sc != OZ_NOSCALE;
    const unsigned long long F = in ? fixed_biased(A[(size_t)i * nrow + k], sc) : OZ_BIAS;
    char *ch = base + (size_t)(k / OZ_KC) * A_BYTES + sw64_off(d, (k % OZ_KC) >> 3) + (k & 7) * 2;
#pragma unroll
    for (int p = 0; p < OZ_S; p++) *(__nv_bfloat16 *)(ch + p * AS_BYTES) = __float2bfloat16_rn(digit(F, p));
  }
}

// the operand images of X for the sample columns j0 .. of one block, one CTA
// per 32 samples: per tile of 128 samples and K-chunk, 7 slices of 128 rows
// (samples) x 32 k; sx[j - j0] the column exponents.  The second reading of
// the columns comes from L1 / L2.  A thread turns 8 values of k of one sample
// into 7 16-byte groups; a warp's groups fill 8 rows (512 contiguous bytes).
__global__ void __launch_bounds__(256) k_oz_slice_x(const double *__restrict__ X, int64_t ldx, int nrow, int nkc,
                                                    int64_t j0, int64_t ncol, int *__restrict__ sx,
                                                    char *__restrict__ img) {
  __shared__ unsigned long long sh[8][32];
  __shared__ int ssc[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t js = (int64_t)blockIdx.x * 32;  // first sample, relative to j0
  const int64_t j = j0 + js + lane;
  unsigned long long m = 0;
  if (j < ncol) {
#pragma unroll 8
    for (int k = warp; k < nrow; k += 8) {
      const unsigned long long a = abs_bits(__ldg(X + k * ldx + j));
      m = a > m ? a : m;
    }
  }
  sh[warp][lane] = m;
  __syncthreads();
  if (warp == 0) {
    for (int w = 1; w < 8; w++) m = sh[w][lane] > m ? sh[w][lane] : m;
    const int sc = scale_of(m);
    ssc[lane] = sc;
    sx[js + lane] = sc;
  }
  __syncthreads();
  const int kg = lane >> 3;
  char *tile = img + (size_t)(js / OZ_M) * nkc * X_BYTES;
  for (int u = warp; u < 4 * nkc; u += 8) {
    const int kc = u >> 2, s = (u & 3) * 8 + (lane & 7);  // sample within the CTA's 32
    const int sc = ssc[s];
    const int64_t js_ = j0 + js + s;
    unsigned long long F[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int k = kc * OZ_KC + kg * 8 + e;
      const bool in = k < nrow && js_ < ncol && sc != OZ_NOSCALE;
      F[e] = in ? fixed_biased(__ldg(X + k * ldx + js_), sc) : OZ_BIAS;
    }
    char *dst = tile + (size_t)kc * X_BYTES + sw64_off((uint32_t)(js % OZ_M) + s, kg);
#pragma unroll
    for (int p = 0; p < OZ_S; p++) {
      uint4 v;
      v.x = pack2(digit(F[0], p), digit(F[1], p));
      v.y = pack2(digit(F[2], p), digit(F[3], p));
      v.z = pack2(digit(F[4], p), digit(F[5], p));
      v.w = pack2(digit(F[6], p), digit(F[7], p));
      *(uint4 *)(dst + p * XS_BYTES) = v;
    }
  }
}

// shared-memory matrix descriptor: K-major, SWIZZLE_64B, 8-row groups 512 B apart
__device__ __forceinline__ uint64_t sdesc64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;              // leading byte offset (unused)
  d |= (uint64_t)(512u >> 4) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;              // descriptor version (tcgen05)
  d |= (uint64_t)4 << 61;              // swizzle: 64B
  return d;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum));
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// bounded wait that also polls the CTA's abort flag (set on a timeout)
__device__ __forceinline__ bool oz_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  for (uint32_t i = 0; i < SPIN_LIMIT; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 31u) == 31u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// (hi 2^32 + lo) 2^(e - 62) rounded once to FP64, in integers (GB300 runs two
// FP64 operations per clock and SM)
__device__ __forceinline__ double combine(long long hi, long long lo, int e) {
  const __int128 S = (((__int128)hi) << 32) + lo;
  const bool neg = S < 0;
  const unsigned __int128 U = neg ? -(unsigned __int128)S : (unsigned __int128)S;
  const unsigned long long h = (unsigned long long)(U >> 64), l = (unsigned long long)U;
  if ((h | l) == 0) return 0.0;
  unsigned long long w;
  bool sticky = false;
  int top;  // position of U's leading bit
  if (h) {
    const int z = __clzll((long long)h);  // h < 2^32: z >= 32
    w = (h << z) | (l >> (64 - z));
    sticky = (l << z) != 0;
    top = 127 - z;
  } else {
    const int z = __clzll((long long)l);
    w = l << z;
    top = 63 - z;
  }
  unsigned long long m = w >> 11;
  const unsigned r = (unsigned)(w & 0x7FFu);
  if (r > 0x400u || (r == 0x400u && (sticky || (m & 1)))) m++;  // a carry to 2^53 moves into the exponent below
  const int E = top - 62 + e;
  const unsigned long long sign = neg ? 0x8000000000000000ull : 0ull;
  if (E > -1022 && E < 1023) return __longlong_as_double((long long)((((unsigned long long)(E + 1022)) << 52) + m + sign));
  return ldexp(__longlong_as_double((long long)((1022ull << 52) + m + sign)), E);
}

// R for ntile tiles of OZ_M samples (the first at column j0) and ndb blocks of
// OZ_ND detectors; item i = (tile i / ndb, block i % ndb), so the CTAs that
// run together share X chunks in L2
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_oz_gemm(const char *__restrict__ ximg, const char *__restrict__ aimg, const int *__restrict__ sx,
              const int *__restrict__ sa, double *__restrict__ R, int64_t ldr, int nrow, int nkc, int ndb, int nitem,
              int64_t j0, int64_t ncol, int *__restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char *const asm_ = smem + XSTG * X_BYTES;  // A stages: zero rows, then the chunk
  __shared__ uint64_t full_x[XSTG], empty_x[XSTG], full_a[ASTG], empty_a[ASTG], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  volatile int *abort_flag = &abort_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < XSTG; s++) {
      mbar_init(&full_x[s], 1);
      mbar_init(&empty_x[s], 1);
    }
    for (int s = 0; s < ASTG; s++) {
      mbar_init(&full_a[s], 1);
      mbar_init(&empty_a[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], EPI_WARPS * 32);
    }
    abort_sh = 0;
    mbar_init_fence();
  }
  for (uint32_t o = tid * 16; o < ASTG * Z_BYTES; o += OZ_THREADS * 16)
    *(uint4 *)(asm_ + (o / Z_BYTES) * (Z_BYTES + A_BYTES) + o % Z_BYTES) = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base_sh;
  const int ndrain = (nkc + OZ_DRAIN - 1) / OZ_DRAIN;
  uint32_t issued = 0, g_mma = 0;  // chunks whose copies were issued / whose MMAs were committed

  if (warp == EPI_WARPS) {
    // ---- producer (one thread)
    if (lane == 0) {
      for (int i = blockIdx.x; i < nitem && !*abort_flag; i += gridDim.x) {
        const char *xs = ximg + (size_t)(i / ndb) * nkc * X_BYTES;
        const char *as = aimg + (size_t)(i % ndb) * nkc * A_BYTES;
        for (int kc = 0; kc < nkc; kc++) {
          const uint32_t g = issued, x = g % XSTG, a = g % ASTG;
          if (g >= XSTG && !oz_wait(&empty_x[x], (g / XSTG - 1) & 1, abort_flag)) break;
          if (g >= ASTG && !oz_wait(&empty_a[a], (g / ASTG - 1) & 1, abort_flag)) break;
          mbar_expect_tx(&full_x[x], X_BYTES);
          bulk_g2s(smem + x * X_BYTES, xs + (size_t)kc * X_BYTES, X_BYTES, &full_x[x]);
          mbar_expect_tx(&full_a[a], A_BYTES);
          bulk_g2s(asm_ + a * (Z_BYTES + A_BYTES) + Z_BYTES, as + (size_t)kc * A_BYTES, A_BYTES, &full_a[a]);
          issued = g + 1;
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    // ---- MMA (one thread)
    if (lane == 0) {
      constexpr uint32_t idesc =
          (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);
      uint32_t dr = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < nitem && ok; i += gridDim.x) {
        for (int kc = 0; kc < nkc; kc++) {
          const uint32_t g = g_mma, x = g % XSTG, a = g % ASTG, ab = dr & 1;
          const uint32_t dacc = tmem + ab * 256;
          const bool first = kc % OZ_DRAIN == 0;
          if (first && dr >= 2 && !oz_wait(&acc_empty[ab], (dr / 2 - 1) & 1, abort_flag)) ok = false;
          if (!ok || !oz_wait(&full_x[x], (g / XSTG) & 1, abort_flag) ||
              !oz_wait(&full_a[a], (g / ASTG) & 1, abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t sxa = smem_u32(smem + x * X_BYTES), saa = smem_u32(asm_ + a * (Z_BYTES + A_BYTES));
#pragma unroll
          for (int k16 = 0; k16 < OZ_KC / 16; k16++)
#pragma unroll
            for (int q = 0; q < OZ_S; q++)
              mma_bf16(dacc, sdesc64(sxa + q * XS_BYTES + k16 * 32), sdesc64(saa + (OZ_S - 1 - q) * AS_BYTES + k16 * 32),
                       idesc, first && k16 == 0 && q == 0 ? 0u : 1u);
          mma_commit(&empty_x[x]);
          mma_commit(&empty_a[a]);
          g_mma = g + 1;
          if (kc % OZ_DRAIN == OZ_DRAIN - 1 || kc == nkc - 1) {
            mma_commit(&acc_full[ab]);
            dr++;
          }
        }
      }
    }
  } else {
    // ---- epilogue: lane = sample, 16 detectors per thread
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t base = tmem + ((uint32_t)(32 * quarter) << 16) + 16 * half;
    uint32_t dr = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < nitem && ok; i += gridDim.x) {
      const int js = (i / ndb) * OZ_M + 32 * quarter + lane;
      const int d0 = (i % ndb) * OZ_ND + 16 * half;
      long long hi[16], lo[16];
#pragma unroll
      for (int d = 0; d < 16; d++) hi[d] = lo[d] = 0;
      for (int n = 0; n < ndrain; n++, dr++) {
        // every lane waits; the warp goes on only if all of them saw the
        // phase complete (tcgen05.ld needs the whole warp converged)
        const bool okw = oz_wait(&acc_full[dr & 1], (dr / 2) & 1, abort_flag);
        if (!__all_sync(0xffffffffu, okw)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int t = 0; t < OZ_S; t++) {
          float v[16];
          tmem_ld16(base + (dr & 1) * 256 + t * OZ_ND, v);
#pragma unroll
          for (int d = 0; d < 16; d++) {
            const long long s = (long long)__float2int_rn(v[d]);
            if (t < 3)
              hi[d] += s * (1 << (8 * (2 - t)));
            else
              lo[d] += s * (1 << (8 * (6 - t)));
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        mbar_arrive(&acc_empty[dr & 1]);
      }
      const int64_t j = j0 + js;
      if (ok && j < ncol) {
        const int c = sx[js];
#pragma unroll
        for (int d = 0; d < 16; d++) {
          if (d0 + d >= nrow) continue;
          const int a = sa[d0 + d];
          // NaN, as the FP64 product of a non-finite entry
          const double r = a == OZ_NOSCALE || c == OZ_NOSCALE ? __longlong_as_double(0x7FF8000000000000ll)
                                                              : combine(hi[d], lo[d], a + c);
          __stcs(R + (int64_t)(d0 + d) * ldr + j, r);
        }
      }
    }
  }
  __syncthreads();
  if (*abort_flag) {
    // after a timeout: bounded waits for the copies and MMAs still in flight
    if (tid == EPI_WARPS * 32)
      for (uint32_t g = issued > XSTG ? issued - XSTG : 0; g < issued; g++) {
        (void)mbar_wait(&full_x[g % XSTG], (g / XSTG) & 1);
        if (g + ASTG >= issued) (void)mbar_wait(&full_a[g % ASTG], (g / ASTG) & 1);
      }
    if (tid == (EPI_WARPS + 1) * 32) {
      atomicExch(err, 1);
      for (uint32_t g = g_mma > XSTG ? g_mma - XSTG : 0; g < g_mma; g++)
        (void)mbar_wait(&empty_x[g % XSTG], (g / XSTG) & 1);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

size_t al256(size_t x) { return (x + 255) / 256 * 256; }

struct Layout {
  int nkc, ndb;
  int64_t tiles;  // most sample tiles of one block
  size_t sa, a, sx, x, total;
};

Layout layout(int64_t nrow) {
  Layout L;
  L.nkc = (int)((nrow + OZ_KC - 1) / OZ_KC);
  L.ndb = (int)((nrow + OZ_ND - 1) / OZ_ND);
  L.tiles = OZ_IMG_BYTES / ((int64_t)L.nkc * X_BYTES);
  if (L.tiles > OZ_TILES) L.tiles = OZ_TILES;
  size_t o = 0;
  L.sa = o;
  o += al256((size_t)L.ndb * OZ_ND * sizeof(int));
  L.a = o;
  o += al256((size_t)L.ndb * L.nkc * A_BYTES);
  L.sx = o;
  o += al256((size_t)L.tiles * OZ_M * sizeof(int));
  L.x = o;
  o += (size_t)L.tiles * L.nkc * X_BYTES;
  L.total = o;
  return L;
}

}  // namespace

bool ozaki_supported(int64_t nrow) { return nrow >= 1 && nrow <= OZ_MAXROW; }

size_t ozaki_ws_bytes(int64_t nrow) { return ozaki_supported(nrow) ? layout(nrow).total : 0; }

int ozaki_rotate_f64(const double *A, const double *X, int64_t ldx, double *R, int64_t ldr, int64_t nrow,
                     int64_t ncol, void *ws, size_t ws_bytes, int *err, cudaStream_t st) {
  MK_CHECK_ARG(ozaki_supported(nrow), "sliced FP64 rotation: ndet %lld is out of its range", (long long)nrow);
  const Layout L = layout(nrow);
  MK_CHECK_ARG(ws && err && ws_bytes >= L.total && ((uintptr_t)ws % 256) == 0,
               "sliced FP64 rotation: workspace too small (%zu < %zu)", ws_bytes, L.total);
  if (ncol <= 0) return MK_OK;
  static int attr_set[64] = {0};
  int dev = 0;
  MK_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    MK_CUDA(cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OZ_SMEM));
    attr_set[dev] = 1;
  }
  char *w = (char *)ws;
  int *sa = (int *)(w + L.sa), *sx = (int *)(w + L.sx);
  k_oz_prep_a<<<L.ndb * OZ_ND, 128, 0, st>>>(A, (int)nrow, L.nkc, sa, w + L.a);
  int rc = launch_status("sliced FP64 rotation: A slices");
  if (rc) return rc;
  const int64_t ntile = (ncol + OZ_M - 1) / OZ_M, nblk = (ntile + L.tiles - 1) / L.tiles;
  const int64_t per = (ntile + nblk - 1) / nblk;  // blocks of equal size
  for (int64_t t0 = 0; t0 < ntile; t0 += per) {
    const int64_t nt = ntile - t0 < per ? ntile - t0 : per, j0 = t0 * OZ_M;
    k_oz_slice_x<<<(unsigned)(nt * (OZ_M / 32)), 256, 0, st>>>(X, ldx, (int)nrow, L.nkc, j0, ncol, sx, w + L.x);
    if ((rc = launch_status("sliced FP64 rotation: X slices"))) return rc;
    const int nitem = (int)(nt * L.ndb);
    const int grid = nitem < sm_count() ? nitem : sm_count();
    k_oz_gemm<<<grid, OZ_THREADS, OZ_SMEM, st>>>(w + L.x, w + L.a, sx, sa, R, ldr, (int)nrow, L.nkc, L.ndb, nitem, j0,
                                                 ncol, err);
    if ((rc = launch_status("sliced FP64 rotation"))) return rc;
  }
  return MK_OK;
}

}  // namespace mk
