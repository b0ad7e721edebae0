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
// Roles: warps 0-15 drain (warp w: TMEM lanes 32 (w % 4), 8 of the block's 32
// detectors), warp 16 streams operand chunks with bulk copies (X: ring of 3 x
// 56 KB, A: ring of 2), warp 17 issues the MMAs.
//
// What bounds it, in the order found on 256 x 130,978 (products 0.56 ms with 8
// drain warps and one thread in charge of the MMAs): the drain's latency (two
// warps a scheduler; sums in 64-bit shifts), then the issuing thread, 2050
// cycles a chunk for MMAs that take 1570 (operands moved to uniform registers
// for each of them, two barriers and two commits a chunk).  With 16 drain warps,
// 32-bit combination steps and a converged MMA warp with one barrier and one
// commit a chunk: 0.46 ms, 85 % of the tensor core's time for this shape; the
// slices 0.23 -> 0.16 ms (one pass over X, 97 -> 65 instructions per value).
// One rotation, before and after: 256 x 130,978 821 -> 628 us, 128 x 100,000 244
// -> 170, 64 x 65,341 80 -> 53, 300 x 50,000 473 -> 365, 26 x 60,000 46 -> 32.  (8
// slices of 7 bits multiplied by 12 cuBLAS bf16 GEMMs whose FP32 results, 96 B
// per sample, a last kernel combined: 3.49 ms; DGEMM 15.7 ms.)
// Tried: accumulators of 7, 5 and 3 blocks for the slices from 1, 3 and 5 on (33
// block products instead of 49): 868 us, the tensor core pays for each change of
// accumulator.
#include <cuda_bf16.h>

#include "mk_async.cuh"
#include "mk_common.cuh"
#include "mk_ozaki.cuh"

namespace mk {
namespace {

constexpr int OZ_S = 7;               // slices per operand
static_assert(8 * OZ_S - 1 == 55, "fixed-point bits of a scaled entry");
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
constexpr int EPI_WARPS = 16, OZ_THREADS = (EPI_WARPS + 2) * 32;
constexpr int EPI_ND = 4 * OZ_ND / EPI_WARPS;  // detectors of one epilogue thread (8)
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

// round(x 2^(55 - sc)) + OZ_BIAS for |x| < 2^sc (half away from zero); OZ_BIAS
// for sc far above x
__device__ __forceinline__ unsigned long long fixed_biased(double x, int sc) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int ef = (int)((hi >> 20) & 0x7FFu);
  const uint32_t mh = (hi & 0xFFFFFu) | (ef ? 0x100000u : 0u);
  // |x| 2^(55 - sc) = w 2^-(r + 1) with w = 8 m: r >= 0, since |x| < 2^sc
  const unsigned long long w = ((unsigned long long)__funnelshift_l(lo, mh, 3) << 32) | (lo << 3);
  const int r = min(1022 + sc - (ef ? ef : 1), 63);
  const unsigned long long m = ((w >> r) + 1) >> 1;
  return ((int)hi < 0 ? 0ull - m : m) + OZ_BIAS;
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

// digits p of two biased fixed-point values as a bf16 pair.  Below the top
// digit u = digit + 128 is a byte: (128 + u % 128) - (u < 128 ? 256 : 128) in
// bf16, every term and the result exact; the top one reaches 256.
__device__ __forceinline__ uint32_t digits2(unsigned long long F, unsigned long long G, int p) {
  if (p == 0) return pack2(digit(F, 0), digit(G, 0));
  const uint32_t f = p <= 2 ? (uint32_t)(F >> 32) : (uint32_t)F, g = p <= 2 ? (uint32_t)(G >> 32) : (uint32_t)G;
  const uint32_t at = p <= 2 ? 2 - p : 6 - p;
  const uint32_t u = __byte_perm(f, g, at | (4 + at) << 8);  // bytes 0 and 2; 1 and 3 are masked off
  const uint32_t a = (u & 0x007F007Fu) | 0x43004300u, b = (u & 0x00800080u) ^ 0x43804380u;
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// the operand images of X for the sample columns j0 .. of one block, one CTA
// per 32 samples: per tile of 128 samples and K-chunk, 7 slices of 128 rows
// (samples) x 32 k; sx[j - j0] the column exponents.  A thread has one sample
// and NU groups of 8 values of k: they are all in flight at once and are kept
// in registers from the search for the column's exponent to the digits.  A
// warp's 16-byte groups fill 8 rows (512 contiguous bytes) of a slice.  NU = 0:
// any nrow, the values are read twice (from L1 / L2 the second time).
template <int NU>
__global__ void __launch_bounds__(256, NU == 4 ? 2 : 0) k_oz_slice_x(const double *__restrict__ X, int64_t ldx, int nrow, int nkc,
                                                    int64_t j0, int64_t ncol, int *__restrict__ sx,
                                                    char *__restrict__ img) {
  __shared__ uint32_t sh[8][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t js = (int64_t)blockIdx.x * 32;  // first sample, relative to j0
  const int s = (warp & 3) * 8 + (lane & 7);    // sample within the CTA's 32
  const int kg = lane >> 3;
  const int64_t j = j0 + js + s;
  const int nr = j < ncol ? nrow : 0;
  // group i: k = 32 kc + 8 kg .. + 7, kc = warp / 4 + 2 i
  const int k0 = (warp >> 2) * OZ_KC + kg * 8;
  const double *const xp = X + (int64_t)k0 * ldx + j;
  double v[NU ? NU : 1][8];
  uint32_t m = 0;  // largest high word; a value below 2^-1042 counts as 1
  const auto load = [&](int i, double *v8) {
    const int k = k0 + 2 * OZ_KC * i;
#pragma unroll
    for (int e = 0; e < 8; e++) v8[e] = k + e < nr ? __ldg(xp + (int64_t)(2 * OZ_KC * i + e) * ldx) : 0.0;
  };
  const auto largest = [&](const double *v8) {
#pragma unroll
    for (int e = 0; e < 8; e++)
      m = max(m, ((uint32_t)__double2hiint(v8[e]) & 0x7FFFFFFFu) | (__double2loint(v8[e]) ? 1u : 0u));
  };
  if constexpr (NU > 0) {
#pragma unroll
    for (int i = 0; i < NU; i++) load(i, v[i]);
#pragma unroll
    for (int i = 0; i < NU; i++) largest(v[i]);
  } else {
    for (int i = 0; 2 * i < nkc; i++) {
      load(i, v[0]);
      largest(v[0]);
    }
  }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
  if (lane < 8) sh[warp][lane] = m;
  __syncthreads();
  m = max(m, sh[warp ^ 4][lane & 7]);
  const int sc = scale_of((unsigned long long)m << 32);
  if (warp < 4 && lane < 8) sx[js + s] = sc;
  const int scx = sc == OZ_NOSCALE ? -OZ_NOSCALE : sc;  // no digits
  char *const dst = img + (size_t)(js / OZ_M) * nkc * X_BYTES + sw64_off((uint32_t)(js % OZ_M) + s, kg);
  const auto store = [&](int i, const double *v8) {
    const int kc = (warp >> 2) + 2 * i;
    if (kc >= nkc) return;
    unsigned long long F[8];
#pragma unroll
    for (int e = 0; e < 8; e++) F[e] = fixed_biased(v8[e], scx);
#pragma unroll
    for (int p = 0; p < OZ_S; p++)
      *(uint4 *)(dst + (size_t)kc * X_BYTES + p * XS_BYTES) =
          make_uint4(digits2(F[0], F[1], p), digits2(F[2], F[3], p), digits2(F[4], F[5], p), digits2(F[6], F[7], p));
  };
  if constexpr (NU > 0) {
#pragma unroll
    for (int i = 0; i < NU; i++) store(i, v[i]);
  } else {
    for (int i = 0; 2 * i < nkc; i++) {
      load(i, v[0]);
      store(i, v[0]);
    }
  }
}

// shared-memory matrix descriptors: K-major, SWIZZLE_64B, 8-row groups 512 B
// apart.  Low word: address / 16 (and an unused leading offset), so a step
// within a stage is an addition; high word: stride 512 B, version (tcgen05),
// swizzle 64B
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t saddr) { return (saddr >> 4) | (1u << 16); }
constexpr uint32_t SDESC_HI = (512u >> 4) | (1u << 14) | (4u << 29);

// one lane of a converged warp, the same one at every call
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(e));
  return e;
}

// MMA by the lane whose lead is set (executed by the whole warp, so that the
// operands stay in uniform registers); acc: add to the accumulator
__device__ __forceinline__ void mma_bf16(uint32_t lead, uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p, l;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 l, %6, 0;\n"
      " mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
      " @l tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(alo), "r"(blo), "r"(idesc), "r"(acc), "n"(SDESC_HI), "r"(lead));
}

__device__ __forceinline__ void mma_commit(uint32_t lead, uint64_t *bar) {
  asm volatile("{\n .reg .pred l;\n setp.ne.b32 l, %1, 0;\n"
               " @l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_u32(bar)),
               "r"(lead)
               : "memory");
}

// 8 accumulator columns of this thread's lane; valid after tmem_wait
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// the registers of N loads may be read from here on (listed, so that their
// uses stay below the wait)
template <int N>
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[N][8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int n = 0; n < N; n++)
#pragma unroll
    for (int i = 0; i < 8; i++) asm volatile("" : "+r"(r[n][i]));
}

// bounded wait that also polls the CTA's abort flag (set on a timeout)
__device__ __forceinline__ bool oz_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  for (uint32_t i = 0; i < ROLE_SPIN_LIMIT; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 31u) == 31u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// a converged warp waits for a barrier; true if every lane saw it complete
// (tcgen05.ld and the MMA warp's instructions need the whole warp converged)
__device__ __forceinline__ bool acc_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  const bool ok = __all_sync(0xffffffffu, oz_wait(bar, parity, abort_flag));
  asm volatile("tcgen05.fence::after_thread_sync;");
  return ok;
}

// acc + v w in 64 bits, one instruction
__device__ __forceinline__ long long mad_wide(int v, int w, long long acc) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(v), "r"(w), "l"(acc));
  return r;
}

// (hi 2^32 + lo) 2^(e - 62) rounded once to FP64 for any |hi|, |lo| < 2^62 and
// e; NaN for e below -50000 (a scale of OZ_NOSCALE)
__device__ __noinline__ double combine_any(long long hi, long long lo, int e) {
  if (e < -50000) return __longlong_as_double(0x7FF8000000000000ll);
  // magnitude T 2^32 + L
  long long t = hi + (lo >> 32);
  uint32_t L = (uint32_t)lo;
  const bool neg = t < 0;
  if (neg) {
    t = ~t + (L == 0 ? 1 : 0);
    L = 0u - L;
  }
  unsigned long long T = (unsigned long long)t;
  int top = 95;  // position of the leading bit after the shift below
  if (T == 0) {  // L alone
    T = (unsigned long long)L << 32;
    L = 0;
    top = 31;
    if (T == 0) return 0.0;
  }
  const int z = __clzll((long long)T);
  const unsigned long long l = (unsigned long long)L << 32;
  const unsigned long long w = (T << z) | (z ? l >> (64 - z) : 0ull);
  const uint32_t sticky = (l << z) != 0 ? 1u : 0u;
  unsigned long long m = w >> 11;
  // to nearest, ties to even; a carry to 2^53 moves into the exponent below
  if ((((uint32_t)w & 0x7FFu) | sticky) + ((uint32_t)m & 1u) > 0x400u) m++;
  const int E = top - z - 62 + e;
  const unsigned long long sign = neg ? 0x8000000000000000ull : 0ull;
  if (E > -1022 && E < 1023) return __longlong_as_double((long long)((((unsigned long long)(E + 1022)) << 52) + m + sign));
  return ldexp(__longlong_as_double((long long)((1022ull << 52) + m + sign)), E);
}

// combine_any's result in 32-bit steps where the sum has more than 32 bits and
// the result is a normal number (integers: GB300 runs two FP64 operations per
// clock and SM, and 64-bit shifts by a variable are several instructions)
__device__ __forceinline__ double combine(long long hi, long long lo, int e) {
  const long long t = hi + (lo >> 32);
  const uint32_t s = (uint32_t)((int)(t >> 63));  // all ones if negative
  uint32_t a2, a1, a0;
  asm("sub.cc.u32 %0, %3, %6;\n subc.cc.u32 %1, %4, %6;\n subc.u32 %2, %5, %6;"
      : "=&r"(a0), "=&r"(a1), "=r"(a2)
      : "r"((uint32_t)lo ^ s), "r"((uint32_t)t ^ s), "r"((uint32_t)(t >> 32) ^ s), "r"(s));
  const bool big = a2 != 0;
  const uint32_t w1 = big ? a2 : a1, w2 = big ? a1 : a0, w3 = big ? a0 : 0u;
  const int z = __clz((int)w1);
  const int E = (big ? 1022 + 95 - 62 : 1022 + 63 - 62) - z + e;  // exponent field - 1
  if (w1 == 0 || (uint32_t)(E - 1) >= 2044u) return combine_any(hi, lo, e);
  const uint32_t m1 = __funnelshift_l(w2, w1, z), m2 = __funnelshift_l(w3, w2, z);
  const uint32_t rem = (m2 & 0x7FFu) | (w3 << z ? 1u : 0u);
  uint32_t rl = __funnelshift_r(m2, m1, 11);
  uint32_t rh = (m1 >> 11) + ((uint32_t)E << 20) + (s & 0x80000000u);
  const uint32_t up = rem + (rl & 1u) > 0x400u ? 1u : 0u;  // to nearest, ties to even
  asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, 0;" : "+r"(rl), "+r"(rh) : "r"(up));
  return __hiloint2double((int)rh, (int)rl);
}

// NaN where this CTA writes R (not inlined: the kernel around it keeps its code
// and its time; inlined, 256 x 130,978 took 643 us for 628)
__device__ __noinline__ void fill_nan(double *R, int64_t ldr, int nrow, int ndb, int nitem, int64_t j0, int64_t ncol) {
  for (int i = blockIdx.x; i < nitem; i += gridDim.x)
    for (int e = threadIdx.x; e < OZ_M * OZ_ND; e += OZ_THREADS) {
      const int64_t j = j0 + (int64_t)(i / ndb) * OZ_M + e % OZ_M;
      const int d = (i % ndb) * OZ_ND + e / OZ_M;
      if (j < ncol && d < nrow) R[(int64_t)d * ldr + j] = __longlong_as_double(0x7FF8000000000000ll);
    }
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
  __shared__ uint64_t full[XSTG], done[XSTG], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  volatile int *abort_flag = &abort_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < XSTG; s++) {
      mbar_init(&full[s], 2);  // X's copy and A's
      mbar_init(&done[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], EPI_WARPS);
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
          // X goes where chunk g - XSTG was, A where chunk g - ASTG was
          const uint32_t g = issued, x = g % XSTG, a = g % ASTG;
          if (g >= XSTG && !oz_wait(&done[x], (g / XSTG - 1) & 1, abort_flag)) break;
          mbar_expect_tx(&full[x], X_BYTES);
          bulk_g2s(smem + x * X_BYTES, xs + (size_t)kc * X_BYTES, X_BYTES, &full[x]);
          if (g >= ASTG && !oz_wait(&done[(g - ASTG) % XSTG], ((g - ASTG) / XSTG) & 1, abort_flag)) {
            mbar_arrive(&full[x]);  // no A: the phase ends with X's copy
            issued = g + 1;
            break;
          }
          mbar_expect_tx(&full[x], A_BYTES);
          bulk_g2s(asm_ + a * (Z_BYTES + A_BYTES) + Z_BYTES, as + (size_t)kc * A_BYTES, A_BYTES, &full[x]);
          issued = g + 1;
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    // ---- MMA (one lane issues; the warp stays converged)
    const uint32_t lead = elect_one();
    constexpr uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);
    uint32_t dr = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < nitem && ok; i += gridDim.x) {
      for (int kc = 0; kc < nkc; kc++) {
        const uint32_t g = g_mma, x = g % XSTG, a = g % ASTG, ab = dr & 1;
        const uint32_t dacc = tmem + ab * 256;
        const bool first = kc % OZ_DRAIN == 0;
        if (first && dr >= 2) ok = acc_wait(&acc_empty[ab], (dr / 2 - 1) & 1, abort_flag);
        ok = ok && acc_wait(&full[x], (g / XSTG) & 1, abort_flag);
        if (!__all_sync(0xffffffffu, ok && !*abort_flag)) {
          ok = false;
          break;
        }
        // (these instructions are the kernel's serial part: 14 MMAs take the
        // tensor core 1570 cycles)
        const uint32_t xd = sdesc_lo(smem_u32(smem + x * X_BYTES)),
                       ad = sdesc_lo(smem_u32(asm_ + a * (Z_BYTES + A_BYTES)));
#pragma unroll
        for (int n = 0; n < OZ_S * (OZ_KC / 16); n++) {
          const int q = n % OZ_S, k16 = n / OZ_S;
          mma_bf16(lead, dacc, xd + (q * XS_BYTES + k16 * 32) / 16, ad + ((OZ_S - 1 - q) * AS_BYTES + k16 * 32) / 16, idesc,
                   n == 0 && first ? 0u : 1u);
        }
        mma_commit(lead, &done[x]);
        g_mma = g + 1;
        if (kc % OZ_DRAIN == OZ_DRAIN - 1 || kc == nkc - 1) {
          mma_commit(lead, &acc_full[ab]);
          dr++;
        }
      }
    }
  } else {
    // ---- epilogue: lane = sample, EPI_ND detectors per thread
    const int quarter = warp & 3, part = warp >> 2;
    const uint32_t base = tmem + ((uint32_t)(32 * quarter) << 16) + EPI_ND * part;
    uint32_t dr = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < nitem && ok; i += gridDim.x) {
      const int js = (i / ndb) * OZ_M + 32 * quarter + lane;
      const int d0 = (i % ndb) * OZ_ND + EPI_ND * part;
      const int c = sx[js];
      int a[EPI_ND];
#pragma unroll
      for (int d = 0; d < EPI_ND; d++) a[d] = __ldg(sa + d0 + d);
      long long hi[EPI_ND], lo[EPI_ND];
#pragma unroll
      for (int d = 0; d < EPI_ND; d++) hi[d] = lo[d] = 0;
      for (int n = 0; n < ndrain; n++, dr++) {
        ok = acc_wait(&acc_full[dr & 1], (dr / 2) & 1, abort_flag);
        if (!ok) break;
        const uint32_t acc = base + (dr & 1) * 256;
        uint32_t v[3][8], u[4][8];
#pragma unroll
        for (int t = 0; t < 3; t++) tmem_ld8(acc + t * OZ_ND, v[t]);
        tmem_wait(v);
#pragma unroll
        for (int t = 0; t < 4; t++) tmem_ld8(acc + (3 + t) * OZ_ND, u[t]);
#pragma unroll
        for (int d = 0; d < EPI_ND; d++)
#pragma unroll
          for (int t = 0; t < 3; t++) hi[d] = mad_wide(__float2int_rn(__uint_as_float(v[t][d])), 1 << (8 * (2 - t)), hi[d]);
        tmem_wait(u);
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[dr & 1]);
#pragma unroll
        for (int d = 0; d < EPI_ND; d++)
#pragma unroll
          for (int t = 0; t < 4; t++) lo[d] = mad_wide(__float2int_rn(__uint_as_float(u[t][d])), 1 << (8 * (3 - t)), lo[d]);
      }
      const int64_t j = j0 + js;
      if (ok && j < ncol) {
#pragma unroll
        for (int d = 0; d < EPI_ND; d++) {
          if (d0 + d >= nrow) continue;
          // (a NOSCALE row or column: NaN, as the FP64 product of a non-finite entry)
          const double r = combine(hi[d], lo[d], a[d] + c);
          __stcs(R + (int64_t)(d0 + d) * ldr + j, r);
        }
      }
    }
  }
  __syncthreads();
  const bool failed = *abort_flag;
  if (failed) {
    // after a timeout: bounded waits for the copies and MMAs still in flight
    if (tid == EPI_WARPS * 32)
      for (uint32_t g = issued > XSTG ? issued - XSTG : 0; g < issued; g++) {
        (void)mbar_wait(&full[g % XSTG], (g / XSTG) & 1);
      }
    if (tid == (EPI_WARPS + 1) * 32) {
      atomicExch(err, 1);
      for (uint32_t g = g_mma > XSTG ? g_mma - XSTG : 0; g < g_mma; g++)
        (void)mbar_wait(&done[g % XSTG], (g / XSTG) & 1);
    }
  }
  if (failed) fill_nan(R, ldr, nrow, ndb, nitem, j0, ncol);  // no caller takes this CTA's part for a result
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
  // blocks of equal size; a little larger where that gives every SM the same
  // number of items (256 x 130,978: 54 items in a row instead of 56)
  int64_t per = (ntile + nblk - 1) / nblk;
  for (int64_t q = per; q <= L.tiles; q++)
    if (q * L.ndb % sm_count() == 0) {
      per = q;
      break;
    }
  for (int64_t t0 = 0; t0 < ntile; t0 += per) {
    const int64_t nt = ntile - t0 < per ? ntile - t0 : per, j0 = t0 * OZ_M;
    const int nu = (L.nkc + 1) / 2;
    auto slice = nu == 1 ? k_oz_slice_x<1> : nu == 2 ? k_oz_slice_x<2> : nu <= 4 ? k_oz_slice_x<4> : k_oz_slice_x<0>;
    slice<<<(unsigned)(nt * (OZ_M / 32)), 256, 0, st>>>(X, ldx, (int)nrow, L.nkc, j0, ncol, sx, w + L.x);
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
