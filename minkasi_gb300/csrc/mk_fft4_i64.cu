// FP64 DCT-I by the four-step FFT of mk_fft4.cuh in 64-bit block fixed point.
//
// GB300 runs two FP64 operations per clock and SM, and the FP64 passes needed
// about 47 per point: they kept the FP64 pipe busy and everything else idle.
// Its integer units are 16-32 times as wide, so the passes for smooth lengths
// run on int64 values with one exponent per CTA tile:
//   * pass A converts the rows of a pair to v = x 2^(f - e0), 2^e0 > max |x|
//     over both rows, f about 58 bits (exact for the largest samples);
//   * before each stage of radix R the tile's largest magnitude (the OR of all
//     high words, reduced over the CTA) decides how many bits the values are
//     shifted down, so that the stage cannot overflow; the tile's exponent
//     follows;
//   * T holds the int64 values, with (exponent, bits) per tile of pass A; pass
//     B aligns them to the pair's largest exponent;
//   * pass B's last stage converts to FP64 (rounded to nearest) and applies the
//     weights or the halving in FP64.
// A product by a twiddle (62 fraction bits) or a butterfly constant (61) keeps
// 64 bits, rounded.  So a stage rounds at about 2^-58 of the tile's largest
// value where FP64 rounds at 2^-53 of each value.  Both spread over all
// outputs in the stages that follow; relative error (2-norm) of a DCT-I of
// 130,978 points against extended precision, FP64 passes in brackets: white
// noise 7.4e-17 (7.0e-16), 1/f noise 1.0e-16 (5.7e-16), noise on an offset of
// 1e4 1.2e-16 (3.5e-16; its upper spectrum 1.3e-12, 3.6e-12), one sample 1e6
// times the others 4.3e-16 (6.9e-16), a 1/f power spectrum 7.6e-16 (7.9e-16).
// A pair with a NaN or infinity becomes NaN throughout, as its FP64 transform
// (which mixes the two rows in every product) does.
//
// One DCT-I of 256 x 130,978 takes 0.98 ms against 2.52 ms in FP64, of 64 x
// 65,341 0.18 against 0.31 ms, of 256 x 450,561 2.80 against 7.88 ms.
#include <algorithm>

#include "mk_common.cuh"
#include "mk_fft4.cuh"

namespace mk {
namespace {

using i64 = long long;
struct __align__(16) Z {  // a fixed-point complex value
  i64 x, y;
};
struct __align__(16) W {  // a twiddle: 2^62 (cos, -sin), each as 2^32 h + l with a signed low word
  int xh, xl, yh, yl;
};

constexpr int NT = 256;             // threads per CTA
constexpr int FBH = 8, FBL = 4;     // transforms per CTA (wide and narrow tile, as the FP64 kernels)
constexpr int LIM = 61;             // a stage's outputs stay below 2^(LIM + 1/2)
constexpr int MAXT = 256;           // most tiles of a pass per pair
constexpr int PRE = 16;             // slices of the pre-pass over a pair's rows
constexpr int NAN_TILE = 1 << 28;   // exponent of a tile that holds a non-finite value

__device__ __forceinline__ Z mkz(i64 x, i64 y) {
  Z z;
  z.x = x;
  z.y = y;
  return z;
}
__device__ __forceinline__ Z operator+(Z a, Z b) { return mkz(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ Z operator-(Z a, Z b) { return mkz(a.x - b.x, a.y - b.y); }

// a = 2^32 h + l, l signed
struct HL {
  int h, l;
};
__host__ __device__ __forceinline__ constexpr HL split(i64 a) {
  const int l = (int)a;
  return HL{(int)(a >> 32) + (int)((unsigned)l >> 31), l};
}
__device__ __forceinline__ i64 wide(int a, int b) { return (i64)a * b; }

// a w for |a| < 2^61.5, w with 62 fraction bits, rounded to nearest.  Rounding
// down instead would add the same offset to every value, and the next stages
// sum those coherently; leaving the low x low products out would add a third
// of a unit of noise per product.
__device__ __forceinline__ Z cmul(Z a, W w) {
  const HL x = split(a.x), y = split(a.y);
  const i64 hr = wide(x.h, w.xh) - wide(y.h, w.yh), hi = wide(x.h, w.yh) + wide(y.h, w.xh);
  // the low x low products from the upper halves of the low words
  const int x2 = x.l >> 16, y2 = y.l >> 16, wx = w.xl >> 17, wy = w.yl >> 17;
  const i64 lr = (i64)(x2 * wx - y2 * wy) * 2, li = (i64)(x2 * wy + y2 * wx) * 2;
  const i64 cr = (1ll << 29) + lr + wide(x.h, w.xl) + wide(x.l, w.xh) - wide(y.h, w.yl) - wide(y.l, w.yh);
  const i64 ci = (1ll << 29) + li + wide(x.h, w.yl) + wide(x.l, w.yh) + wide(y.h, w.xl) + wide(y.l, w.xh);
  return mkz((hr << 2) + (cr >> 30), (hi << 2) + (ci >> 30));
}
__device__ __forceinline__ Z cmulc(Z a, i64 c, i64 s) {  // a (c + i s), constants with 62 bits
  const HL k = split(c), t = split(s);
  return cmul(a, W{k.h, k.l, t.h, t.l});
}
__device__ __forceinline__ i64 mulq62(i64 a, i64 k) {
  const HL x = split(a), c = split(k);
  return (wide(x.h, c.h) << 2) + (((1ll << 29) + (wide(x.l, c.l) >> 32) + wide(x.h, c.l) + wide(x.l, c.h)) >> 30);
}
__device__ __forceinline__ Z mul_mi(Z z) { return mkz(z.y, -z.x); }  // -i z

// forward DFT of R points in registers, as in mk_fft4_kern.cuh.  With
// |components| < 2^(LIM - ceil(log2 R) + 1/2) on entry nothing overflows:
// the outputs are at most R times the largest modulus.
template <int R>
struct Dft;
template <>
struct Dft<2> {
  __device__ static __forceinline__ void run(Z *v) {
    const Z a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  }
};
template <>
struct Dft<4> {
  __device__ static __forceinline__ void run(Z *v) {
    const Z s02 = v[0] + v[2], d02 = v[0] - v[2], s13 = v[1] + v[3], d13 = v[1] - v[3];
    v[0] = s02 + s13;
    v[2] = s02 - s13;
    v[1] = mkz(d02.x + d13.y, d02.y - d13.x);
    v[3] = mkz(d02.x - d13.y, d02.y + d13.x);
  }
};
constexpr i64 Q62_H = 3260954456333195553ll;  // sqrt(1/2)
template <>
struct Dft<8> {
  __device__ static __forceinline__ void run(Z *v) {
    Z e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4>::run(e);
    Dft<4>::run(o);
    o[1] = mkz(mulq62(o[1].x + o[1].y, Q62_H), mulq62(o[1].y - o[1].x, Q62_H));
    o[2] = mul_mi(o[2]);
    o[3] = mkz(mulq62(o[3].y - o[3].x, Q62_H), -mulq62(o[3].x + o[3].y, Q62_H));
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[k] = e[k] + o[k];
      v[k + 4] = e[k] - o[k];
    }
  }
};

// cos(2 pi t / R) and sin(2 pi q / R) with 61 fraction bits, 1 <= t, q <= (R - 1) / 2
template <int R>
__device__ __forceinline__ constexpr i64 odd_c(int t) {
  constexpr i64 k3[] = {-1152921504606846976ll};
  constexpr i64 k5[] = {712544676207699905ll, -1865466180814546881ll};
  constexpr i64 k7[] = {1437669600931991917ll, -513098339966869658ll, -2077492765571969234ll};
  constexpr i64 k11[] = {1939798577655101867ll, 957881803652815594ll, -328155674939831993ll, -1510006045376284332ll,
                         -2212440165598648113ll};
  return R == 3 ? k3[t - 1] : R == 5 ? k5[t - 1] : R == 7 ? k7[t - 1] : k11[t - 1];
}
template <int R>
__device__ __forceinline__ constexpr i64 odd_s(int q) {
  constexpr i64 k3[] = {1996918623117814388ll};
  constexpr i64 k5[] = {2192987019466309470ll, 1355340514917506542ll};
  constexpr i64 k7[] = {1802780658232085260ll, 2248030710791760100ll, 1000467786655719552ll};
  constexpr i64 k11[] = {1246632849425566526ll, 2097468577445319519ll, 2282372852130967407ll, 1742639872740991266ll,
                         649631046660710334ll};
  return R == 3 ? k3[q - 1] : R == 5 ? k5[q - 1] : R == 7 ? k7[q - 1] : k11[q - 1];
}

// sum_r k_r a_r over split operands: the high and the cross products apart
// (each sum stays below 2^63 for the magnitudes above), and the low products
// from the upper halves of the low words
struct Acc {
  i64 hh = 0, cr = 1ll << 28;
  int ll = 0;
  __device__ __forceinline__ void add(HL a, HL k) {
    hh += wide(a.h, k.h);
    cr += wide(a.h, k.l) + wide(a.l, k.h);
    ll += (a.l >> 16) * (k.l >> 18);
  }
  __device__ __forceinline__ i64 q61() const { return (hh << 3) + ((cr + (i64)ll * 4) >> 29); }
};

template <int R>
struct DftOdd {
  __device__ static __forceinline__ void run(Z *v) {
    constexpr int H = (R - 1) / 2;
    HL sx[H + 1], sy[H + 1], dx[H + 1], dy[H + 1];
    Z x0 = v[0];
#pragma unroll
    for (int r = 1; r <= H; r++) {
      const Z s = v[r] + v[R - r], d = v[r] - v[R - r];
      x0 = x0 + s;
      sx[r] = split(s.x);
      sy[r] = split(s.y);
      dx[r] = split(d.x);
      dy[r] = split(d.y);
    }
#pragma unroll
    for (int q = 1; q <= H; q++) {
      Acc ax, ay, bx, by;
#pragma unroll
      for (int r = 1; r <= H; r++) {
        const int t = (r * q) % R;
        const HL c = split(odd_c<R>(t <= H ? t : R - t));
        const HL s = split(t <= H ? odd_s<R>(t) : -odd_s<R>(R - t));
        ax.add(sx[r], c);
        ay.add(sy[r], c);
        bx.add(dx[r], s);
        by.add(dy[r], s);
      }
      const i64 Ax = v[0].x + ax.q61(), Ay = v[0].y + ay.q61(), Bx = bx.q61(), By = by.q61();
      v[q] = mkz(Ax + By, Ay - Bx);
      v[R - q] = mkz(Ax - By, Ay + Bx);
    }
    v[0] = x0;
  }
};
template <>
struct Dft<3> : DftOdd<3> {};
template <>
struct Dft<5> : DftOdd<5> {};
template <>
struct Dft<7> : DftOdd<7> {};
template <>
struct Dft<11> : DftOdd<11> {};

template <>
struct Dft<9> {
  __device__ static __forceinline__ void run(Z *v) {
    Z y[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < 3; n1++) y[n2][n1] = v[3 * n1 + n2];
      Dft<3>::run(y[n2]);
    }
    constexpr i64 c1 = 3532756447825785444ll, s1 = 2964334632409774423ll, c2 = 800810873071977681ll,
                  s2 = 4541624145405292212ll, c4 = -4333567320897763126ll, s4 = 1577289512995517789ll;
    y[1][1] = cmulc(y[1][1], c1, -s1);
    y[1][2] = cmulc(y[1][2], c2, -s2);
    y[2][1] = cmulc(y[2][1], c2, -s2);
    y[2][2] = cmulc(y[2][2], c4, -s4);
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++) {
      Z t[3] = {y[0][k1], y[1][k1], y[2][k1]};
      Dft<3>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < 3; k2++) v[k1 + 3 * k2] = t[k2];
    }
  }
};
template <>
struct Dft<16> {
  __device__ static __forceinline__ void run(Z *v) {
    constexpr i64 c1 = 4260642322793532497ll, s1 = 1764815834521887442ll, h = Q62_H;
    Z y[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < 4; n1++) y[n2][n1] = v[4 * n1 + n2];
      Dft<4>::run(y[n2]);
    }
    y[1][1] = cmulc(y[1][1], c1, -s1);
    y[1][2] = cmulc(y[1][2], h, -h);
    y[1][3] = cmulc(y[1][3], s1, -c1);
    y[2][1] = cmulc(y[2][1], h, -h);
    y[2][2] = mul_mi(y[2][2]);
    y[2][3] = cmulc(y[2][3], -h, -h);
    y[3][1] = cmulc(y[3][1], s1, -c1);
    y[3][2] = cmulc(y[3][2], -h, -h);
    y[3][3] = cmulc(y[3][3], -c1, s1);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      Z t[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
      Dft<4>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < 4; k2++) v[k1 + 4 * k2] = t[k2];
    }
  }
};

constexpr int inv_mod(int a, int m) {
  for (int x = 1; x < m; x++)
    if ((a * x) % m == 1) return x;
  return 1;
}
template <int R1, int R2>
struct DftPfa {  // Good-Thomas
  __device__ static __forceinline__ void run(Z *v) {
    constexpr int R = R1 * R2, e1 = inv_mod(R2 % R1, R1), e2 = inv_mod(R1 % R2, R2);
    Z a[R2][R1];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) a[n2][n1] = v[(n1 * R2 + n2 * R1) % R];
      Dft<R1>::run(a[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
      Z c[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; n2++) c[n2] = a[n2][k1];
      Dft<R2>::run(c);
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) v[(k1 * R2 * e1 + k2 * R1 * e2) % R] = c[k2];
    }
  }
};
template <>
struct Dft<6> : DftPfa<2, 3> {};
template <>
struct Dft<10> : DftPfa<2, 5> {};
template <>
struct Dft<12> : DftPfa<4, 3> {};
template <>
struct Dft<14> : DftPfa<2, 7> {};
template <>
struct Dft<15> : DftPfa<3, 5> {};

static_assert(MK_FFT4_RMAX64 == 16, "the radix switch below covers 2 .. 16");
#define MK_RADIX_SWITCH(R, CALL)                     \
  switch (R) {                                       \
    case 2: { constexpr int RR = 2; CALL; } break;   \
    case 3: { constexpr int RR = 3; CALL; } break;   \
    case 4: { constexpr int RR = 4; CALL; } break;   \
    case 5: { constexpr int RR = 5; CALL; } break;   \
    case 6: { constexpr int RR = 6; CALL; } break;   \
    case 7: { constexpr int RR = 7; CALL; } break;   \
    case 8: { constexpr int RR = 8; CALL; } break;   \
    case 9: { constexpr int RR = 9; CALL; } break;   \
    case 10: { constexpr int RR = 10; CALL; } break; \
    case 12: { constexpr int RR = 12; CALL; } break; \
    case 14: { constexpr int RR = 14; CALL; } break; \
    case 15: { constexpr int RR = 15; CALL; } break; \
    case 16: { constexpr int RR = 16; CALL; } break; \
    default: { constexpr int RR = 11; CALL; } break; \
  }

__device__ __forceinline__ W ldw(const W *p) {
  const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
  return W{v.x, v.y, v.z, v.w};
}

// ---- magnitudes and exponents ---------------------------------------------
__device__ __forceinline__ int mag(i64 v) {  // high word of |v| (or of |v| - 1)
  const int h = (int)(v >> 32);
  return h ^ (h >> 31);
}
__device__ __forceinline__ int mag(Z v) { return mag(v.x) | mag(v.y); }
// |v| <= 2^bits for every value whose mag() went into the OR
__device__ __forceinline__ int bits_of(int o) { return o ? 64 - __clz(o) : 32; }
__device__ __forceinline__ int lg_ceil(int R) { return 32 - __clz(R - 1); }
// bits to shift values below 2^bits (in units of 2^ex) down by before a stage
// of radix R: its outputs are below R times that, and below the pair's
// 2^bsum >= sum |e_j| whatever the stage (an impulse never grows)
__device__ __forceinline__ int stage_shift(int bits, int R, int bsum, int ex) {
  return max(0, min(bits + lg_ceil(R), bsum - ex) - LIM);
}
// (v + half) >> sh with half = 2^(sh - 1), or 0 for sh = 0
struct Shift {
  int sh;
  i64 half;
  __device__ __forceinline__ explicit Shift(int s) : sh(s), half((1ll << s) >> 1) {}
  __device__ __forceinline__ Z operator()(Z v) const { return mkz((v.x + half) >> sh, (v.y + half) >> sh); }
};
// the CTA's OR of `o` into *word (zero before); a barrier follows
__device__ __forceinline__ void or_into(int *word, int o) {
  o = __reduce_or_sync(0xffffffffu, (unsigned)o);
  if ((threadIdx.x & 31) == 0 && o) atomicOr(word, o);
}

// x 2^(frac - e0) rounded, for |x| < 2^e0
__device__ __forceinline__ i64 to_fixed(double x, int e0, int frac) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ef = (int)((b >> 52) & 0x7FF);
  unsigned long long m = b & 0x000FFFFFFFFFFFFFull;
  if (ef) m |= 0x0010000000000000ull;
  const int sh = (ef ? ef : 1) - 1075 + frac - e0;  // at most frac - 53
  if (sh >= 0)
    m <<= sh;
  else
    m = sh > -64 ? (m + (1ull << (-sh - 1))) >> (-sh) : 0ull;
  return b >> 63 ? -(i64)m : (i64)m;
}

// v 2^ex rounded to nearest
__device__ __forceinline__ double to_double(i64 v, int ex) {
  const unsigned long long sign = (unsigned long long)v & 0x8000000000000000ull;
  const unsigned long long a = sign ? 0ull - (unsigned long long)v : (unsigned long long)v;
  if (a == 0) return 0.0;
  const int z = __clzll((i64)a);
  const unsigned long long w = a << z;
  unsigned long long m = w >> 11;
  const unsigned r = (unsigned)w & 0x7FFu;
  if (r > 0x400u || (r == 0x400u && (m & 1))) m++;  // a carry to 2^53 moves into the exponent below
  const int E = 63 - z + ex;
  if (E > -1022 && E < 1023)
    return __longlong_as_double((i64)((((unsigned long long)(E + 1022)) << 52) + m + sign));
  return ldexp(__longlong_as_double((i64)((1022ull << 52) + m + sign)), E);
}

__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7FFFFFFF; }

// |x| of a high word as a float, at least 2^-126, infinite from 2^128 on (20
// bits of the significand; the sums below carry 0.1 % of slack)
__device__ __forceinline__ float hi_float(int h) {
  return __int_as_float(h >= (1151 << 20) ? 0x7F800000 : (max(h, 897 << 20) - (896 << 20)) << 3);
}

// (largest high word, sum of |x|) of a thread's values reduced over the CTA;
// thread 0 stores the exponent field and the sum
__device__ __forceinline__ void store_stats(int2 *dst, int mx, float sum, int2 *sh) {
  mx = __reduce_max_sync(0xffffffffu, mx);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_int2(mx, __float_as_int(sum));
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)blockDim.x / 32; w++) {
      mx = max(mx, sh[w].x);
      sum += __int_as_float(sh[w].y);
    }
    *dst = make_int2(mx >> 20, __float_as_int(sum));
  }
}

// stat[pair][slice] = (exponent field of the largest |x|, sum of |x|) of a
// slice of the pair's rows
__global__ void __launch_bounds__(NT) k_i64_stats(const double *__restrict__ x, int64_t ldx, int64_t nrow, int64_t n,
                                                  int2 *__restrict__ stat) {
  const int64_t pair = blockIdx.y;
  const int64_t a = n * blockIdx.x / PRE, b = n * (blockIdx.x + 1) / PRE;
  int m = 0;
  float sum = 0.f;
  for (int r = 0; r < 2; r++) {
    if (2 * pair + r >= nrow) break;
    const double *row = x + (2 * pair + r) * ldx;
#pragma unroll 8
    for (int64_t i = a + threadIdx.x; i < b; i += NT) {
      const int h = abs_hi(__ldg(row + i));
      m = max(m, h);
      sum += hi_float(h);
    }
  }
  __shared__ int2 sh[NT / 32];
  store_stats(stat + pair * MAXT + blockIdx.x, m, sum, sh);
}

// a decimation-in-time stage in shared memory on one slot; inputs shifted down by sh
template <int R, int FB>
__device__ __forceinline__ int stage_dit(Z *slot, int Ls, int Ns, float invNs, const W *stw, Shift sh) {
  const int nq = Ls / R;
  int o = 0;
  for (int q = threadIdx.x / FB; q < nq; q += (int)blockDim.x / FB) {
    const int g = __float2int_rz(((float)q + 0.5f) * invNs);
    const int k = q - g * Ns;
    Z *a = slot + g * Ns * R + k;
    Z v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = sh(a[r * Ns]);
      if (r) v[r] = cmul(v[r], ldw(stw + (r - 1) * Ns + k));
    }
    Dft<R>::run(v);
#pragma unroll
    for (int r = 0; r < R; r++) {
      a[r * Ns] = v[r];
      o |= mag(v[r]);
    }
  }
  return o;
}

__host__ __device__ __forceinline__ int pitch_odd(int Ls) { return Ls | 1; }
__device__ __forceinline__ const W *wtab(const void *t) { return static_cast<const W *>(t); }

// ---- pass A: rows of a pair -> T[pair] and texp[pair][tile] = (exponent, bits, the pair's bsum)
template <int R, int FB>
__device__ __forceinline__ int astage_first(Z *sbuf, int pitch, const double *x1, const double *x2, bool has2, int j1_0,
                                            int nb, int e0, int frac, const Fft4Dev &p) {
  const int nq = p.L2 / R, b = threadIdx.x % FB, L = (int)p.L;
  int o = 0;
  if (b >= nb) return o;
  const int step = p.L1 * nq;
  for (int q = threadIdx.x / FB; q < nq; q += (int)blockDim.x / FB) {
    const int j = j1_0 + b + p.L1 * __ldg(p.iperm2 + q * R);
    double u[R], w[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int jj = min(j + step * r, L - (j + step * r));
      u[r] = __ldg(x1 + jj);
      w[r] = has2 ? __ldg(x2 + jj) : 0.0;
    }
    Z v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = mkz(to_fixed(u[r], e0, frac), to_fixed(w[r], e0, frac));
    Dft<R>::run(v);
    Z *a = sbuf + b * pitch + q * R;
#pragma unroll
    for (int r = 0; r < R; r++) {
      a[r] = v[r];
      o |= mag(v[r]);
    }
  }
  return o;
}

// output k2 of row j1 into T with its four-step twiddle
__device__ __forceinline__ int put_t(Z *row, const W *tw, int e, Z v) {
  const Z t = cmul(v, ldw(tw + e));
  row[e] = t;
  return mag(t);
}

template <int R, int FB>
__device__ __forceinline__ int astage_last(const Z *sbuf, int pitch, int Ns, const W *stw, Shift sh, int j1_0, int nb,
                                           const Fft4Dev &p, Z *Tp) {
  const int h2 = p.L2 / 2;
  int o = 0;
  for (int bf = threadIdx.x; bf < FB * Ns; bf += (int)blockDim.x) {
    const int b = bf / Ns, q = bf - b * Ns;
    if (b >= nb) break;  // b grows with bf
    const Z *a = sbuf + b * pitch + q;
    Z v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = sh(a[r * Ns]);
      if (r) v[r] = cmul(v[r], ldw(stw + (r - 1) * Ns + q));
    }
    Dft<R>::run(v);
    const int j1 = j1_0 + b;
    const W *tw = wtab(p.tfull) + j1 * p.P;
    Z *row = Tp + j1 * p.P;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k2 = q + r * Ns;
      o |= put_t(row, tw, k2 + (k2 > h2 ? p.pad : 0), v[r]);
    }
    if (q == p.qh) {  // L2 even: entry L2 / 2 again with the other sign's twiddle
#pragma unroll
      for (int r = 0; r < R; r++)
        if (q + r * Ns == h2) o |= put_t(row, tw, h2 + p.pad, v[r]);
    }
  }
  return o;
}

template <int FB>
__global__ void __launch_bounds__(NT, 2) k_i64_a(const double *__restrict__ x, int64_t ldx, int64_t nrow,
                                                 Z *__restrict__ T, const int2 *__restrict__ stat, int nstat,
                                                 int4 *__restrict__ texp, const Fft4Dev p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Z *const sbuf = reinterpret_cast<Z *>(smem_raw);
  __shared__ int s_or[FFT4_MAXR + 1], s_e;
  __shared__ float s_sum;
  const int L2 = p.L2, pitch = pitch_odd(L2), tid = threadIdx.x;
  const int64_t pair = blockIdx.y, r0 = 2 * pair;
  const bool has2 = r0 + 1 < nrow;
  const double *x1 = x + r0 * ldx, *x2 = has2 ? x1 + ldx : x1;
  const int j1_0 = blockIdx.x * FB, nb = min(FB, p.H1 - j1_0);
  Z *Tp = T + pair * p.tsz;
  if (tid < FFT4_MAXR + 1) s_or[tid] = 0;
  if (tid < 32) {
    int m = 0;
    float sum = 0.f;
    for (int i = tid; i < nstat; i += 32) {
      const int2 t = stat[pair * MAXT + i];
      m = max(m, t.x);
      sum += __int_as_float(t.y);
    }
    m = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (tid == 0) {
      s_e = m;
      s_sum = 2.002f * sum;  // the extension holds every inner sample twice
    }
  }
  __syncthreads();
  const int ef = s_e;
  if (ef == 0x7FF) {
    if (tid == 0) texp[pair * MAXT + blockIdx.x] = make_int4(NAN_TILE, 0, 0, 0);
    return;
  }
  const int S = p.nr2, e0 = ef - 1022;  // |x| < 2^e0
  // 2^bsum > the sum; no bound (2^4000) where FP32 cannot hold it
  const int bsum = s_sum < 3e38f ? (__float_as_int(s_sum) >> 23) - 126 : 4000;
  // the most fraction bits with which the first stage stays below 2^LIM
  const int frac = LIM - max(0, min(S ? lg_ceil(p.r2[0]) : 0, bsum - e0));
  int ex = e0 - frac, o = 0;
  if (S >= 1)
    MK_RADIX_SWITCH(p.r2[0], (o = astage_first<RR, FB>(sbuf, pitch, x1, x2, has2, j1_0, nb, e0, frac, p)));
  if (S >= 2) {
    for (int s = 1; s < S; s++) {
      or_into(&s_or[s], o);
      __syncthreads();
      const Shift sh(stage_shift(bits_of(s_or[s]), p.r2[s], bsum, ex));
      ex += sh.sh;
      o = 0;
      const W *stw = wtab(p.stw2) + p.to2[s];
      if (s < S - 1) {
        if (tid % FB < nb)
          MK_RADIX_SWITCH(p.r2[s],
                          (o = stage_dit<RR, FB>(sbuf + (tid % FB) * pitch, L2, p.ns2[s], p.inv2[s], stw, sh)));
      } else {
        MK_RADIX_SWITCH(p.r2[s], (o = astage_last<RR, FB>(sbuf, pitch, p.ns2[s], stw, sh, j1_0, nb, p, Tp)));
      }
    }
  } else {
    // one stage at most (L2 <= 16): each warp twiddles and stores rows b
    if (S == 0 && tid < nb) {  // L2 == 1
      const int jj = min(j1_0 + tid, (int)p.L - (j1_0 + tid));
      sbuf[tid * pitch] = mkz(to_fixed(x1[jj], e0, frac), has2 ? to_fixed(x2[jj], e0, frac) : 0);
    }
    __syncthreads();
    const int k2 = tid & 31, h2 = L2 / 2;
    o = 0;
    for (int b = tid >> 5; b < nb; b += (int)blockDim.x / 32) {
      const int j1 = j1_0 + b;
      if (k2 < L2) {
        const Z v = sbuf[b * pitch + k2];
        const W *tw = wtab(p.tfull) + j1 * p.P;
        o |= put_t(Tp + j1 * p.P, tw, k2 + (k2 > h2 ? p.pad : 0), v);
        if (k2 == h2 && L2 % 2 == 0) o |= put_t(Tp + j1 * p.P, tw, h2 + p.pad, v);
      }
    }
  }
  or_into(&s_or[0], o);
  __syncthreads();
  if (tid == 0) texp[pair * MAXT + blockIdx.x] = make_int4(ex, bits_of(s_or[0]), bsum, 0);
}

// ---- pass B: T[pair] -> DCT rows of out with the epilogue
struct PassB {
  int L2, L, k2, m;
  bool has2, self;  // self: the column is its own mirror
  double *o1, *o2;
  const double *w1, *w2;
};

// largest high word and sum of what a thread wrote (EPI FFT4_FILTER)
struct Stats {
  int mx = 0;
  float sum = 0.f;
  __device__ __forceinline__ void add(double x) {
    const int h = abs_hi(x);
    mx = max(mx, h);
    sum += hi_float(h);
  }
};

// outputs k1 = q + r Ns of the column, scaled by 2^ex
template <int R, int EPI>
__device__ __forceinline__ void bput(const Z *v, int q, int Ns, int ex, const PassB &pb, Stats &st) {
#pragma unroll
  for (int r = 0; r < R; r++) {
    int kk = pb.k2 + pb.L2 * (q + r * Ns);
    if (pb.self && kk > pb.m) continue;  // a self-mirrored column holds both values of a pair
    kk = min(kk, pb.L - kk);
    double a = to_double(v[r].x, ex), c = to_double(v[r].y, ex);
    if (EPI == FFT4_FILTER) {
      a *= __ldg(pb.w1 + kk);
      st.add(a);
      if (pb.has2) {
        c *= __ldg(pb.w2 + kk);
        st.add(c);
      }
    } else if (EPI == FFT4_HALVE && (kk == 0 || kk == pb.m)) {
      a *= 0.5;
      c *= 0.5;
    }
    pb.o1[kk] = a;
    if (pb.has2) pb.o2[kk] = c;
  }
}
template <int R>
__device__ __forceinline__ void bput_epi(const Z *v, int q, int Ns, int ex, int epi, const PassB &pb, Stats &st) {
  if (epi == FFT4_FILTER) bput<R, FFT4_FILTER>(v, q, Ns, ex, pb, st);
  else if (epi == FFT4_HALVE) bput<R, FFT4_HALVE>(v, q, Ns, ex, pb, st);
  else bput<R, FFT4_PLAIN>(v, q, Ns, ex, pb, st);
}

// element j1 of the column: row j1 (2 j1 <= L1) or row L1 - j1's mirrored entry
struct TCol {
  const Z *fwd, *rev;
  int L1, P, lgfa;
  const int *shift;  // per tile of pass A
  __device__ __forceinline__ Z at(int j1) const {
    const bool mir = 2 * j1 > L1;
    const int o = j1 * P, sh = shift[(mir ? L1 - j1 : j1) >> lgfa];
    return Shift(sh)(*(mir ? rev - o : fwd + o));
  }
};

template <int R, int FB, bool LAST>
__device__ __forceinline__ int bstage_first(Z *slot, int Ls, const TCol &col, const int *iperm, int ex, int epi,
                                            const PassB &pb, Stats &st) {
  const int nq = Ls / R;
  int o = 0;
  for (int q = threadIdx.x / FB; q < nq; q += (int)blockDim.x / FB) {
    const int j = __ldg(iperm + q * R);
    Z v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = col.at(j + nq * r);
    Dft<R>::run(v);
    if (LAST) {
      bput_epi<R>(v, q, 1, ex, epi, pb, st);
    } else {
      Z *a = slot + q * R;
#pragma unroll
      for (int r = 0; r < R; r++) {
        a[r] = v[r];
        o |= mag(v[r]);
      }
    }
  }
  return o;
}

template <int R, int FB>
__device__ __forceinline__ void bstage_last(const Z *slot, int Ns, const W *stw, Shift sh, int ex, int epi,
                                            const PassB &pb, Stats &st) {
  for (int q = threadIdx.x / FB; q < Ns; q += (int)blockDim.x / FB) {
    const Z *a = slot + q;
    Z v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = sh(a[r * Ns]);
      if (r) v[r] = cmul(v[r], ldw(stw + (r - 1) * Ns + q));
    }
    Dft<R>::run(v);
    bput_epi<R>(v, q, Ns, ex, epi, pb, st);
  }
}

template <int FB>
__global__ void __launch_bounds__(NT, 2) k_i64_b(const Z *__restrict__ T, int64_t nrow, double *__restrict__ out,
                                                 int64_t ldo, const double *__restrict__ w, int64_t ldw, int epi,
                                                 const int4 *__restrict__ texp, int ntile, int2 *__restrict__ stat,
                                                 const Fft4Dev p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Z *const sbuf = reinterpret_cast<Z *>(smem_raw);
  __shared__ int s_or[FFT4_MAXR + 1], s_shift[MAXT], s_ec, s_bits;
  __shared__ int2 s_stat[NT / 32];
  const int L1 = p.L1, L2 = p.L2, tid = threadIdx.x, b = tid % FB, S = p.nr1;
  const int64_t pair = blockIdx.y, r0 = 2 * pair;
  if (tid < FFT4_MAXR + 1) s_or[tid] = 0;
  if (tid < 32) {
    // the pair's largest exponent, and the bits of its values at that exponent
    int ec = -(1 << 28), top = -(1 << 28);
    for (int i = tid; i < ntile; i += 32) {
      const int4 t = texp[pair * MAXT + i];
      ec = max(ec, t.x);
      top = max(top, t.x + t.y);
    }
    ec = __reduce_max_sync(0xffffffffu, ec);
    top = __reduce_max_sync(0xffffffffu, top);
    if (tid == 0) {
      s_ec = ec;
      s_bits = top - ec;
    }
  }
  __syncthreads();
  PassB pb;
  pb.has2 = r0 + 1 < nrow;
  pb.k2 = blockIdx.x * FB + b;
  pb.self = pb.k2 == 0 || 2 * pb.k2 == L2;
  const bool on = pb.k2 < p.H2;
  pb.L2 = L2;
  pb.L = (int)p.L;
  pb.m = (int)p.m;
  pb.o1 = out + r0 * ldo;
  pb.o2 = pb.o1 + ldo;
  pb.w1 = pb.w2 = nullptr;
  if (epi == FFT4_FILTER) {
    pb.w1 = w + r0 * ldw;
    pb.w2 = pb.has2 ? pb.w1 + ldw : pb.w1;
  }
  if (s_ec == NAN_TILE) {
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    for (int k1 = tid / FB; on && k1 < L1; k1 += (int)blockDim.x / FB) {
      int kk = pb.k2 + L2 * k1;
      if (pb.self && kk > pb.m) continue;
      kk = min(kk, pb.L - kk);
      pb.o1[kk] = nan;
      if (pb.has2) pb.o2[kk] = nan;
    }
    if (tid == 0 && epi == FFT4_FILTER) stat[pair * MAXT + blockIdx.x] = make_int2(0x7FF, 0);
    return;
  }
  const int bsum = texp[pair * MAXT].z, sh0 = stage_shift(s_bits, p.r1[0], bsum, s_ec);
  for (int i = tid; i < ntile; i += (int)blockDim.x) s_shift[i] = min(62, s_ec - texp[pair * MAXT + i].x + sh0);
  __syncthreads();
  int ex = s_ec + sh0, o = 0;
  Z *const slot = sbuf + b * pitch_odd(L1);
  Stats st;
  TCol col;
  const int k2 = on ? pb.k2 : 0;
  col.fwd = T + pair * p.tsz + k2;
  col.rev = T + pair * p.tsz + L1 * p.P + (k2 ? L2 - k2 + p.pad : 0);
  col.L1 = L1;
  col.P = p.P;
  col.lgfa = 31 - __clz(p.fba);
  col.shift = s_shift;
  if (S == 1) {
    if (on) MK_RADIX_SWITCH(p.r1[0], (bstage_first<RR, FB, true>(slot, L1, col, p.iperm1, ex, epi, pb, st)));
  } else {
    if (on) MK_RADIX_SWITCH(p.r1[0], (o = bstage_first<RR, FB, false>(slot, L1, col, p.iperm1, ex, epi, pb, st)));
    for (int s = 1; s < S; s++) {
      or_into(&s_or[s], o);
      __syncthreads();
      const Shift sh(stage_shift(bits_of(s_or[s]), p.r1[s], bsum, ex));
      ex += sh.sh;
      o = 0;
      const W *stw = wtab(p.stw1) + p.to1[s];
      if (on) {
        if (s < S - 1)
          MK_RADIX_SWITCH(p.r1[s], (o = stage_dit<RR, FB>(slot, L1, p.ns1[s], p.inv1[s], stw, sh)))
        else
          MK_RADIX_SWITCH(p.r1[s], (bstage_last<RR, FB>(slot, p.ns1[s], stw, sh, ex, epi, pb, st)))
      }
    }
  }
  if (epi == FFT4_FILTER) store_stats(stat + pair * MAXT + blockIdx.x, st.mx, st.sum, s_stat);
}
#undef MK_RADIX_SWITCH

// cos and -sin of 2 pi t / L with 62 fraction bits; the angle is reduced to an
// eighth of the circle in integers, so that its rounding stays below 2^-54
__device__ W unit_w(int64_t t, int64_t L) {
  t %= L;
  if (t < 0) t += L;
  const bool neg = 2 * t > L;  // -(L - t)
  if (neg) t = L - t;
  const bool half = 4 * t > L;  // pi - angle
  const int64_t u = half ? L - 2 * t : 2 * t;  // angle = pi u / L, u <= L / 2
  const bool swap = 4 * u > L;  // pi / 2 - angle
  double s, c;
  sincospi((swap ? (double)(L - 2 * u) * 0.5 : (double)u) / (double)L, &s, &c);
  if (swap) {
    const double q = s;
    s = c;
    c = q;
  }
  if (half) c = -c;
  if (neg) s = -s;
  const HL x = split(__double2ll_rn(c * 0x1p62)), y = split(__double2ll_rn(-s * 0x1p62));
  return W{x.h, x.l, y.h, y.l};
}

// the four-step twiddles of every entry of T
__global__ void k_i64_tfull(W *__restrict__ out, const Fft4Dev p) {
  const int n = p.H1 * p.P;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int j1 = i / p.P, e = i - j1 * p.P;
    const int k = e < p.up() ? e : e - p.pad - p.L2;  // the entry's signed column
    out[i] = unit_w((int64_t)j1 * k, p.L);
  }
}

bool g_attr[64] = {false};

int tiles(int H, int fb) { return (H + fb - 1) / fb; }

size_t t_bytes(const Fft4Dev &d, int64_t npairs) {
  return ((size_t)npairs * (size_t)d.tsz * sizeof(Z) + 255) / 256 * 256;
}

}  // namespace

size_t fft4_i64_bytes(const Fft4Dev &d, int64_t nrow) {
  const int64_t npairs = (nrow + 1) / 2;
  return t_bytes(d, npairs) + (size_t)npairs * MAXT * (sizeof(int4) + sizeof(int2));
}

int fft4_i64_tfull(const Fft4Dev &d, void *out) {
  k_i64_tfull<<<mk_grid((int64_t)d.H1 * d.P, 256, 8), 256>>>((W *)out, d);
  const int rc = launch_status("fft4 twiddle table");
  if (rc) return rc;
  MK_CUDA(cudaStreamSynchronize(0));
  return MK_OK;
}

// threads of a pass of ntile CTAs with smem bytes each: NT, or half of it where
// CTAs of NT threads (two per SM) would need a second, mostly empty wave and
// half-size ones (four per SM: the registers are those of 2 NT threads) all run
// at once.  Larger TODs keep NT (256 x 130,978: 0.97 ms for 1.15).  DCT with NT and
// with half: 53 x 20,001 (351 tiles a pass) 55.6 and 43.1 us, 64 x 26,245 63.0 and
// 50.7 us.
static int threads_for(int64_t ntile, size_t smem) {
  const int64_t sms = sm_count(), fit = 227 * 1024 / (int64_t)(smem + 2048);
  return ntile > std::min<int64_t>(2, fit) * sms && ntile <= std::min<int64_t>(4, fit) * sms ? NT / 2 : NT;
}

int fft4_dct_i64(const Fft4Plan &p, const double *x, int64_t ldx, int64_t nrow, void *scratch, double *out, int64_t ldo,
                 int epi, const double *w, int64_t ldw, bool chained, cudaStream_t st) {
  const Fft4Dev &d = p.d;
  const int64_t npairs = (nrow + 1) / 2;
  MK_CHECK_ARG(npairs >= 1 && npairs <= 65535, "fft4: %lld rows out of range", (long long)nrow);
  MK_CHECK_ARG(ldx >= d.n && ldo >= d.n, "fft4: leading dimensions below the row length");
  MK_CHECK_ARG(epi != FFT4_FILTER || (w && ldw >= d.n), "fft4: filter weights missing");
  MK_CHECK_ARG(d.f64 && !d.blue, "fft4: plan does not match the call");
  const int ta = tiles(d.H1, d.fba), tb = tiles(d.H2, d.fbb);
  MK_CHECK_ARG(ta <= MAXT && tb <= MAXT, "fft4: too many tiles");
  int dev = 0;
  MK_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !g_attr[dev]) {
    const int mx = FBH * (FFT4_LMAX + 1) * (int)sizeof(Z), mn = FBL * (FFT4_LMAX + 1) * (int)sizeof(Z);
    MK_CUDA(cudaFuncSetAttribute(k_i64_a<FBH>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    MK_CUDA(cudaFuncSetAttribute(k_i64_b<FBH>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    MK_CUDA(cudaFuncSetAttribute(k_i64_a<FBL>, cudaFuncAttributeMaxDynamicSharedMemorySize, mn));
    MK_CUDA(cudaFuncSetAttribute(k_i64_b<FBL>, cudaFuncAttributeMaxDynamicSharedMemorySize, mn));
    g_attr[dev] = true;
  }
  Z *T = (Z *)scratch;
  int4 *texp = (int4 *)((char *)scratch + t_bytes(d, npairs));
  int2 *stat = (int2 *)(texp + npairs * MAXT);
  const unsigned np = (unsigned)npairs;
  int rc;
  if (!chained) {
    k_i64_stats<<<dim3(PRE, np), NT, 0, st>>>(x, ldx, nrow, d.n, stat);
    if ((rc = launch_status("fft4 row statistics"))) return rc;
  }
  const int nstat = chained ? tb : PRE;
  const size_t sa = (size_t)d.fba * pitch_odd(d.L2) * sizeof(Z), sb = (size_t)d.fbb * pitch_odd(d.L1) * sizeof(Z);
  if (d.fba == FBH)
    k_i64_a<FBH><<<dim3(ta, np), threads_for((int64_t)ta * np, sa), sa, st>>>(x, ldx, nrow, T, stat, nstat, texp, d);
  else
    k_i64_a<FBL><<<dim3(ta, np), threads_for((int64_t)ta * np, sa), sa, st>>>(x, ldx, nrow, T, stat, nstat, texp, d);
  if ((rc = launch_status("fft4 pass A"))) return rc;
  if (d.fbb == FBH)
    k_i64_b<FBH><<<dim3(tb, np), threads_for((int64_t)tb * np, sb), sb, st>>>(T, nrow, out, ldo, w, ldw, epi, texp, ta, stat, d);
  else
    k_i64_b<FBL><<<dim3(tb, np), threads_for((int64_t)tb * np, sb), sb, st>>>(T, nrow, out, ldo, w, ldw, epi, texp, ta, stat, d);
  return launch_status("fft4 pass B");
}

}  // namespace mk
