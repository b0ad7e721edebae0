// Device side of the four-step FFT DCT-I (see mk_fft4.cuh), written once
// for both precisions: the including file defines
//   MK_FFT4_NS   the namespace (one per precision)
//   MK_FFT4_C    the complex type (float2 or double2)
//   MK_FFT4_RT   the real type (float or double)
//   MK_FFT4_FBHI / MK_FFT4_FBLO        transforms per CTA, wide and narrow tile
//   MK_FFT4_NTHI / MK_FFT4_NTLO        threads per CTA for each
//   MK_FFT4_MINBLO                     CTAs per SM the narrow tile's registers are sized for
//   (MK_FFT4_MINBHI, default 2: the same for the wide tile)
//   MK_FFT4_SMOOTH                     1: lengths without Bluestein too (0 in FP64: mk_fft4_i64.cu has those)
// and includes this file once.  dct_launch is the host entry of the
// precision.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <utility>

#include "mk_common.cuh"
#include "mk_fft4.cuh"

namespace mk {
namespace MK_FFT4_NS {

using C = MK_FFT4_C;
using RT = MK_FFT4_RT;
constexpr bool F32 = sizeof(RT) == 4;
static_assert(MK_FFT4_RMAX >= 11, "every prime of a supported length is a radix");
#ifndef MK_FFT4_PACK
#define MK_FFT4_PACK 1
#endif
constexpr int FB_HI = MK_FFT4_FBHI, FB_LO = MK_FFT4_FBLO;
#ifndef MK_FFT4_MINBHI
#define MK_FFT4_MINBHI 2
#endif
constexpr int NT_HI = MK_FFT4_NTHI, NT_LO = MK_FFT4_NTLO, MINB_LO = MK_FFT4_MINBLO, MINB_HI = MK_FFT4_MINBHI;

__host__ __device__ __forceinline__ C mkc(RT x, RT y) {
  C c;
  c.x = x;
  c.y = y;
  return c;
}

__device__ __forceinline__ C cmul(C a, C b) {
  return mkc(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// additions and real scalings: in FP32 both components in one f32x2
// instruction (the same roundings); the FP32 passes are bound by issue
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cfma(double2 a, double s, double2 b) {  // a s + b
  return make_double2(fma(a.x, s, b.x), fma(a.y, s, b.y));
}
#if MK_FFT4_PACK
#define MK_F32X2(OP)                                                                                             \
  float2 r;                                                                                                      \
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n " OP ".rn.f32x2 x, x, y;\n"           \
      " mov.b64 {%0, %1}, x;\n}"                                                                                 \
      : "=f"(r.x), "=f"(r.y)                                                                                     \
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                                 \
  return r;
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { MK_F32X2("add") }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { MK_F32X2("sub") }
#undef MK_F32X2
__device__ __forceinline__ float2 cfma(float2 a, float s, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mov.b64 z, {%5, %6};\n"
      " fma.rn.f32x2 z, x, y, z;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(s), "f"(b.x), "f"(b.y));
  return r;
}
#else
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cfma(float2 a, float s, float2 b) {
  return make_float2(fmaf(a.x, s, b.x), fmaf(a.y, s, b.y));
}
#endif
// -i z
__device__ __forceinline__ C mul_mi(C z) { return mkc(z.y, -z.x); }

// forward DFT of R points in registers: v_q <- sum_r v_r W_R^{rq}
template <int R>
struct Dft;

template <>
struct Dft<2> {
  __device__ static __forceinline__ void run(C *v) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <>
struct Dft<4> {
  __device__ static __forceinline__ void run(C *v) {
    const C s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
    const C s13 = cadd(v[1], v[3]), d13 = csub(v[1], v[3]);
    v[0] = cadd(s02, s13);
    v[2] = csub(s02, s13);
    v[1] = mkc(d02.x + d13.y, d02.y - d13.x);
    v[3] = mkc(d02.x - d13.y, d02.y + d13.x);
  }
};

template <>
struct Dft<8> {
  __device__ static __forceinline__ void run(C *v) {
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4>::run(e);
    Dft<4>::run(o);
    const RT h = (RT)0.70710678118654752440;
    // o_k *= W_8^k
    o[1] = mkc(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
    o[2] = mul_mi(o[2]);
    o[3] = mkc(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[k] = cadd(e[k], o[k]);
      v[k + 4] = csub(e[k], o[k]);
    }
  }
};

// constants of the odd prime radices: c(t) = cos(2 pi t / R), s(q) =
// sin(2 pi q / R) for 1 <= t, q <= H = (R - 1) / 2, and rho(q, r) =
// sin(2 pi q r / R) / s(q)
template <int R>
struct OddConst;
template <>
struct OddConst<3> {
  __device__ static __forceinline__ constexpr RT c(int t) {
    constexpr double k[] = {-0.5000000000000000000000};
    return (RT)k[t - 1];
  }
  __device__ static __forceinline__ constexpr RT s(int q) {
    constexpr double k[] = {0.8660254037844386467637};
    return (RT)k[q - 1];
  }
  __device__ static __forceinline__ constexpr RT rho(int q, int r) {
    constexpr double k[] = {1.0000000000000000000000};
    return (RT)k[(q - 1) * 1 + r - 1];
  }
};
template <>
struct OddConst<5> {
  __device__ static __forceinline__ constexpr RT c(int t) {
    constexpr double k[] = {0.3090169943749474241023, -0.8090169943749474241023};
    return (RT)k[t - 1];
  }
  __device__ static __forceinline__ constexpr RT s(int q) {
    constexpr double k[] = {0.9510565162951535721164, 0.5877852522924731291687};
    return (RT)k[q - 1];
  }
  __device__ static __forceinline__ constexpr RT rho(int q, int r) {
    constexpr double k[] = {1.0000000000000000000000, 0.6180339887498948482046,
                            1.0000000000000000000000, -1.6180339887498948482046};
    return (RT)k[(q - 1) * 2 + r - 1];
  }
};
template <>
struct OddConst<7> {
  __device__ static __forceinline__ constexpr RT c(int t) {
    constexpr double k[] = {0.6234898018587335305250, -0.2225209339563144042889,
                            -0.9009688679024191262361};
    return (RT)k[t - 1];
  }
  __device__ static __forceinline__ constexpr RT s(int q) {
    constexpr double k[] = {0.7818314824680298087084, 0.9749279121818236070181,
                            0.4338837391175581204758};
    return (RT)k[q - 1];
  }
  __device__ static __forceinline__ constexpr RT rho(int q, int r) {
    constexpr double k[] = {1.0000000000000000000000, 1.2469796037174670610500,
                            0.5549581320873711914222, 1.0000000000000000000000,
                            -0.4450418679126288085778, -0.8019377358048382524722,
                            1.0000000000000000000000, -1.8019377358048382524722,
                            2.2469796037174670610500};
    return (RT)k[(q - 1) * 3 + r - 1];
  }
};
template <>
struct OddConst<11> {
  __device__ static __forceinline__ constexpr RT c(int t) {
    constexpr double k[] = {0.8412535328311811688618, 0.4154150130018864255293,
                            -0.1423148382732851404438, -0.6548607339452850640569,
                            -0.9594929736144973898904};
    return (RT)k[t - 1];
  }
  __device__ static __forceinline__ constexpr RT s(int q) {
    constexpr double k[] = {0.5406408174555975821076, 0.9096319953545183714117,
                            0.9898214418809327323761, 0.7557495743542582837740,
                            0.2817325568414296977114};
    return (RT)k[q - 1];
  }
  __device__ static __forceinline__ constexpr RT rho(int q, int r) {
    constexpr double k[] = {1.0000000000000000000000, 1.6825070656623623377236,
                            1.8308300260037728510585, 1.3978773891157920568360,
                            0.5211085581132027229447, 1.0000000000000000000000,
                            0.8308300260037728510585, -0.3097214678905701281139,
                            -1.0881559212252219287222, -0.5943511444371404090014,
                            1.0000000000000000000000, -0.2846296765465702808876,
                            -0.9189859472289947797807, 0.5462003494572025701710,
                            0.7635211184333675579429, 1.0000000000000000000000,
                            -1.3097214678905701281139, 0.7153703234534297191124,
                            0.3727855977717922096098, -1.2036156237755650606683,
                            1.0000000000000000000000, -1.9189859472289947797807,
                            2.6825070656623623377236, -3.2287074151195649078946,
                            3.5133370916661351887822};
    return (RT)k[(q - 1) * 5 + r - 1];
  }
};

// odd prime R: with s_r = v_r + v_{R-r} and d_r = v_r - v_{R-r},
//   V_q, V_{R-q} = A_q -+ i s(q) E_q,  A_q = v_0 + sum_r cos(2 pi q r / R) s_r,
//                                      E_q = d_1 + sum_{r>1} rho(q, r) d_r.
// s(q) is factored out so that it joins the last additions as an FMA: 4 H^2 +
// 8 H operations (the FP64 passes are bound by the FP64 pipe).
template <int R>
struct DftOdd {
  __device__ static __forceinline__ void run(C *v) {
    constexpr int H = (R - 1) / 2;
    using K = OddConst<R>;
    C s[H + 1], d[H + 1];
    C x0 = v[0];
#pragma unroll
    for (int r = 1; r <= H; r++) {
      s[r] = cadd(v[r], v[R - r]);
      d[r] = csub(v[r], v[R - r]);
      x0 = cadd(x0, s[r]);
    }
#pragma unroll
    for (int q = 1; q <= H; q++) {
      C A = v[0], E = d[1];
#pragma unroll
      for (int r = 1; r <= H; r++) {
        const int t = (r * q) % R;
        A = cfma(s[r], K::c(t <= H ? t : R - t), A);
        if (r > 1) E = cfma(d[r], K::rho(q, r), E);
      }
      const RT sn = K::s(q);
      v[q] = mkc(fma(E.y, sn, A.x), fma(-E.x, sn, A.y));
      v[R - q] = mkc(fma(-E.y, sn, A.x), fma(E.x, sn, A.y));
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

__device__ __forceinline__ C cmulc(C a, RT c, RT s) {  // a (c + i s)
  return mkc(a.x * c - a.y * s, a.x * s + a.y * c);
}

// 9 = 3 x 3: three 3-point DFTs of the stride-3 subsequences, the twiddles
// W_9^{n2 k1}, three 3-point DFTs across them
template <>
struct Dft<9> {
  __device__ static __forceinline__ void run(C *v) {
    C y[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < 3; n1++) y[n2][n1] = v[3 * n1 + n2];
      Dft<3>::run(y[n2]);
    }
    const RT c1 = (RT)0.7660444431189780352024, s1 = (RT)0.6427876096865393263226;
    const RT c2 = (RT)0.1736481776669303488517, s2 = (RT)0.9848077530122080593667;
    const RT c4 = (RT)-0.9396926207859083840541, s4 = (RT)0.3420201433256687330441;
    y[1][1] = cmulc(y[1][1], c1, -s1);
    y[1][2] = cmulc(y[1][2], c2, -s2);
    y[2][1] = cmulc(y[2][1], c2, -s2);
    y[2][2] = cmulc(y[2][2], c4, -s4);
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++) {
      C t[3] = {y[0][k1], y[1][k1], y[2][k1]};
      Dft<3>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < 3; k2++) v[k1 + 3 * k2] = t[k2];
    }
  }
};

// 16 = 4 x 4 (decimation in time): four 4-point DFTs of the stride-4
// subsequences, the twiddles W_16^{n2 k1}, four 4-point DFTs across them
template <>
struct Dft<16> {
  __device__ static __forceinline__ void run(C *v) {
    const RT c1 = (RT)0.92387953251128674785, s1 = (RT)0.38268343236508977173, h = (RT)0.70710678118654752440;
    C y[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < 4; n1++) y[n2][n1] = v[4 * n1 + n2];
      Dft<4>::run(y[n2]);
    }
    // W_16^j = cos(pi j / 8) - i sin(pi j / 8)
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
      C t[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
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

// R = R1 R2 with R1, R2 coprime, by the Good-Thomas index maps (no twiddles):
// input n = (n1 R2 + n2 R1) mod R, output k = (k1 R2 e1 + k2 R1 e2) mod R with
// e1 = R2^-1 mod R1, e2 = R1^-1 mod R2, and X_k = sum W_R1^{n1 k1} W_R2^{n2 k2} x_n
template <int R1, int R2>
struct DftPfa {
  __device__ static __forceinline__ void run(C *v) {
    constexpr int R = R1 * R2, e1 = inv_mod(R2 % R1, R1), e2 = inv_mod(R1 % R2, R2);
    C a[R2][R1];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) a[n2][n1] = v[(n1 * R2 + n2 * R1) % R];
      Dft<R1>::run(a[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
      C c[R2];
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

// CALL with RR the compile-time radix R
#if MK_FFT4_RMAX >= 12
#define MK_RCASE12(CALL) case 12: { constexpr int RR = 12; CALL; } break;
#else
#define MK_RCASE12(CALL)
#endif
#if MK_FFT4_RMAX >= 14
#define MK_RCASE14(CALL) case 14: { constexpr int RR = 14; CALL; } break;
#else
#define MK_RCASE14(CALL)
#endif
#if MK_FFT4_RMAX >= 15
#define MK_RCASE15(CALL) case 15: { constexpr int RR = 15; CALL; } break;
#else
#define MK_RCASE15(CALL)
#endif
#if MK_FFT4_RMAX >= 16
#define MK_RCASE16(CALL) case 16: { constexpr int RR = 16; CALL; } break;
#else
#define MK_RCASE16(CALL)
#endif
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
    MK_RCASE12(CALL)                                 \
    MK_RCASE14(CALL)                                 \
    MK_RCASE15(CALL)                                 \
    MK_RCASE16(CALL)                                 \
    default: { constexpr int RR = 11; CALL; } break; \
  }

__device__ __forceinline__ const C *tab(const void *t) { return static_cast<const C *>(t); }

// threads per CTA by transforms per CTA (FB_HI on passes short enough for
// two such CTAs per SM, FB_LO on longer ones), and the CTAs per SM the
// register budget is sized for
template <int FB>
struct Cfg {
  static constexpr int NT = FB == FB_HI ? NT_HI : NT_LO;
  static constexpr int MINB = FB == FB_HI ? MINB_HI : MINB_LO;
  static_assert(NT % FB == 0, "a thread keeps its slot through a stage");
};

// threads to launch for ntile tiles of FB transforms with smem bytes each: NT,
// or half of it where CTAs of NT threads would need a second, mostly empty
// wave and CTAs of half the size, of which twice as many fit the registers, all
// run at once.  Beyond one wave the larger CTAs hide latency better (256 x
// 130,978 FP32: 165 us for 198).  DCT with NT and with half, FP32: 64 x 65,341
// (384 tiles a pass; 304 CTAs of 512 threads run at once) 29.4 and 24.1 us, 96 x
// 65,341 34.0 and 29.8, 48 x 130,978 41.6 and 35.6; FP64 (Bluestein) 53 x 2,340
// 90.6 and 76.2, 64 x 2,000 107 and 79.
template <int FB>
int threads_for(int64_t ntile, size_t smem) {
  constexpr int NT = Cfg<FB>::NT, HALF = NT / 2;
  const int64_t sms = sm_count(), fit = 227 * 1024 / (int64_t)(smem + 1024);
  const int64_t full = std::min<int64_t>(Cfg<FB>::MINB, fit), half = std::min<int64_t>(2 * Cfg<FB>::MINB, fit);
  return ntile > full * sms && ntile <= half * sms ? HALF : NT;
}

// row pitch (C) of a tile of FB interleaved transforms: odd, so the
// rows fall in distinct shared-memory banks
__host__ __device__ __forceinline__ int pitch_odd(int Ls) { return Ls | 1; }

// Stage indexing: the FB transforms of a CTA (slots) are interleaved over its
// threads, so thread t works on slot t % FB in every butterfly of a stage and
// the FB lanes of a slot group touch FB consecutive columns in global memory.
// Butterfly q of a stage with span Ns is group g = q / Ns, offset k = q % Ns.
// The division is done as trunc((q + 1/2) / Ns) in FP32: q < 1536 and Ns <=
// 1536, so (q + 1/2) / Ns lies at least 1/(2 Ns) from an integer, far above
// the rounding error of the product (checked exhaustively for all q, Ns <
// 2048).

// a decimation-in-time stage in shared memory (twiddles before the butterfly)
// on slot a (Ls elements)
template <int R, int FB>
__device__ __forceinline__ void stage_dit(C *slot, int Ls, int Ns, float invNs, const C *stw) {
  const int nq = Ls / R;
  for (int q = threadIdx.x / FB; q < nq; q += (int)blockDim.x / FB) {
    const int g = __float2int_rz(((float)q + 0.5f) * invNs);
    const int k = q - g * Ns;
    C *a = slot + g * Ns * R + k;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = a[r * Ns];
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(stw + (r - 1) * Ns + k));
    Dft<R>::run(v);
#pragma unroll
    for (int r = 0; r < R; r++) a[r * Ns] = v[r];
  }
}

// ---- pass A ------------------------------------------------------------
// A CTA runs FB transforms (FB consecutive j1 of the H1 = L1 / 2 + 1 that the
// evenness of the input leaves).  The first stage reads its inputs straight
// from the detector rows, forming the even extension, and the middle stages
// run in shared memory with CTA barriers.  The last stage maps the threads
// row by row instead (32 consecutive butterflies of one row per warp): it
// reads shared memory without conflicts (its span is the whole row), twiddles
// its outputs k2 (natural order) and stores them straight to T, one contiguous
// span per instruction.
// what pass A's first stage reads: the rows' even extension (DCT), or the
// same times the Bluestein chirp (zero past m, the ends at +-m halved)
enum { AM_DCT = 0, AM_BLUE = 1 };

struct PassA {
  const RT *x1, *x2;
  const C *chirp;
  bool has2;
  int L1, j1_0, nb, m, L;
  const int *iperm;
};

// input at position j of the circle of length L: the even extension e_j (index
// j or L - j, whichever is smaller); for Bluestein z_{|i|} c_{|i|} at
// j = i mod L, |i| <= m (entry m of the chirp table carries the factor 1/2 of
// the two ends), and zero in between
template <int AM>
__device__ __forceinline__ C a_input(const PassA &pa, int j) {
  const int jj = min(j, pa.L - j);
  if (AM == AM_BLUE && jj > pa.m) return mkc((RT)0, (RT)0);
  const C z = mkc(__ldg(pa.x1 + jj), pa.has2 ? __ldg(pa.x2 + jj) : (RT)0);
  return AM == AM_BLUE ? cmul(z, __ldg(pa.chirp + jj)) : z;
}

template <int R, int AM, int FB>
__device__ __forceinline__ void astage_first(C *sbuf, int pitch, int Ls, const PassA &pa) {
  const int nq = Ls / R, b = threadIdx.x % FB;
  if (b >= pa.nb) return;
  const int step = pa.L1 * nq;
  for (int q = threadIdx.x / FB; q < nq; q += (int)blockDim.x / FB) {
    const int j = pa.j1_0 + b + pa.L1 * __ldg(pa.iperm + q * R);
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = a_input<AM>(pa, j + step * r);
    Dft<R>::run(v);
    C *a = sbuf + b * pitch + q * R;
#pragma unroll
    for (int r = 0; r < R; r++) a[r] = v[r];
  }
}

// four-step twiddle of entry e of row j1 of T (see mk_fft4.cuh): the FP64 build
// keeps the whole table (16 B per entry from L2 instead of 4 operations on the
// FP64 pipe that bounds it), the FP32 one multiplies two short tables
struct RowTw {
  const C *tl, *tb;
};
__device__ __forceinline__ RowTw row_tw(const Fft4Dev &p, int j1) {
  if (!F32) return {nullptr, tab(p.tfull) + (int64_t)j1 * p.P};
  return {tab(p.tlane) + 32 * j1, tab(p.tblk) + j1 * p.nb32};
}
__device__ __forceinline__ C tw_at(const RowTw &t, int e) {
  if (!F32) return __ldg(t.tb + e);
  return cmul(__ldg(t.tb + (e >> 5)), __ldg(t.tl + (e & 31)));
}

// the last stage of pass A (Ns R = L2, so every butterfly has g = 0): rows
// mapped warp by warp, outputs k2 = q + r Ns twiddled and stored to this
// pair's T (row j1 = j1_0 + b)
template <int R, int FB>
__device__ __forceinline__ void astage_last(const C *sbuf, int pitch, int Ns, const C *stw, const PassA &pa,
                                            const Fft4Dev &p, C *Tp) {
  const int h2 = p.L2 / 2;
  for (int bf = threadIdx.x; bf < FB * Ns; bf += (int)blockDim.x) {
    const int b = bf / Ns, q = bf - b * Ns;
    if (b >= pa.nb) break;  // b grows with bf
    const C *a = sbuf + b * pitch + q;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = a[r * Ns];
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(stw + (r - 1) * Ns + q));
    Dft<R>::run(v);
    const int j1 = pa.j1_0 + b;
    const RowTw tw = row_tw(p, j1);
    C *row = Tp + j1 * p.P;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k2 = q + r * Ns, e = k2 + (k2 > h2 ? p.pad : 0);
      row[e] = cmul(v[r], tw_at(tw, e));
    }
    if (q == p.qh) {  // L2 even: entry L2 / 2 again with the other sign's twiddle
#pragma unroll
      for (int r = 0; r < R; r++)
        if (q + r * Ns == h2) row[h2 + p.pad] = cmul(v[r], tw_at(tw, h2 + p.pad));
    }
  }
}

// pass A: rows (2 pair, 2 pair + 1) of x -> T[pair] (H1 x P, twiddled)
template <int AM, int FB>
__global__ void __launch_bounds__(Cfg<FB>::NT, Cfg<FB>::MINB) k_fft4_a(const RT *__restrict__ x, int64_t ldx,
                                                    int64_t nrow, C *__restrict__ T, const Fft4Dev p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *const sbuf = reinterpret_cast<C *>(smem_raw);
  const int L2 = p.L2, pitch = pitch_odd(L2), tid = threadIdx.x;
  const int64_t pair = blockIdx.y, r0 = 2 * pair;
  PassA pa;
  pa.has2 = r0 + 1 < nrow;
  pa.x1 = x + r0 * ldx;
  pa.x2 = pa.has2 ? pa.x1 + ldx : pa.x1;
  pa.chirp = tab(p.chirp);
  pa.L1 = p.L1;
  pa.j1_0 = blockIdx.x * FB;
  pa.nb = min(FB, p.H1 - pa.j1_0);
  pa.m = (int)p.m;
  pa.L = (int)p.L;
  pa.iperm = p.iperm2;
  C *Tp = T + pair * p.tsz;
  const int S = p.nr2;
  if (S >= 1) MK_RADIX_SWITCH(p.r2[0], (astage_first<RR, AM, FB>(sbuf, pitch, L2, pa)));
  if (S >= 2) {
    for (int s = 1; s < S - 1; s++) {
      __syncthreads();
      if (tid % FB < pa.nb)
        MK_RADIX_SWITCH(p.r2[s], (stage_dit<RR, FB>(sbuf + (tid % FB) * pitch, L2, p.ns2[s], p.inv2[s],
                                                    tab(p.stw2) + p.to2[s])));
    }
    __syncthreads();
    MK_RADIX_SWITCH(p.r2[S - 1], (astage_last<RR, FB>(sbuf, pitch, p.ns2[S - 1], tab(p.stw2) + p.to2[S - 1], pa, p, Tp)));
    return;
  }
  // one stage at most (L2 <= 16): into shared memory, then each warp
  // twiddles and stores rows b
  if (S == 0 && tid < pa.nb) sbuf[tid * pitch] = a_input<AM>(pa, pa.j1_0 + tid);  // L2 == 1
  __syncthreads();
  const int k2 = tid & 31, h2 = L2 / 2;
  for (int b = tid >> 5; b < pa.nb; b += (int)blockDim.x / 32) {
    const int j1 = pa.j1_0 + b;
    const RowTw tw = row_tw(p, j1);
    C *row = Tp + j1 * p.P;
    if (k2 < L2) {
      const C v = sbuf[b * pitch + k2];
      const int e = k2 + (k2 > h2 ? p.pad : 0);
      row[e] = cmul(v, tw_at(tw, e));
      if (k2 == h2 && L2 % 2 == 0) row[h2 + p.pad] = cmul(v, tw_at(tw, h2 + p.pad));
    }
  }
}

// ---- pass B ------------------------------------------------------------
// The first stage reads its inputs straight from T (natural order: position
// g R0 + r of the digit-reversed layout holds index iperm[g R0] + (L1 / R0) r),
// and the last stage writes its outputs straight to the DCT rows with the
// epilogue.
// BM_DCT: the H2 columns k2 <= L2 / 2 of the even transform.  Input j1 is
// entry k2 of row j1 of T for j1 <= L1 / 2, and the entry of L2 - k2 in row
// L1 - j1 beyond it; output kk = k2 + L2 k1 is the DCT's value kk, or L - kk
// when kk > m (the column L2 - k2, which is not computed).
// BM_BLUE: every column of V; output kk <= m is c_kk conj(F_kk).
enum { BM_DCT = 0, BM_BLUE = 1 };

// column k2 <= L2 / 2 of a pair's T
struct TCol {
  const C *fwd, *rev;  // element j1 at fwd[j1 P] (2 j1 <= L1) or rev[-j1 P]
  int L1, P;
  __device__ __forceinline__ TCol(const C *Tp, const Fft4Dev &p, int k2)
      : fwd(Tp + k2), rev(Tp + p.L1 * p.P + (k2 ? p.L2 - k2 + p.pad : 0)), L1(p.L1), P(p.P) {}
  __device__ __forceinline__ C at(int j1) const {
    const int o = j1 * P;
    return *(2 * j1 > L1 ? rev - o : fwd + o);
  }
};

struct PassB {
  const C *chirp;
  int L2, L, k2, m, epi;
  bool has2, self;  // self: the column is its own mirror
  RT *o1, *o2;
  const RT *w1, *w2;
};

template <int R, int BM, int FB>
__device__ __forceinline__ void bload(C *v, const TCol &col, int j, int step) {
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = BM == BM_DCT ? col.at(j + step * r) : col.fwd[(j + step * r) * col.P];
}

// outputs k1 = q + r Ns of the column to the rows
template <int R, int BM, int EPI>
__device__ __forceinline__ void bput(C *v, int q, int Ns, const PassB &pb) {
#pragma unroll
  for (int r = 0; r < R; r++) {
    // Bluestein keeps the outputs kk <= m < M / 3: none has r >= R / 3, and the
    // butterfly that forms them drops out
    if (BM == BM_BLUE && 3 * r >= R) continue;
    int kk = pb.k2 + pb.L2 * (q + r * Ns);
    if (BM == BM_DCT) {
      if (pb.self && kk > pb.m) continue;  // a self-mirrored column holds both values of a pair
      kk = min(kk, pb.L - kk);
    } else {
      if (kk > pb.m) continue;
      v[r] = cmul(mkc(v[r].x, -v[r].y), __ldg(pb.chirp + (kk == pb.m ? kk + 1 : kk)));
    }
    RT a = v[r].x, c = v[r].y;
    if (EPI == FFT4_FILTER) {
      a *= __ldg(pb.w1 + kk);
      if (pb.has2) c *= __ldg(pb.w2 + kk);
    } else if (EPI == FFT4_HALVE && (kk == 0 || kk == pb.m)) {
      a *= (RT)0.5;
      c *= (RT)0.5;
    }
    pb.o1[kk] = a;
    if (pb.has2) pb.o2[kk] = c;
  }
}

template <int R, int BM>
__device__ __forceinline__ void bput_epi(C *v, int q, int Ns, const PassB &pb) {
  if (pb.epi == FFT4_FILTER) bput<R, BM, FFT4_FILTER>(v, q, Ns, pb);
  else if (pb.epi == FFT4_HALVE) bput<R, BM, FFT4_HALVE>(v, q, Ns, pb);
  else bput<R, BM, FFT4_PLAIN>(v, q, Ns, pb);
}

template <int R, int BM, int FB, bool LAST>
__device__ __forceinline__ void bstage_first(C *slot, int Ls, const TCol &col, const int *iperm, const PassB &pb) {
  const int nq = Ls / R;
  for (int q = threadIdx.x / FB; q < nq; q += (int)blockDim.x / FB) {
    C v[R];
    bload<R, BM, FB>(v, col, __ldg(iperm + q * R), nq);
    Dft<R>::run(v);
    if (LAST) {
      bput_epi<R, BM>(v, q, 1, pb);
    } else {
      C *a = slot + q * R;
#pragma unroll
      for (int r = 0; r < R; r++) a[r] = v[r];
    }
  }
}

template <int R, int BM, int FB>
__device__ __forceinline__ void bstage_last(const C *slot, int Ns, const C *stw, const PassB &pb) {
  for (int q = threadIdx.x / FB; q < Ns; q += (int)blockDim.x / FB) {
    const C *a = slot + q;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = a[r * Ns];
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(stw + (r - 1) * Ns + q));
    Dft<R>::run(v);
    bput_epi<R, BM>(v, q, Ns, pb);
  }
}

// pass B: T[pair] (BM_DCT) or V[pair] (BM_BLUE) -> DCT rows 2 pair, 2 pair + 1
// of out (k <= m) with the epilogue
template <int BM, int FB>
__global__ void __launch_bounds__(Cfg<FB>::NT, Cfg<FB>::MINB) k_fft4_b(const C *__restrict__ T, int64_t nrow,
                                                    RT *__restrict__ out, int64_t ldo, const RT *__restrict__ w,
                                                    int64_t ldw, int epi, const Fft4Dev p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *const sbuf = reinterpret_cast<C *>(smem_raw);
  const int L1 = p.L1, b = threadIdx.x % FB;
  const int64_t pair = blockIdx.y, r0 = 2 * pair;
  C *const slot = sbuf + b * pitch_odd(L1);
  PassB pb;
  pb.has2 = r0 + 1 < nrow;
  pb.k2 = blockIdx.x * FB + b;
  pb.self = pb.k2 == 0 || 2 * pb.k2 == p.L2;
  const bool on = pb.k2 < (BM == BM_DCT ? p.H2 : p.L2);
  const int k2 = on ? pb.k2 : 0;
  TCol col(T + pair * (BM == BM_DCT ? p.tsz : p.vsz), p, k2);
  if (BM == BM_BLUE) col.P = p.PV;
  pb.chirp = tab(p.chirp);
  pb.L2 = p.L2;
  pb.L = (int)p.L;
  pb.m = (int)p.m;
  pb.epi = epi;
  pb.o1 = out + r0 * ldo;
  pb.o2 = pb.o1 + ldo;
  pb.w1 = pb.w2 = nullptr;
  if (epi == FFT4_FILTER) {
    pb.w1 = w + r0 * ldw;
    pb.w2 = pb.has2 ? pb.w1 + ldw : pb.w1;
  }
  const int S = p.nr1;
  if (S == 1) {
    if (on) MK_RADIX_SWITCH(p.r1[0], (bstage_first<RR, BM, FB, true>(slot, L1, col, p.iperm1, pb)));
    return;
  }
  if (on) MK_RADIX_SWITCH(p.r1[0], (bstage_first<RR, BM, FB, false>(slot, L1, col, p.iperm1, pb)));
  __syncthreads();
  for (int s = 1; s < S - 1; s++) {
    if (on)
      MK_RADIX_SWITCH(p.r1[s], (stage_dit<RR, FB>(slot, L1, p.ns1[s], p.inv1[s], tab(p.stw1) + p.to1[s])));
    __syncthreads();
  }
  if (on) MK_RADIX_SWITCH(p.r1[S - 1], (bstage_last<RR, BM, FB>(slot, p.ns1[S - 1], tab(p.stw1) + p.to1[S - 1], pb)));
}

// ---- Bluestein's middle pass ----------------------------------------------
// Between pass A (a -> T) and the last pass, Bluestein needs
// U = conj(DFT_M(a) B^) and then DFT_M(U).  With M = L1 L2, U is indexed
// i = i2 + L2 i1 (i2 = k2 of the first transform, i1 = k1), and
//   DFT(U)[o1 + L1 o2] = sum_i2 W_L2^{i2 o2} W_M^{i2 o1} sum_i1 W_L1^{i1 o1} U[i2 + L2 i1],
// so for each column k2 the last step of the first transform (length L1
// over j1 -> k1), the product with B^ and the first step of the second
// transform (length L1 over i1 -> o1) run in one CTA without leaving shared
// memory.  The first transform runs by decimation in frequency (natural
// input read from T, digit-reversed output, twiddles after each butterfly),
// which leaves exactly the digit-reversed input order the second transform's
// decimation-in-time stages take, so no permutation is needed: its stage 0
// and the second transform's stage 0 share one butterfly pass with the
// product in between.  The last stage stores V[k2][o1] = W_M^{k2 o1} (.)
// row by row (o1 contiguous), and pass B over the transposed shape (length
// L2 over i2 -> o2, rows o1) finishes with the chirp and the epilogue.
//
// a is even, so DFT(a) is even: F[(L2 - k2) + L2 (L1 - 1 - k1)] = F[k2 + L2 k1],
// and one first-transform column serves both columns k2 and L2 - k2 of the
// second transform (B^ is not even, so that one needs them all).  A CTA takes
// FB / 2 column pairs: the first transform runs on slots 0 .. FB / 2 - 1, the
// shared butterfly pass writes column k2 back into its slot and column
// L2 - k2 into slot FB / 2 + b, and the second transform runs on all slots.
struct PassC {
  C *Vp;  // this pair's V (L2 x PV)
  const C *bhat;
  int L1, L2, PV, k2_0, nh;  // nh: column pairs of this CTA
};

// the column in slot b (pairs' first columns, then their partners), or -1
template <int FB>
__device__ __forceinline__ int c_col(const PassC &pc, int b) {
  constexpr int H = FB / 2;
  if (b < H) return b < pc.nh ? pc.k2_0 + b : -1;
  const int k2 = pc.k2_0 + b - H;
  return b - H < pc.nh && k2 != 0 && 2 * k2 != pc.L2 ? pc.L2 - k2 : -1;
}

// the first decimation-in-frequency stage (span Ns = L1 / R): natural-order
// inputs q + r Ns from T's column, butterfly, twiddle after it
template <int R, int FB>
__device__ __forceinline__ void cstage_first(C *slot, int Ns, const C *stw, const TCol &col) {
  constexpr int H = FB / 2;
  for (int q = threadIdx.x / H; q < Ns; q += (int)blockDim.x / H) {
    C v[R];
    bload<R, BM_DCT, FB>(v, col, q, Ns);
    Dft<R>::run(v);
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(stw + (r - 1) * Ns + q));
    C *a = slot + q;
#pragma unroll
    for (int r = 0; r < R; r++) a[r * Ns] = v[r];
  }
}

// a decimation-in-frequency stage in shared memory (twiddles after the
// butterfly), same butterfly indexing as the decimation-in-time stages
template <int R, int FB>
__device__ __forceinline__ void cstage_dif(C *slot, int Ls, int Ns, float invNs, const C *stw) {
  constexpr int H = FB / 2;
  const int nq = Ls / R;
  for (int q = threadIdx.x / H; q < nq; q += (int)blockDim.x / H) {
    const int g = __float2int_rz(((float)q + 0.5f) * invNs);
    const int k = q - g * Ns;
    C *a = slot + g * Ns * R + k;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = a[r * Ns];
    Dft<R>::run(v);
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(stw + (r - 1) * Ns + k));
#pragma unroll
    for (int r = 0; r < R; r++) a[r * Ns] = v[r];
  }
}

// stage 0 of both transforms: the last DIF butterflies give F at k1 =
// iperm[q R] + (L1 / R) r; U = conj(F B^) there, for the column and, with k1
// mirrored to L1 - 1 - k1 (another butterfly, its legs reversed), for its
// partner (kp, slot_p; kp < 0: the column is its own mirror); then the first
// DIT butterflies of the second transform on each.  F goes through shared
// memory in between, so that one set of R values is live at a time.  LOAD
// (one-stage passes): the inputs come straight from T.
template <int R, int FB, bool LOAD>
__device__ __forceinline__ void cstage_mid(C *slot, C *slot_p, int k2, int kp, int L1, const int *iperm,
                                           const int *perm, const TCol &col, const PassC &pc) {
  constexpr int H = FB / 2;
  const int nq = L1 / R, step = pc.L2 * nq;
  for (int q = threadIdx.x / H; q < nq; q += (int)blockDim.x / H) {
    const int kq = __ldg(iperm + q * R);
    C *a = slot + q * R;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = LOAD ? col.at(r) : a[r];
    Dft<R>::run(v);
    if (kp >= 0) {
#pragma unroll
      for (int r = 0; r < R; r++) a[r] = v[r];
      const C *bh = pc.bhat + kp + pc.L2 * (L1 - 1 - kq);
      C u[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        const C f = cmul(v[r], __ldg(bh - step * r));
        u[R - 1 - r] = mkc(f.x, -f.y);
      }
      Dft<R>::run(u);
      C *ap = slot_p + __ldg(perm + (nq - 1 - kq));
#pragma unroll
      for (int r = 0; r < R; r++) ap[r] = u[r];
      asm volatile("" ::: "memory");
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = a[r];
    }
    const C *bh = pc.bhat + k2 + pc.L2 * kq;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const C f = cmul(v[r], __ldg(bh + step * r));
      v[r] = mkc(f.x, -f.y);
    }
    Dft<R>::run(v);
#pragma unroll
    for (int r = 0; r < R; r++) a[r] = v[r];
  }
}

// element o1 of column k2, twiddled by W_M^{k2 o1}, into row k2 of V
__device__ __forceinline__ void put_v(const PassC &pc, const Fft4Dev &p, int k2, int o1, C v) {
  const C *tl = tab(p.tlane2) + 32 * k2, *tb = tab(p.tblk2) + k2 * p.nb32b;
  pc.Vp[k2 * pc.PV + o1] = cmul(v, cmul(__ldg(tb + (o1 >> 5)), __ldg(tl + (o1 & 31))));
}

// the last DIT stage (Ns R = L1): rows warp by warp, outputs o1 = q + r Ns
// twiddled and stored to V
template <int R, int FB>
__device__ __forceinline__ void cstage_last(const C *sbuf, int pitch, int Ns, const C *stw, const PassC &pc,
                                            const Fft4Dev &p) {
  for (int bf = threadIdx.x; bf < FB * Ns; bf += (int)blockDim.x) {
    const int b = bf / Ns, q = bf - b * Ns;
    const int k2 = c_col<FB>(pc, b);
    if (k2 < 0) continue;
    const C *a = sbuf + b * pitch + q;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = a[r * Ns];
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(stw + (r - 1) * Ns + q));
    Dft<R>::run(v);
#pragma unroll
    for (int r = 0; r < R; r++) put_v(pc, p, k2, q + r * Ns, v[r]);
  }
}

// T[pair] (from pass A on the chirped rows) -> V[pair] (L2 x PV)
template <int FB>
__global__ void __launch_bounds__(Cfg<FB>::NT, Cfg<FB>::MINB) k_fft4_conv(const C *__restrict__ T, C *__restrict__ V,
                                                     const Fft4Dev p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *const sbuf = reinterpret_cast<C *>(smem_raw);
  constexpr int H = FB / 2;
  const int L1 = p.L1, pitch = pitch_odd(L1), S = p.nr1, b = threadIdx.x % H;
  const int64_t pair = blockIdx.y;
  PassC pc;
  pc.Vp = V + pair * p.vsz;
  pc.bhat = tab(p.bhat);
  pc.L1 = L1;
  pc.L2 = p.L2;
  pc.PV = p.PV;
  pc.k2_0 = blockIdx.x * H;
  pc.nh = min(H, p.H2 - pc.k2_0);
  const bool on = b < pc.nh;
  const int k2 = on ? pc.k2_0 + b : 0, kp = c_col<FB>(pc, H + b);
  const TCol col(T + pair * p.tsz, p, k2);
  C *const slot = sbuf + b * pitch, *const slot_p = slot + H * pitch;
  if (S == 1) {  // L1 <= 16: the shared butterfly pass alone, then the rows
    if (on)
      MK_RADIX_SWITCH(p.r1[0], (cstage_mid<RR, FB, true>(slot, slot_p, k2, kp, L1, p.iperm1, p.perm1, col, pc)));
    __syncthreads();
    for (int e = threadIdx.x; e < FB * L1; e += (int)blockDim.x) {
      const int be = e / L1, o1 = e - be * L1, ke = c_col<FB>(pc, be);
      if (ke >= 0) put_v(pc, p, ke, o1, sbuf[be * pitch + o1]);
    }
    return;
  }
  if (on)
    MK_RADIX_SWITCH(p.r1[S - 1], (cstage_first<RR, FB>(slot, p.ns1[S - 1], tab(p.stw1) + p.to1[S - 1], col)));
  __syncthreads();
  for (int s = S - 2; s >= 1; s--) {
    if (on)
      MK_RADIX_SWITCH(p.r1[s], (cstage_dif<RR, FB>(slot, L1, p.ns1[s], p.inv1[s], tab(p.stw1) + p.to1[s])));
    __syncthreads();
  }
  if (on)
    MK_RADIX_SWITCH(p.r1[0], (cstage_mid<RR, FB, false>(slot, slot_p, k2, kp, L1, p.iperm1, p.perm1, col, pc)));
  __syncthreads();
  const bool on2 = c_col<FB>(pc, threadIdx.x % FB) >= 0;
  for (int s = 1; s < S - 1; s++) {
    if (on2)
      MK_RADIX_SWITCH(p.r1[s], (stage_dit<RR, FB>(sbuf + (threadIdx.x % FB) * pitch, L1, p.ns1[s], p.inv1[s],
                                                  tab(p.stw1) + p.to1[s])));
    __syncthreads();
  }
  MK_RADIX_SWITCH(p.r1[S - 1], (cstage_last<RR, FB>(sbuf, pitch, p.ns1[S - 1], tab(p.stw1) + p.to1[S - 1], pc, p)));
}
#undef MK_RADIX_SWITCH
#undef MK_RCASE12
#undef MK_RCASE14
#undef MK_RCASE15
#undef MK_RCASE16

bool g_attr[64] = {false};

// out rows = DCT-I of x rows with the epilogue (see mk_fft4.cuh)
int dct_launch(const Fft4Plan &p, const RT *x, int64_t ldx, int64_t nrow, C *T, RT *out, int64_t ldo, int epi,
               const RT *w, int64_t ldw, cudaStream_t st) {
  const Fft4Dev &d = p.d;
  const int64_t npairs = (nrow + 1) / 2;
  MK_CHECK_ARG(npairs >= 1 && npairs <= 65535, "fft4: %lld rows out of range", (long long)nrow);
  MK_CHECK_ARG(ldx >= d.n && ldo >= d.n, "fft4: leading dimensions below the row length");
  MK_CHECK_ARG(epi != FFT4_FILTER || (w && ldw >= d.n), "fft4: filter weights missing");
  MK_CHECK_ARG(d.f64 == (sizeof(RT) == 8), "fft4: plan precision does not match the call");
  int dev = 0;
  MK_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !g_attr[dev]) {
    const int mhi = FB_HI * (FFT4_LMAX + 1) * (int)sizeof(C);
    const int mlo = FB_LO * (FFT4_LMAX + 1) * (int)sizeof(C);
#define MK_FFT4_ATTR(k, v) MK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, v))
    MK_FFT4_ATTR((k_fft4_a<AM_BLUE, FB_LO>), mlo);
    MK_FFT4_ATTR((k_fft4_b<BM_BLUE, FB_LO>), mlo);
    MK_FFT4_ATTR((k_fft4_a<AM_BLUE, FB_HI>), mhi);
    MK_FFT4_ATTR((k_fft4_b<BM_BLUE, FB_HI>), mhi);
    MK_FFT4_ATTR((k_fft4_conv<FB_LO>), mlo);
    MK_FFT4_ATTR((k_fft4_conv<FB_HI>), mhi);
#if MK_FFT4_SMOOTH
    MK_FFT4_ATTR((k_fft4_a<AM_DCT, FB_LO>), mlo);
    MK_FFT4_ATTR((k_fft4_b<BM_DCT, FB_LO>), mlo);
    MK_FFT4_ATTR((k_fft4_a<AM_DCT, FB_HI>), mhi);
    MK_FFT4_ATTR((k_fft4_b<BM_DCT, FB_HI>), mhi);
#endif
#undef MK_FFT4_ATTR
    g_attr[dev] = true;
  }
  const bool hia = d.fba == FB_HI, hib = d.fbb == FB_HI;
  const int fa = hia ? FB_HI : FB_LO, fb = hib ? FB_HI : FB_LO;
  const unsigned np = (unsigned)npairs;
  const size_t smem_a = (size_t)fa * pitch_odd(d.L2) * sizeof(C);  // transforms of length L2
  const size_t smem_b = (size_t)fb * pitch_odd(d.L1) * sizeof(C);  // transforms of length L1
  const dim3 ga((d.H1 + fa - 1) / fa, np);
  int rc;
#if MK_FFT4_SMOOTH
  if (!d.blue) {
    const dim3 gb((d.H2 + fb - 1) / fb, np);
    if (hia) k_fft4_a<AM_DCT, FB_HI><<<ga, threads_for<FB_HI>((int64_t)ga.x * np, smem_a), smem_a, st>>>(x, ldx, nrow, T, d);
    else k_fft4_a<AM_DCT, FB_LO><<<ga, threads_for<FB_LO>((int64_t)ga.x * np, smem_a), smem_a, st>>>(x, ldx, nrow, T, d);
    if ((rc = launch_status("fft4 pass A"))) return rc;
    if (hib) k_fft4_b<BM_DCT, FB_HI><<<gb, threads_for<FB_HI>((int64_t)gb.x * np, smem_b), smem_b, st>>>(T, nrow, out, ldo, w, ldw, epi, d);
    else k_fft4_b<BM_DCT, FB_LO><<<gb, threads_for<FB_LO>((int64_t)gb.x * np, smem_b), smem_b, st>>>(T, nrow, out, ldo, w, ldw, epi, d);
    return launch_status("fft4 pass B");
  }
#else
  MK_CHECK_ARG(d.blue, "fft4: plan does not match the call");
#endif
  C *V = T + npairs * d.tsz;
  if (hia) k_fft4_a<AM_BLUE, FB_HI><<<ga, threads_for<FB_HI>((int64_t)ga.x * np, smem_a), smem_a, st>>>(x, ldx, nrow, T, d);
  else k_fft4_a<AM_BLUE, FB_LO><<<ga, threads_for<FB_LO>((int64_t)ga.x * np, smem_a), smem_a, st>>>(x, ldx, nrow, T, d);
  if ((rc = launch_status("fft4 Bluestein pass A"))) return rc;
  const dim3 gc((d.H2 + fb / 2 - 1) / (fb / 2), np);
  if (hib) k_fft4_conv<FB_HI><<<gc, threads_for<FB_HI>((int64_t)gc.x * np, smem_b), smem_b, st>>>(T, V, d);
  else k_fft4_conv<FB_LO><<<gc, threads_for<FB_LO>((int64_t)gc.x * np, smem_b), smem_b, st>>>(T, V, d);
  if ((rc = launch_status("fft4 Bluestein middle pass"))) return rc;
  // pass B on the transposed shape: length L2 over the rows of V, outputs
  // o1 + L1 o2
  Fft4Dev tr = d;
  std::swap(tr.L1, tr.L2);
  std::swap(tr.nr1, tr.nr2);
  std::swap(tr.r1, tr.r2);
  std::swap(tr.ns1, tr.ns2);
  std::swap(tr.to1, tr.to2);
  std::swap(tr.inv1, tr.inv2);
  std::swap(tr.stw1, tr.stw2);
  std::swap(tr.iperm1, tr.iperm2);
  const dim3 gt((tr.L2 + fa - 1) / fa, np);
  if (hia) k_fft4_b<BM_BLUE, FB_HI><<<gt, threads_for<FB_HI>((int64_t)gt.x * np, smem_a), smem_a, st>>>(V, nrow, out, ldo, w, ldw, epi, tr);
  else k_fft4_b<BM_BLUE, FB_LO><<<gt, threads_for<FB_LO>((int64_t)gt.x * np, smem_a), smem_a, st>>>(V, nrow, out, ldo, w, ldw, epi, tr);
  return launch_status("fft4 Bluestein last pass");
}

}  // namespace MK_FFT4_NS
}  // namespace mk
