// Polarized projections (PolMap).  Stokes maps are pixel-major:
// map[p * npol + k], p = x * ny + y, as the reference's (nx, ny, npol) array.
// With c = cos(twogamma[i]), s = sin(twogamma[i]) and d = dat[i]:
//
//   map2tod  IQU        dat (+)= I + Q c + U s                minkasi/lib/minkasi.c:146-159
//            QU         dat (+)= Q c + U s                    minkasi.c:162-174
//   tod2map  IQU        (I, Q, U)      += (d, d c, d s)       minkasi.c:176-185
//            QU         (Q, U)         += (d c, d s)          minkasi.c:187-194
//            QU_PRECON  (QQ, UU, QU)   += (d c c, d s s, d s c)              minkasi.c:196-207
//            IQU_PRECON (I, Q, U, QQ, QU, UU) += (d, d c, d s, d c c, d s c, d s s)
//                                                              minkasi.c:231-245
//
// The reference evaluates cos/sin of every sample on every call.  Here the
// angle terms are either computed in the kernel from twogamma (the drop-in
// form, FP64) or read from a cos/sin pair computed once per TOD by
// mk_pol_sincos (the pointing is fixed across PCG iterations, so this trades
// 8 more bytes per sample for no FP64 transcendental work on GB300's narrow
// FP64 pipe).  tod2map sums runs of equal pixels over windows of 256 samples
// per warp and issues one atomic per Stokes component per run.
#include <math.h>

#include "mk_common.cuh"
#include "mk_wide.cuh"

namespace {

template <int MODE>
struct Pol;
// npol per mode; the integer values are the MK_POL_* codes
template <> struct Pol<MK_POL_QU> { static constexpr int N = 2; };
template <> struct Pol<MK_POL_IQU> { static constexpr int N = 3; };
template <> struct Pol<MK_POL_QU_PRECON> { static constexpr int N = 3; };
template <> struct Pol<MK_POL_IQU_PRECON> { static constexpr int N = 6; };

// acc (or 0 if `fresh`; FIRST: nothing yet) plus the sample's Stokes weights: one FP64 operation
// per term where the last product joins the sum as an FMA (the FP64 pipe bounds
// the kernel)
template <int MODE, typename T, bool FIRST>
__device__ __forceinline__ void pol_add(T (&acc)[Pol<MODE>::N], bool fresh, T d, T c, T s) {
  T b[Pol<MODE>::N];
#pragma unroll
  for (int k = 0; k < Pol<MODE>::N; k++) b[k] = fresh ? T(0) : acc[k];
  if constexpr (MODE == MK_POL_QU) {
    acc[0] = fma(d, c, b[0]);
    acc[1] = fma(d, s, b[1]);
  } else if constexpr (MODE == MK_POL_IQU) {
    acc[0] = FIRST ? d : b[0] + d;
    acc[1] = fma(d, c, b[1]);
    acc[2] = fma(d, s, b[2]);
  } else {
    const T dc = d * c, ds = d * s;
    if constexpr (MODE == MK_POL_QU_PRECON) {
      acc[0] = fma(dc, c, b[0]);
      acc[1] = fma(ds, s, b[1]);
      acc[2] = fma(ds, c, b[2]);
    } else {
      acc[0] = FIRST ? d : b[0] + d;
      acc[1] = FIRST ? dc : b[1] + dc;
      acc[2] = FIRST ? ds : b[2] + ds;
      acc[3] = fma(dc, c, b[3]);
      acc[4] = fma(ds, c, b[4]);
      acc[5] = fma(ds, s, b[5]);
    }
  }
}

// angle terms of sample i: from the cached pair, or sincos of twogamma
template <typename T, bool TRIG>
__device__ __forceinline__ void angle(const T *__restrict__ cs, const T *__restrict__ sn,
                                      const double *__restrict__ tg, int64_t i, T &c, T &s) {
  if constexpr (TRIG) {
    double sd, cd;
    sincos(__ldcs(tg + i), &sd, &cd);
    c = (T)cd;
    s = (T)sd;
  } else {
    c = __ldcs(cs + i);
    s = __ldcs(sn + i);
  }
}

template <int MODE, typename T, bool TRIG, bool ADD>
__global__ void __launch_bounds__(256) k_polmap2tod(T *__restrict__ dat, const T *__restrict__ map,
                                                    const T *__restrict__ cs, const T *__restrict__ sn,
                                                    const double *__restrict__ tg,
                                                    const int32_t *__restrict__ ipix, int64_t n, int64_t npix) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t p = __ldcs(ipix + i);
    T c, s;
    angle<T, TRIG>(cs, sn, tg, i, c, s);
    T v = T(0);
    if ((uint32_t)p < (uint64_t)npix) {
      if constexpr (MODE == MK_POL_IQU) {
        const T *m = map + 3 * (int64_t)p;
        v = __ldg(m) + __ldg(m + 1) * c + __ldg(m + 2) * s;
      } else {
        const T *m = map + 2 * (int64_t)p;
        v = __ldg(m) * c + __ldg(m + 1) * s;
      }
    }
    if (ADD) v = dat[i] + v;
    __stcs(dat + i, v);
  }
}

// Scatter: a warp takes windows of 256 consecutive samples, 8 per lane (32-byte
// loads if VEC: every array 32-byte aligned).  Runs of equal pixels are summed
// in registers, joined across lanes, written to shared memory in sample order
// and added to the map component by component: 32 consecutive (run, component)
// pairs per instruction, which are neighbouring words of the map, as in
// tod2map's warp_runs.  IQU on 64 x 65,341 samples, 256^2 pixels: FP64 43 us (45
// with 16-byte loads) for 51 with an atomic per component and 4-sample run in
// each thread, FP32 13 for 46; on 256 x 130,978, 1024^2: 225 (235) for 405 and
// 104 for 304.
// ROWS: d = rowval[i / ndata] (1 if rowval is NULL): hit / weight maps
constexpr unsigned FULL = 0xffffffffu;
template <int MODE>
constexpr int PW = Pol<MODE>::N > 3 ? 2 : 4;  // warps per CTA (their runs fit in shared memory)

template <int MODE, typename T, bool TRIG, bool ROWS, bool VEC>
__global__ void __launch_bounds__(PW<MODE> * 32) k_tod2polmap(T *__restrict__ map, const T *__restrict__ dat,
                                                        const T *__restrict__ cs, const T *__restrict__ sn,
                                                        const double *__restrict__ tg,
                                                        const int32_t *__restrict__ ipix, int64_t n, int64_t npix,
                                                        const T *__restrict__ rowval, int64_t ndata) {
  constexpr int NP = Pol<MODE>::N;
  __shared__ T rsum[PW<MODE>][256 * NP];
  __shared__ int32_t rkey[PW<MODE>][256];
  const int lane = threadIdx.x & 31;
  T *const sum = rsum[threadIdx.x >> 5];
  int32_t *const key = rkey[threadIdx.x >> 5];
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = warp * 256; base < n; base += nwarp * 256) {
    const int64_t i0 = base + 8 * lane, left = n - i0;
    const int m = left <= 0 ? 0 : (left >= 8 ? 8 : (int)left);  // valid samples, a prefix of the window
    int32_t p[8];
    T d[8], c[8], s[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      p[j] = INT32_MIN;
      d[j] = c[j] = s[j] = T(0);
    }
    if (VEC && m == 8) {
      mk::ld32(ipix + i0, p);
      if constexpr (!ROWS) mk::ld8_wide(dat + i0, d);
      if constexpr (!TRIG) {
        mk::ld8_wide(cs + i0, c);
        mk::ld8_wide(sn + i0, s);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (j >= m) continue;
        p[j] = __ldcs(ipix + i0 + j);
        if constexpr (!ROWS) d[j] = __ldcs(dat + i0 + j);
        if constexpr (!TRIG) angle<T, TRIG>(cs, sn, tg, i0 + j, c[j], s[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (j >= m) continue;
      if constexpr (ROWS) d[j] = rowval ? rowval[(i0 + j) / ndata] : T(1);
      if constexpr (TRIG) angle<T, TRIG>(cs, sn, tg, i0 + j, c[j], s[j]);
    }
    // which samples end a run, and the places of the lane's closed runs
    int32_t kf = INT32_MIN, kl = INT32_MIN;
    unsigned ends = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (j < m) {
        if (j == 0) kf = p[0];
        else if (p[j] != p[j - 1]) ends |= 1u << (j - 1);
        kl = p[j];
      }
    }
    const bool single = ends == 0;
    const int32_t kl_prev = __shfl_up_sync(FULL, kl, 1), kf_next = __shfl_down_sync(FULL, kf, 1);
    const bool cont_in = lane > 0 && m > 0 && kl_prev == kf;
    const bool cont_out = lane < 31 && kf_next == kl && m > 0;
    if (m > 0 && !cont_out) ends |= 1u << (m - 1);
    const int cnt = __popc(ends);
    int at = cnt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int up = __shfl_up_sync(FULL, at, off);
      if (lane >= off) at += up;
    }
    const int total = __shfl_sync(FULL, at, 31), first = at - cnt;
    at = first;
    T acc[NP];
#pragma unroll
    for (int k = 0; k < NP; k++) acc[k] = T(0);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (j >= m) continue;
      if (j == 0) pol_add<MODE, T, true>(acc, true, d[0], c[0], s[0]);
      else pol_add<MODE, T, false>(acc, ends >> (j - 1) & 1, d[j], c[j], s[j]);
      if (ends >> j & 1) {
        key[at] = p[j];
#pragma unroll
        for (int k = 0; k < NP; k++) sum[at * NP + k] = acc[k];
        at++;
      }
    }
    // what a lane hands on (see warp_runs in mk_proj.cu)
    bool pend = single && cont_in;
    for (int off = 1; __any_sync(FULL, pend); off <<= 1) {
      const bool pup = __shfl_up_sync(FULL, (int)pend, off) != 0;
#pragma unroll
      for (int k = 0; k < NP; k++) {
        const T up = __shfl_up_sync(FULL, acc[k], off);
        if (pend) acc[k] += up;
      }
      if (pend) pend = pup;
    }
#pragma unroll
    for (int k = 0; k < NP; k++) {
      const T prev = __shfl_up_sync(FULL, acc[k], 1);
      if (cont_in && cnt > 0) sum[first * NP + k] += prev;
    }
    __syncwarp();
    for (int e = lane; e < total * NP; e += 32) {
      const int r = e / NP;
      const int32_t q = key[r];
      if ((uint32_t)q < (uint64_t)npix) atomicAdd(map + (int64_t)q * NP + (e - r * NP), sum[e]);
    }
    __syncwarp();
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_pol_sincos(T *__restrict__ cs, T *__restrict__ sn,
                                                    const double *__restrict__ tg, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    double s, c;
    sincos(tg[i], &s, &c);
    cs[i] = (T)c;
    sn[i] = (T)s;
  }
}

// out = P . m per pixel for a PRECON map P and a map m (PolMap.__mul__,
// minkasi/maps/polmap.py:624-684):
//   QU_PRECON (QQ, UU, QU) . (Q, U)
//   IQU_PRECON (I, Q, U, QQ, QU, UU) as the symmetric [a0 a1 a2; a1 a3 a4; a2 a4 a5] . (I, Q, U)
template <typename T>
__global__ void __launch_bounds__(256) k_pol_precon_mul(T *__restrict__ out, const T *__restrict__ P,
                                                        const T *__restrict__ m, int64_t npix, int iqu) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += stride) {
    if (iqu) {
      const T *a = P + 6 * p;
      const T *x = m + 3 * p;
      const T x0 = x[0], x1 = x[1], x2 = x[2];
      out[3 * p] = a[0] * x0 + a[1] * x1 + a[2] * x2;
      out[3 * p + 1] = a[1] * x0 + a[3] * x1 + a[4] * x2;
      out[3 * p + 2] = a[2] * x0 + a[4] * x1 + a[5] * x2;
    } else {
      const T *a = P + 3 * p;
      const T *x = m + 2 * p;
      const T x0 = x[0], x1 = x[1];
      out[2 * p] = a[0] * x0 + a[2] * x1;
      out[2 * p + 1] = a[2] * x0 + a[1] * x1;
    }
  }
}

template <int MODE, typename T, bool TRIG>
int polmap2tod_t(void *dat, const void *map, const void *cs, const void *sn, const double *tg,
                 const int32_t *ipix, int64_t n, int64_t npix, int do_add, cudaStream_t st) {
  if (do_add) {
    auto k = k_polmap2tod<MODE, T, TRIG, true>;
    k<<<mk_grid_fit(k, n, 256), 256, 0, st>>>((T *)dat, (const T *)map, (const T *)cs, (const T *)sn, tg,
                                               ipix, n, npix);
  } else {
    auto k = k_polmap2tod<MODE, T, TRIG, false>;
    k<<<mk_grid_fit(k, n, 256), 256, 0, st>>>((T *)dat, (const T *)map, (const T *)cs, (const T *)sn, tg,
                                               ipix, n, npix);
  }
  return mk::launch_status("mk_polmap2tod");
}

template <int MODE, typename T, bool TRIG, bool ROWS>
int tod2polmap_t(void *map, const void *dat, const void *cs, const void *sn, const double *tg,
                 const int32_t *ipix, int64_t n, int64_t npix, const void *rowval, int64_t ndata,
                 cudaStream_t st) {
  const bool vec = mk::aligned32(ipix) && (ROWS || mk::aligned32(dat)) && (TRIG || (mk::aligned32(cs) && mk::aligned32(sn)));
  auto k = vec ? k_tod2polmap<MODE, T, TRIG, ROWS, true> : k_tod2polmap<MODE, T, TRIG, ROWS, false>;
  k<<<mk_grid((n + 7) / 8, PW<MODE> * 32, 64), PW<MODE> * 32, 0, st>>>((T *)map, (const T *)dat, (const T *)cs, (const T *)sn, tg,
                                                            ipix, n, npix, (const T *)rowval, ndata);
  return mk::launch_status("mk_tod2polmap");
}

template <typename T, bool TRIG, bool ROWS>
int tod2polmap_mode(int mode, void *map, const void *dat, const void *cs, const void *sn, const double *tg,
                    const int32_t *ipix, int64_t n, int64_t npix, const void *rowval, int64_t ndata,
                    cudaStream_t st) {
  switch (mode) {
    case MK_POL_QU:
      return tod2polmap_t<MK_POL_QU, T, TRIG, ROWS>(map, dat, cs, sn, tg, ipix, n, npix, rowval, ndata, st);
    case MK_POL_IQU:
      return tod2polmap_t<MK_POL_IQU, T, TRIG, ROWS>(map, dat, cs, sn, tg, ipix, n, npix, rowval, ndata, st);
    case MK_POL_QU_PRECON:
      return tod2polmap_t<MK_POL_QU_PRECON, T, TRIG, ROWS>(map, dat, cs, sn, tg, ipix, n, npix, rowval, ndata,
                                                           st);
    default:
      return tod2polmap_t<MK_POL_IQU_PRECON, T, TRIG, ROWS>(map, dat, cs, sn, tg, ipix, n, npix, rowval, ndata,
                                                            st);
  }
}

bool pol_mode_ok(int mode) {
  return mode == MK_POL_QU || mode == MK_POL_IQU || mode == MK_POL_QU_PRECON || mode == MK_POL_IQU_PRECON;
}

}  // namespace

extern "C" int mk_pol_npol(int mode) {
  switch (mode) {
    case MK_POL_QU: return 2;
    case MK_POL_IQU: return 3;
    case MK_POL_QU_PRECON: return 3;
    case MK_POL_IQU_PRECON: return 6;
    default: return 0;
  }
}

extern "C" int mk_pol_sincos(void *cs, void *sn, const double *twogamma, int64_t n, int dtype, void *stream) {
  MK_CHECK_ARG(n >= 0, "mk_pol_sincos: negative size");
  MK_CHECK_ARG(MK_DTYPE_OK(dtype), "mk_pol_sincos: bad dtype %d", dtype);
  if (n == 0) return MK_OK;
  MK_CHECK_ARG(cs && sn && twogamma, "mk_pol_sincos: null pointer");
  cudaStream_t st = mk::as_stream(stream);
  if (dtype == MK_F64)
    k_pol_sincos<double><<<mk_grid_fit(k_pol_sincos<double>, n, 256), 256, 0, st>>>((double *)cs, (double *)sn,
                                                                                   twogamma, n);
  else
    k_pol_sincos<float><<<mk_grid_fit(k_pol_sincos<float>, n, 256), 256, 0, st>>>((float *)cs, (float *)sn,
                                                                                 twogamma, n);
  return mk::launch_status("mk_pol_sincos");
}

extern "C" int mk_polmap2tod(void *dat, const void *map, const void *cos2g, const void *sin2g,
                             const double *twogamma, const int32_t *ipix, int64_t ndet, int64_t ndata,
                             int64_t npix, int mode, int dtype, int do_add, void *stream) {
  MK_CHECK_ARG(ndet >= 0 && ndata >= 0 && npix >= 0, "mk_polmap2tod: negative size");
  MK_CHECK_ARG(mode == MK_POL_QU || mode == MK_POL_IQU,
               "mk_polmap2tod: mode %d not implemented (QU and IQU only, as the reference)", mode);
  MK_CHECK_ARG(MK_DTYPE_OK(dtype), "mk_polmap2tod: bad dtype %d", dtype);
  const int64_t n = ndet * ndata;
  if (n == 0) return MK_OK;
  MK_CHECK_ARG(dat && map && ipix, "mk_polmap2tod: null pointer");
  const bool trig = (cos2g == nullptr);
  MK_CHECK_ARG(trig ? (twogamma != nullptr) : (sin2g != nullptr),
               "mk_polmap2tod: give cos2g and sin2g, or twogamma");
  MK_CHECK_ARG(!trig || dtype == MK_F64, "mk_polmap2tod: the twogamma form is FP64 only");
  cudaStream_t st = mk::as_stream(stream);
  if (trig)
    return mode == MK_POL_IQU
               ? polmap2tod_t<MK_POL_IQU, double, true>(dat, map, nullptr, nullptr, twogamma, ipix, n, npix, do_add, st)
               : polmap2tod_t<MK_POL_QU, double, true>(dat, map, nullptr, nullptr, twogamma, ipix, n, npix, do_add, st);
  if (dtype == MK_F64)
    return mode == MK_POL_IQU
               ? polmap2tod_t<MK_POL_IQU, double, false>(dat, map, cos2g, sin2g, nullptr, ipix, n, npix, do_add, st)
               : polmap2tod_t<MK_POL_QU, double, false>(dat, map, cos2g, sin2g, nullptr, ipix, n, npix, do_add, st);
  return mode == MK_POL_IQU
             ? polmap2tod_t<MK_POL_IQU, float, false>(dat, map, cos2g, sin2g, nullptr, ipix, n, npix, do_add, st)
             : polmap2tod_t<MK_POL_QU, float, false>(dat, map, cos2g, sin2g, nullptr, ipix, n, npix, do_add, st);
}

extern "C" int mk_tod2polmap(void *map, const void *dat, const void *cos2g, const void *sin2g,
                             const double *twogamma, const int32_t *ipix, int64_t ndet, int64_t ndata,
                             int64_t npix, int mode, int dtype, const void *rowval, void *stream) {
  MK_CHECK_ARG(ndet >= 0 && ndata >= 0 && npix >= 0, "mk_tod2polmap: negative size");
  MK_CHECK_ARG(pol_mode_ok(mode), "mk_tod2polmap: unknown mode %d", mode);
  MK_CHECK_ARG(MK_DTYPE_OK(dtype), "mk_tod2polmap: bad dtype %d", dtype);
  const int64_t n = ndet * ndata;
  if (n == 0) return MK_OK;
  MK_CHECK_ARG(map && ipix, "mk_tod2polmap: null pointer");
  const bool rows = (dat == nullptr);
  const bool trig = (cos2g == nullptr);
  MK_CHECK_ARG(trig ? (twogamma != nullptr) : (sin2g != nullptr),
               "mk_tod2polmap: give cos2g and sin2g, or twogamma");
  MK_CHECK_ARG(!trig || dtype == MK_F64, "mk_tod2polmap: the twogamma form is FP64 only");
  cudaStream_t st = mk::as_stream(stream);
  if (trig)
    return rows ? tod2polmap_mode<double, true, true>(mode, map, dat, nullptr, nullptr, twogamma, ipix, n, npix,
                                                      rowval, ndata, st)
                : tod2polmap_mode<double, true, false>(mode, map, dat, nullptr, nullptr, twogamma, ipix, n, npix,
                                                       rowval, ndata, st);
  if (dtype == MK_F64)
    return rows ? tod2polmap_mode<double, false, true>(mode, map, dat, cos2g, sin2g, nullptr, ipix, n, npix,
                                                       rowval, ndata, st)
                : tod2polmap_mode<double, false, false>(mode, map, dat, cos2g, sin2g, nullptr, ipix, n, npix,
                                                        rowval, ndata, st);
  return rows ? tod2polmap_mode<float, false, true>(mode, map, dat, cos2g, sin2g, nullptr, ipix, n, npix, rowval,
                                                    ndata, st)
              : tod2polmap_mode<float, false, false>(mode, map, dat, cos2g, sin2g, nullptr, ipix, n, npix, rowval,
                                                     ndata, st);
}

extern "C" int mk_pol_precon_mul(void *out, const void *precon, const void *map, int64_t npix, int mode,
                                 int dtype, void *stream) {
  MK_CHECK_ARG(npix >= 0, "mk_pol_precon_mul: negative size");
  MK_CHECK_ARG(mode == MK_POL_QU_PRECON || mode == MK_POL_IQU_PRECON,
               "mk_pol_precon_mul: mode must be QU_PRECON or IQU_PRECON");
  MK_CHECK_ARG(MK_DTYPE_OK(dtype), "mk_pol_precon_mul: bad dtype %d", dtype);
  if (npix == 0) return MK_OK;
  MK_CHECK_ARG(out && precon && map, "mk_pol_precon_mul: null pointer");
  cudaStream_t st = mk::as_stream(stream);
  const int iqu = mode == MK_POL_IQU_PRECON;
  if (dtype == MK_F64)
    k_pol_precon_mul<double><<<mk_grid_fit(k_pol_precon_mul<double>, npix, 256), 256, 0, st>>>(
        (double *)out, (const double *)precon, (const double *)map, npix, iqu);
  else
    k_pol_precon_mul<float><<<mk_grid_fit(k_pol_precon_mul<float>, npix, 256), 256, 0, st>>>(
        (float *)out, (const float *)precon, (const float *)map, npix, iqu);
  return mk::launch_status("mk_pol_precon_mul");
}
