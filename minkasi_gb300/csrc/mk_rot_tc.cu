// Detector rotation R = A . X on the 5th-generation tensor cores, FP32 in /
// FP32 out: the apply_noise rotations np.dot(v, dat), np.dot(vT, .) of
// minkasi/mapmaking/noise.py:704,709.
//
// Split: an FP32 value is the exact sum of three bf16 values, x = h + m + l (8
// significant bits each, every part rounded to nearest) for 2^-110 <= |x| <
// 2^128 (1 - 2^-9); below, the low part loses bits to bf16's smallest denormal
// (2^-133: an absolute error of at most 2^-134), above, h rounds to infinity and
// the sample becomes NaN.  Then
//   R ~= h h + h m + m h + m m + h l + l h   (tcgen05.mma kind::f16, FP32
// accumulation in tensor memory); the dropped products are below 2^-25
// relative.  (Two TF32 parts need 8 B per value where three bf16 parts need
// 6 B, at the same MMA time, and drop products of 2^-22.)
//
// Tile mapping (all operands K-major, 64-byte swizzle):
//   D^T (128 samples x ndet) = X^T (128 samples x K=ndet) . A^T (K x N=ndet)
//   MMA A-operand: the X^T tile.  A split thread owns one sample; it loads the
//     32 detector values of a K-chunk (coalesced across the warp: 32
//     consecutive samples of one detector row) one chunk ahead into registers,
//     splits them, and writes three rows of 64 B into shared memory.
//   MMA B-operand: rows j = output detector, K contiguous = A[j][k0..k0+31],
//     i.e. A row-major.  Its split is built by k_bprep in exactly the
//     shared-memory image and bulk-copied (cp.async.bulk) per K-chunk.
//   Accumulator: 128 TMEM lanes (= samples) x ndet columns (= detectors).
//
// MT tiles of 128 samples share one pass over the operand image: it is
// 6 ndet^2 bytes per pass against 512 ndet bytes of X per tile, so at 256
// detectors one tile per pass reads three times as much of A's image from L2
// as of X from memory, which is what bounded the kernel (with the 8 B TF32
// image: 0.156 ms on 256 x 130,978).  MT = 2 there (one CTA per SM: two
// accumulators of 256 columns fill tensor memory) once there are more tiles than
// SMs; MT = 1 for fewer, which an item of two would put on half as many SMs
// (256 x 1,000 .. 19,000: 30.9 us with MT = 2, 22.7 with 1), and MT = 1 below 256
// detectors, where two CTAs fit an SM and each has two accumulators.
//
// Roles: MT x 4 split warps; MT x 4 epilogue warps (warp w reads TMEM lanes
// 32 (w % 4) .. of its tile and stores per detector 32 consecutive samples);
// one warp of which one lane issues the image copies and the MMAs (the warp
// stays converged: with operands in uniform registers a chunk's MMAs issue
// faster than they run; 256 x 450,561 309 -> 292 us, 256 x 130,978 111 -> 105, no
// change below 256 detectors).  Two shared-memory stages: the MMAs of chunk g
// run while chunk g + 1 is split.
// Measured against the 3xTF32 kernels before it (8 B per value, one tile per
// pass; error against FP64 in brackets): 256 x 450,561 0.29 ms (1.7e-6) for
// 0.47 (1.9e-6), 256 x 130,978 0.105 for 0.146, 128 x 563,201 0.151 (8.2e-7)
// for 0.259 (9.7e-7), 64 x 65,341 0.017 for 0.025.
// Every wait is bounded and also polls the CTA's abort flag, so a timeout in
// one role ends all of them; the MMA thread then drains its outstanding
// copies and MMAs (bounded) before the tensor memory is freed.
//
// A tile's inputs are all read before its outputs are written, so R may be X.
// One launch covers a table of TODs (per-TOD pointers, lengths, images).
#include "mk_async.cuh"
#include "mk_common.cuh"
#include "mk_rot.cuh"

namespace {

using mk::bulk_g2s;
using mk::mbar_expect_tx;
using mk::mbar_init;
using mk::mbar_wait;
using mk::smem_u32;

constexpr int TILE_M = 128;  // samples per MMA tile
constexpr int KC = 32;       // K per chunk: one 64-byte swizzle row of bf16
constexpr int NSTAGE = 2;
constexpr uint32_t A_PART = TILE_M * 64;   // one of the three parts of an X tile chunk (8 KB)
constexpr uint32_t A_TILE = 3 * A_PART;

// two floats rounded to bf16 (nearest; NaN and infinity stay), and the parts as
// floats again
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float lo_part(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float hi_part(uint32_t p) { return __uint_as_float(p & 0xFFFF0000u); }

// the three bf16 parts of two values
__device__ __forceinline__ void split2(float a, float b, uint32_t &h, uint32_t &m, uint32_t &l) {
  h = bf16_pair(a, b);
  a -= lo_part(h);
  b -= hi_part(h);
  m = bf16_pair(a, b);
  l = bf16_pair(a - lo_part(m), b - hi_part(m));
}

// byte offset of the 16-byte group c (8 values of k) of row r in a K-major
// tile of 64-byte rows with the 64-byte swizzle
__device__ __forceinline__ uint32_t sw64_off(uint32_t r, uint32_t c) { return r * 64u + ((c ^ ((r >> 1) & 3u)) << 4); }

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

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// B-operand image in global memory: per K-chunk c the h, m and l tiles, each
// ndet rows x 32 k in the swizzled layout above
__global__ void k_bprep(const float *__restrict__ A, int ndet, char *__restrict__ img) {
  const size_t part = (size_t)ndet * 64;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < ndet * ndet; idx += gridDim.x * blockDim.x) {
    const int j = idx / ndet, k = idx % ndet;
    uint32_t h, m, l;
    split2(A[idx], 0.f, h, m, l);
    char *p = img + (size_t)(k / KC) * 3 * part + sw64_off(j, (k % KC) >> 3) + (k & 7) * 2;
    *(uint16_t *)p = (uint16_t)h;
    *(uint16_t *)(p + part) = (uint16_t)m;
    *(uint16_t *)(p + 2 * part) = (uint16_t)l;
  }
}

__device__ __forceinline__ bool ws_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  for (uint32_t i = 0; i < mk::ROLE_SPIN_LIMIT; i++) {
    if (mk::mbar_try_wait(bar, parity)) return true;
    if ((i & 31u) == 31u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// a converged warp waits; true if every lane saw the phase complete
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  const bool ok = __all_sync(0xffffffffu, ws_wait(bar, parity, abort_flag));
  asm volatile("tcgen05.fence::after_thread_sync;");
  return ok;
}

// The job (TOD) that owns tile t of the launch; jobs are sorted by tile0 and
// each role walks its tiles in increasing order, so the cursor only moves on.
__device__ __forceinline__ int job_at(const mk::RotJob *jobs, int njobs, int64_t t, int cur) {
  while (cur + 1 < njobs && jobs[cur + 1].tile0 <= t) cur++;
  return cur;
}

// plain (R may be X) streaming load; zero past the TOD's end
__device__ __forceinline__ float load1(const float *p, bool ok) { return ok ? __ldcs(p) : 0.f; }

// NaN where this CTA writes its jobs' R (not inlined: the kernel around it keeps
// its code)
template <int MT>
__device__ __noinline__ void fill_nan(const mk::RotJob *jobs, int njobs, int64_t nitem, int ndet, int64_t mirror_n) {
  const float nan = __int_as_float(0x7FC00000);
  int cur = 0;
  for (int64_t item = blockIdx.x; item < nitem; item += gridDim.x) {
    cur = job_at(jobs, njobs, item, cur);
    const mk::RotJob &J = jobs[cur];
    for (int e = threadIdx.x; e < MT * TILE_M * ndet; e += (int)blockDim.x) {
      const int64_t my = (item - J.tile0) * MT * TILE_M + e % (MT * TILE_M);
      float *row = J.R + (int64_t)(e / (MT * TILE_M)) * J.ldr;
      if (my >= J.ncol) continue;
      row[my] = nan;
      if (mirror_n > 0 && my >= 1 && my <= J.ncol - 2) row[mirror_n - my] = nan;
    }
  }
}

// One item = MT tiles of 128 samples of one job (RotJob::tile0 counts items).
// `jobs` (device memory, sorted by tile0) lists the TODs of a grouped launch,
// all with ndet detectors; for one TOD it is null and `j0` is that TOD.
// mirror_n, xs and halve_ends apply to single-TOD launches (0, 1, 0 in groups).
template <int MT>
__global__ void __launch_bounds__((8 * MT + 1) * 32, 3 - MT)
    k_rot_tc(const mk::RotJob *jobs_in, int njobs, const mk::RotJob j0, int64_t nitem, int ndet, int nbuf,
             uint32_t tcols, int *err, int64_t mirror_n, int64_t xs, int halve_ends) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int NSPLIT = 4 * MT, NEPI = 4 * MT;
  const uint32_t b_part = (uint32_t)ndet * 64;
  const uint32_t stage_bytes = MT * A_TILE + 3 * b_part;
  __shared__ uint64_t full_a[NSTAGE], full_b[NSTAGE], mma_done[NSTAGE], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  volatile int *abort_flag = &abort_sh;
  const mk::RotJob *jobs = jobs_in ? jobs_in : &j0;
  if (!jobs_in) njobs = 1;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nchunk = ndet / KC;
  if (tid == 0) {
    for (int s = 0; s < NSTAGE; s++) {
      mbar_init(&full_a[s], NSPLIT * 32);
      mbar_init(&full_b[s], 1);
      mbar_init(&mma_done[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], NEPI * 32);
    }
    abort_sh = 0;
    mk::mbar_init_fence();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"(tcols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base_sh;
  uint32_t g_copied = 0, g_issued = 0;  // MMA thread: chunks whose image copy / MMAs were issued

  if (warp < NSPLIT) {
    // ---- split role: thread = sample; the values of the next chunk are
    // loaded into the registers that the current one leaves
    const int mt = warp >> 2, row = (warp & 3) * 32 + lane;
    int cur = 0;
    uint32_t g = 0;
    float v[KC];
    int64_t item = blockIdx.x, ldx = 0;
    const float *src = nullptr;
    bool ok = false;
    float hs = 1.f, hs_next = 1.f;
    auto open = [&]() {  // this thread's sample of `item`
      cur = job_at(jobs, njobs, item, cur);
      const mk::RotJob &J = jobs[cur];
      const int64_t my = ((item - J.tile0) * MT + mt) * TILE_M + row;
      ok = my < J.ncol;
      ldx = J.ldx;
      src = J.X + (ok ? my : 0) * xs;
      hs_next = halve_ends && (my == 0 || my == J.ncol - 1) ? 0.5f : 1.0f;
    };
    if (item < nitem) {
      open();
#pragma unroll
      for (int kk = 0; kk < KC; kk++) v[kk] = load1(src + kk * ldx, ok);
    }
    for (bool stop = false; item < nitem && !stop && !*abort_flag;) {
      hs = hs_next;
      for (int c = 0; c < nchunk; c++, g++) {
        const uint32_t s = g % NSTAGE;
        if (g >= NSTAGE && !ws_wait(&mma_done[s], (g / NSTAGE - 1) & 1, abort_flag)) {
          stop = true;
          break;
        }
        if (c + 1 < nchunk) {
          src += KC * ldx;
        } else {
          item += gridDim.x;
          ok = false;
          if (item < nitem) open();
        }
        unsigned char *at = smem + s * stage_bytes + mt * A_TILE;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint32_t h[4], m[4], l[4];
#pragma unroll
          for (int i = 0; i < 4; i++) split2(v[8 * q + 2 * i] * hs, v[8 * q + 2 * i + 1] * hs, h[i], m[i], l[i]);
#pragma unroll
          for (int i = 0; i < 8; i++) v[8 * q + i] = load1(src + (8 * q + i) * ldx, ok);
          const uint32_t off = sw64_off(row, q);
          *(uint4 *)(at + off) = make_uint4(h[0], h[1], h[2], h[3]);
          *(uint4 *)(at + A_PART + off) = make_uint4(m[0], m[1], m[2], m[3]);
          *(uint4 *)(at + 2 * A_PART + off) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        mk::fence_proxy_async_smem();
        mk::mbar_arrive(&full_a[s]);
      }
    }
  } else if (warp == NSPLIT + NEPI) {
    // ---- image copies and MMAs (one lane issues; the warp stays converged)
    const uint32_t lead = elect_one();
    const uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ndet >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);
    uint32_t it = 0;
    int cur = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; item < nitem && ok; item += gridDim.x, it++) {
      cur = job_at(jobs, njobs, item, cur);
      const char *bimg = jobs[cur].bimg;
      const uint32_t ab = nbuf == 2 ? it & 1 : 0, au = nbuf == 2 ? it >> 1 : it;
      for (int c = 0; c < nchunk; c++) {
        const uint32_t g = g_issued, s = g % NSTAGE, use = g / NSTAGE;
        unsigned char *st = smem + s * stage_bytes;
        if (g >= NSTAGE && !warp_wait(&mma_done[s], (use - 1) & 1, abort_flag)) {
          ok = false;
          break;
        }
        if (lead) {
          mbar_expect_tx(&full_b[s], 3 * b_part);
          bulk_g2s(st + MT * A_TILE, bimg + (size_t)c * 3 * b_part, 3 * b_part, &full_b[s]);
        }
        g_copied = g + 1;
        if (c == 0 && au >= 1) ok = warp_wait(&acc_empty[ab], (au - 1) & 1, abort_flag);
        ok = ok && warp_wait(&full_b[s], use & 1, abort_flag) && warp_wait(&full_a[s], use & 1, abort_flag);
        if (!ok) break;
        const uint32_t ad = sdesc_lo(smem_u32(st)), bd = sdesc_lo(smem_u32(st + MT * A_TILE));
        constexpr uint32_t AP = A_PART / 16;
        const uint32_t bp = b_part / 16;
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
          const uint32_t dacc = tmem + (ab * MT + mt) * (uint32_t)ndet;
#pragma unroll
          for (int k16 = 0; k16 < KC / 16; k16++) {
            const uint32_t h = ad + (mt * A_TILE + k16 * 32) / 16, b = bd + k16 * 2;
            mma_bf16(lead, dacc, h, b + 2 * bp, idesc, c == 0 && k16 == 0 ? 0u : 1u);
            mma_bf16(lead, dacc, h + 2 * AP, b, idesc, 1u);
            mma_bf16(lead, dacc, h + AP, b + bp, idesc, 1u);
            mma_bf16(lead, dacc, h, b + bp, idesc, 1u);
            mma_bf16(lead, dacc, h + AP, b, idesc, 1u);
            mma_bf16(lead, dacc, h, b, idesc, 1u);
          }
        }
        mma_commit(lead, &mma_done[s]);
        g_issued = g + 1;
      }
      if (!ok) break;
      mma_commit(lead, &acc_full[ab]);
    }
  } else {
    // ---- epilogue role
    const int ew = warp - NSPLIT, mt = ew >> 2;
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    const int row = 32 * q + lane;
    uint32_t it = 0;
    int cur = 0;
    for (int64_t item = blockIdx.x; item < nitem; item += gridDim.x, it++) {
      cur = job_at(jobs, njobs, item, cur);
      const uint32_t ab = nbuf == 2 ? it & 1 : 0, au = nbuf == 2 ? it >> 1 : it;
      if (!warp_wait(&acc_full[ab], au & 1, abort_flag)) break;
      const mk::RotJob &J = jobs[cur];
      const int64_t my = ((item - J.tile0) * MT + mt) * TILE_M + row, ncol = J.ncol, ldr = J.ldr;
      float *R = J.R;
      const uint32_t base = tmem + ((uint32_t)(32 * q) << 16) + (ab * MT + mt) * (uint32_t)ndet;
      for (int c0 = 0; c0 < ndet; c0 += 32) {
        float v[32];
        tmem_ld32(base + (uint32_t)c0, v);
        if (my < ncol) {
#pragma unroll
          for (int j = 0; j < 32; j++) __stcs(R + (int64_t)(c0 + j) * ldr + my, v[j]);
          // even extension for the DCT-I that follows: R[., mirror_n - my] = R[., my]
          if (mirror_n > 0 && my >= 1 && my <= ncol - 2) {
#pragma unroll
            for (int j = 0; j < 32; j++) __stcs(R + (int64_t)(c0 + j) * ldr + (mirror_n - my), v[j]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      mk::mbar_arrive(&acc_empty[ab]);
    }
  }
  __syncthreads();
  const bool failed = *abort_flag;
  if (failed && tid == (NSPLIT + NEPI) * 32) {
    atomicExch(err, 1);
    // bounded waits for the copies and MMAs this thread issued
    for (uint32_t g = (g_copied > NSTAGE ? g_copied - NSTAGE : 0); g < g_copied; g++)
      (void)mbar_wait(&full_b[g % NSTAGE], (g / NSTAGE) & 1);
    for (uint32_t g = (g_issued > NSTAGE ? g_issued - NSTAGE : 0); g < g_issued; g++)
      (void)mbar_wait(&mma_done[g % NSTAGE], (g / NSTAGE) & 1);
  }
  if (failed) fill_nan<MT>(jobs, njobs, nitem, ndet, mirror_n);  // no caller takes this CTA's part for a result
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols));
}

template <int MT>
int launch(const mk::RotJob *jobs, int njobs, const mk::RotJob &j0, int64_t nitem, int nd, int *err, cudaStream_t st,
           int64_t mirror_n, int64_t xs, int halve_ends) {
  const auto bytes = [](int ndet) { return NSTAGE * ((size_t)MT * A_TILE + 3 * (size_t)ndet * 64) + 1024; };
  const size_t smem = bytes(nd);
  // the limit of the largest detector count of the instantiation, whatever this
  // call's: threads that set it at the same time set the same value
  static bool attr[64] = {false};
  int dev = 0;
  MK_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr[dev]) {
    MK_CUDA(cudaFuncSetAttribute(k_rot_tc<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)bytes(256)));
    attr[dev] = true;
  }
  const int nbuf = MT * nd * 2 <= 512 / (MT == 1 ? 2 : 1) ? 2 : 1;  // accumulators; MT = 1: two CTAs per SM
  const uint32_t tcols = (uint32_t)(MT * nd * nbuf);
  int64_t grid = (int64_t)mk::sm_count() * (MT == 1 ? 2 : 1);
  if (grid > nitem) grid = nitem;
  k_rot_tc<MT><<<(unsigned)grid, (8 * MT + 1) * 32, smem, st>>>(jobs, njobs, j0, nitem, nd, nbuf, tcols, err, mirror_n,
                                                                xs, halve_ends);
  return mk::launch_status("rot_tc");
}

int launch_mt(int mt, const mk::RotJob *jobs, int njobs, const mk::RotJob &j0, int64_t nitem, int nd, int *err,
              cudaStream_t st, int64_t mirror_n, int64_t xs, int halve_ends) {
  if (mt == 2) return launch<2>(jobs, njobs, j0, nitem, nd, err, st, mirror_n, xs, halve_ends);
  return launch<1>(jobs, njobs, j0, nitem, nd, err, st, mirror_n, xs, halve_ends);
}

}  // namespace

namespace mk {

bool rot_tc_supported(int64_t nrow) {
  return nrow == 32 || nrow == 64 || nrow == 128 || nrow == 256;
}

size_t rot_tc_bimg_bytes(int64_t nrow) { return (size_t)nrow * (size_t)nrow * 6; }

int64_t rot_tc_tiles(int64_t ncol) { return (ncol + TILE_M - 1) / TILE_M; }

int rot_tc_tiles_per_item(int64_t nrow, int64_t ntile) { return nrow == 256 && ntile > sm_count() ? 2 : 1; }

int64_t rot_tc_items(int64_t ncol, int mt) { return (rot_tc_tiles(ncol) + mt - 1) / mt; }

int rot_tc_f32(const float *A, const float *X, int64_t ldx, float *R, int64_t ldr, int64_t nrow,
               int64_t ncol, void *bimg, int *err, cudaStream_t st, int64_t mirror_n, int64_t x_stride,
               int halve_ends) {
  MK_CHECK_ARG(mirror_n == 0 || (mirror_n == 2 * (ncol - 1) && ldr >= mirror_n),
               "tensor-core rotation: bad mirror extent");
  MK_CHECK_ARG(x_stride == 1 || x_stride == 2, "tensor-core rotation: element stride must be 1 or 2");
  MK_CHECK_ARG(err, "tensor-core rotation: bad scratch");
  if (ncol <= 0) return MK_OK;
  const int rc = rot_tc_bprep(A, nrow, bimg, st);
  if (rc) return rc;
  const RotJob j0{X, R, (const char *)bimg, ldx, ldr, ncol, 0};
  const int mt = rot_tc_tiles_per_item(nrow, rot_tc_tiles(ncol));
  return launch_mt(mt, nullptr, 1, j0, rot_tc_items(ncol, mt), (int)nrow, err, st, mirror_n, x_stride, halve_ends);
}

int rot_tc_bprep(const float *A, int64_t nrow, void *bimg, cudaStream_t st) {
  MK_CHECK_ARG(rot_tc_supported(nrow), "tensor-core rotation supports ndet in {32,64,128,256}, got %lld",
               (long long)nrow);
  MK_CHECK_ARG(A && bimg && ((uintptr_t)bimg % 16) == 0, "tensor-core rotation: bad operand image");
  const int nd = (int)nrow;
  k_bprep<<<(nd * nd + 255) / 256, 256, 0, st>>>(A, nd, (char *)bimg);
  return launch_status("rot_tc_bprep");
}

int rot_tc_group(const RotJob *jobs_dev, int njobs, int64_t nitem, int mt, int64_t nrow, int *err, cudaStream_t st) {
  MK_CHECK_ARG(rot_tc_supported(nrow), "tensor-core rotation supports ndet in {32,64,128,256}, got %lld",
               (long long)nrow);
  MK_CHECK_ARG(jobs_dev && njobs >= 1 && err, "tensor-core rotation group: bad arguments");
  if (nitem <= 0) return MK_OK;
  return launch_mt(mt, jobs_dev, njobs, RotJob{}, nitem, (int)nrow, err, st, 0, 1, 0);
}

}  // namespace mk
