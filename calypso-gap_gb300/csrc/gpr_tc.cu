// gpr_tc.cu - the sparse-GPR contraction on the 5th-generation tensor cores.
//
// Same quantities as gpr.cu (GET_COV and the energy / dE/dG loops of
// FGAP_CALC, gappy/libgap/gap_calc.f90:143-166, 268-288), computed as two
// GEMMs with split-BF16 operands and FP32 accumulation in tensor memory:
//
//   centred, scaled descriptors  x'' = x/theta - mu,  m'' = m/theta - mu
//   (mu = mean of the sparse points; differences are unchanged by centring)
//   s_ik  = |x''_i|^2 + |m''_k|^2 - 2 x''_i . m''_k
//   GEMM1 (N x M, K = D):  x''.m'' ~ xh.mh + xh.ml + xl.mh  (3-term BF16 split,
//                          x'' = xh + xl, m'' = mh + ml, every product exact in FP32)
//                          as two MMAs per K step: xh.[mh; ml] (N = 128) into
//                          columns [0, 64) and [64, 128), and xl.mh (N = 64)
//                          into [0, 64); the epilogue adds the two halves
//   w_ik  = c_k exp(-s_ik / 2),  e_i = sum_k w_ik  (compensated FP32, Kahan)
//   GEMM2 (N x D, K = M):  (W M'')_id ~ wh.mh + wh.ml + wl.mh, the same way:
//                          wh.[mhT; mlT] (N = 128) and wl.mhT (N = 64)
//   dE/dG_id = -(1/theta_d) (x''_id e_i - (W M'')_id)
//
// One CTA owns 128 atoms and walks the sparse points in tiles of 64.  Roles:
// two sets of eight epilogue warps (thread = atom row and half of a tile's
// columns) that take tiles in turn, a warp that issues GEMM1, one that issues
// GEMM2, one that keeps a ring of five tiles loading.  C1 has three buffers of
// 128 TMEM columns, so GEMM1 runs up to three tiles ahead; an epilogue warp
// writes W (wh 16 + wl 16 columns) over the columns that it alone has read, and
// GEMM2 takes W from there as its A operand.  C2 is the other 128 columns: one
// CTA per SM.  Per SM an M = 128, K = 16 MMA takes 16 + N/2 cycles with A in
// tensor memory and 48 + N/2 with A in shared memory (measured, N = 64 to 256),
// so fewer, wider MMAs, and W in tensor memory: 760 + 500 cycles a tile.
// Two warps issue because a warp's next barrier poll waits for the MMAs that it
// has queued: with one, the pipe idles 350 cycles after each batch of eight.
// Measured: a tile (128 atoms x 64 points) takes about 1650 cycles, 43 to 47 %
// of the tensor pipe's cycles and 57 to 62 % of the issue slots; a wave of up to
// 152 x 128 atoms takes 61 us at M = 4000 and 108 at M = 8000, where a kernel of
// 4 warps per 128 atoms and two CTAs per SM, each with its GEMMs and epilogue in
// turn and A and W in shared memory, took 131 and 241.  The [mh; ml] and
// [mhT; mlT] pairs are adjacent 64-row blocks in shared memory, which is the
// 128-row B operand of the same canonical layout.
//
// Operand tiles use the no-swizzle K-major canonical layout: 8-row x 16-byte
// core matrices, K-adjacent cores 128 B apart (LBO), 8-row groups
// (K/8)*128 B apart (SBO).  The model's tiles are built once on the host in
// that layout, so a tile is a contiguous block and needs no tensor map.
//
// Every mbarrier wait is bounded; a wait that gives up sets an error flag,
// the CTA skips the rest of its work, frees its tensor memory and returns.
#include <cuda_bf16.h>

#include <cstring>

#include "gapgb_internal.h"
#include "tc_util.cuh"

namespace gapgb {
namespace {

using namespace tc;

constexpr int kRows = 128;   // atoms per CTA (UMMA M)
constexpr int kTileK = 64;   // sparse points per tile (GEMM1 N, GEMM2 K)
constexpr int kDP = 64;      // padded descriptor length (GEMM1 K, GEMM2 N)
constexpr int kXBytes16 = kRows * kDP * 2;           // 128 x 64 bf16: 16 KB
constexpr int kMBytes16 = kTileK * kDP * 2;          // 64 x 64 bf16: 8 KB
// per sparse tile image: mh, ml (64 x 64), mhT, mlT (64 x 64), b2[64], c[64]
constexpr int kImgTile = 4 * kMBytes16 + 2 * kTileK * 4;     // 32.5 KB
constexpr int kImgAtoms = 2 * kXBytes16;                      // xh, xl per 128 atoms

// shared memory map (bytes from the 1024-aligned base): the ring of tile images
constexpr int kStages = 5;
constexpr int kStage = 33 * 1024;  // one tile image, padded
constexpr int kOffMh = 0;
constexpr int kOffMl = kOffMh + kMBytes16;
constexpr int kOffMhT = kOffMl + kMBytes16;
constexpr int kOffMlT = kOffMhT + kMBytes16;
constexpr int kOffMnc = kOffMlT + kMBytes16;  // b2 and c
static_assert(kImgTile <= kStage, "tile image beyond its stage");
// [mh; ml] and [mhT; mlT] as one 128-row B operand: the second block starts
// eight 8-row groups (the canonical layout's SBO apart) after the first
static_assert(kOffMl - kOffMh == 8 * (kDP / 8) * 128, "mh / ml not one 128-row operand");
static_assert(kOffMlT - kOffMhT == 8 * (kTileK / 8) * 128, "mhT / mlT not one 128-row operand");
constexpr int kOffX = kStages * kStage;                  // xh, xl
constexpr int kOffBar = kOffX + kImgAtoms;
constexpr int kOffEp = kOffBar + 512;                    // partial energies [128] (FP64)
constexpr int kOffPart = kOffEp + kRows * 8;             // odd tiles' partial sums [3][256] float4
constexpr int kSmemBytes = kOffPart + 3 * 2 * kRows * 16 + 1024;  // + alignment slack
// two sets of 8 epilogue warps: w and w + 4 share TMEM lanes and split the columns
constexpr int kEpiWarps = 16;
constexpr int kGprThreads = 32 * (kEpiWarps + 3);  // and a warp each for GEMM1, GEMM2 and copies
// TMEM columns
constexpr int kC1 = 3;  // C1 / W buffers
constexpr int kColC1 = 0, kColC2 = 128 * kC1;

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// v = (16 columns at taddr) + (16 columns at taddr + off), as tmem_ld32_sum2
__device__ __forceinline__ void tmem_ld16_sum2(uint32_t taddr, uint32_t off, float (&v)[16]) {
  uint32_t r[16], s[16];
#define GAPGB_LD16(dst, addr)                                                                     \
  asm volatile(                                                                                  \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"   \
      "%14,%15}, [%16];"                                                                         \
      : "=r"(dst[0]), "=r"(dst[1]), "=r"(dst[2]), "=r"(dst[3]), "=r"(dst[4]), "=r"(dst[5]),     \
        "=r"(dst[6]), "=r"(dst[7]), "=r"(dst[8]), "=r"(dst[9]), "=r"(dst[10]), "=r"(dst[11]),   \
        "=r"(dst[12]), "=r"(dst[13]), "=r"(dst[14]), "=r"(dst[15])                              \
      : "r"(addr))
  GAPGB_LD16(r, taddr);
  GAPGB_LD16(s, taddr + off);
#undef GAPGB_LD16
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    asm volatile("" : "+r"(r[q]), "+r"(s[q]));  // uses stay behind the wait
    v[q] = __uint_as_float(r[q]) + __uint_as_float(s[q]);
  }
}
// s += x with Kahan compensation c
__device__ __forceinline__ void kahan(float &s, float &c, float x) {
  const float y = x - c;
  const float t = s + y;
  c = (t - s) - y;
  s = t;
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__global__ void __launch_bounds__(kGprThreads, 1)
    k_gpr_tc(int N, int ntiles, const unsigned char *__restrict__ img_model,
             const unsigned char *__restrict__ img_atoms, const float *__restrict__ xs,
             const float *__restrict__ xn, const float *__restrict__ invth, int D,
             double *__restrict__ e_out, float *__restrict__ dedg, int *__restrict__ flags) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>(
      ((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // epilogue warps: set, TMEM lane quadrant, column half
  const int set = warp >> 3, quad = warp & 3, half = (warp >> 2) & 1;
  const uint32_t s_base = smem_u32(sm);
  // a tile's image has arrived / is free (its GEMM2 done); C1 computed; W
  // written; the atoms have arrived; given up; odd tiles' sums stored [3][8]
  const uint32_t mfull = s_base + kOffBar, mempty = mfull + 8 * kStages,
                 c1full = mempty + 8 * kStages, wfull = c1full + 8 * kC1, xfull = wfull + 8 * kC1,
                 dead = xfull + 8, pfull = dead + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + kOffBar + 384);
  volatile int *abort_flag = reinterpret_cast<int *>(sm + kOffBar + 392);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int q = 0; q < kStages; ++q) {
      mbar_init(mfull + 8 * q, 1);
      mbar_init(mempty + 8 * q, 1);
    }
    for (int q = 0; q < kC1; ++q) {
      mbar_init(c1full + 8 * q, 1);
      mbar_init(wfull + 8 * q, 8);
    }
    mbar_init(xfull, 1);
    mbar_init(dead, 1);
    mbar_init(dead + 8, 1);
    for (int q = 0; q < 3 * 8; ++q) mbar_init(pfull + 8 * q, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);  // this warp's TMEM lanes
  const int row = quad * 32 + lane;                                  // atom row of this thread
  const int i = blockIdx.x * kRows + row;
  bool ok = true;
  if (warp == kEpiWarps + 2) {
    if (lane == 0) {
      int t = 0;
      mbar_expect_tx(xfull, kImgAtoms);
      bulk_g2s(s_base + kOffX, img_atoms + (size_t)blockIdx.x * kImgAtoms, kImgAtoms, xfull);
      for (; t < ntiles; ++t) {
        const int q = t % kStages;
        if (t >= kStages && !mbar_wait(mempty + 8 * q, (t / kStages - 1) & 1, flags)) break;
        if (*abort_flag) break;
        mbar_expect_tx(mfull + 8 * q, kImgTile);
        bulk_g2s(s_base + q * kStage, img_model + (size_t)t * kImgTile, kImgTile, mfull + 8 * q);
      }
      if (t < ntiles) {
        // gave up: one more bounded wait for each copy still in flight
        *abort_flag = 1;
        for (int u = t > kStages ? t - kStages : 0; u < t; ++u)
          mbar_wait(mfull + 8 * (u % kStages), (u / kStages) & 1, flags);
      }
      mbar_wait(xfull, 0, flags);  // (also where there was no tile to use it)
    }
  } else if (warp >= kEpiWarps) {
    // N = 128: [mh; ml] (GEMM1) or [mhT; mlT] (GEMM2); N = 64: mh or mhT alone
    const uint32_t id_pair = instr_desc(kRows, 128), id1 = instr_desc(kRows, kTileK);
    auto wait = [&](uint32_t bar, uint32_t parity) {  // the warp as one
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, flags) && !*abort_flag) != 0;
    };
    int t = 0;
    if (warp == kEpiWarps) {
      // C1[:, 0:64] + C1[:, 64:128] = xh.mh + xh.ml + xl.mh over K = 64 (4 steps
      // of 16): xh.[mh; ml] into both halves, then xl.mh into the first
      const uint64_t da = smem_desc(s_base + kOffX, 128, (kDP / 8) * 128);
      ok = ntiles > 0 && wait(xfull, 0);
      for (; t < ntiles && ok; ++t) {
        if (!(ok = wait(mfull + 8 * (t % kStages), (t / kStages) & 1))) break;
        // W of tile t - 3 lies where C1 goes: its GEMM2 has to be done
        const int u = t - kC1;
        if (u >= 0 && !(ok = wait(mempty + 8 * (u % kStages), (u / kStages) & 1))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t c1 = tmem + kColC1 + 128 * (t % kC1);
        const uint64_t db =
            smem_desc(s_base + (t % kStages) * kStage + kOffMh, 128, (kDP / 8) * 128);
        if (elect_one()) {
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int kk = 0; kk < kDP / 16; ++kk)
              umma(c1, da + p * (kXBytes16 >> 4) + 16 * kk, db + 16 * kk, p == 0 ? id_pair : id1,
                   (p > 0 || kk > 0) ? 1u : 0u);
          umma_commit(c1full + 8 * (t % kC1));
        }
        __syncwarp();
      }
    } else {
      // C2[:, 0:64] + C2[:, 64:128] += wh.mhT + wh.mlT + wl.mhT over K = 64
      // (4 steps of 16): wh.[mhT; mlT] into both halves, wl.mhT into the first
      for (; t < ntiles && ok; ++t) {
        if (!(ok = wait(wfull + 8 * (t % kC1), (t / kC1) & 1))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t w = tmem + kColC1 + 128 * (t % kC1);
        const uint64_t db =
            smem_desc(s_base + (t % kStages) * kStage + kOffMhT, 128, (kTileK / 8) * 128);
        if (elect_one()) {
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int kk = 0; kk < kTileK / 16; ++kk)
              umma_ta(tmem + kColC2, w + 32 * (kk >> 1) + 16 * p + 8 * (kk & 1), db + 16 * kk,
                      p == 0 ? id_pair : id1, (t > 0 || p > 0 || kk > 0) ? 1u : 0u);
          umma_commit(mempty + 8 * (t % kStages));
        }
        __syncwarp();
      }
    }
    if (t < ntiles) {
      // gave up: a last bounded wait for the MMAs issued so far
      *abort_flag = 1;
      const uint32_t bar = dead + 8 * (warp - kEpiWarps);
      if (elect_one()) umma_commit(bar);
      __syncwarp();
      mbar_wait(bar, 0, flags);
    }
  } else {
    const float xnorm = (i < N) ? xn[i] : 0.f;
    // w = c exp(-s/2) = c 2^(log2e v + a2_i + b2_k) with a2_i = -log2e |x''_i|^2 / 2
    // and b2_k = -log2e |m''_k|^2 / 2 (the image stores b2): one add, one FMA
    // and ex2 per element.  The sets take tiles in turn, so that one computes
    // while the other waits for TMEM.  e = sum w: each thread sums its 32
    // elements of a tile into four plain partial sums (8 elements each), which
    // enter four independent Kahan chains per (row, half) once per tile, in tile
    // order.  Set 0 keeps the chains; set 1 hands it its sums through shared
    // memory: three slots, since C1 of tile t + 6 waits for the W of tile t + 3,
    // which set 0 writes after it has taken the sums of tile t.
    const float a2 = -0.5f * kLog2e * xnorm;
    float es[4] = {0.f, 0.f, 0.f, 0.f}, ec[4] = {0.f, 0.f, 0.f, 0.f};
    float4 *slots = reinterpret_cast<float4 *>(sm + kOffPart) + half * kRows + row;
    const uint32_t my_pfull = pfull + 8 * (warp & 7);
    // the sums of odd tile t into set 0's chains
    auto take = [&](int t) {
      const int sl = (t >> 1) % 3;
      if (!mbar_wait_w(my_pfull + 64 * sl, ((t >> 1) / 3) & 1, flags)) return false;
      const float4 p = slots[sl * 2 * kRows];
      kahan(es[0], ec[0], p.x);
      kahan(es[1], ec[1], p.y);
      kahan(es[2], ec[2], p.z);
      kahan(es[3], ec[3], p.w);
      return true;
    };
    for (int t = set; t < ntiles; t += 2) {
      const int q = t % kStages;
      ok = __all_sync(0xffffffffu, mbar_wait(mfull + 8 * q, (t / kStages) & 1, flags) &&
                                       mbar_wait(c1full + 8 * (t % kC1), (t / kC1) & 1, flags) &&
                                       !*abort_flag);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float *smn = reinterpret_cast<const float *>(sm + q * kStage + kOffMnc);
      const float *sc = smn + kTileK;
      const uint32_t c1 = lane_base + kColC1 + 128 * (t % kC1) + 32 * half;
      float part[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t hpk[16], lpk[16];
#pragma unroll
      for (int gg = 0; gg < 2; ++gg) {
        float v[16];
        tmem_ld16_sum2(c1 + 16 * gg, kTileK, v);
#pragma unroll
        for (int g = 2 * gg; g < 2 * gg + 2; ++g) {
          const int kg = half * 32 + g * 8;
          const float4 b0 = *reinterpret_cast<const float4 *>(smn + kg);
          const float4 b1 = *reinterpret_cast<const float4 *>(smn + kg + 4);
          const float4 f0 = *reinterpret_cast<const float4 *>(sc + kg);
          const float4 f1 = *reinterpret_cast<const float4 *>(sc + kg + 4);
          const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
          const float cv[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            float w2[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int e = h * 2 + u;
              const float w = cv[e] * ex2_approx(fmaf(v[(g & 1) * 8 + e], kLog2e, a2 + bv[e]));
              part[h] += w;
              w2[u] = w;
            }
            const __nv_bfloat162 hi = __floats2bfloat162_rn(w2[0], w2[1]);
            const float2 hf = __bfloat1622float2(hi);
            hpk[4 * g + h] = *reinterpret_cast<const uint32_t *>(&hi);
            lpk[4 * g + h] = pack_bf16(w2[0] - hf.x, w2[1] - hf.y);
          }
        }
      }
      // over the columns that this warp has just read: wh, wl of 32 points
      tmem_st16(c1, hpk);
      tmem_st16(c1 + 16, lpk);
      tmem_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(wfull + 8 * (t % kC1));
      if (set == 1) {
        const int sl = (t >> 1) % 3;
        slots[sl * 2 * kRows] = make_float4(part[0], part[1], part[2], part[3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(my_pfull + 64 * sl);
      } else {
        if (t > 0 && !(ok = take(t - 1))) break;
#pragma unroll
        for (int h = 0; h < 4; ++h) kahan(es[h], ec[h], part[h]);
      }
    }
    if (set == 0 && ok && ntiles > 0 && (ntiles & 1) == 0) ok = take(ntiles - 1);
    if (ok && ntiles > 0)
      ok = __all_sync(0xffffffffu, mbar_wait(mempty + 8 * ((ntiles - 1) % kStages),
                                             ((ntiles - 1) / kStages) & 1, flags));
    if (!ok) *abort_flag = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // the two column halves' partial energies, summed in a fixed order
    double *ep = reinterpret_cast<double *>(sm + kOffEp);
    auto sync16 = [] { asm volatile("bar.sync 1, 512;" ::: "memory"); };  // the epilogue warps
    double emine = (double)es[0] - (double)ec[0];
    emine += (double)es[1] - (double)ec[1];
    emine += (double)es[2] - (double)ec[2];
    emine += (double)es[3] - (double)ec[3];
    if (set == 0 && half == 1) ep[row] = emine;
    sync16();
    if (set == 0 && half == 0) ep[row] = emine + ep[row];
    sync16();
    if (__all_sync(0xffffffffu, !*abort_flag)) {  // (the TMEM load needs the whole warp)
      // dE/dG: each thread a row and 16 components
      const double etot = ep[row];
      const int d0 = half * 32 + set * 16;
      float c2[16];
      tmem_ld16_sum2(lane_base + kColC2 + d0, kDP, c2);
      if (i < N) {
        if (set == 0 && half == 0) e_out[i] = etot;
        const float ef = (float)etot;
        float x[16];
#pragma unroll
        for (int k = 0; k < 16; k += 4)
          *reinterpret_cast<float4 *>(x + k) =
              *reinterpret_cast<const float4 *>(xs + (size_t)i * kDP + d0 + k);
        float *o = dedg + (size_t)i * D + d0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int d = d0 + k;
          if (d < D) x[k] = -invth[d] * (x[k] * ef - c2[k]);
        }
        if (D % 4 == 0) {  // rows of dedg are then 16-byte aligned
#pragma unroll
          for (int k = 0; k < 16; k += 4)
            if (d0 + k < D)
              *reinterpret_cast<float4 *>(o + k) =
                  make_float4(x[k], x[k + 1], x[k + 2], x[k + 3]);
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (d0 + k < D) o[k] = x[k];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// x'' = G / theta - mu (FP32, row-padded to 64), |x''|^2, and the xh/xl tiles
__global__ void k_tc_prep_atoms(int N, int D, const float *__restrict__ G,
                                const float *__restrict__ invth, const float *__restrict__ mu,
                                float *__restrict__ xs, float *__restrict__ xn,
                                unsigned char *__restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int ntile_rows = ((N + kRows - 1) / kRows) * kRows;
  if (i >= ntile_rows) return;
  unsigned char *tile = img + (size_t)(i / kRows) * kImgAtoms;
  const int r = i % kRows;
  float nrm = 0.f;
  for (int k0 = 0; k0 < kDP; k0 += 8) {
    uint32_t hp[4], lp[4];
    for (int h = 0; h < 4; ++h) {
      float x2[2];
      for (int u = 0; u < 2; ++u) {
        const int d = k0 + h * 2 + u;
        float x = 0.f;
        if (i < N && d < D) x = G[(size_t)i * D + d] * invth[d] - mu[d];
        if (i < N) xs[(size_t)i * kDP + d] = x;
        nrm += x * x;
        x2[u] = x;
      }
      const __nv_bfloat162 hi = __floats2bfloat162_rn(x2[0], x2[1]);
      const float2 hf = __bfloat1622float2(hi);
      hp[h] = *reinterpret_cast<const uint32_t *>(&hi);
      lp[h] = pack_bf16(x2[0] - hf.x, x2[1] - hf.y);
    }
    const int off = kmajor_off(r, k0, kDP / 8);
    *reinterpret_cast<uint4 *>(tile + off) = make_uint4(hp[0], hp[1], hp[2], hp[3]);
    *reinterpret_cast<uint4 *>(tile + kXBytes16 + off) = make_uint4(lp[0], lp[1], lp[2], lp[3]);
  }
  if (i < N) xn[i] = nrm;
}

// host-side bf16 (round to nearest even) for the model image
uint16_t bf16_bits(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)(u >> 16);  // inf / nan
  const uint32_t lsb = (u >> 16) & 1u;
  u += 0x7fffu + lsb;
  return (uint16_t)(u >> 16);
}
float bf16_val(uint16_t b) {
  const uint32_t u = (uint32_t)b << 16;
  float f;
  std::memcpy(&f, &u, 4);
  return f;
}

}  // namespace

size_t tc_smem_bytes() { return kSmemBytes; }

// Builds the model's tensor-core image: per sparse tile mh, ml (K-major over
// D), mhT, mlT (K-major over the tile's points), b2 = -log2e |m''|^2 / 2 and c
// (FP32), plus mu.
gapgb_status build_tc_image(gapgb_model *m, bool refresh) {
  if (m->d_tc && !refresh) return GAPGB_OK;
  const HostModel &h = m->host;
  const int M = h.M, D = h.D;
  if (D > kDP) {
    set_last_error("tensor-core GPR supports D <= 64");
    return GAPGB_ERR_CAP_EXCEEDED;
  }
  const int nt = (M + kTileK - 1) / kTileK;
  std::vector<double> mu(kDP, 0.0);
  std::vector<double> mm2((size_t)M * kDP, 0.0);
  for (int k = 0; k < M; ++k)
    for (int d = 0; d < D; ++d) {
      mm2[(size_t)k * kDP + d] = h.mm[(size_t)k * D + d] / h.theta[d];
      mu[d] += mm2[(size_t)k * kDP + d] / M;
    }
  std::vector<unsigned char> img((size_t)nt * kImgTile, 0);
  for (int t = 0; t < nt; ++t) {
    unsigned char *T = img.data() + (size_t)t * kImgTile;
    float *mn = reinterpret_cast<float *>(T + 4 * kMBytes16);
    float *cf = mn + kTileK;
    for (int kk = 0; kk < kTileK; ++kk) {
      const int k = t * kTileK + kk;
      if (k >= M) continue;
      double nrm = 0.0;
      for (int d = 0; d < kDP; ++d) {
        const double v = (d < D) ? mm2[(size_t)k * kDP + d] - mu[d] : 0.0;
        nrm += v * v;
        const uint16_t hb = bf16_bits((float)v);
        const uint16_t lb = bf16_bits((float)(v - (double)bf16_val(hb)));
        // GEMM1 B operand: rows = sparse points, K = descriptor components
        std::memcpy(T + kmajor_off(kk, d, kDP / 8), &hb, 2);
        std::memcpy(T + kMBytes16 + kmajor_off(kk, d, kDP / 8), &lb, 2);
        // GEMM2 B operand: rows = descriptor components, K = sparse points
        std::memcpy(T + 2 * kMBytes16 + kmajor_off(d, kk, kTileK / 8), &hb, 2);
        std::memcpy(T + 3 * kMBytes16 + kmajor_off(d, kk, kTileK / 8), &lb, 2);
      }
      mn[kk] = (float)(-0.5 * 1.4426950408889634 * nrm);  // b2_k = -log2e |m''_k|^2 / 2
      cf[kk] = (float)h.coeff[k];
    }
  }
  std::vector<float> muf(kDP);
  for (int d = 0; d < kDP; ++d) muf[d] = (float)mu[d];
  const size_t bytes = img.size() + kDP * sizeof(float);
  if (!m->d_tc) GAPGB_CUDA_TRY(cudaMalloc(&m->d_tc, bytes));  // same size on a refresh
  GAPGB_CUDA_TRY(cudaMemcpy(m->d_tc, img.data(), img.size(), cudaMemcpyHostToDevice));
  GAPGB_CUDA_TRY(cudaMemcpy((unsigned char *)m->d_tc + img.size(), muf.data(), kDP * sizeof(float),
                            cudaMemcpyHostToDevice));
  m->tc_bytes = img.size();
  m->tc_tiles = nt;
  return GAPGB_OK;
}

size_t tc_atom_scratch_bytes(int N) {
  const size_t tiles = (size_t)(N + kRows - 1) / kRows;
  return tiles * kImgAtoms + (size_t)N * kDP * sizeof(float) + (size_t)N * sizeof(float) + 1024;
}

void launch_gpr_tc(gapgb_model *m, Workspace &ws, int N, cudaStream_t st, int a0, int a1) {
  const int D = m->host.D;
  if (a1 < 0) a1 = N;
  // the scratch layout is the whole batch's; the range's atoms start at tile a0 / 128
  const int tiles = (N + kRows - 1) / kRows;
  unsigned char *img_atoms = reinterpret_cast<unsigned char *>(ws.tc_scratch);
  float *xs = reinterpret_cast<float *>(img_atoms + (size_t)tiles * kImgAtoms);
  float *xn = xs + (size_t)N * kDP;
  const float *mu = reinterpret_cast<const float *>((const unsigned char *)m->d_tc + m->tc_bytes);
  const int n = a1 - a0, t0 = a0 / kRows, ct = (n + kRows - 1) / kRows;
  if (n <= 0) return;
  unsigned char *img_r = img_atoms + (size_t)t0 * kImgAtoms;
  float *xs_r = xs + (size_t)a0 * kDP, *xn_r = xn + a0;
  k_tc_prep_atoms<<<(ct * kRows + 127) / 128, 128, 0, st>>>(
      n, D, (const float *)ws.G + (size_t)a0 * D, m->d_invth32, mu, xs_r, xn_r, img_r);
  kernel_smem((const void *)k_gpr_tc, kSmemBytes, true);
  k_gpr_tc<<<ct, kGprThreads, kSmemBytes, st>>>(n, m->tc_tiles, (const unsigned char *)m->d_tc,
                                                img_r, xs_r, xn_r, m->d_invth32, D, ws.e + a0,
                                                (float *)ws.dedg + (size_t)a0 * D, ws.d_flags);
}

}  // namespace gapgb
