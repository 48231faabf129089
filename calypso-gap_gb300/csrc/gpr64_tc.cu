// gpr64_tc.cu - the FP64 sparse GPR on the 5th-generation tensor cores.
//
// Same quantities as gpr.cu (GET_COV and the energy / dE/dG loops of
// FGAP_CALC, gappy/libgap/gap_calc.f90:143-166, 268-288), for the FP64 and
// mixed forms.  On the CUDA cores they are bound by the FP64 pipe (1/64 of the
// FP32 rate): 4 N M D operations at 1.06 TFLOP/s.  Here both contractions are
// integer matrix products on tcgen05.mma: every FP64 operand becomes a
// fixed-point integer with a power-of-two scale per row and is cut into signed
// base-256 digits, which BF16 holds exactly; products of digits are at most
// 2^14, so FP32 accumulation of a tile is exact, and the sums of all digit
// pairs (i, j) with equal i + j share one accumulator (the error-free
// splitting of K. Ozaki, T. Ogita, S. Oishi and S. M. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numerical Algorithms 59, 2012).
//
//   x = (G - mean m) sqrt(log2 e) / theta, m likewise; z_ik = x_i.m_k - |x_i|^2/2
//   - |m_k|^2/2 + log2 |c_k|,  w_ik = sgn(c_k) 2^z,  e_i = sum_k w_ik,
//   dE/dG_id = -(x_id e_i - sum_k w_ik m_kd) / (theta_d sqrt(log2 e))
//
// k_g64_w: x.m from 8 + 8 digits (62 bits; the 36 pairs with i + j < 8), so
// that the expansion of |x - m|^2 loses nothing: z is formed modulo 2^64 in
// units of 2^-52, its error is 2^-53 plus 2^-59 max|x_i| max|m_k|, while the
// CUDA-core kernel rounds x/theta and m/theta themselves.  2^z is evaluated in
// integer arithmetic too (a 1024-entry table and a degree-4 polynomial): an
// FP64 instruction costs as much as 64 issue slots of the other pipes.
// k_g64_b: sum_k w m likewise, from the digits of w relative to the row's
// largest and of m relative to the column's, drained into integers every 128
// points.  (With 7 digits and the 28 pairs i + j < 7 the forces of ragged
// cells were 2.5 times as far from 64-bit values as the CUDA cores'.)  Row
// sums and partial sums are integers, so results do not depend on how the
// work is split; x e - sum w m is formed in double-double.
//
// Measured (ncu; all kernels of the stage, CUDA-core kernel -> these): 6.2 k
// ragged atoms x 2000 points 7143 -> 230 us, 512 atoms x 4000 points 1237 -> 80
// us, 64 atoms x 500 points 315 -> 45 us, so no size keeps the CUDA cores; D >
// 80 does (the digits of 128 atoms no longer fit in shared memory), and so
// does a model with scaled points beyond 2^6 (whose fixed point would be
// coarser than FP64).  What bounds it: the integer epilogue of k_g64_w (about
// 100 instructions per kernel value) and the MMAs of k_g64_b.  Rows of 128 atoms and 32 points per
// accumulator, because eight accumulators of 32 columns, twice, fill the 512
// TMEM columns: the MMAs of one tile run under the epilogue of the other.
#include <cuda_bf16.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "gapgb_internal.h"
#include "tc_util.cuh"

namespace gapgb {
namespace {

using namespace tc;
typedef unsigned long long u64;
typedef long long i64;

constexpr int kR = 128;        // rows (atoms) per CTA
constexpr int kT1 = 32;        // sparse points per tile of k_g64_w
constexpr int kS1 = 8;         // digits of x and m in k_g64_w
constexpr int kT2 = 32;        // sparse points per stage of k_g64_b
constexpr int kS2 = 8;         // digits of w and m in k_g64_b
constexpr int kN2 = 64;        // descriptor components per CTA of k_g64_b
constexpr int kDrain = 4;      // stages between drains of k_g64_b (128 points)
constexpr int kThreads = 288;  // 8 epilogue / conversion warps and one that issues
constexpr int kRowNaN = INT_MAX;

// constants of one sparse point: z's column term in units of 2^-52, the scale
// exponent of its digits (low byte, biased by 64) with sgn(c) on top, and the
// column term in FP32
struct Col {
  i64 b;
  unsigned es;
  float bf;
};
struct Row {
  i64 b;    // -|x|^2 / 2 in units of 2^-52
  int e;    // scale exponent of the row's digits
  float bf;  // the same in FP32; -1e30: every w of the row is zero
};

__host__ __device__ constexpr int slice1(int kd) { return kR * kd * 2; }       // bytes
__host__ __device__ constexpr int tile1(int kd) { return kS1 * kT1 * kd * 2; }
__host__ __device__ constexpr int nbuf1(int kd) { return kd <= 64 ? 2 : 1; }
constexpr int kSlice2 = kR * kT2 * 2;
constexpr int kA2 = kS2 * kSlice2;
constexpr int kB2 = kS2 * kN2 * kT2 * 2;

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}
// waits for the loads of all S x 8 registers; the empty statements make every
// use of a register depend on the wait
template <int S>
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[S][8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < S; ++q)
    asm volatile("" : "+r"(r[q][0]), "+r"(r[q][1]), "+r"(r[q][2]), "+r"(r[q][3]), "+r"(r[q][4]),
                      "+r"(r[q][5]), "+r"(r[q][6]), "+r"(r[q][7]));
}
__device__ __forceinline__ int f2i(uint32_t r) { return __float2int_rn(__uint_as_float(r)); }

// BF16 bits (upper half) of byte b of y less 128: exact
__device__ __forceinline__ uint32_t digit_f(uint32_t y, int b) {
  const uint32_t u = __byte_perm(y, 0x4B000000u, 0x7540 | b);  // 2^23 + byte
  return __float_as_uint(__uint_as_float(u) - 8388736.f);
}
__device__ __forceinline__ uint32_t pack_hi(uint32_t lo, uint32_t hi) {
  return __byte_perm(lo, hi, 0x7632);
}

// the S digits of eight K-adjacent values of one row, one 16-byte store per
// slice.  X = sum_i d_i 256^(S-1-i) with -128 <= d_i < 128, |X| < 2^(8 S - 2):
// adding 128 to every digit leaves the bytes d_i + 128
template <int S>
__device__ __forceinline__ void store_digits(const i64 (&X)[8], unsigned char *dst,
                                             int slice_bytes) {
  uint32_t pk[S][4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    uint32_t f[S][2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const u64 Y = (u64)X[2 * h + u] + 0x8080808080808080ull;
      const uint32_t lo = (uint32_t)Y, hi = (uint32_t)(Y >> 32);
#pragma unroll
      for (int i = 0; i < S; ++i) {
        const int byte = S - 1 - i;
        f[i][u] = digit_f(byte < 4 ? lo : hi, byte & 3);
      }
    }
#pragma unroll
    for (int i = 0; i < S; ++i) pk[i][h] = pack_hi(f[i][0], f[i][1]);
  }
#pragma unroll
  for (int i = 0; i < S; ++i)
    *reinterpret_cast<uint4 *>(dst + (size_t)i * slice_bytes) =
        make_uint4(pk[i][0], pk[i][1], pk[i][2], pk[i][3]);
}

// ---- operands ---------------------------------------------------------------

// mean of every descriptor component over the sparse points (fixed order)
__global__ void __launch_bounds__(256)
    k_g64_mean(int M, int D, const double *__restrict__ mm, double *__restrict__ mu) {
  __shared__ double red[256];
  const int d = blockIdx.x;
  double s = 0.0;
  for (int k = threadIdx.x; k < M; k += 256) s += mm[(size_t)k * D + d];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) mu[d] = red[0] / M;
}

// Scaled, centred values of 8 components of one row and the row's exponent,
// digits and norm: 16 lanes per row (8 components each).  Shared by atoms
// and sparse points.  Returns the norm |x|^2/2 in units of 2^-52 modulo 2^64
// on every lane; bf is it in FP32; e the exponent, |x| < 2^e.
__device__ __forceinline__ i64 row_digits(const double (&x)[8], int &e, float &bf,
                                          i64 (&X)[8], bool &nan) {
  int me = -1022;
  bool bad = false;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int h = __double2hiint(x[u]) & 0x7fffffff;
    bad |= x[u] != x[u];
    me = max(me, (h >> 20) - 1023);
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    me = max(me, __shfl_xor_sync(0xffffffffu, me, o));
    bad |= (bool)__shfl_xor_sync(0xffffffffu, (int)bad, o);
  }
  nan = bad;
  e = max(me + 1, -4);
  unsigned __int128 q2 = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    X[u] = e <= 9 ? __double2ll_rn(ldexp(x[u], 62 - e)) : 0;
    const i64 q = (X[u] + 2) >> 2;
    const u64 a = (u64)(q < 0 ? -q : q);
    q2 += (unsigned __int128)a * a;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const u64 lo = __shfl_xor_sync(0xffffffffu, (u64)q2, o);
    const u64 hi = __shfl_xor_sync(0xffffffffu, (u64)(q2 >> 64), o);
    q2 += ((unsigned __int128)hi << 64) | lo;
  }
  // sum q^2 2^(2 (e - 60)) / 2 in units of 2^-52
  const int sh = 69 - 2 * min(e, 9);
  const i64 n = (i64)(u64)((q2 + ((unsigned __int128)1 << (sh - 1))) >> sh);
  const double top = (double)(u64)(q2 >> 64) * 18446744073709551616.0 + (double)(u64)q2;
  bf = (float)ldexp(top, 2 * e - 121);
  return n;
}

// atoms: xh [N][D], the digit image of every 128-atom tile, row constants
template <typename TG>
__global__ void __launch_bounds__(128)
    k_g64_atoms(int N, int D, int KD, const TG *__restrict__ G, const double *__restrict__ mu,
                const double *__restrict__ scale, double *__restrict__ xh,
                unsigned char *__restrict__ img, Row *__restrict__ row, int *__restrict__ rowexp) {
  const int lane16 = threadIdx.x & 15;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 4);
  double x[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int d = lane16 * 8 + u;
    x[u] = 0.0;
    if (i < N && d < D) {
      x[u] = ((double)G[(size_t)i * D + d] - mu[d]) * scale[d];
      xh[(size_t)i * D + d] = x[u];
    }
  }
  int e;
  float bf;
  i64 X[8];
  bool nan;
  const i64 n = row_digits(x, e, bf, X, nan);
  unsigned char *tile = img + (size_t)(i / kR) * kS1 * slice1(KD);
  if (lane16 * 8 < KD)
    store_digits<kS1>(X, tile + kmajor_off(i % kR, lane16 * 8, KD / 8), slice1(KD));
  if (lane16 == 0) {
    // beyond 2^9 (every |m| is below 2^6) and past the last atom: all w zero
    const bool far = i >= N || nan || e > 9;
    row[i] = {far ? 0 : -n, far ? 0 : e, far ? -1e30f : -bf};
    rowexp[i] = nan && i < N ? kRowNaN : INT_MIN;
  }
}

// sparse points: mh [M][D] scaled and centred, the stacked digit image of
// every 32-point tile (rows slice * 32 + point), the column constants without
// coefficients, and the largest exponent of the model
__global__ void __launch_bounds__(128)
    k_g64_points(int M, int Mp, int D, int KD, const double *__restrict__ mm,
                 const double *__restrict__ mu, const double *__restrict__ scale,
                 double *__restrict__ mh, unsigned char *__restrict__ img, Col *__restrict__ col,
                 int *__restrict__ emax) {
  const int lane16 = threadIdx.x & 15;
  const int k = blockIdx.x * 8 + (threadIdx.x >> 4);
  double x[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int d = lane16 * 8 + u;
    x[u] = 0.0;
    if (k < M && d < D) {
      x[u] = (mm[(size_t)k * D + d] - mu[d]) * scale[d];
      mh[(size_t)k * D + d] = x[u];
    }
  }
  int e;
  float bf;
  i64 X[8];
  bool nan;
  const i64 n = row_digits(x, e, bf, X, nan);
  if (k >= Mp) return;
  unsigned char *tile = img + (size_t)(k / kT1) * tile1(KD);
  if (lane16 * 8 < KD)
    store_digits<kS1>(X, tile + kmajor_off(k % kT1, lane16 * 8, KD / 8), kT1 * KD * 2);
  if (lane16 == 0) {
    col[k] = {k < M ? -n : 0, (unsigned)(e + 64), k < M ? -bf : -1e30f};
    if (k < M) atomicMax(emax, nan ? 99 : e);
  }
}

// column constants with the coefficients: + log2 |c_k|, and sgn(c_k)
__global__ void k_g64_coeff(int M, int Mp, const Col *__restrict__ unit,
                            const double *__restrict__ c, Col *__restrict__ col) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= Mp) return;
  Col o = unit[k];
  if (k < M) {
    const double a = fabs(c[k]);
    if (a == 0.0) {
      o.b = 0;
      o.bf = -1e30f;
    } else {
      int ex;
      const double f = frexp(a, &ex);  // [0.5, 1)
      o.b += ((i64)ex << 52) + __double2ll_rn(ldexp(log2(f), 52));
      o.bf += (float)ex + (float)log2(f);
    }
    if (c[k] < 0.0) o.es |= 0x80000000u;
  }
  col[k] = o;
}

// per component: exponent of the largest |m|, then the digit image of every
// 32-point stage (rows slice * 64 + component, K = points) of column tile y
__global__ void __launch_bounds__(256)
    k_g64_image2(int M, int nst, int D, const double *__restrict__ mh,
                 unsigned char *__restrict__ img, int *__restrict__ eD) {
  __shared__ int red[256];
  const int d = blockIdx.x, tid = threadIdx.x;
  int me = -1022;
  if (d < D)
    for (int k = tid; k < M; k += 256)
      me = max(me, ((__double2hiint(mh[(size_t)k * D + d]) & 0x7fffffff) >> 20) - 1023);
  red[tid] = me;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) red[tid] = max(red[tid], red[tid + w]);
    __syncthreads();
  }
  const int e = max(red[0] + 1, -60);
  if (tid == 0) eD[d] = e;
  unsigned char *base = img + (size_t)(d / kN2) * nst * kB2;
  for (int g = tid; g < nst * (kT2 / 8); g += 256) {
    const int st = g / (kT2 / 8), k0 = (g % (kT2 / 8)) * 8;
    i64 X[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = st * kT2 + k0 + u;
      X[u] = d < D && k < M ? __double2ll_rn(ldexp(mh[(size_t)k * D + d], 62 - e)) : 0;
    }
    store_digits<kS2>(X, base + (size_t)st * kB2 + kmajor_off(d % kN2, k0, kT2 / 8),
                      kN2 * kT2 * 2);
  }
}

// ---- kernel values ------------------------------------------------------------

// 2^f, f in units of 2^-52 below one, as a 1.63 fixed-point number
__device__ __forceinline__ u64 exp2_fix(u64 f, const u64 *__restrict__ T) {
  const u64 t = T[(uint32_t)(f >> 42) & (kExpN - 1)];
  // y = rho ln 2 in units of 2^-74, rho the part below 2^-10
  const u64 y = __umul64hi((f & ((1ull << 42) - 1)) << 22, 0xB17217F7D1CF79ACull);
  const u64 y2 = __umul64hi(y, y);                                   // 2^-84
  const uint32_t yh = (uint32_t)(y >> 32);                           // 2^-42
  const uint32_t y3 = __umulhi((uint32_t)(y2 >> 32), yh);            // 2^-62
  const uint32_t y4 = __umulhi(y3, yh);                              // 2^-72
  const u64 p = y + (y2 >> 11) +
                ((u64)(__umulhi(y3, 0x2AAAAAABu) + (__umulhi(y4, 0x0AAAAAABu) >> 10)) << 12);
  return t + (__umul64hi(t, p) >> 10);
}

template <int KD>
__global__ void __launch_bounds__(kThreads, 1)
    k_g64_w(int ntile, int Mp, const unsigned char *__restrict__ ximg,
            const Row *__restrict__ row, const unsigned char *__restrict__ mimg,
            const Col *__restrict__ col, const u64 *__restrict__ tab, double *__restrict__ W,
            int *__restrict__ rowexp, int *__restrict__ flags) {
  constexpr int NB = nbuf1(KD), kc = KD / 8;
  constexpr int oB = kS1 * slice1(KD), oT = oB + NB * tile1(KD), oC = oT + kExpN * 8,
                oBar = oC + 4 * kT1 * 16;
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sb = smem_u32(sm);
  const uint32_t bfull = sb + oBar, bempty = bfull + 16, dfull = bempty + 16, dempty = dfull + 16;
  uint32_t *slot = reinterpret_cast<uint32_t *>(sm + oBar + 64);
  volatile int *abort_flag = reinterpret_cast<int *>(sm + oBar + 72);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(bfull + 8 * b, 1);
      mbar_init(bempty + 8 * b, 1);
      mbar_init(dfull + 8 * b, 1);
      mbar_init(dempty + 8 * b, 8);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int q = tid; q < kExpN; q += kThreads) reinterpret_cast<u64 *>(sm + oT)[q] = tab[q];
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *slot;
  const int per = (ntile + gridDim.y - 1) / gridDim.y;
  const int t0 = blockIdx.y * per, t1 = min(ntile, t0 + per), nt = t1 - t0;
  if (warp == 8) {
    if (lane == 0 && nt > 0) {
      auto load = [&](int t) {  // tile t0 + t
        const uint32_t bar = bfull + 8 * (t % NB);
        mbar_expect_tx(bar, tile1(KD) + kT1 * 16 + (t == 0 ? kS1 * slice1(KD) : 0));
        if (t == 0)
          for (int i = 0; i < kS1; ++i)
            bulk_g2s(sb + i * slice1(KD),
                     ximg + ((size_t)blockIdx.x * kS1 + i) * slice1(KD), slice1(KD), bar);
        bulk_g2s(sb + oB + (t % NB) * tile1(KD), mimg + (size_t)(t0 + t) * tile1(KD), tile1(KD), bar);
        bulk_g2s(sb + oC + (t & 3) * kT1 * 16, col + (size_t)(t0 + t) * kT1, kT1 * 16, bar);
      };
      int loaded = 0, waited = 0;
      for (; loaded < NB && loaded < nt; ++loaded) load(loaded);
      bool ok = true;
      int t = 0, issued = 0;  // tiles whose MMAs are under way
      for (; t < nt && ok; ++t) {
        ok = mbar_wait(bfull + 8 * (t % NB), (t / NB) & 1, flags);
        if (!ok) break;
        ++waited;
        if (t >= 2) ok = mbar_wait(dempty + 8 * (t & 1), ((t >> 1) - 1) & 1, flags);
        if (!ok || *abort_flag) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t D = tmem + (t & 1) * 256, B = sb + oB + (t % NB) * tile1(KD);
        for (int kk = 0; kk < KD / 16; ++kk)
          for (int i = 0; i < kS1; ++i)
            umma(D + kT1 * i, smem_desc(sb + i * slice1(KD) + kk * 256, 128, kc * 128),
                 smem_desc(B + kk * 256, 128, kc * 128), instr_desc(kR, kT1 * (kS1 - i)),
                 (kk > 0 || i > 0) ? 1u : 0u);
        umma_commit(dfull + 8 * (t & 1));
        umma_commit(bempty + 8 * (t % NB));
        issued = t + 1;
        const int f = t - (NB - 1);  // the tile whose buffer is refilled
        if (loaded < nt && f >= 0) {
          ok = mbar_wait(bempty + 8 * (f % NB), (f / NB) & 1, flags);
          if (!ok) break;
          load(loaded++);
        }
      }
      if (t < nt) *abort_flag = 1;
      // a wait gave up: one more bounded wait for each copy still in flight; and
      // for the last MMAs, before the tensor memory goes
      for (; waited < loaded; ++waited) mbar_wait(bfull + 8 * (waited % NB), (waited / NB) & 1, flags);
      if (issued > 0) mbar_wait(bempty + 8 * ((issued - 1) % NB), ((issued - 1) / NB) & 1, flags);
    }
  } else {
    const int quad = warp & 3, half = warp >> 2;
    const int r = quad * 32 + lane;
    const Row rw = row[(size_t)blockIdx.x * kR + r];
    const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16) + 16 * half;
    const u64 *T = reinterpret_cast<const u64 *>(sm + oT);
    int emax = INT_MIN;
    for (int t = 0; t < nt; ++t) {
      // (a warp gives up as one: the TMEM loads and __syncwarp below need all of it)
      if (!__all_sync(0xffffffffu, mbar_wait(dfull + 8 * (t & 1), (t >> 1) & 1, flags) &&
                                       !*abort_flag)) {
        *abort_flag = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const Col *cs = reinterpret_cast<const Col *>(sm + oC + (t & 3) * kT1 * 16) + 16 * half;
      double *out = W + ((size_t)blockIdx.x * Mp + (size_t)(t0 + t) * kT1 + 16 * half) * kR + r;
#pragma unroll 1
      for (int g = 0; g < 2; ++g) {
        uint32_t a[kS1][8];
#pragma unroll
        for (int w = 0; w < kS1; ++w) tmem_ld8(lb + (t & 1) * 256 + kT1 * w + 8 * g, a[w]);
        tmem_ld_wait(a);
        if (g == 1) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(dempty + 8 * (t & 1));
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const Col c = cs[8 * g + q];
          const int E = rw.e + (int)(c.es & 255u) - 64;
          // sum_w a_w 2^(40 - 8 w + E) in units of 2^-52, modulo 2^64
          const i64 H = (i64)(f2i(a[0][q]) * 256 + f2i(a[1][q])) * 65536 +
                        (f2i(a[2][q]) * 256 + f2i(a[3][q]));
          const i64 L = (i64)(f2i(a[4][q]) * 256 + f2i(a[5][q])) * 65536 +
                        ((i64)f2i(a[6][q]) * 256 + f2i(a[7][q]));
          const i64 z = (H << (16 + E)) + ((L + (1ll << (15 - E))) >> (16 - E)) + rw.b + c.b;
          // the same in FP32 decides whether z is in range at all
          const float zf = fmaf(fmaf(__uint_as_float(a[2][q]), 1.f / 65536.f,
                                     fmaf(__uint_as_float(a[1][q]), 1.f / 256.f,
                                          __uint_as_float(a[0][q]))),
                                __int_as_float((E + 127 - 12) << 23), rw.bf + c.bf);
          const bool in = zf > -1020.f;
          const int n = (int)(z >> 52);
          const u64 m = exp2_fix((u64)z & ((1ull << 52) - 1), T);
          u64 bits = ((u64)(uint32_t)(n + 1022) << 52) + (m >> 11) + ((m >> 10) & 1);
          bits |= (u64)(c.es & 0x80000000u) << 32;
          if (in) emax = max(emax, n);
          out[(size_t)(8 * g + q) * kR] = in ? __longlong_as_double((i64)bits) : 0.0;
        }
      }
    }
    if (rowexp && emax > INT_MIN) atomicMax(rowexp + (size_t)blockIdx.x * kR + r, emax);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ---- sum_k w_ik m_kd -----------------------------------------------------------

__global__ void __launch_bounds__(kThreads, 1)
    k_g64_b(int nst, int Mp, const double *__restrict__ W, const int *__restrict__ rowexp,
            const unsigned char *__restrict__ img, longlong2 *__restrict__ part,
            longlong2 *__restrict__ epart, int *__restrict__ flags) {
  constexpr int oB = 2 * kA2, oBar = oB + 2 * kB2;
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sb = smem_u32(sm);
  const uint32_t afull = sb + oBar, bfull = afull + 16, sempty = bfull + 16, dfull = sempty + 16,
                 dempty = dfull + 8;
  uint32_t *slot = reinterpret_cast<uint32_t *>(sm + oBar + 64);
  volatile int *abort_flag = reinterpret_cast<int *>(sm + oBar + 72);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(afull + 8 * b, 8);
      mbar_init(bfull + 8 * b, 1);
      mbar_init(sempty + 8 * b, 1);
    }
    mbar_init(dfull, 1);
    mbar_init(dempty, 8);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *slot;
  // this split's stages, whole drain groups
  const int ng = (nst + kDrain - 1) / kDrain, pg = (ng + gridDim.y - 1) / gridDim.y;
  const int s0 = min(nst, (int)blockIdx.y * pg * kDrain), s1 = min(nst, s0 + pg * kDrain);
  const int ns = s1 - s0;
  const size_t pslot = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  if (warp == 8) {
    if (lane == 0 && ns > 0) {
      const unsigned char *src = img + ((size_t)blockIdx.z * nst + s0) * kB2;
      auto load = [&](int s) {
        mbar_expect_tx(bfull + 8 * (s & 1), kB2);
        bulk_g2s(sb + oB + (s & 1) * kB2, src + (size_t)s * kB2, kB2, bfull + 8 * (s & 1));
      };
      int loaded = 0, waited = 0;
      for (; loaded < 2 && loaded < ns; ++loaded) load(loaded);
      bool ok = true;
      int s = 0, issued = 0;
      for (; s < ns && ok; ++s) {
        ok = mbar_wait(bfull + 8 * (s & 1), (s >> 1) & 1, flags);
        if (!ok) break;
        ++waited;
        ok = mbar_wait(afull + 8 * (s & 1), (s >> 1) & 1, flags);
        if (ok && s > 0 && s % kDrain == 0) ok = mbar_wait(dempty, (s / kDrain - 1) & 1, flags);
        if (!ok || *abort_flag) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t A = sb + (s & 1) * kA2, B = sb + oB + (s & 1) * kB2;
        for (int kk = 0; kk < kT2 / 16; ++kk)
          for (int i = 0; i < kS2; ++i) {
            const uint64_t ad = smem_desc(A + i * kSlice2 + kk * 256, 128, (kT2 / 8) * 128);
            const int n = kN2 * (kS2 - i), n0 = n < 256 ? n : 256;
            const uint32_t acc = (s % kDrain > 0 || kk > 0 || i > 0) ? 1u : 0u;
            umma(tmem + kN2 * i, ad, smem_desc(B + kk * 256, 128, (kT2 / 8) * 128),
                 instr_desc(kR, n0), acc);
            if (n > 256)
              umma(tmem + kN2 * i + 256, ad,
                   smem_desc(B + (256 / 8) * (kT2 / 8) * 128 + kk * 256, 128, (kT2 / 8) * 128),
                   instr_desc(kR, n - 256), acc);
          }
        umma_commit(sempty + 8 * (s & 1));
        issued = s + 1;
        if (s % kDrain == kDrain - 1 || s == ns - 1) umma_commit(dfull);
        if (loaded < ns && s > 0) {
          ok = mbar_wait(sempty + 8 * ((s - 1) & 1), ((s - 1) >> 1) & 1, flags);
          if (!ok) break;
          load(loaded++);
        }
      }
      if (s < ns) *abort_flag = 1;
      for (; waited < loaded; ++waited) mbar_wait(bfull + 8 * (waited & 1), (waited >> 1) & 1, flags);
      if (issued > 0) mbar_wait(sempty + 8 * ((issued - 1) & 1), ((issued - 1) >> 1) & 1, flags);
    }
  } else {
    const int quad = warp & 3, half = warp >> 2;
    const int r = quad * 32 + lane;
    const int re = rowexp[(size_t)blockIdx.x * kR + r];
    const double *w = W + ((size_t)blockIdx.x * Mp + (size_t)s0 * kT2 + 16 * half) * kR + r;
    const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16) + 32 * half;
    i64 aH[32], aL[32];
#pragma unroll
    for (int q = 0; q < 32; ++q) aH[q] = aL[q] = 0;
    __int128 es = 0;
    bool ok = true;
    double nx[16];  // the next stage's values, loaded one stage ahead
#pragma unroll
    for (int q = 0; q < 16; ++q) nx[q] = ns > 0 ? w[(size_t)q * kR] : 0.0;
    for (int s = 0; s < ns; ++s) {
      double v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = nx[q];
      if (s + 1 < ns) {
#pragma unroll
        for (int q = 0; q < 16; ++q) nx[q] = w[((size_t)(s + 1) * kT2 + q) * kR];
      }
      // (a warp gives up as one, here and below)
      ok = s < 2 || mbar_wait(sempty + 8 * (s & 1), ((s >> 1) - 1) & 1, flags);
      ok = __all_sync(0xffffffffu, ok && !*abort_flag) != 0;
      if (!ok) break;
      unsigned char *dst = sm + (s & 1) * kA2;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        i64 X[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          // w / 2^(re + 1 - 62), rounded: |X| < 2^62
          const u64 b = (u64)__double_as_longlong(v[8 * g + q]);
          const int ex = (int)(b >> 52) & 0x7ff;
          const u64 mant = ((b & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 9;
          const int d = re + 1023 - ex;
          i64 x = d <= 0 ? (i64)mant : (d < 63 ? (i64)((mant + (1ull << (d - 1))) >> d) : 0);
          if (ex == 0) x = 0;
          X[q] = (b >> 63) ? -x : x;
          es += X[q];
        }
        store_digits<kS2>(X, dst + kmajor_off(r, 16 * half + 8 * g, kT2 / 8), kSlice2);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(afull + 8 * (s & 1));
      if (s % kDrain == kDrain - 1 || s == ns - 1) {
        ok = __all_sync(0xffffffffu, mbar_wait(dfull, (s / kDrain) & 1, flags) && !*abort_flag) != 0;
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t a[kS2][8];
#pragma unroll
          for (int c = 0; c < kS2; ++c) tmem_ld8(lb + kN2 * c + 8 * g, a[c]);
          tmem_ld_wait(a);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            aH[8 * g + q] += (i64)(f2i(a[0][q]) * 256 + f2i(a[1][q])) * 65536 +
                             ((i64)f2i(a[2][q]) * 256 + f2i(a[3][q]));
            aL[8 * g + q] += ((i64)f2i(a[4][q]) * 256 + f2i(a[5][q])) * 65536 +
                             ((i64)f2i(a[6][q]) * 256 + f2i(a[7][q]));
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(dempty);
      }
    }
    if (!ok) *abort_flag = 1;
#pragma unroll
    for (int q = 0; q < 32; ++q)
      part[(pslot * kN2 + 32 * half + q) * kR + r] = make_longlong2(aH[q], aL[q]);
    if (blockIdx.z == 0)
      epart[(((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 2 + half) * kR + r] =
          make_longlong2((i64)(u64)es, (i64)(es >> 64));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// e and dE/dG of one tile of 128 atoms: the splits' integer sums, in FP64
template <typename TG>
__global__ void __launch_bounds__(kR)
    k_g64_final(int N, int D, int i0, int splits, int ntile, const longlong2 *__restrict__ part,
                const longlong2 *__restrict__ epart, const int *__restrict__ rowexp,
                const int *__restrict__ eD, const double *__restrict__ xh,
                const double *__restrict__ unscale, double *__restrict__ e_out,
                TG *__restrict__ dedg) {
  const int tile = blockIdx.x, r = threadIdx.x, d = blockIdx.y;
  const int i = i0 + tile * kR + r;
  if (i >= N) return;
  const int re = rowexp[i];
  __int128 s = 0;
  for (int p = 0; p < splits; ++p)
    for (int h = 0; h < 2; ++h) {
      const longlong2 v = epart[(((size_t)p * ntile + tile) * 2 + h) * kR + r];
      s += ((__int128)v.y << 64) | (u64)v.x;
    }
  const int sc = re == INT_MIN || re == kRowNaN ? 0 : re + 1;
  // e and v = sum w m as unevaluated sums of two doubles, and x e - v from them
  const double eh = (double)(i64)(s >> 24) * 16777216.0;
  const double el = (double)(i64)(s - (__int128)(i64)(s >> 24) * 16777216) +
                    16777216.0 * (double)((i64)(s >> 24) - (i64)(double)(i64)(s >> 24));
  double e = ldexp(eh + el, sc - 62);
  if (re == kRowNaN) e = nan("");
  if (d == 0) e_out[i] = e;
  i64 H = 0, L = 0;
  const int z = d / kN2, c = d % kN2;
  for (int p = 0; p < splits; ++p) {
    const longlong2 v = part[((((size_t)z * splits + p) * ntile + tile) * kN2 + c) * kR + r];
    H += v.x;
    L += v.y;
  }
  const double vs = ldexp(1.0, eD[d] - 6);  // v / e's unit: 2^(eD - 68 + 62)
  const double vh = (double)H * 4294967296.0 * vs;
  const double vl = ((double)L + 4294967296.0 * (double)(H - (i64)(double)H)) * vs;
  const double x = xh[(size_t)i * D + d];
  const double ph = x * eh;
  const double pl = fma(x, eh, -ph) + x * el;
  const double g = ldexp((ph - vh) + (pl - vl), sc - 62);
  dedg[(size_t)i * D + d] = (TG)(re == kRowNaN ? e : -unscale[d] * g);
}

// phi[s][k] += sum over the structures' atoms within [i0, i1) of K_ik (W: the
// kernel values of the row tiles from i0 on); the first part of a structure
// sets.  A warp per (structure, point), lanes over rows: fixed order.  An atom
// whose descriptors are not numbers (its W is zero) makes the sum NaN.
__global__ void __launch_bounds__(256)
    k_g64_phi(int i0, int i1, int Mp, int Mf, const int *__restrict__ off,
              const int *__restrict__ rowexp, const double *__restrict__ W,
              double *__restrict__ phi) {
  const int s = blockIdx.y, lane = threadIdx.x & 31;
  const int k = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int a0 = max(off[s], i0), a1 = min(off[s + 1], i1);
  if (k >= Mf || (a0 >= a1 && off[s] != off[s + 1])) return;
  double v = 0.0;
  for (int i = a0 + lane; i < a1; i += 32)
    v += rowexp[i] == kRowNaN ? nan("") : W[((size_t)((i - i0) / kR) * Mp + k) * kR + (i - i0) % kR];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) {
    double *p = phi + (size_t)s * Mf + k;
    *p = off[s] >= i0 ? v : *p + v;
  }
}

// A[i0 + r][k] = K(m_r, m_k) of one row tile (rows and columns below M; the
// padded columns zero), transposed through shared memory
__global__ void __launch_bounds__(256)
    k_g64_kmm(int M, int i0, int Mp, int Mf, const double *__restrict__ W, double *__restrict__ A) {
  __shared__ double t[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int r0 = blockIdx.y * 32, k0 = blockIdx.x * 32;  // r0 within the chunk's rows
  for (int q = ty; q < 32; q += 8)
    t[q][tx] = W[((size_t)(r0 / kR) * Mp + k0 + q) * kR + r0 % kR + tx];
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int r = i0 + r0 + q, k = k0 + tx;
    if (r < M && k < Mf) A[(size_t)r * Mf + k] = k < M ? t[tx][q] : 0.0;
  }
}

size_t smem1(int kd) {
  return (size_t)kS1 * slice1(kd) + nbuf1(kd) * tile1(kd) + kExpN * 8 + 4 * kT1 * 16 + 128 + 1024;
}
constexpr size_t kSmem2 = 2 * (size_t)(kA2 + kB2) + 128 + 1024;

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

const u64 *exp2_table() {
  static const std::vector<u64> T = [] {
    // 2^(j/1024) in 1.63 fixed point: products of the successive square roots of 2
    typedef unsigned __int128 u128;
    std::vector<u64> v(kExpN, (u64)1 << 63);
    u128 sq = (u128)1 << 127;  // 2 in 2.126
    for (int b = kExpN / 2; b > 0; b >>= 1) {
      u64 x = (u64)(std::sqrt((double)(u64)(sq >> 64)) * 4294967296.0);
      for (int it = 0; it < 3; ++it) x = (u64)(((u128)x + sq / x) >> 1);
      for (int j = 0; j < kExpN; ++j)
        if (j & b) v[j] = (u64)(((u128)v[j] * x + ((u128)1 << 62)) >> 63);
      sq = (u128)x << 63;
    }
    return v;
  }();
  return T.data();
}

// device image of a model: layout offsets from m->d_g64
struct G64 {
  int KD, Mp, nt1, nst, nz;
  size_t mu, scale, unscale, mh, img1, col, colc, img2, eD, tab, emax, mm, bytes;
};
static G64 g64_layout(int M, int D) {
  G64 g;
  g.KD = D <= 64 ? 64 : 80;
  g.Mp = (M + kDrain * kT2 - 1) / (kDrain * kT2) * (kDrain * kT2);
  g.nt1 = g.Mp / kT1;
  g.nst = g.Mp / kT2;
  g.nz = (D + kN2 - 1) / kN2;
  size_t o = 0;
  auto take = [&](size_t &at, size_t n) { at = o, o += up256(n); };
  take(g.mu, 8 * (size_t)D);
  take(g.scale, 8 * (size_t)D);
  take(g.unscale, 8 * (size_t)D);
  take(g.mh, 8 * (size_t)M * D);
  take(g.mm, 8 * (size_t)M * D);
  take(g.img1, (size_t)g.nt1 * tile1(g.KD));
  take(g.col, sizeof(Col) * (size_t)g.Mp);
  take(g.colc, sizeof(Col) * (size_t)g.Mp);
  take(g.img2, (size_t)g.nz * g.nst * kB2);
  take(g.eD, 4 * (size_t)g.nz * kN2);
  take(g.tab, 8 * (size_t)kExpN);
  take(g.emax, 16);
  g.bytes = o;
  return g;
}

// The image, for models of D <= 80 whose scaled sparse points stay below 2^6
// (others keep the CUDA-core kernel); coefficients are refreshed in place.
gapgb_status g64_prepare(gapgb_model *m, bool refresh) {
  const HostModel &h = m->host;
  if (refresh && !m->d_g64) return GAPGB_OK;
  if (!refresh && m->g64_tried) return GAPGB_OK;
  m->g64_tried = true;
  m->g64_finite = std::all_of(h.coeff.begin(), h.coeff.end(), [](double c) { return std::isfinite(c); });
  const int M = h.M, D = h.D;
  if (D > 80) return GAPGB_OK;
  const G64 g = g64_layout(M, D);
  unsigned char *p = m->d_g64;
  if (!refresh) {
    GAPGB_CUDA_TRY(cudaMalloc(&p, g.bytes));
    const double root = std::sqrt(1.4426950408889634074);
    std::vector<double> sc(2 * (size_t)up256(8 * (size_t)D) / 8);
    for (int d = 0; d < D; ++d) {
      sc[d] = root / h.theta[d];
      sc[up256(8 * (size_t)D) / 8 + d] = 1.0 / (h.theta[d] * root);
    }
    cudaError_t e = cudaMemcpyAsync(p + g.scale, sc.data(), 8 * sc.size(), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(p + g.mm, h.mm.data(), 8 * h.mm.size(), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(p + g.tab, exp2_table(), 8 * (size_t)kExpN, cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(p + g.emax, 0x80, 16, m->stream);
    const double *mu = (const double *)(p + g.mu), *scale = (const double *)(p + g.scale);
    k_g64_mean<<<D, 256, 0, m->stream>>>(M, D, (const double *)(p + g.mm), (double *)(p + g.mu));
    k_g64_points<<<(g.Mp + 7) / 8, 128, 0, m->stream>>>(M, g.Mp, D, g.KD, (const double *)(p + g.mm),
                                                        mu, scale, (double *)(p + g.mh), p + g.img1,
                                                        (Col *)(p + g.col), (int *)(p + g.emax));
    k_g64_image2<<<g.nz * kN2, 256, 0, m->stream>>>(M, g.nst, D, (const double *)(p + g.mh),
                                                    p + g.img2, (int *)(p + g.eD));
    int emax = 99;
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(&emax, p + g.emax, 4, cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess || emax > 6) {
      cudaFree(p);
      if (e != cudaSuccess) {
        set_last_error(std::string("GPR image: ") + cudaGetErrorString(e));
        return GAPGB_ERR_CUDA;
      }
      return GAPGB_OK;
    }
  }
  k_g64_coeff<<<(g.Mp + 127) / 128, 128, 0, m->stream>>>(M, g.Mp, (const Col *)(p + g.col),
                                                         m->d_coeff, (Col *)(p + g.colc));
  GAPGB_CUDA_TRY(cudaGetLastError());
  GAPGB_CUDA_TRY(cudaStreamSynchronize(m->stream));
  m->d_g64 = p;
  return GAPGB_OK;
}

// scratch of one launch over N atoms: operands of all of them, kernel values
// and partial sums of `ct` row tiles at a time
struct G64Run {
  int tiles, ct, sa, sb, slots;
  size_t xh, img, row, rowexp, W, part, epart, bytes;
};
static G64Run g64_run(const G64 &g, int N, int D) {
  G64Run r;
  r.tiles = (N + kR - 1) / kR;
  const int sms = device_sms();
  // at most one row tile per SM at a time, and 768 MB of kernel values
  const size_t per = (size_t)g.Mp * kR * 8;
  r.ct = (int)std::max<size_t>(1, std::min<size_t>({(size_t)r.tiles, (size_t)sms, ((size_t)768 << 20) / per}));
  r.sa = std::max(1, std::min(g.nt1, sms / r.ct));
  r.sb = std::max(1, std::min(g.nst / kDrain, sms / (r.ct * g.nz)));
  // partial sums: the most that any batch up to N takes (sb ct is not monotone
  // in N), so that a smaller batch fits into a larger one's scratch
  r.slots = std::max(r.ct, std::min(r.ct * (g.nst / kDrain), sms / g.nz));
  size_t o = 0;
  auto take = [&](size_t &at, size_t n) { at = o, o += up256(n); };
  take(r.xh, 8 * (size_t)N * D);
  take(r.img, (size_t)r.tiles * kS1 * slice1(g.KD));
  take(r.row, sizeof(Row) * (size_t)r.tiles * kR);
  take(r.rowexp, 4 * (size_t)r.tiles * kR);
  take(r.W, per * r.ct);
  take(r.part, sizeof(longlong2) * (size_t)g.nz * r.slots * kN2 * kR);
  take(r.epart, sizeof(longlong2) * (size_t)r.slots * 2 * kR);
  r.bytes = o;
  return r;
}

static bool g64_scratch(const G64 &g, Workspace &ws, int N, int D, const G64Run &r, cudaStream_t st) {
  return grow_scratch(ws, &ws.g64_scratch, &ws.g64_bytes, g64_run(g, std::max(N, ws.N), D).bytes,
                      r.bytes, st);
}

// The FP64 GPR of N atoms; false (nothing launched) when the model has no
// image, a coefficient is not finite (fixed point has no NaN: the CUDA-core
// kernel carries it into the results) or the scratch cannot be had (grow_scratch).
template <typename TG>
bool launch_gpr64(const gapgb_model *m, Workspace &ws, int N, cudaStream_t st) {
  if (!m->d_g64 || !m->g64_finite) return false;
  const int M = m->host.M, D = m->host.D;
  const G64 g = g64_layout(M, D);
  const G64Run r = g64_run(g, N, D);
  if (!g64_scratch(g, ws, N, D, r, st)) return false;
  const unsigned char *p = m->d_g64;
  unsigned char *q = (unsigned char *)ws.g64_scratch;
  Row *row = (Row *)(q + r.row);
  int *rowexp = (int *)(q + r.rowexp);
  double *xh = (double *)(q + r.xh);
  k_g64_atoms<TG><<<r.tiles * (kR / 8), 128, 0, st>>>(
      N, D, g.KD, (const TG *)ws.G, (const double *)(p + g.mu), (const double *)(p + g.scale), xh,
      q + r.img, row, rowexp);
  auto fw = g.KD == 64 ? k_g64_w<64> : k_g64_w<80>;
  kernel_smem((const void *)fw, (int)smem1(g.KD), true);
  kernel_smem((const void *)k_g64_b, (int)kSmem2, true);
  for (int c0 = 0; c0 < r.tiles; c0 += r.ct) {
    const int ct = std::min(r.ct, r.tiles - c0);
    fw<<<dim3(ct, r.sa), kThreads, smem1(g.KD), st>>>(
        g.nt1, g.Mp, q + r.img + (size_t)c0 * kS1 * slice1(g.KD), row + (size_t)c0 * kR,
        p + g.img1, (const Col *)(p + g.colc), (const u64 *)(p + g.tab), (double *)(q + r.W),
        rowexp + (size_t)c0 * kR, ws.d_flags);
    k_g64_b<<<dim3(ct, r.sb, g.nz), kThreads, kSmem2, st>>>(
        g.nst, g.Mp, (const double *)(q + r.W), rowexp + (size_t)c0 * kR, p + g.img2,
        (longlong2 *)(q + r.part), (longlong2 *)(q + r.epart), ws.d_flags);
    k_g64_final<TG><<<dim3(ct, D), kR, 0, st>>>(
        N, D, c0 * kR, r.sb, ct, (const longlong2 *)(q + r.part), (const longlong2 *)(q + r.epart),
        rowexp, (const int *)(p + g.eD), xh, (const double *)(p + g.unscale), ws.e, (TG *)ws.dedg);
  }
  return true;
}

// Kernel values without coefficients, for the fit: row tiles in chunks.
// use(first row, row tiles, every row's rowexp, W) enqueues what reads them.
template <typename F>
static bool g64_kernel_values(const gapgb_model *m, Workspace &ws, int N, const double *X,
                              cudaStream_t st, F use) {
  if (!m->d_g64) return false;
  const int M = m->host.M, D = m->host.D;
  const G64 g = g64_layout(M, D);
  const G64Run r = g64_run(g, N, D);
  if (!g64_scratch(g, ws, N, D, r, st)) return false;
  const unsigned char *p = m->d_g64;
  unsigned char *q = (unsigned char *)ws.g64_scratch;
  Row *row = (Row *)(q + r.row);
  k_g64_atoms<double><<<r.tiles * (kR / 8), 128, 0, st>>>(
      N, D, g.KD, X, (const double *)(p + g.mu), (const double *)(p + g.scale),
      (double *)(q + r.xh), q + r.img, row, (int *)(q + r.rowexp));
  auto fw = g.KD == 64 ? k_g64_w<64> : k_g64_w<80>;
  kernel_smem((const void *)fw, (int)smem1(g.KD), true);
  for (int c0 = 0; c0 < r.tiles; c0 += r.ct) {
    const int ct = std::min(r.ct, r.tiles - c0);
    fw<<<dim3(ct, r.sa), kThreads, smem1(g.KD), st>>>(
        g.nt1, g.Mp, q + r.img + (size_t)c0 * kS1 * slice1(g.KD), row + (size_t)c0 * kR,
        p + g.img1, (const Col *)(p + g.col), (const u64 *)(p + g.tab), (double *)(q + r.W),
        nullptr, ws.d_flags);
    use(c0 * kR, ct, (const int *)(q + r.rowexp), (const double *)(q + r.W));
  }
  return true;
}

// phi[S][Mf]: sums of the kernel values over each structure's atoms
bool launch_phi64(const gapgb_model *m, Workspace &ws, int N, int S, int Mf, const int *d_off,
                  const double *G, double *phi, cudaStream_t st) {
  const int Mp = g64_layout(m->host.M, m->host.D).Mp;
  return g64_kernel_values(m, ws, N, G, st, [&](int i0, int ct, const int *rowexp, const double *W) {
    k_g64_phi<<<dim3((Mf + 7) / 8, S), 256, 0, st>>>(i0, std::min(N, i0 + ct * kR), Mp, Mf, d_off,
                                                     rowexp, W, phi);
  });
}

// A[M][Mf] = K_MM
bool launch_kmm64(const gapgb_model *m, Workspace &ws, int Mf, double *A, cudaStream_t st) {
  const int M = m->host.M;
  const G64 g = g64_layout(M, m->host.D);
  if (!m->d_g64) return false;
  return g64_kernel_values(m, ws, M, (const double *)(m->d_g64 + g.mm), st,
                           [&](int i0, int ct, const int *, const double *W) {
                             k_g64_kmm<<<dim3((Mf + 31) / 32, ct * (kR / 32)), 256, 0, st>>>(
                                 M, i0, g.Mp, Mf, W, A);
                           });
}

template bool launch_gpr64<double>(const gapgb_model *, Workspace &, int, cudaStream_t);
template bool launch_gpr64<float>(const gapgb_model *, Workspace &, int, cudaStream_t);

}  // namespace gapgb
