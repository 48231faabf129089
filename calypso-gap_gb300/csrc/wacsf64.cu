// wacsf64.cu - FP64 wACSF descriptors and slot gradients for the usual SF sets
// (the same functions as wacsf.cu, which holds the reference citations).
//
// Taken when every angular SF has an integer zeta of at most 4 and each
// angular cutoff holds at most 4 distinct alphas; other sets keep wacsf.cu's
// generic kernels.  GB300 issues FP64 at 1/64 of its FP32 rate (measured 1.06
// against 78.5 TFLOP/s), so these kernels are bound by the FP64 pipe and are
// built to issue as few FP64 instructions as possible:
//  - the pairs of slots within each angular cutoff are found in FP32 from the
//    neighbour kernel's FP32 records (a conservative screen; the exact squared
//    distance decides) and compacted into lists, so every lane of an FP64
//    instruction works on a contributing pair;
//  - fc(r) = (cos(pi r / rc) + 1) / 2 is an even, entire function of r: a
//    polynomial of degree 11 in r^2, with fc'(r)/r from its derivative, so neither
//    the slots nor the pairs take a cosine, and a pair takes no square root
//    and no division either (every factor is written in r^2 and 1/r_slot);
//  - a pair's geometry (c^2, a^2 + b^2 + c^2, the dot product), that polynomial
//    and the exponential (a 1024-entry table of 2^(j/1024) and a degree-4
//    polynomial, argument reduction included) run in 64-bit fixed point on the
//    integer pipe, where an instruction costs an SM sub-partition 1 to 2
//    cycles, not 64; errors of the two functions below 0.5 and 1 ulp, pairs too
//    close for the units in FP64 (pair_of);
//  - the (1 +- cos)^zeta of a cutoff group are combinations of the products
//    u^n w^(DEG-n) (u = (1 + cos)/2, w = 1 - u) with non-negative weights: a
//    pair adds those products, times each alpha's exponential, to moments;
//  - the gradient contracts dE/dG onto a polynomial in cos per alpha first,
//    so a pair needs one Horner pass for value and derivative, and it yields
//    three scalars (s1 + s3, s2 + s3, s3); a slot's gradient is then
//    d_q sum(s_own + s3) - sum(s3 d_other), gathered per slot.
// Per pair of the standard set that is about 35 FP64 instructions for the
// descriptors and 55 for the gradient, where the generic kernels issue about
// 520 and 770.  Measured (ncu, both generic kernels -> these, split launches
// included): 512 alloy atoms (56 slots, 690 pairs each) 520 -> 82 us and
// 665 -> 133 us; 64 carbon atoms (158 slots, 7 cutoffs) 2380 -> 102 us and
// 1858 -> 211 us; 6.4 k atoms of ragged cells 5444 -> 604 and 10177 -> 1094
// us (842 and 1330 with the geometry and the exponential's argument in FP64,
// 1139 and 1691 with all of the polynomials there).
//
// A block of 4 warps works on one atom.  The pair list of each cutoff group
// is cut into units of 512 pairs.  Small batches spread an atom's units over
// several blocks (`split`); the arithmetic is arranged so that the result
// does not depend on it: moments are summed per unit, units per residue class
// (unit mod 8) in order, and classes in order; a slot's gradient is summed
// over its pairs in order after the pairs' scalars are written, by the same
// block (split = 1) or by a second kernel.  Nothing is atomic, so results are
// the same bit for bit in every run and in every batch (short of one whose scratch
// cannot be allocated, which takes wacsf.cu's kernels).
#include <algorithm>
#include <cmath>
#include <vector>

#include "gapgb_internal.h"

namespace gapgb {
namespace {

constexpr int kBlk = 128;        // threads per block (4 warps)
constexpr int kUnit = 512;       // pairs per unit
constexpr int kClasses = 8;      // residue classes of units (bounds the split)

typedef unsigned long long u64;
typedef long long i64;
struct __align__(32) I64x4 {
  i64 x, y, z, w;
};

// x 2^sc as a double, rounded (0 < x < 2^63; otherwise zero)
__device__ __forceinline__ double fix_double(u64 x, int sc) {
  const int lz = __clzll((i64)x);
  const u64 m = x << (lz & 63);
  const u64 b = ((u64)(uint32_t)(1022 + 63 - lz + sc) << 52) + (m >> 11) + ((m >> 10) & 1);
  return (i64)x > 0 ? __longlong_as_double((i64)b) : 0.0;
}

// x in units of 2^(E - 64), top = the biased exponent of 2^(E - 1) (x >= 0;
// 2^E and more: the largest)
__device__ __forceinline__ u64 to_fix(double x, int top) {
  const u64 b = (u64)__double_as_longlong(x);
  const int sh = top - (int)(b >> 52);
  const u64 m = ((b & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 11;
  return sh < 0 ? ~0ull : (sh >= 64 ? 0 : m >> sh);
}
__device__ __forceinline__ i64 to_fix_signed(double x, int top) {
  const i64 m = (i64)to_fix(fabs(x), top);
  return x < 0.0 ? -m : m;
}
__device__ __forceinline__ double signed_double(i64 x, int sc) {
  const i64 sg = x >> 63;
  return __longlong_as_double(__double_as_longlong(fix_double((u64)((x ^ sg) - sg), sc)) |
                              (sg & (i64)(1ull << 63)));
}

// w = r^2 / rc^2 (kv r^2 / 2) in units of 2^-64, below one; r^2 in units of
// 2^(E - 64), rc^2 <= 2^E
__device__ __forceinline__ u64 fc_arg(u64 r2, const W64Cut &c) {
  const u64 w = __umul64hi(r2, c.ratio);
  return (w >> 63) ? ~0ull : w << 1;
}
__device__ __forceinline__ u64 slot_arg(double r2, const W64Cut &c) {
  return fc_arg(to_fix(r2, c.top), c);
}
// of a pair within the cutoff: r^2 in the pairs' unit, `up` bits finer
__device__ __forceinline__ u64 pair_arg(u64 r2, const W64Cut &c) {
  return (r2 >> (64 - c.up)) ? ~0ull : fc_arg(r2 << c.up, c);
}
// fc = sum (-1)^n c_n w^n in integer arithmetic (units of 2^-61), and -d fc / dw
__device__ __forceinline__ double fc_fix(const W64Cut &c, u64 w) {
  u64 p = c.c[kFcN - 1];
#pragma unroll
  for (int n = kFcN - 2; n >= 0; --n) p = c.c[n] - __umul64hi(w, p);
  return fix_double(p, -61);
}
__device__ __forceinline__ void fc_fix2(const W64Cut &c, u64 w, double &f, double &d) {
  u64 p = c.c[kFcN - 1], e = 0;
#pragma unroll
  for (int n = kFcN - 2; n >= 0; --n) {
    e = p - __umul64hi(w, e);
    p = c.c[n] - __umul64hi(w, p);
  }
  f = fix_double(p, -61);
  // past pi (the format's pi is 4e-10 above it) the derivative changes sign
  d = (i64)e < 0 ? -fix_double(0ull - e, -61) : fix_double(e, -61);
}

// exp(a v), a <= 0, of v = x 2^(e - 64): m x is |a| v 1024 / ln 2 with `frac`
// fractional bits in its high word; its floor and fraction give 2^(k/1024) from
// a table (P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15, 1989) and
// 2^(r/1024) by a degree-4 polynomial, all in integer arithmetic (exp2_fix of
// gpr64_tc.cu).  The fraction is cut at 2^-50 (and 2^-50 off where it is zero):
// a relative 2^-60.  Past the normal range (|a v| >= 708), for a > 0 (frac < 0),
// and where x is so small that its units are too coarse for the exponent
// (c.steep and the caller's `small`), the value in FP64, f().
template <typename F>
__device__ __forceinline__ double exp_neg(const W64Exp &c, u64 x, const u64 *__restrict__ T,
                                          bool small, F f) {
  const u64 hi = __umul64hi(x, c.m), lo = x * c.m;
  const u64 ki = hi >> (c.frac & 63);
  if (c.frac < 0 || (c.steep && small) || ki >= 1045929) return f();
  const u64 fr = c.frac >= 50 ? hi >> (c.frac - 50) : (hi << (50 - c.frac)) | (lo >> (14 + c.frac));
  const int k = -1 - (int)ki;
  const u64 t = T[k & (kExpN - 1)];
  // y = the fraction of 1/1024 times ln 2, in units of 2^-74
  const u64 y = __umul64hi((~fr & ((1ull << 50) - 1)) << 14, 0xB17217F7D1CF79ACull);
  const u64 y2 = __umul64hi(y, y);                         // 2^-84
  const uint32_t yh = (uint32_t)(y >> 32);                 // 2^-42
  const uint32_t y3 = __umulhi((uint32_t)(y2 >> 32), yh);  // 2^-62
  const uint32_t y4 = __umulhi(y3, yh);                    // 2^-72
  const u64 p = y + (y2 >> 11) +
                ((u64)(__umulhi(y3, 0x2AAAAAABu) + (__umulhi(y4, 0x0AAAAAABu) >> 10)) << 12);
  // rounded after the shift: at a zero argument m is 55 below 2^64, m + 1024
  // would wrap, and the carry into the exponent is what makes the result 1
  const u64 m = t + (__umul64hi(t, p) >> 10);
  return __longlong_as_double(
      (i64)(((u64)(uint32_t)((k >> 10) + 1022) << 52) + (m >> 11) + ((m >> 10) & 1)));
}

// exp(a u2) of a slot's (r - rs)^2
__device__ __forceinline__ double slot_exp(const W64Exp &c, double u2, const W64Fc &fc,
                                           const u64 *__restrict__ T) {
  const u64 x = to_fix(u2, fc.er - 1 + 1023);
  return exp_neg(c, x, T, (x >> 53) == 0, [&] { return exp(c.a * u2); });
}

// sums v[0..N) over the warp's lanes by halving exchanges: at each step a
// lane hands half of its values to its partner and adds the half it keeps
// (N - 1 additions in all instead of 5 N).  On return *out holds the total of
// value `idx` (idx < 0: none).  The order of the additions is fixed.
template <int N>
__device__ __forceinline__ void warp_fold(double (&v)[N], int lane, double *out, int *idx) {
  constexpr int P = 32;
  double a[P];
#pragma unroll
  for (int n = 0; n < P; ++n) a[n] = n < N ? v[n] : 0.0;
  int base = 0;
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int n = 0; n < h; ++n) {
      // values n (kept by the lower lanes) and n + h (kept by the upper ones)
      const bool low_live = n < N, high_live = n + h < N;  // before this step: < min(N, 2h)
      if (!low_live) continue;
      if (high_live) {
        const double give = up ? a[n] : a[n + h];
        const double got = __shfl_xor_sync(0xffffffffu, give, h);
        a[n] = (up ? a[n + h] : a[n]) + got;
      } else {
        const double got = __shfl_xor_sync(0xffffffffu, a[n], h);
        a[n] = a[n] + got;  // every lane keeps it; the lower lanes' copy counts
      }
    }
    if (up) base += h;
  }
  *out = a[0];
  *idx = base < N ? base : -1;
}

// shared-memory layout (bytes), common to the kernels
struct Lay {
  size_t A, B, I, fc, f4, idx, mask, pre, row, list, rest, total;
};
__host__ __device__ inline size_t up32(size_t x) { return (x + 31) / 32 * 32; }
__host__ __device__ inline Lay layout(int capS, int nrc, size_t rest) {
  const int W = (capS + 31) / 32;
  const size_t c = capS;
  Lay l;
  size_t o = kExpN * 8;
  l.A = o, o += c * 32;                  // dx, dy, dz, r
  l.I = o, o += c * 32;                  // dx, dy, dz, r^2/2 in fixed point
  l.B = o, o += up32(c * 16);            // 1/r, weight
  l.fc = o, o += up32(c * nrc * 16);     // fc, fc'/r of every cutoff
  l.f4 = o, o += up32(c * 16);           // FP32 dx, dy, dz, r
  l.idx = o, o += up32(c * 2);           // the group's slots (those within its cutoff)
  l.mask = o, o += up32(c * W * 4);      // pair bits of the group's slots, a row's words adjacent
  l.pre = o, o += up32(c * W * 2);       // the row's pairs k > j before each word
  l.row = o, o += up32((c + 2) * 4);     // first pair of each row
  l.list = o, o += kUnit * 4;            // the unit's pairs
  l.rest = o, o += up32(rest);
  l.total = o;
  return l;
}

struct View {
  const u64 *T;
  double4 *A;
  double2 *B, *fc;
  I64x4 *I;
  float4 *f4;
  unsigned *mask;
  unsigned short *idx, *pre;
  int *row;
  unsigned *list;
};
__device__ __forceinline__ View view(unsigned char *sm, const Lay &l) {
  View v;
  v.T = reinterpret_cast<const u64 *>(sm);
  v.A = reinterpret_cast<double4 *>(sm + l.A);
  v.B = reinterpret_cast<double2 *>(sm + l.B);
  v.fc = reinterpret_cast<double2 *>(sm + l.fc);
  v.I = reinterpret_cast<I64x4 *>(sm + l.I);
  v.f4 = reinterpret_cast<float4 *>(sm + l.f4);
  v.idx = reinterpret_cast<unsigned short *>(sm + l.idx);
  v.mask = reinterpret_cast<unsigned *>(sm + l.mask);
  v.pre = reinterpret_cast<unsigned short *>(sm + l.pre);
  v.row = reinterpret_cast<int *>(sm + l.row);
  v.list = reinterpret_cast<unsigned *>(sm + l.list);
  return v;
}

// slots of atom i into shared memory (fc'/r only for the gradient).
// want_fc: the gather kernel reads positions alone.
template <bool GRAD>
__device__ __forceinline__ int stage(const View &s, const W64Tab &t, const W64Fc &fc, int i, int cap, int capS,
                                     const int *__restrict__ cnt, const double4 *__restrict__ xyzr,
                                     const int *__restrict__ nj, const double4 *__restrict__ apos,
                                     const float4 *__restrict__ d32, bool want_fc) {
  const int P = min(cnt[i], capS);
  const double4 pi = apos[i];
  for (int q = threadIdx.x; q < P; q += blockDim.x) {
    const size_t g = (size_t)i * cap + q;
    const double4 e = xyzr[g];
    const double r = e.w;
    const double dx = e.x - pi.x, dy = e.y - pi.y, dz = e.z - pi.z;
    s.A[q] = make_double4(dx, dy, dz, r);
    s.f4[q] = d32[g];
    if (!want_fc) continue;
    const int top = fc.e - 1 + 1023;
    I64x4 v;
    v.x = to_fix_signed(dx, top), v.y = to_fix_signed(dy, top), v.z = to_fix_signed(dz, top);
    v.w = (i64)to_fix(0.5 * (r * r), 2 * fc.e - 1 + 1023);
    s.I[q] = v;
    s.B[q] = make_double2(1.0 / r, apos[nj[g]].w);
    for (int c = 0; c < t.nrc; ++c) {
      double f = 0.0, d = 0.0;
      if (r <= t.rc[c]) {
        if (GRAD) {
          fc_fix2(fc.c[c], slot_arg(r * r, fc.c[c]), f, d);
          d *= t.kd[c];
        } else {
          f = fc_fix(fc.c[c], slot_arg(r * r, fc.c[c]));
        }
      }
      s.fc[(size_t)c * capS + q] = make_double2(f, d);
    }
  }
  return P;
}

// The pairs j < k of cutoff group g among its n slots (the slots within the
// cutoff, renumbered in order: idx): bit k of row j's mask words (FULL: for
// every k, not only k > j), the row's pairs before each word, and the rows'
// first pairs (row[n] is their number).  FP32 screen with a relative margin
// of 4e-5 on the squared lengths (the FP32 records are off by less than 1e-6
// of rc^2): pairs just outside the cutoff may be listed, and contribute
// exactly zero.  The screen's arithmetic is even in (j, k), so bits (j, k) and
// (k, j) agree, and its rounding is spelled out, so the lists of k_w64_bwd and
// k_w64_gather do (a pair's scalars are found by its place).  Ends with a barrier.
template <bool FULL>
__device__ __forceinline__ int build_pairs(const View &s, const W64Tab &t, int g, int P, int &n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float rcf = (float)t.rc[t.grp_rc[g]];
  const float rm = rcf * 1.00002f, c2m = rcf * rcf * 1.00004f;
  if (warp == 0) {
    int m = 0;
    for (int b = 0; b < P; b += 32) {
      const bool in = b + lane < P && s.f4[b + lane].w <= rm;
      const unsigned v = __ballot_sync(0xffffffffu, in);
      if (in) s.idx[m + __popc(v & ((1u << lane) - 1u))] = (unsigned short)(b + lane);
      m += __popc(v);
    }
    if (lane == 0) s.row[P + 1] = m;
  }
  __syncthreads();
  n = s.row[P + 1];
  const int W = (n + 31) >> 5;
  for (int j = warp; j < n; j += nw) {
    const float4 aj = s.f4[s.idx[j]];
    int c = 0;
    for (int w = FULL ? 0 : j >> 5; w < W; ++w) {
      const int k = 32 * w + lane;
      bool in = k < n && (FULL ? k != j : k > j);
      const float4 ak = s.f4[s.idx[in ? k : j]];
      const float cx = aj.x - ak.x, cy = aj.y - ak.y, cz = aj.z - ak.z;
      in = in && __fmaf_rn(cz, cz, __fmaf_rn(cy, cy, __fmul_rn(cx, cx))) <= c2m;
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (lane == 0) {
        s.mask[j * W + w] = m;
        s.pre[j * W + w] = (unsigned short)c;
      }
      c += __popc(__ballot_sync(0xffffffffu, in && k > j));
    }
    if (lane == 0) s.row[j] = c;
  }
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the row counts
    int carry = 0;
    for (int b = 0; b < n; b += 32) {
      const int v = b + lane < n ? s.row[b + lane] : 0;
      int x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      __syncwarp();
      if (b + lane < n) s.row[b + lane] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) s.row[n] = carry;
  }
  __syncthreads();
  return s.row[n];
}

// the bits k > j of word w of row j
__device__ __forceinline__ unsigned upper(const View &s, int W, int j, int w) {
  const unsigned m = s.mask[j * W + w];
  return w > (j >> 5) ? m : (w < (j >> 5) ? 0u : m & ~((2u << (j & 31)) - 1u));
}

// A pair of slots: s3 = a^2 + b^2 + c^2 in units of 2^(2 e - 64), the argument of
// fc(c), the cosine, and whether c is within the group's cutoff.  Formed in
// fixed point: integer instructions, two FP64 ones less per coordinate.  The
// differences are below the cutoff, 2^(e - 1), whatever wraps before; the dot
// product is off by at most 2.5 of those units, so the cosine by less than
// 2^-53 as long as a b is at least 2^(2 e - 9) (0.5 A^2 at a cutoff of 6 A, 8 at
// 20).  Closer slots, and with them every pair within a cutoff far below the
// longest, are formed in FP64 (fc.close: the high word of the largest 1/(ab)
// that is not), and so are their steep exponentials.
struct Pair {
  u64 s3, w;
  double cosv;
  bool in, close;
};
__device__ __forceinline__ double pair_c2(const double4 &a, const double4 &b) {
  const double x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
  return fma(x, x, fma(y, y, z * z));
}
// exp(al s3), a factor per side (rare: a loop, so that it takes few registers)
__device__ __forceinline__ double pair_exp(const double4 *A, int j, int k, double al) {
  double e = 1.0;
#pragma unroll 1
  for (int u = 0; u < 3; ++u) {
    const double r = A[u ? k : j].w;
    e *= exp(al * (u < 2 ? r * r : pair_c2(A[j], A[k])));
  }
  return e;
}
__device__ __forceinline__ Pair pair_of(const View &s, int j, int k, double iab, const W64Fc &fc,
                                        const W64Cut &cut) {
  Pair p;
  p.close = __double2hiint(iab) > fc.close;
  if (p.close) {
    const double4 a = s.A[j], b = s.A[k];
    const double c2 = pair_c2(a, b);
    p.s3 = to_fix(fma(a.w, a.w, fma(b.w, b.w, c2)), 2 * fc.e - 1 + 1023);
    p.w = slot_arg(c2, cut);
    p.in = c2 <= cut.rc2d;
    p.cosv = fma(a.x, b.x, fma(a.y, b.y, a.z * b.z)) * iab;
    return p;
  }
  const I64x4 a = s.I[j], b = s.I[k];
  auto sq = [](i64 d) {
    const u64 m = (u64)(d < 0 ? -d : d);
    return __umul64hi(m, m);
  };
  const u64 c2 = sq((i64)((u64)a.x - (u64)b.x)) + sq((i64)((u64)a.y - (u64)b.y)) +
                 sq((i64)((u64)a.z - (u64)b.z));
  const u64 h = (u64)a.w + (u64)b.w;
  p.s3 = 2 * h + c2;
  p.w = pair_arg(c2, cut);
  p.in = c2 <= cut.rc2;
  // costheta = (rij^2 + rik^2 - rjk^2) / (2 rij rik) (wacsf.f90:271-273)
  p.cosv = signed_double((i64)(h - (c2 >> 1)), 2 * fc.e - 64) * iab;
  return p;
}

// list[p - p0] = j | k << 16 (slots) for the pairs p in [p0, p1).  Ends with a
// barrier.
__device__ __forceinline__ void expand(const View &s, int n, int p0, int p1) {
  const int W = (n + 31) >> 5;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    int p = s.row[j];
    if (p >= p1 || s.row[j + 1] <= p0) continue;
    const unsigned js = s.idx[j];
    for (int w = j >> 5; w < W && p < p1; ++w) {
      unsigned m = upper(s, W, j, w);
      while (m) {
        const int k = 32 * w + __ffs(m) - 1;
        m &= m - 1;
        if (p >= p0 && p < p1) s.list[p - p0] = js | ((unsigned)s.idx[k] << 16);
        ++p;
      }
    }
  }
  __syncthreads();
}

// Descriptors.  grid (atoms, split); block (i, y) takes the units whose
// residue class is y modulo the split, the last one also the radial terms.
// split > 1: the classes' moments go to part[i][group][class][moment], summed
// by k_w64_final.
template <int NAL, int DEG>
__global__ void __launch_bounds__(kBlk, NAL * (DEG + 1) <= 10 ? 5 : 3)
    k_w64_fwd(int N, int cap, int capS, const int *__restrict__ cnt,
              const double4 *__restrict__ xyzr, const int *__restrict__ nj,
              const double4 *__restrict__ apos, const float4 *__restrict__ d32,
              const W64Tab *__restrict__ tab, const __grid_constant__ W64Fc fc,
              const u64 *__restrict__ expt,
              double *__restrict__ G, double *__restrict__ part, int split) {
  constexpr int NB = DEG + 1, NM = 2 * NAL * NB;
  extern __shared__ __align__(32) unsigned char smraw[];
  const W64Tab &t = *tab;
  const Lay l = layout(capS, t.nrc, 0);
  const View s = view(smraw, l);
  double *wpart = reinterpret_cast<double *>(smraw + l.rest);      // [4][NM]
  double *S = wpart + 4 * NM;                                      // [group][class][NM]
  double *rp = S + (size_t)t.ngrp * kClasses * NM;                 // [2][kBlk]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int q = tid; q < kExpN; q += kBlk) reinterpret_cast<u64 *>(smraw)[q] = expt[q];
  const int y = blockIdx.y;
  for (int i = blockIdx.x; i < N; i += gridDim.x) {
    __syncthreads();
    const int P = stage<false>(s, t, fc, i, cap, capS, cnt, xyzr, nj, apos, d32, true);
    for (int q = tid; q < t.ngrp * kClasses * NM; q += kBlk) S[q] = 0.0;
    __syncthreads();
    double *Gi = G + (size_t)i * t.D;
    if (t.nrad > 0 && y == split - 1) {
      // radial terms: thread = (slot group, SF), so the lanes stay busy for
      // any number of SFs; the slot groups are summed in pairs
      const int ng = kBlk / t.nrad, sr = tid % t.nrad, gr = tid / t.nrad;
      double acc = 0.0, accw = 0.0;
      if (gr < ng) {
        const W64Exp ex = t.rad_e[sr];
        const double rs = t.rad_rs[sr];
        const double2 *f = s.fc + (size_t)t.rad_rc[sr] * capS;
        for (int q = gr; q < P; q += ng) {
          const double fq = f[q].x, u = s.A[q].w - rs, u2 = u * u;
          const double e = slot_exp(ex, u2, fc, s.T);
          const double v = __double2hiint(fq) != 0 ? e * fq : 0.0;  // beyond the cutoff: zero
          acc += v;
          accw = fma(v, s.B[q].y, accw);
        }
      }
      rp[tid] = acc;
      rp[kBlk + tid] = accw;
      __syncthreads();
      for (int w = ng; w > 1;) {
        const int h = (w + 1) / 2;
        if (gr < w - h) {
          rp[tid] += rp[tid + h * t.nrad];
          rp[kBlk + tid] += rp[kBlk + tid + h * t.nrad];
        }
        w = h;
        __syncthreads();
      }
      if (tid < t.nrad) {
        Gi[t.rad_d[tid]] = rp[tid];
        Gi[t.rad_d[tid] + t.nsf] = rp[kBlk + tid];
      }
    }
    int u0 = 0;  // index of the group's first unit
    for (int g = 0; g < t.ngrp; ++g) {
      __syncthreads();
      int n;
      const int np = build_pairs<false>(s, t, g, P, n);
      const int rci = t.grp_rc[g];
      const double2 *f = s.fc + (size_t)rci * capS;
      W64Exp ex[NAL];
#pragma unroll
      for (int q = 0; q < NAL; ++q) ex[q] = t.alpha[g][q];
      const int nu = (np + kUnit - 1) / kUnit;
      for (int u = 0; u < nu; ++u) {
        const int cls = (u0 + u) % kClasses;
        if (cls % split != y) continue;
        const int p0 = u * kUnit, p1 = min(np, p0 + kUnit);
        expand(s, n, p0, p1);
        double acc[NM];
#pragma unroll
        for (int n = 0; n < NM; ++n) acc[n] = 0.0;
        for (int p = p0 + tid; p - lane < p1; p += kBlk) {
          const bool live = p < p1;
          const unsigned jk = live ? s.list[p - p0] : 0u;
          const int j = jk & 0xffff, k = jk >> 16;
          const double2 bj = s.B[j], bk = s.B[k];
          const Pair pr = pair_of(s, j, k, bj.x * bk.x, fc, fc.c[rci]);
          double fcc = fc_fix(fc.c[rci], pr.w);
          const bool in = live && pr.in;  // else exactly zero
          fcc = in ? fcc : 0.0;
          const double cosv = pr.cosv;
          const double F = f[j].x * f[k].x * fcc;
          const double wjk = bj.y * bk.y;
          const double uu = fma(0.5, cosv, 0.5), ww = fma(-0.5, cosv, 0.5);
          double basis[NB];
          if constexpr (DEG == 1) {
            basis[0] = ww;
            basis[1] = uu;
          } else if constexpr (DEG == 2) {
            basis[0] = ww * ww;
            basis[1] = uu * ww;
            basis[2] = uu * uu;
          } else {
            const double u2 = uu * uu, w2 = ww * ww, uw = uu * ww;
            basis[0] = w2 * w2;
            basis[1] = uw * w2;
            basis[2] = u2 * w2;
            basis[3] = uw * u2;
            basis[4] = u2 * u2;
          }
#pragma unroll
          for (int q = 0; q < NAL; ++q) {
            const double ef = in ? exp_neg(ex[q], pr.s3, s.T, pr.close,
                                           [&] { return pair_exp(s.A, j, k, ex[q].a); }) * F
                                 : 0.0;
            const double efw = ef * wjk;
#pragma unroll
            for (int n = 0; n < NB; ++n) {
              acc[q * NB + n] = fma(basis[n], ef, acc[q * NB + n]);
              acc[(NAL + q) * NB + n] = fma(basis[n], efw, acc[(NAL + q) * NB + n]);
            }
          }
        }
        if constexpr (NM <= 32) {
          double tot;
          int idx;
          warp_fold<NM>(acc, lane, &tot, &idx);
          if (idx >= 0) wpart[warp * NM + idx] = tot;
        } else {
          double lo[32], hi[NM - 32], tot;
          int idx;
#pragma unroll
          for (int n = 0; n < NM; ++n) (n < 32 ? lo[n & 31] : hi[n < 32 ? 0 : n - 32]) = acc[n];
          warp_fold<32>(lo, lane, &tot, &idx);
          if (idx >= 0) wpart[warp * NM + idx] = tot;
          warp_fold<NM - 32>(hi, lane, &tot, &idx);
          if (idx >= 0) wpart[warp * NM + 32 + idx] = tot;
        }
        __syncthreads();
        if (tid < NM)
          S[(g * kClasses + cls) * NM + tid] +=
              ((wpart[tid] + wpart[NM + tid]) + wpart[2 * NM + tid]) + wpart[3 * NM + tid];
      }
      u0 += nu;
    }
    __syncthreads();
    if (split > 1) {
      for (int e = tid; e < t.ngrp * kClasses * NM; e += kBlk)
        if ((e / NM) % kClasses % split == y)
          part[(size_t)i * t.ngrp * kClasses * NM + e] = S[e];
    } else {
      // classes in order, then the moments combine into the SFs
      for (int e = tid; e < t.ngrp * NM; e += kBlk) {
        const int g = e / NM, n = e % NM;
        double v = 0.0;
        for (int c = 0; c < kClasses; ++c) v += S[(g * kClasses + c) * NM + n];
        S[(g * kClasses) * NM + n] = v;
      }
      __syncthreads();
      for (int a = tid; a < t.nang; a += kBlk) {
        const double *m = S + (size_t)t.ang_g[a] * kClasses * NM + t.ang_q[a] * NB;
        double x = 0.0, w = 0.0;
#pragma unroll
        for (int n = 0; n < NB; ++n) {
          x = fma(t.bern[a][n], m[n], x);
          w = fma(t.bern[a][n], m[NAL * NB + n], w);
        }
        Gi[t.ang_d[a]] = x;
        Gi[t.ang_d[a] + t.nsf] = w;
      }
    }
  }
}

// split > 1: the class sums and the combination of moments, as above
__global__ void __launch_bounds__(kBlk)
    k_w64_final(int N, int NB, int NM, const W64Tab *__restrict__ tab,
                const double *__restrict__ part, double *__restrict__ G) {
  const W64Tab &t = *tab;
  const int i = blockIdx.x;
  for (int a = threadIdx.x; a < t.nang; a += kBlk) {
    const double *m =
        part + (size_t)i * t.ngrp * kClasses * NM + (size_t)t.ang_g[a] * kClasses * NM + t.ang_q[a] * NB;
    double x = 0.0, w = 0.0;
    for (int n = 0; n < NB; ++n) {
      double mx = 0.0, mw = 0.0;
      for (int c = 0; c < kClasses; ++c) {
        mx += m[c * NM + n];
        mw += m[c * NM + NM / 2 + n];
      }
      x = fma(t.bern[a][n], mx, x);
      w = fma(t.bern[a][n], mw, w);
    }
    G[(size_t)i * t.D + t.ang_d[a]] = x;
    G[(size_t)i * t.D + t.ang_d[a] + t.nsf] = w;
  }
}

// adds group g's pairs to the slots' sums: acc[q] = (sum of the neighbour
// vectors' terms x, y, z; the sum that multiplies d_q).  Two threads per slot,
// which take the mask words of even and of odd number, each in ascending
// order; `sc` holds a pair's (s1 + s3, s2 + s3, s3) in one 32-byte sector.
__device__ __forceinline__ void gather(const View &s, int n, const double4 *sc, double4 *acc) {
  const int W = (n + 31) >> 5, per = blockDim.x >> 1;
  for (int q0 = 0; q0 < n; q0 += per) {
    const int q = q0 + (int)(threadIdx.x >> 1);
    const bool own = q < n;
    double4 a = make_double4(0.0, 0.0, 0.0, 0.0);
    const int wq = q >> 5;
    const unsigned below = (1u << (q & 31)) - 1u;
    if (own)
      for (int w = threadIdx.x & 1; w < W; w += 2) {
        unsigned m = s.mask[q * W + w];
        int up = s.row[q] + s.pre[q * W + w];  // the row's next pair (q, k > q)
        while (m) {
          const int k = 32 * w + __ffs(m) - 1;
          m &= m - 1;
          const bool first = k > q;
          const int e = first ? up++
                              : s.row[k] + s.pre[k * W + wq] + __popc(upper(s, W, k, wq) & below);
          const double *v = reinterpret_cast<const double *>(sc + e);
          const double4 d = s.A[s.idx[k]];
          const double c = v[2];
          a.x = fma(-c, d.x, a.x);
          a.y = fma(-c, d.y, a.y);
          a.z = fma(-c, d.z, a.z);
          a.w += v[first ? 0 : 1];
        }
      }
    a.x += __shfl_xor_sync(0xffffffffu, a.x, 1);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, 1);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, 1);
    a.w += __shfl_xor_sync(0xffffffffu, a.w, 1);
    if (own && !(threadIdx.x & 1)) {
      double4 &o = acc[s.idx[q]];
      o = make_double4(o.x + a.x, o.y + a.y, o.z + a.z, o.w + a.w);
    }
  }
}

// slot gradients and the per-atom virial from the finished sums (the block's
// first kBlk threads, so that every launch adds in the same order)
__device__ __forceinline__ void finish(const View &s, int i, int cap, int P, const double4 *acc,
                                       double *vir, double4 *__restrict__ gslot,
                                       double *__restrict__ wvir) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kBlk) {
    double V[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int q = threadIdx.x; q < P; q += kBlk) {
      const double4 a = acc[q], d = s.A[q];
      const double gx = fma(a.w, d.x, a.x), gy = fma(a.w, d.y, a.y), gz = fma(a.w, d.z, a.z);
      gslot[(size_t)i * cap + q] = make_double4(gx, gy, gz, 0.0);
      const double dd[3] = {d.x, d.y, d.z}, gg[3] = {gx, gy, gz};
#pragma unroll
      for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int y = 0; y < 3; ++y) V[x * 3 + y] = fma(dd[x], gg[y], V[x * 3 + y]);
    }
    double tot;
    int idx;
    warp_fold<9>(V, lane, &tot, &idx);
    if (idx >= 0) vir[warp * 9 + idx] = tot;
  }
  __syncthreads();
  if (threadIdx.x < 9)
    wvir[(size_t)i * 9 + threadIdx.x] =
        ((vir[threadIdx.x] + vir[9 + threadIdx.x]) + vir[18 + threadIdx.x]) + vir[27 + threadIdx.x];
}

// Slot gradients.  split = 1: grid-stride over atoms; a group's scalars pass
// through the block's own scratch (sc + blockIdx.x * nsc) and are gathered
// before the next group.  split > 1: block (i, y) writes its units' scalars
// to sc + i * nsc + (group's first unit) * kUnit, the radial sums to
// rad[i][slot] and the groups' first units to first[i][g], for k_w64_gather.
template <int NAL, int DEG>
__global__ void __launch_bounds__(kBlk, 4)
    k_w64_bwd(int N, int cap, int capS, const int *__restrict__ cnt,
              const double4 *__restrict__ xyzr, const int *__restrict__ nj,
              const double4 *__restrict__ apos, const float4 *__restrict__ d32,
              const W64Tab *__restrict__ tab, const __grid_constant__ W64Fc fc,
              const u64 *__restrict__ expt, const double *__restrict__ dedg,
              double4 *__restrict__ gslot, double *__restrict__ wvir, double4 *scr,
              double *__restrict__ rad, int *__restrict__ first, size_t nsc, int split) {
  constexpr int NB = DEG + 1;
  extern __shared__ __align__(32) unsigned char smraw[];
  const W64Tab &t = *tab;
  const Lay l = layout(capS, t.nrc, 0);
  const View s = view(smraw, l);
  double4 *acc = reinterpret_cast<double4 *>(smraw + l.rest);             // [capS]
  double *dg = reinterpret_cast<double *>(acc + capS);                    // [D]
  double *sU = dg + t.D;                                                  // [2][NAL][NB]
  double *vir = sU + 2 * NAL * NB;                                        // [4][9]
  const int tid = threadIdx.x, lane = tid & 31;
  for (int q = tid; q < kExpN; q += kBlk) reinterpret_cast<u64 *>(smraw)[q] = expt[q];
  const int y = blockIdx.y;
  for (int i = blockIdx.x; i < N; i += gridDim.x) {
    __syncthreads();
    const int P = stage<true>(s, t, fc, i, cap, capS, cnt, xyzr, nj, apos, d32, true);
    for (int d = tid; d < t.D; d += kBlk) dg[d] = dedg[(size_t)i * t.D + d];
    __syncthreads();
    // radial terms, thread = slot: sum_s dE/dG_s G_s'(r)/r, with
    // (exp fc)'/r = exp (-2 alpha (1 - rs/r) fc + fc'/r)
    if (y == split - 1)
      for (int q = tid; q < P; q += kBlk) {
        const double r = s.A[q].w, r2 = r * r;
        const double2 b = s.B[q];
        double sum = 0.0;
        for (int a = 0; a < t.nrad; ++a) {
          const double2 f = s.fc[(size_t)t.rad_rc[a] * capS + q];
          if ((__double2hiint(f.x) | __double2hiint(f.y)) == 0) continue;  // beyond the cutoff
          const double al = t.rad_e[a].a, rs = t.rad_rs[a];
          double u2 = r2, ur = 1.0;
          if (rs != 0.0) {  // uniform over the block
            const double u = r - rs;
            u2 = u * u;
            ur = u * b.x;
          }
          const double e = slot_exp(t.rad_e[a], u2, fc, s.T);
          const double g = fma(2.0 * al * ur, f.x, f.y);
          sum = fma(fma(dg[t.rad_d[a] + t.nsf], b.y, dg[t.rad_d[a]]) * e, g, sum);
        }
        if (split > 1) rad[(size_t)i * capS + q] = sum;
        else acc[q] = make_double4(0.0, 0.0, 0.0, sum);
      }
    int u0 = 0;
    for (int g = 0; g < t.ngrp; ++g) {
      __syncthreads();
      int n;
      const int np = build_pairs<true>(s, t, g, P, n);
      const int rci = t.grp_rc[g];
      const double kd = t.kd[rci];
      const double2 *f = s.fc + (size_t)rci * capS;
      // dE/dG contracted onto polynomials in cos: cell (weighting, alpha, power)
      for (int c = tid; c < 2 * NAL * NB; c += kBlk) {
        const int h = c / (NAL * NB), q = (c / NB) % NAL, m = c % NB;
        double v = 0.0;
        for (int a = t.grp_start[g]; a < t.grp_start[g + 1]; ++a)
          if (t.ang_q[a] == q) v = fma(t.mono[a][m], dg[t.ang_d[a] + (h ? t.nsf : 0)], v);
        sU[c] = v;
      }
      W64Exp ex[NAL];
#pragma unroll
      for (int q = 0; q < NAL; ++q) ex[q] = t.alpha[g][q];
      __syncthreads();
      double4 *sc = split > 1 ? scr + (size_t)i * nsc + (size_t)u0 * kUnit
                              : scr + (size_t)blockIdx.x * nsc;
      if (split > 1 && y == 0 && tid == 0) first[i * t.ngrp + g] = u0;
      const int nu = (np + kUnit - 1) / kUnit;
      for (int u = 0; u < nu; ++u) {
        if ((u0 + u) % kClasses % split != y) continue;
        const int p0 = u * kUnit, p1 = min(np, p0 + kUnit);
        __syncthreads();  // the previous unit's list has been read
        expand(s, n, p0, p1);
        for (int p = p0 + tid; p - lane < p1; p += kBlk) {
          const bool live = p < p1;
          const unsigned jk = live ? s.list[p - p0] : 0u;
          const int j = jk & 0xffff, k = jk >> 16;
          const double2 bj = s.B[j], bk = s.B[k], fj = f[j], fk = f[k];
          const double iab = bj.x * bk.x;
          const Pair pr = pair_of(s, j, k, iab, fc, fc.c[rci]);
          double fcc, fcd;
          fc_fix2(fc.c[rci], pr.w, fcc, fcd);
          fcd *= kd;
          const bool in = live && pr.in;
          fcc = in ? fcc : 0.0;
          fcd = in ? fcd : 0.0;
          const double cosv = pr.cosv;
          const double wjk = bj.y * bk.y;
          double SP = 0.0, SQ = 0.0, SU = 0.0;
#pragma unroll
          for (int q = 0; q < NAL; ++q) {
            const double e = in ? exp_neg(ex[q], pr.s3, s.T, pr.close,
                                          [&] { return pair_exp(s.A, j, k, ex[q].a); })
                                : 0.0;
            const double *U0 = sU + q * NB, *U1 = sU + (NAL + q) * NB;
            double pv = fma(wjk, U1[DEG], U0[DEG]), pd = 0.0;
#pragma unroll
            for (int m = DEG - 1; m >= 0; --m) {
              pd = m == DEG - 1 ? pv : fma(pd, cosv, pv);
              pv = fma(pv, cosv, fma(wjk, U1[m], U0[m]));
            }
            const double x = e * pv;
            SQ += x;
            SU = fma(-2.0 * ex[q].a, x, SU);
            SP = fma(e, pd, SP);
          }
          // d/da of [P(cos) E fc(a) fc(b) fc(c)], over a; likewise b and c:
          //   dcos/da / a = 1/(ab) - cos/a^2,  dcos/dc / c = -1/(ab)
          const double fab = fj.x * fk.x;
          const double F = fab * fcc, Qc = SQ * fcc;
          const double t1 = fma(SP, fma(-cosv, bj.x * bj.x, iab), -SU);
          const double t2 = fma(SP, fma(-cosv, bk.x * bk.x, iab), -SU);
          const double t3 = fma(-SP, iab, -SU);
          const double c3 = fma(F, t3, SQ * fab * fcd);
          const double c1 = fma(F, t1, Qc * fk.x * fj.y) + c3;
          const double cc = fma(F, t2, Qc * fj.x * fk.y) + c3;
          if (live) sc[p] = make_double4(c1, cc, c3, 0.0);
        }
      }
      u0 += nu;
      __syncthreads();
      if (split == 1) gather(s, n, sc, acc);
    }
    __syncthreads();
    if (split == 1) finish(s, i, cap, P, acc, vir, gslot, wvir);
  }
}

// split > 1: the gathers that k_w64_bwd does with split 1, a block per atom and
// group.  Latency bound (a load of 32 bytes and an index search per pair, two
// threads per slot), so groups in turn cost their sum: 64 carbon atoms with
// seven groups 133 us by one block per atom, 70 + 14 us so.  One group: the block finishes
// the atom; several: the groups' sums pass through gp[i][g][slot] to
// k_w64_finish, which adds them in order.
constexpr int kGatherThreads = 512;
__global__ void __launch_bounds__(kGatherThreads)
    k_w64_gather(int cap, int capS, const int *__restrict__ cnt,
                 const double4 *__restrict__ xyzr, const int *__restrict__ nj,
                 const double4 *__restrict__ apos, const float4 *__restrict__ d32,
                 const W64Tab *__restrict__ tab, const __grid_constant__ W64Fc fc,
                 double4 *__restrict__ gslot, double *__restrict__ wvir, const double4 *scr,
                 const double *__restrict__ rad, const int *__restrict__ first,
                 double4 *__restrict__ gp, size_t nsc) {
  extern __shared__ __align__(32) unsigned char smraw[];
  const W64Tab &t = *tab;
  const Lay l = layout(capS, t.nrc, 0);
  const View s = view(smraw, l);
  double4 *acc = reinterpret_cast<double4 *>(smraw + l.rest);
  double *vir = reinterpret_cast<double *>(acc + capS);
  const int i = blockIdx.x, g = blockIdx.y;
  const int P = stage<false>(s, t, fc, i, cap, capS, cnt, xyzr, nj, apos, d32, false);
  for (int q = threadIdx.x; q < P; q += blockDim.x)
    acc[q] = make_double4(0.0, 0.0, 0.0, gp ? 0.0 : rad[(size_t)i * capS + q]);
  __syncthreads();
  if (g < t.ngrp) {  // (a set may have no angular SF)
    int n;
    build_pairs<true>(s, t, g, P, n);
    gather(s, n, scr + (size_t)i * nsc + (size_t)first[i * t.ngrp + g] * kUnit, acc);
  }
  __syncthreads();
  if (gp)
    for (int q = threadIdx.x; q < P; q += blockDim.x)
      gp[((size_t)i * t.ngrp + g) * capS + q] = acc[q];
  else
    finish(s, i, cap, P, acc, vir, gslot, wvir);
}
__global__ void __launch_bounds__(kBlk)
    k_w64_finish(int cap, int capS, const int *__restrict__ cnt, const double4 *__restrict__ xyzr,
                 const int *__restrict__ nj, const double4 *__restrict__ apos,
                 const float4 *__restrict__ d32, const W64Tab *__restrict__ tab,
                 const __grid_constant__ W64Fc fc, double4 *__restrict__ gslot,
                 double *__restrict__ wvir, const double *__restrict__ rad,
                 const double4 *__restrict__ gp) {
  extern __shared__ __align__(32) unsigned char smraw[];
  const W64Tab &t = *tab;
  const Lay l = layout(capS, t.nrc, 0);
  const View s = view(smraw, l);
  double4 *acc = reinterpret_cast<double4 *>(smraw + l.rest);
  double *vir = reinterpret_cast<double *>(acc + capS);
  const int i = blockIdx.x;
  const int P = stage<false>(s, t, fc, i, cap, capS, cnt, xyzr, nj, apos, d32, false);
  for (int q = threadIdx.x; q < P; q += kBlk) {
    double4 a = make_double4(0.0, 0.0, 0.0, rad[(size_t)i * capS + q]);
    for (int g = 0; g < t.ngrp; ++g) {
      const double4 v = gp[((size_t)i * t.ngrp + g) * capS + q];
      a = make_double4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w);
    }
    acc[q] = a;
  }
  __syncthreads();
  finish(s, i, cap, P, acc, vir, gslot, wvir);
}

// unevaluated sums of two doubles (about 106 bits), for the table below
struct DD {
  double h, l;
};
DD dd_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
DD dd_add(DD a, DD b) {
  DD s = dd_sum(a.h, b.h);
  return dd_sum(s.h, s.l + a.l + b.l);
}
DD dd_mul(DD a, DD b) {
  const double p = a.h * b.h;
  return dd_sum(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
DD dd_div(DD a, double b) {
  const double q = a.h / b;
  const double r = std::fma(-q, b, a.h) + a.l;
  return dd_sum(q, r / b);
}

// fc(r) = (cos(k r) + 1) / 2, k = pi / rc, in powers of w = kv r^2 / 2, with
// kv = 2 / rc^2 cut down to 24 bits (so that kv itself brings no error, and w
// stays at most 1): the power series of cos(sqrt(t)), t = (2 k^2 / kv) w,
// in powers of v = 2 w - 1 to degree 18, economised to degree 11 by Chebyshev
// polynomials (largest error 2e-17, the derivative's 5e-17), then in powers of
// w, whose signs alternate.  Coefficients in units of 2^-61.  Returns kv.
double fc_series(double rc, W64Cut *cut) {
  const double k = kPiRef / rc;
  const double k2 = 2.0 / (rc * rc);
  float kf = (float)k2;
  if ((double)kf > k2) kf = std::nextafter(kf, 0.f);
  const double kv = (double)kf;
  constexpr int kDeg = 18, kTerms = 28;
  const DD w = dd_div(dd_mul({k, 0.0}, {k, 0.0}), kv);
  DD a[kDeg + 1] = {};
  DD u = {0.5, 0.0};  // (-w)^n / (2 (2n)!)
  double row[kTerms + 1] = {1.0};  // C(n, m)
  for (int n = 0; n <= kTerms; ++n) {
    for (int m = 0; m <= std::min(n, kDeg); ++m) a[m] = dd_add(a[m], dd_mul(u, {row[m], 0.0}));
    u = dd_div(dd_mul(u, {-w.h, -w.l}), (2.0 * n + 1.0) * (2.0 * n + 2.0));
    for (int m = std::min(n + 1, kTerms); m > 0; --m) row[m] += row[m - 1];
  }
  a[0] = dd_add(a[0], {0.5, 0.0});
  double T[kDeg + 1][kDeg + 1] = {};  // T_n in powers of v (exact integers)
  T[0][0] = 1.0;
  T[1][1] = 1.0;
  for (int n = 2; n <= kDeg; ++n)
    for (int m = 0; m <= n; ++m) T[n][m] = (m ? 2.0 * T[n - 1][m - 1] : 0.0) - T[n - 2][m];
  for (int n = kDeg; n >= kFcN; --n) {
    const DD q = dd_div(a[n], -T[n][n]);
    for (int m = 0; m < n; ++m) a[m] = dd_add(a[m], dd_mul(q, {T[n][m], 0.0}));
  }
  // v = 2 w - 1: coefficient of w^m is sum_n a_n C(n, m) 2^m (-1)^(n - m)
  double bin[kFcN][kFcN] = {};
  for (int n = 0; n < kFcN; ++n)
    for (int m = 0; m <= n; ++m) bin[n][m] = m == 0 || m == n ? 1.0 : bin[n - 1][m - 1] + bin[n - 1][m];
  for (int m = 0; m < kFcN; ++m) {
    DD c = {0.0, 0.0};
    for (int n = m; n < kFcN; ++n)
      c = dd_add(c, dd_mul(a[n], {std::ldexp(bin[n][m], m) * ((n & 1) ? -1.0 : 1.0), 0.0}));
    // times (-1)^(n - m) (-1)^m = (-1)^n: the alternating form's coefficient
    cut->c[m] = (unsigned long long)((__int128)std::ldexp(c.h, 61) + (__int128)std::llround(std::ldexp(c.l, 61)));
  }
  // 2^(E - 1) < rc^2 <= 2^E; kv / 2 in units of 2^(-63 - E)
  int E;
  if (std::frexp(2.0 / kv, &E) == 0.5) --E;  // rc^2 a power of two
  cut->top = E - 1 + 1023;
  cut->ratio = (unsigned long long)std::ldexp(kv * 0.5, E + 63);
  return kv;
}

// The Jacobian J[i][slot][xyz][d] = dG_id / dp_slot of atoms [0, N): what the
// gradient contracts with one dE/dG, kept for contractions with many (the
// force rows of a fit).  One block per atom; a pair's scalars (as in
// k_w64_bwd, one triple per angular SF of the group) pass through the block's
// scratch and are gathered by thread = (slot, SF).
template <int NAL, int DEG>
__global__ void __launch_bounds__(kBlk)
    k_w64_jac(int N, int cap, int capS, const int *__restrict__ cnt,
              const double4 *__restrict__ xyzr, const int *__restrict__ nj,
              const double4 *__restrict__ apos, const float4 *__restrict__ d32,
              const W64Tab *__restrict__ tab, const __grid_constant__ W64Fc fc,
              const u64 *__restrict__ expt, double *__restrict__ J, double4 *scr, size_t nsc,
              int namax) {
  extern __shared__ __align__(32) unsigned char smraw[];
  const W64Tab &t = *tab;
  const Lay l = layout(capS, t.nrc, 0);
  const View s = view(smraw, l);
  const int tid = threadIdx.x, lane = tid & 31;
  for (int q = tid; q < kExpN; q += kBlk) reinterpret_cast<u64 *>(smraw)[q] = expt[q];
  for (int i = blockIdx.x; i < N; i += gridDim.x) {
    __syncthreads();
    const int P = stage<true>(s, t, fc, i, cap, capS, cnt, xyzr, nj, apos, d32, true);
    double *Ji = J + (size_t)i * capS * 3 * t.D;
    __syncthreads();
    for (int e = tid; e < P * 3 * t.D; e += kBlk) Ji[e] = 0.0;
    __syncthreads();
    for (int e = tid; e < P * t.nrad; e += kBlk) {
      const int q = e / t.nrad, a = e - q * t.nrad;
      const double2 f = s.fc[(size_t)t.rad_rc[a] * capS + q], b = s.B[q];
      if ((__double2hiint(f.x) | __double2hiint(f.y)) == 0) continue;  // beyond the cutoff
      const double4 d = s.A[q];
      const double al = t.rad_e[a].a, u = d.w - t.rad_rs[a];
      const double v = slot_exp(t.rad_e[a], u * u, fc, s.T) * fma(2.0 * al * (u * b.x), f.x, f.y);
      const double dd[3] = {d.x, d.y, d.z};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double *o = Ji + ((size_t)q * 3 + c) * t.D + t.rad_d[a];
        o[0] = v * dd[c];
        o[t.nsf] = v * b.y * dd[c];
      }
    }
    for (int g = 0; g < t.ngrp; ++g) {
      __syncthreads();
      int n;
      const int np = build_pairs<true>(s, t, g, P, n);
      const int rci = t.grp_rc[g], s0 = t.grp_start[g], na = t.grp_start[g + 1] - s0;
      const double kd = t.kd[rci];
      const double2 *f = s.fc + (size_t)rci * capS;
      double4 *sc = scr + (size_t)blockIdx.x * nsc;
      for (int p0 = 0; p0 < np; p0 += kUnit) {
        const int p1 = min(np, p0 + kUnit);
        __syncthreads();
        expand(s, n, p0, p1);
        for (int p = p0 + tid; p - lane < p1; p += kBlk) {
          if (p >= p1) continue;
          const unsigned jk = s.list[p - p0];
          const int j = jk & 0xffff, k = jk >> 16;
          const double2 bj = s.B[j], bk = s.B[k], fj = f[j], fk = f[k];
          const double iab = bj.x * bk.x;
          const Pair pr = pair_of(s, j, k, iab, fc, fc.c[rci]);
          double fcc, fcd;
          fc_fix2(fc.c[rci], pr.w, fcc, fcd);
          const bool in = pr.in;
          fcc = in ? fcc : 0.0;
          fcd = in ? fcd * kd : 0.0;
          const double cosv = pr.cosv;
          double E[NAL];
#pragma unroll
          for (int q = 0; q < NAL; ++q)
            E[q] = in ? exp_neg(t.alpha[g][q], pr.s3, s.T, pr.close,
                                [&] { return pair_exp(s.A, j, k, t.alpha[g][q].a); })
                      : 0.0;
          const double fab = fj.x * fk.x, F = fab * fcc;
          const double ca = fma(-cosv, bj.x * bj.x, iab), cb = fma(-cosv, bk.x * bk.x, iab);
          const double ga = fcc * fk.x * fj.y, gb = fcc * fj.x * fk.y, gc = fab * fcd;
          for (int a = 0; a < na; ++a) {
            const double *m = t.mono[s0 + a];
            double pv = m[DEG], pd = 0.0;
#pragma unroll
            for (int o = DEG - 1; o >= 0; --o) {
              pd = fma(pd, cosv, pv);
              pv = fma(pv, cosv, m[o]);
            }
            const int q = t.ang_q[s0 + a];
            double e = E[0];
#pragma unroll
            for (int z = 1; z < NAL; ++z) e = q == z ? E[z] : e;
            const double SQ = e * pv, SP = e * pd, SU = -2.0 * t.alpha[g][q].a * SQ;
            const double c3 = fma(F, fma(-SP, iab, -SU), SQ * gc);
            const double c1 = fma(F, fma(SP, ca, -SU), SQ * ga) + c3;
            const double cc = fma(F, fma(SP, cb, -SU), SQ * gb) + c3;
            sc[(size_t)p * namax + a] = make_double4(c1, cc, c3, 0.0);
          }
        }
      }
      __syncthreads();
      const int W = (n + 31) >> 5;
      for (int e = tid; e < n * na; e += kBlk) {
        const int q = e / na, a = e - q * na, wq = q >> 5;
        const unsigned below = (1u << (q & 31)) - 1u;
        double x = 0, y = 0, z = 0, o = 0, xw = 0, yw = 0, zw = 0, ow = 0;
        for (int w = 0; w < W; ++w) {
          unsigned m = s.mask[q * W + w];
          int up = s.row[q] + s.pre[q * W + w];
          while (m) {
            const int k = 32 * w + __ffs(m) - 1;
            m &= m - 1;
            const bool first = k > q;
            const int pr = first ? up++
                                 : s.row[k] + s.pre[k * W + wq] + __popc(upper(s, W, k, wq) & below);
            const double4 v = sc[(size_t)pr * namax + a];
            const int sk = s.idx[k];
            const double4 d = s.A[sk];
            const double wk = s.B[sk].y, c = v.z, own = first ? v.x : v.y;
            const double cw = c * wk;
            x = fma(-c, d.x, x), y = fma(-c, d.y, y), z = fma(-c, d.z, z), o += own;
            xw = fma(-cw, d.x, xw), yw = fma(-cw, d.y, yw), zw = fma(-cw, d.z, zw);
            ow = fma(own, wk, ow);
          }
        }
        const int sq = s.idx[q], dst = t.ang_d[s0 + a];
        const double4 d = s.A[sq];
        const double wq2 = s.B[sq].y;
        const double v[3] = {fma(o, d.x, x), fma(o, d.y, y), fma(o, d.z, z)};
        const double vw[3] = {fma(ow, d.x, xw), fma(ow, d.y, yw), fma(ow, d.z, zw)};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          double *out = Ji + ((size_t)sq * 3 + c) * t.D + dst;
          out[0] = v[c];
          out[t.nsf] = wq2 * vw[c];
        }
      }
    }
  }
}

// C(n, k) for n <= 4
double binom(int n, int k) {
  double b = 1.0;
  for (int q = 1; q <= k; ++q) b = b * (n - q + 1) / q;
  return b;
}

using Jac = decltype(&k_w64_jac<1, 1>);
template <int NAL>
Jac pick_jac(int deg) {
  return deg <= 1 ? k_w64_jac<NAL, 1> : (deg <= 2 ? k_w64_jac<NAL, 2> : k_w64_jac<NAL, 4>);
}

using Fwd = decltype(&k_w64_fwd<1, 1>);
using Bwd = decltype(&k_w64_bwd<1, 1>);

template <int NAL>
void pick_deg(int deg, Fwd *f, Bwd *b) {
  if (deg <= 1) { *f = k_w64_fwd<NAL, 1>; *b = k_w64_bwd<NAL, 1>; }
  else if (deg <= 2) { *f = k_w64_fwd<NAL, 2>; *b = k_w64_bwd<NAL, 2>; }
  else { *f = k_w64_fwd<NAL, 4>; *b = k_w64_bwd<NAL, 4>; }
}
void pick(int nal, int deg, Fwd *f, Bwd *b) {
  if (nal <= 1) pick_deg<1>(deg, f, b);
  else if (nal <= 2) pick_deg<2>(deg, f, b);
  else pick_deg<4>(deg, f, b);
}

int nal_pad(int n) { return n <= 1 ? 1 : (n <= 2 ? 2 : 4); }
int deg_pad(int d) { return d <= 1 ? 1 : (d <= 2 ? 2 : 4); }

constexpr size_t kSmemMax = 227 * 1024;

// blocks per atom: enough that every SM has about 8 blocks, at most the number
// of classes (one block per atom from 8 atoms per SM)
int split_of(int N) {
  const int want = 8 * device_sms();
  int s = 1;
  while (s < kClasses && N * s < want) s *= 2;
  return s;
}

}  // namespace

namespace {

// e = -alpha as exp_neg takes it, for arguments in units of 2^(E - 64) that are off
// by up to `units` of them (a pair's s3: 4, a slot's (r - rs)^2: 1).  Steep: that
// passes 2^-52 of the exponent (pairs from alpha = 4 at a cutoff of 6 A, slots
// from 64), so only arguments large enough for FP64 products to be off by as
// much take the units.
W64Exp exp_scale(double alpha, int E, int units) {
  W64Exp c = {-alpha, 0, 50, std::ldexp(std::fabs(alpha) * units, E) > 4096.0};
  if (alpha == 0.0) return c;
  const DD v = dd_mul({alpha, 0.0}, {0x1.71547652b82fep+10, 0x1.777d0ffda0d24p-46});
  int ea;
  std::frexp(v.h, &ea);
  c.frac = 64 - E - ea;
  if (!(alpha > 0.0 && std::isfinite(v.h)) || c.frac <= 0) {
    c.frac = -1;
    return c;
  }
  c.frac = std::min(c.frac, 63);
  const int bits = c.frac + E;  // m = 1024 alpha / ln 2 2^bits
  c.m = (unsigned long long)((__int128)std::ldexp(v.h, bits) +
                             (__int128)std::llround(std::ldexp(v.l, bits)));
  return c;
}

// The table of a model, or false when its SF set keeps the generic kernels.
bool w64_table(const SFDev &s, W64Tab *t, W64Fc *fc) {
  *t = W64Tab{};
  *fc = W64Fc{};
  t->nsf = s.nsf;
  t->D = s.D;
  t->nrad = s.nrad;
  t->nang = s.nang;
  t->nrc = s.nrc;
  t->ngrp = s.n_ang_grp;
  // the fixed-point units: 2^(e - 1) above every cutoff (with the screen's
  // margin), 2^er above every (r - rs)^2 within its cutoff
  double rmax = 0.0, u2max = 0.0;
  for (int q = 0; q < s.nrc; ++q) rmax = std::max(rmax, s.rc_val[q]);
  for (int q = 0; q < s.nrad; ++q) {
    const double u = std::max(std::fabs(s.rad_rs[q]), std::fabs(s.rc_val[s.rad_rc[q]] - s.rad_rs[q]));
    u2max = std::max(u2max, u * u);
  }
  std::frexp(1.001 * rmax, &fc->e);
  fc->e += 1;
  fc->close = (1023 + 9 - 2 * fc->e) * (1 << 20) - 1;
  std::frexp(std::max(u2max, 1e-30) * 1.001, &fc->er);
  for (int q = 0; q < s.nrc; ++q) {
    t->rc[q] = s.rc_val[q];
    const double kv = fc_series(s.rc_val[q], &fc->c[q]);
    // (a cutoff 2^30 times shorter than the longest: left to the generic kernels)
    fc->c[q].up = 2 * fc->e - (fc->c[q].top - 1022);
    if (fc->c[q].up > 62) return false;
    fc->c[q].rc2 = (unsigned long long)std::ldexp(s.rc_val[q] * s.rc_val[q], 64 - 2 * fc->e);
    fc->c[q].rc2d = s.rc_val[q] * s.rc_val[q];
    t->kd[q] = -kv;  // fc'(r) / r = (d fc / dw) kv
  }
  for (int q = 0; q < s.nrad; ++q) {
    t->rad_d[q] = s.rad_d[q];
    t->rad_rc[q] = s.rad_rc[q];
    t->rad_e[q] = exp_scale(s.rad_alpha[q], fc->er, 1);
    t->rad_rs[q] = s.rad_rs[q];
  }
  int nal = 1, deg = 1;
  for (int g = 0; g < s.n_ang_grp; ++g) {
    t->grp_rc[g] = s.ang_grp_rc[g];
    t->grp_start[g] = s.ang_grp_start[g];
    t->grp_start[g + 1] = s.ang_grp_start[g + 1];
    int n = 0;
    for (int a = s.ang_grp_start[g]; a < s.ang_grp_start[g + 1]; ++a) {
      if (s.ang_izeta[a] < 1 || s.ang_izeta[a] > 4) return false;
      deg = deg > s.ang_izeta[a] ? deg : s.ang_izeta[a];
      const double al = s.alpha_val[s.ang_alpha[a]];
      int q = 0;
      while (q < n && t->alpha[g][q].a != -al) ++q;
      if (q == 4) return false;
      if (q == n) {
        t->alpha[g][n++] = exp_scale(al, 2 * fc->e, 4);
      }
      t->ang_d[a] = s.ang_d[a];
      t->ang_g[a] = g;
      t->ang_q[a] = q;
    }
    nal = nal > n ? nal : n;
  }
  t->nal = nal_pad(nal);
  t->deg = deg_pad(deg);
  for (int a = 0; a < s.nang; ++a) {
    const int z = s.ang_izeta[a], R = t->deg - z;
    const bool neg = s.ang_lambda[a] < 0;
    for (int n = 0; n <= t->deg; ++n) {
      // (1 +- cos)^z = (2u)^z or (2w)^z, times (u + w)^R
      const int m = neg ? t->deg - n : n;
      t->bern[a][n] = m >= z ? s.ang_pref[a] * std::ldexp(binom(R, m - z), z) : 0.0;
      t->mono[a][n] = n <= z ? s.ang_pref[a] * binom(z, n) * ((neg && (n & 1)) ? -1.0 : 1.0) : 0.0;
    }
  }
  return true;
}

}  // namespace

// The model's table and 2^(j/1024) on the device; called when a model that
// is on the device takes, or is switched to, the FP64 form.
gapgb_status w64_prepare(gapgb_model *m) {
  if (m->d_w64 || m->w64_tried) return GAPGB_OK;
  m->w64_tried = true;
  if (!w64_table(m->sfh, &m->w64h, &m->w64fc)) return GAPGB_OK;
  GAPGB_CUDA_TRY(cudaMalloc(&m->d_exp64, 8 * kExpN));
  GAPGB_CUDA_TRY(cudaMemcpy(m->d_exp64, exp2_table(), 8 * kExpN, cudaMemcpyHostToDevice));
  GAPGB_CUDA_TRY(cudaMalloc(&m->d_w64, sizeof(W64Tab)));
  GAPGB_CUDA_TRY(cudaMemcpy(m->d_w64, &m->w64h, sizeof(W64Tab), cudaMemcpyHostToDevice));
  return GAPGB_OK;
}

namespace {

size_t fwd_smem(const gapgb_model *m, int capS) {
  const W64Tab &t = m->w64h;
  const size_t nm = 2 * t.nal * (t.deg + 1);
  return layout(capS, t.nrc, 8 * (4 * nm + (size_t)t.ngrp * kClasses * nm + 2 * kBlk)).total;
}
size_t bwd_smem(const gapgb_model *m, int capS) {
  const W64Tab &t = m->w64h;
  return layout(capS, t.nrc,
                (size_t)capS * 32 + 8 * ((size_t)t.D + 2 * t.nal * (t.deg + 1) + 36))
      .total;
}
// units of one group at most, and scalar records of a block's scratch
size_t group_units(int capS) {
  const size_t pairs = (size_t)capS * (capS - 1) / 2;
  return std::max<size_t>(1, (pairs + kUnit - 1) / kUnit);
}

constexpr size_t kScratchMax = (size_t)1 << 30;

// Scratch of one launch.  Descriptors: the moments of N atoms, split.
size_t fwd_bytes(const W64Tab &t, int N) {
  return sizeof(double) * (size_t)N * t.ngrp * kClasses * 2 * t.nal * (t.deg + 1);
}
// Gradient, split: scalars [N][nsc], group sums [N][ngrp][capS], radial sums,
// first units.
size_t split_nsc(const W64Tab &t, int capS) {
  return group_units(capS) * kUnit * std::max(1, t.ngrp);
}
size_t bwd_bytes(const W64Tab &t, int N, int capS) {
  return (size_t)N * (split_nsc(t, capS) * 32 + (t.ngrp > 1 ? (size_t)t.ngrp * capS * 32 : 0) +
                      (size_t)capS * 8 + (size_t)t.ngrp * 4);
}
// Gradient, one block per atom: a region per resident block.
size_t region_bytes(int capS) { return group_units(capS) * kUnit * 32; }
int resident(const W64Tab &t, int N, int capS, size_t smem) {
  Fwd f;
  Bwd b;
  pick(t.nal, t.deg, &f, &b);
  kernel_smem((const void *)b, (int)smem, true);
  const int gx = std::min(N, device_sms() * kernel_occupancy((const void *)b, kBlk, smem));
  return (int)std::min<size_t>(gx, std::max<size_t>(1, kScratchMax / region_bytes(capS)));
}
// The most that any batch of up to N atoms with capS slots takes.  A launch
// splits atoms only below kScratchMax; the largest batch of each split bounds
// the smaller ones.
size_t scratch_bound(const gapgb_model *m, int N, int capS) {
  const W64Tab &t = m->w64h;
  size_t b = resident(t, N, capS, bwd_smem(m, capS)) * region_bytes(capS);
  for (int s = 2; s <= kClasses; s *= 2) {
    const int n = std::min(N, (8 * device_sms() - 1) / (s / 2));  // the most atoms that take s
    b = std::max(b, std::min(kScratchMax, std::max(fwd_bytes(t, n), bwd_bytes(t, n, capS))));
  }
  return b;
}

}  // namespace

// Whether the kernels take a batch with capS slots per atom.  Also sizes their
// scratch: at least a region of the gradient's launch with one block per atom, so
// that the gradient of a batch always takes the kernels that its descriptors
// took; the launches split atoms, or keep more blocks resident, as far as it
// reaches (the results are the same).
bool w64_applies(const gapgb_model *m, Workspace &ws, int capS, cudaStream_t st) {
  return m->d_w64 && capS < 65536 && fwd_smem(m, capS) <= kSmemMax &&
         bwd_smem(m, capS) <= kSmemMax &&
         grow_scratch(ws, &ws.w64_scratch, &ws.w64_bytes, scratch_bound(m, ws.N, capS),
                      region_bytes(capS), st);
}

void launch_w64_fwd(const gapgb_model *m, Workspace &ws, int N, int cap, int capS, cudaStream_t st) {
  const W64Tab &t = m->w64h;
  const int NB = t.deg + 1, NM = 2 * t.nal * NB;
  Fwd f;
  Bwd b;
  pick(t.nal, t.deg, &f, &b);
  const size_t smem = fwd_smem(m, capS);
  kernel_smem((const void *)f, (int)smem, true);
  int split = split_of(N);
  if (fwd_bytes(t, N) > std::min(kScratchMax, ws.w64_bytes)) split = 1;
  const int gx = std::min(N, 1 << 20);
  f<<<dim3(gx, split), kBlk, smem, st>>>(N, cap, capS, ws.nbr_cnt, ws.nbr_xyz, ws.nbr_j, ws.apos,
                                         ws.nbr_d32, m->d_w64, m->w64fc, m->d_exp64,
                                         (double *)ws.G, (double *)ws.w64_scratch, split);
  if (split > 1 && t.nang > 0)
    k_w64_final<<<N, kBlk, 0, st>>>(N, NB, NM, m->d_w64, (const double *)ws.w64_scratch,
                                    (double *)ws.G);
}

void launch_w64_bwd(const gapgb_model *m, Workspace &ws, int N, int cap, int capS, cudaStream_t st) {
  const W64Tab &t = m->w64h;
  Fwd f;
  Bwd b;
  pick(t.nal, t.deg, &f, &b);
  const size_t smem = bwd_smem(m, capS);
  kernel_smem((const void *)b, (int)smem, true);
  int split = split_of(N), gx = N;
  size_t nsc = split_nsc(t, capS);
  if (bwd_bytes(t, N, capS) > std::min(kScratchMax, ws.w64_bytes)) split = 1;
  if (split == 1) {
    nsc = group_units(capS) * kUnit;
    gx = (int)std::min<size_t>(resident(t, N, capS, smem), ws.w64_bytes / region_bytes(capS));
  }
  double4 *sc = (double4 *)ws.w64_scratch;
  double4 *gp = split > 1 ? sc + (size_t)N * nsc : nullptr;
  double *rad = (double *)(gp + (split > 1 && t.ngrp > 1 ? (size_t)N * t.ngrp * capS : 0));
  int *first = (int *)(rad + (split > 1 ? (size_t)N * capS : 0));
  if (t.ngrp <= 1) gp = nullptr;
  b<<<dim3(gx, split), kBlk, smem, st>>>(N, cap, capS, ws.nbr_cnt, ws.nbr_xyz, ws.nbr_j, ws.apos,
                                         ws.nbr_d32, m->d_w64, m->w64fc, m->d_exp64,
                                         (const double *)ws.dedg, (double4 *)ws.gslot, ws.wvir, sc,
                                         rad, first, nsc, split);
  if (split > 1) {
    const size_t sg = layout(capS, t.nrc, (size_t)capS * 32 + 36 * 8).total;
    kernel_smem((const void *)k_w64_gather, (int)sg, true);
    // two threads per slot: few slots, small blocks (512 alloy atoms, 56 slots:
    // 31 us at 128 threads, 43 at 512)
    const int th = std::min(kGatherThreads, std::max(kBlk, (2 * capS + 63) / 64 * 64));
    k_w64_gather<<<dim3(N, std::max(1, t.ngrp)), th, sg, st>>>(
        cap, capS, ws.nbr_cnt, ws.nbr_xyz, ws.nbr_j, ws.apos, ws.nbr_d32, m->d_w64, m->w64fc,
        (double4 *)ws.gslot, ws.wvir, sc, rad, first, gp, nsc);
    if (gp) {
      kernel_smem((const void *)k_w64_finish, (int)sg, true);
      k_w64_finish<<<N, kBlk, sg, st>>>(cap, capS, ws.nbr_cnt, ws.nbr_xyz, ws.nbr_j, ws.apos,
                                        ws.nbr_d32, m->d_w64, m->w64fc, (double4 *)ws.gslot,
                                        ws.wvir, rad, gp);
    }
  }
}

// The Jacobians of the batch's atoms into J[N][capS][3][D]; false (nothing
// launched) when the batch does not take these kernels.
bool launch_w64_jac(const gapgb_model *m, Workspace &ws, int N, int cap, int capS, double *J,
                    cudaStream_t st) {
  if (!w64_applies(m, ws, capS, st)) return false;
  const W64Tab &t = m->w64h;
  int na = 1;
  for (int g = 0; g < t.ngrp; ++g) na = std::max(na, t.grp_start[g + 1] - t.grp_start[g]);
  const Jac f = t.nal <= 1 ? pick_jac<1>(t.deg) : (t.nal <= 2 ? pick_jac<2>(t.deg) : pick_jac<4>(t.deg));
  const size_t smem = layout(capS, t.nrc, 0).total, nsc = group_units(capS) * kUnit * na;
  kernel_smem((const void *)f, (int)smem, true);
  int gx = std::min(N, device_sms() * kernel_occupancy((const void *)f, kBlk, smem));
  gx = (int)std::min<size_t>(gx, std::max<size_t>(1, kScratchMax / (nsc * 32)));
  if (!grow_scratch(ws, &ws.w64_scratch, &ws.w64_bytes, gx * nsc * 32, gx * nsc * 32, st))
    return false;
  f<<<gx, kBlk, smem, st>>>(N, cap, capS, ws.nbr_cnt, ws.nbr_xyz, ws.nbr_j, ws.apos, ws.nbr_d32,
                            m->d_w64, m->w64fc, m->d_exp64, J, (double4 *)ws.w64_scratch, nsc, na);
  return true;
}

}  // namespace gapgb
