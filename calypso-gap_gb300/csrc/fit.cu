// fit.cu - sparse-GPR coefficients from training energies, on the device.
//
// The reference evaluates E = sum_i sum_k c_k K(x_i, m_k) (GET_COV and the
// energy sum of FGAP_CALC, gappy/libgap/gap_calc.f90:143-154, 268-288) with
// coefficients fitted elsewhere (calypso.x / ngap.x, not part of the
// repository).  This file fits them from structure energies, and optionally
// forces, with the sparse (subset-of-regressors) normal equations:
//   Phi_sk = sum_{i in s} K(x_i, m_k)                  (structure design rows)
//   PhiF_rk = force component r of the model with c = e_k  (force design rows)
//   PhiS_rk = stress component r (GPa) of the model with c = e_k  (stress rows)
//   A      = K_MM + jitter I + sum_s w_s Phi_s^T Phi_s + PhiF^T PhiF / sigma_f^2
//            + PhiS^T PhiS / sigma_s^2
//   b      = sum_s w_s Phi_s^T E_s + PhiF^T F / sigma_f^2 + PhiS^T sigma / sigma_s^2,
//   w_s = 1 / (sigma_e^2 n_s)
//   A c = b                                           (Cholesky, FP64)
// sigma_e is a per-atom energy noise (independent per atom, so a structure of
// n_s atoms has variance n_s sigma_e^2).  Everything is FP64: A inherits
// K_MM's conditioning.
//
// Kernel values (Phi, K_MM) come from the tensor cores where the model has
// their images (gpr64_tc.cu).  Force and stress rows: the descriptors'
// Jacobians once, one FP64 product per atom for all sparse points, then the
// force gather and the virials; a gradient pass per point (the dE/dG of the
// unit coefficient e_k) where the Jacobians are not to be had.  Then a tiled
// FP64 Gram product, a blocked right-looking Cholesky that carries the
// forward substitution, its trailing updates beside the next block's factor
// and panel, and a back substitution of one launch per block.  No kernel
// waits on another CTA.  Measured per call: 48 alloy512 cells and 1500 points
// 45.5 -> 8.4 ms, 8 Si cells of 64 atoms with forces and stresses and 150
// points 91 -> 3.2 ms.
#include <algorithm>
#include <string>
#include <vector>

#include "gapgb_internal.h"

namespace gapgb {
namespace {

constexpr int kT = 64;    // tile / block width
constexpr int kDC = 32;   // descriptor chunk staged in shared memory
constexpr int kRowsPerPass = 32;  // atoms per pass of the design-row kernel
constexpr int kKC = 16;   // contraction chunk of the tiled products

// Phi[s][k] = sum over structure s's atoms of exp(-1/2 |x_i / theta - m_k / theta|^2);
// structure s = atoms [off[s], off[s+1]) of the rows of G.  Block (k tile, s);
// zero for padded columns.
__global__ void __launch_bounds__(256)
    k_fit_phi(int M, int Mp, int D, const int *__restrict__ off, const double *__restrict__ G,
              const double *__restrict__ invth, const double *__restrict__ mmt,
              double *__restrict__ phi) {
  __shared__ double xs[kRowsPerPass][kDC + 1];
  __shared__ double ms[kT][kDC + 1];
  __shared__ double red[4][kT];
  const int tid = threadIdx.x, tx = tid & 63, ty = tid >> 6;
  const int s = blockIdx.y, kb = blockIdx.x * kT, k = kb + tx;
  const int a0 = off[s], a1 = off[s + 1];
  double sum = 0.0;
  for (int r0 = a0; r0 < a1; r0 += kRowsPerPass) {
    double acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.0;
    for (int d0 = 0; d0 < D; d0 += kDC) {
      for (int e = tid; e < kRowsPerPass * kDC; e += 256) {
        const int r = e / kDC, d = d0 + e % kDC, i = r0 + r;
        xs[r][e % kDC] = (i < a1 && d < D) ? G[(size_t)i * D + d] * invth[d] : 0.0;
      }
      for (int e = tid; e < kT * kDC; e += 256) {
        const int kk = kb + e / kDC, d = d0 + e % kDC;
        ms[e / kDC][e % kDC] = (kk < M && d < D) ? mmt[(size_t)kk * D + d] : 0.0;
      }
      __syncthreads();
#pragma unroll 4
      for (int d = 0; d < kDC; ++d) {
        const double mv = ms[tx][d];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const double t = xs[ty + 4 * q][d] - mv;
          acc[q] += t * t;
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (r0 + ty + 4 * q < a1) sum += exp(-0.5 * acc[q]);
  }
  red[ty][tx] = sum;
  __syncthreads();
  if (ty == 0) {
    const double v = ((red[0][tx] + red[1][tx]) + red[2][tx]) + red[3][tx];
    phi[(size_t)s * Mp + k] = k < M ? v : 0.0;
  }
}

// K_MM[r][k] = exp(-1/2 |m_r / theta - m_k / theta|^2) into A (rows < M; zero
// for padded columns).  Block (k tile, 32-row tile).
__global__ void __launch_bounds__(256)
    k_fit_kmm(int M, int Mp, int D, const double *__restrict__ mmt, double *__restrict__ A) {
  __shared__ double xs[kRowsPerPass][kDC + 1];
  __shared__ double ms[kT][kDC + 1];
  const int tid = threadIdx.x, tx = tid & 63, ty = tid >> 6;
  const int rb = blockIdx.y * kRowsPerPass, kb = blockIdx.x * kT;
  double acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.0;
  for (int d0 = 0; d0 < D; d0 += kDC) {
    for (int e = tid; e < kRowsPerPass * kDC; e += 256) {
      const int r = rb + e / kDC, d = d0 + e % kDC;
      xs[e / kDC][e % kDC] = (r < M && d < D) ? mmt[(size_t)r * D + d] : 0.0;
    }
    for (int e = tid; e < kT * kDC; e += 256) {
      const int k = kb + e / kDC, d = d0 + e % kDC;
      ms[e / kDC][e % kDC] = (k < M && d < D) ? mmt[(size_t)k * D + d] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int d = 0; d < kDC; ++d) {
      const double mv = ms[tx][d];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double t = xs[ty + 4 * q][d] - mv;
        acc[q] += t * t;
      }
    }
    __syncthreads();
  }
  const int k = kb + tx;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int r = rb + ty + 4 * q;
    if (r < M) A[(size_t)r * Mp + k] = k < M ? exp(-0.5 * acc[q]) : 0.0;
  }
}

// A[r][c] (lower tiles only) = base[r][c] + sum_s w_s Phi_sr Phi_sc, and the
// padded diagonal set to 1; base = K_MM + jitter I (in A already).  Block
// (c tile, r tile, slice) with c tile <= r tile.  One slice: adds to A.
// Several (few tiles, many rows: 150 points x 1536 force rows were 6 CTAs,
// 1.1 ms): the slices' sums go to part[slice][Mp][Mp], added in order by
// k_fit_gram_add.
__global__ void __launch_bounds__(256)
    k_fit_gram(int S, int M, int Mp, const double *__restrict__ phi, const double *__restrict__ w,
               double *__restrict__ A, double *__restrict__ part) {
  const int rt = blockIdx.y, ct = blockIdx.x;
  if (ct > rt) return;
  __shared__ double Rs[kKC][kT + 1];
  __shared__ double Cs[kKC][kT + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int rb = rt * kT, cb = ct * kT;
  const int per = ((S + gridDim.z - 1) / gridDim.z + kKC - 1) / kKC * kKC;
  const int sb = blockIdx.z * per, se = min(S, sb + per);
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  for (int s0 = sb; s0 < se; s0 += kKC) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = tid + 256 * q, ss = e / kT, j = e % kT, s = s0 + ss;
      const bool live = s < se;
      const double ws = live ? w[s] : 0.0;
      Rs[ss][j] = live ? phi[(size_t)s * Mp + rb + j] * ws : 0.0;
      Cs[ss][j] = live ? phi[(size_t)s * Mp + cb + j] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int ss = 0; ss < kKC; ++ss) {
      double a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a[u] = Rs[ss][ty * 4 + u];
        b[u] = Cs[ss][tx * 4 + u];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = rb + ty * 4 + u, c = cb + tx * 4 + v;
      if (part) {
        part[((size_t)blockIdx.z * Mp + r) * Mp + c] = acc[u][v];
        continue;
      }
      double *p = A + (size_t)r * Mp + c;
      if (r >= M || c >= M) *p = (r == c) ? 1.0 : 0.0;
      else *p += acc[u][v];
    }
}

// the slices' sums in order into A's lower tiles; the padded diagonal as above
__global__ void __launch_bounds__(256)
    k_fit_gram_add(int M, int Mp, int slices, const double *__restrict__ part,
                   double *__restrict__ A) {
  const int c = blockIdx.x * 256 + threadIdx.x, r = blockIdx.y;
  if (c >= Mp || c / kT > r / kT) return;
  double *p = A + (size_t)r * Mp + c;
  if (r >= M || c >= M) {
    *p = (r == c) ? 1.0 : 0.0;
    return;
  }
  double v = 0.0;
  for (int z = 0; z < slices; ++z) v += part[((size_t)z * Mp + r) * Mp + c];
  *p += v;
}

// b[k] += sum_s w_s Phi_sk E_s: 32 row groups per column, added in order
__global__ void __launch_bounds__(1024)
    k_fit_rhs(int S, int Mp, const double *__restrict__ phi, const double *__restrict__ w,
              const double *__restrict__ E, double *__restrict__ b) {
  __shared__ double red[32][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, k = blockIdx.x * 32 + tx;
  double acc = 0.0;
  for (int s = ty; s < S; s += 32) acc = fma(w[s] * E[s], phi[(size_t)s * Mp + k], acc);
  red[ty][tx] = acc;
  __syncthreads();
  if (ty == 0) {
    double v = 0.0;
    for (int q = 0; q < 32; ++q) v += red[q][tx];
    b[k] += v;
  }
}

// dE/dG of the model with c = e_k (one sparse point, unit coefficient), the
// loop of gap_calc.f90:157-166 for one k:
//   dedg_id = -K_ik (x_id - m_kd) / theta_d^2,  K_ik = exp(-1/2 sum_d ((x_id - m_kd)/theta_d)^2)
// one warp per atom
__global__ void __launch_bounds__(128)
    k_fit_dedg_unit(int N, int D, int k, const double *__restrict__ G,
                    const double *__restrict__ invth, const double *__restrict__ mmt,
                    double *__restrict__ dedg) {
  const int lane = threadIdx.x & 31;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= N) return;
  double q[4];
  double s = 0.0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int d = lane + 32 * t;
    q[t] = d < D ? G[(size_t)i * D + d] * invth[d] - mmt[(size_t)k * D + d] : 0.0;
    s += q[t] * q[t];
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  const double K = exp(-0.5 * s);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int d = lane + 32 * t;
    if (d < D) dedg[(size_t)i * D + d] = -K * q[t] * invth[d];
  }
}

// ---- force and stress rows from the descriptors' Jacobians --------------------
// dE/dG of the unit coefficient e_k is B_dk = -K_ik (x_id - m_kd) / theta_d^2
// (above), so the slot gradients of all k are one product per atom,
//   g[slot xyz][k] = sum_d J[slot xyz][d] B_dk,
// at 3 P D multiply-adds per (atom, k), where a gradient pass per k costs a
// hundred FP64 instructions per pair of slots (64-atom cells, 46 slots, 480
// pairs, 150 points: 81 -> 1.7 ms).  FP64-pipe bound.
constexpr int kJK = 32;   // sparse points per block
constexpr int kJR = 48;   // (slot, xyz) rows per pass (16 slots)

// block (atom, tile of 32 points): g[(slot * 3 + xyz) * ld + k - k0] of points
// [k0, k0 + ld)
__global__ void __launch_bounds__(128)
    k_fit_jmul(int D, int capS, int M, int k0, int ld, const int *__restrict__ cnt,
               const double *__restrict__ G, const double *__restrict__ invth,
               const double *__restrict__ mmt, const double *__restrict__ J,
               double *__restrict__ g) {
  extern __shared__ __align__(16) double smj[];
  double *B = smj;                  // [D][kJK]
  double *Js = B + (size_t)D * kJK;  // [kJR][D + 1]
  __shared__ double Ks[4][kJK], xs[128];
  const int tid = threadIdx.x, i = blockIdx.x, kb = k0 + blockIdx.y * kJK;
  const int P = min(cnt[i], capS), rows = 3 * P, ldj = D + 1;
  for (int d = tid; d < D; d += 128) xs[d] = G[(size_t)i * D + d] * invth[d];
  __syncthreads();
  // x - m, and its squared length by four threads per point in a fixed order
  const int kk = tid & 31, part = tid >> 5, k = kb + kk;
  const bool live = k < M && k < k0 + ld;
  double s2 = 0.0;
  for (int d = part; d < D; d += 4) {
    const double q = live ? xs[d] - mmt[(size_t)k * D + d] : 0.0;
    B[d * kJK + kk] = q;
    s2 = fma(q, q, s2);
  }
  Ks[part][kk] = s2;
  __syncthreads();
  const double K = live ? exp(-0.5 * ((Ks[0][kk] + Ks[1][kk]) + (Ks[2][kk] + Ks[3][kk]))) : 0.0;
  for (int d = part; d < D; d += 4) B[d * kJK + kk] *= -K * invth[d];
  const int tx = tid & 7, ty = tid >> 3;  // 8 x 4 columns, 16 x 3 rows
  const double *Ji = J + (size_t)i * capS * 3 * D;
  double *gi = g + (size_t)i * capS * 3 * ld + blockIdx.y * kJK;
  for (int r0 = 0; r0 < rows; r0 += kJR) {
    __syncthreads();
    for (int e = tid; e < kJR * D; e += 128) {
      const int r = e / D, d = e - r * D;
      Js[r * ldj + d] = r0 + r < rows ? Ji[(size_t)(r0 + r) * D + d] : 0.0;
    }
    __syncthreads();
    double acc[3][4] = {};
#pragma unroll 4
    for (int d = 0; d < D; ++d) {
      double a[3], b[4];
#pragma unroll
      for (int u = 0; u < 3; ++u) a[u] = Js[(ty + 16 * u) * ldj + d];
#pragma unroll
      for (int v = 0; v < 4; ++v) b[v] = B[d * kJK + tx + 8 * v];
#pragma unroll
      for (int u = 0; u < 3; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
    }
#pragma unroll
    for (int u = 0; u < 3; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int r = r0 + ty + 16 * u, c = blockIdx.y * kJK + tx + 8 * v;
        if (r < rows && c < ld) gi[(size_t)r * ld + tx + 8 * v] = acc[u][v];
      }
  }
}

// force rows of atom j, points [k0, k0 + ld): F_j = sum_q g[j][q] minus the
// reverse slots' gradients (the gather of k_forces); thread = point
__global__ void __launch_bounds__(128)
    k_fit_jforce(int cap, int capS, int Mp, int k0, int ld, const int *__restrict__ cnt,
                 const int *__restrict__ nj, const int *__restrict__ rev,
                 const double *__restrict__ g, double *__restrict__ PhiF) {
  const int j = blockIdx.x, c = blockIdx.y * 128 + threadIdx.x;
  if (c >= ld) return;
  const int P = min(cnt[j], capS);
  double f[3] = {0.0, 0.0, 0.0};
  for (int q = 0; q < P; ++q) {
    const size_t idx = (size_t)j * cap + q;
    const double *own = g + ((size_t)j * capS + q) * 3 * ld + c;
    const int r = rev[idx];
#pragma unroll
    for (int x = 0; x < 3; ++x) f[x] += own[(size_t)x * ld];
    if (r >= 0) {
      const double *o = g + ((size_t)nj[idx] * capS + r) * 3 * ld + c;
#pragma unroll
      for (int x = 0; x < 3; ++x) f[x] -= o[(size_t)x * ld];
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x) PhiF[((size_t)j * 3 + x) * Mp + k0 + c] = f[x];
}

// slots whose reverse pair was not found (normally none), thread = point
__global__ void __launch_bounds__(128)
    k_fit_jorphans(int cap, int capS, int Mp, int k0, int ld, const int *__restrict__ flags,
                   const int *__restrict__ orphans, int orphan_cap, const int *__restrict__ nj,
                   const double *__restrict__ g, double *__restrict__ PhiF) {
  const int c = blockIdx.x * 128 + threadIdx.x, n = min(flags[2], orphan_cap);
  if (c >= ld) return;
  for (int o = 0; o < n; ++o) {
    const int idx = orphans[o], i = idx / cap, q = idx - i * cap, j = nj[idx];
    for (int x = 0; x < 3; ++x)
      PhiF[((size_t)j * 3 + x) * Mp + k0 + c] -= g[(((size_t)i * capS + q) * 3 + x) * ld + c];
  }
}

// virial of atom i for every point: vir[i][6][ld], sum_q d_q (x) g_q in the
// order 11 12 13 22 23 33
__global__ void __launch_bounds__(128)
    k_fit_jvirial(int cap, int capS, int ld, const int *__restrict__ cnt,
                  const double4 *__restrict__ xyzr, const double4 *__restrict__ apos,
                  const double *__restrict__ g, double *__restrict__ vir) {
  const int i = blockIdx.x, c = blockIdx.y * 128 + threadIdx.x;
  if (c >= ld) return;
  const int P = min(cnt[i], capS);
  const double4 pi = apos[i];
  double v[6] = {0, 0, 0, 0, 0, 0};
  for (int q = 0; q < P; ++q) {
    const double4 e = xyzr[(size_t)i * cap + q];
    const double d[3] = {e.x - pi.x, e.y - pi.y, e.z - pi.z};
    const double *gq = g + ((size_t)i * capS + q) * 3 * ld + c;
    const double x = gq[0], y = gq[ld], z = gq[2 * (size_t)ld];
    v[0] = fma(d[0], x, v[0]), v[1] = fma(d[0], y, v[1]), v[2] = fma(d[0], z, v[2]);
    v[3] = fma(d[1], y, v[3]), v[4] = fma(d[1], z, v[4]), v[5] = fma(d[2], z, v[5]);
  }
#pragma unroll
  for (int u = 0; u < 6; ++u) vir[((size_t)i * 6 + u) * ld + c] = v[u];
}

// stress rows of structure s: the atoms' virials in order, in GPa
__global__ void __launch_bounds__(128)
    k_fit_jstress(int Mp, int k0, int ld, const StructInfo *__restrict__ sinfo,
                  const double *__restrict__ vir, double *__restrict__ PhiS) {
  const int s = blockIdx.x, u = blockIdx.z, c = blockIdx.y * 128 + threadIdx.x;
  if (c >= ld) return;
  const int a0 = sinfo[s].a0, na = sinfo[s].na;
  double v = 0.0;
  for (int i = a0; i < a0 + na; ++i) v += vir[((size_t)i * 6 + u) * ld + c];
  const int at[6] = {0, 3, 5, 1, 4, 2};  // XX YY ZZ XY YZ ZX of 11 12 13 22 23 33
  PhiS[((size_t)s * 6 + at[u]) * Mp + k0 + c] = -v * (1.0 / kGPa2eVPang) / sinfo[s].volume;
}

// column k of the force design matrix: PhiF[r][k] = F_r for the unit coefficient
__global__ void k_fit_col(int R, int k, int Mp, const double *__restrict__ F,
                          double *__restrict__ PhiF) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < R) PhiF[(size_t)r * Mp + k] = F[r];
}

__global__ void k_fit_fill(int n, double v, double *__restrict__ x) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) x[r] = v;
}

__global__ void k_fit_weights(int S, const int *__restrict__ off, double inv_var,
                              double *__restrict__ w) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < S) w[s] = inv_var / (double)max(1, off[s + 1] - off[s]);
}

__global__ void k_fit_jitter(int M, int Mp, double jitter, double *__restrict__ A) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < M) A[(size_t)k * Mp + k] += jitter;
}

// ---- blocked Cholesky, lower, row-major, in place --------------------------

// Both kernels below work in sub-blocks of 16 columns whose code is run four
// times: the same steps unrolled over all 64 columns (each instruction run
// once) took 154 and 107 us, waiting for instructions.
constexpr int kSB = 16;

// the 64 x 64 diagonal block at (j0, j0), its part of L y = b and the
// diagonal's reciprocals.  One CTA: 16 lanes factor a 16 x 16 block (a row
// per lane in registers, columns by shuffles), the rows below it are solved a
// row per thread, all threads update the rest.  One dependent chain of 64
// square roots and of the FMAs one warp issues (64 cycles each): 99 us under
// ncu; it and the panel run beside the previous step's update.
__global__ void __launch_bounds__(256)
    k_chol_diag(int Mp, int j0, double *__restrict__ A, const double *__restrict__ b,
                double *__restrict__ y, double *__restrict__ inv, int *__restrict__ flags) {
  __shared__ double T[kT][kT + 1];
  __shared__ double iv[kT], ys[kT];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < kT * kT; e += 256) T[e / kT][e % kT] = A[(size_t)(j0 + e / kT) * Mp + j0 + e % kT];
  if (tid < kT) ys[tid] = b[j0 + tid];
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < kT; k += kSB) {
    if (tid < 32) {
      double a[kSB];
      const int r = k + (lane & (kSB - 1));
#pragma unroll
      for (int c = 0; c < kSB; ++c) a[c] = T[r][k + c];
      double t = ys[r];
#pragma unroll
      for (int c = 0; c < kSB; ++c) {
        double d = __shfl_sync(0xffffffffu, a[c], c);
        if (!(d > 0.0)) {  // not positive definite: flag it, keep going on a floor
          if (lane == 0) atomicOr(flags, kFlagNotPositiveDefinite);
          d = 1e-300;
        }
        // root and reciprocal from one reciprocal root, each corrected once
        const double v = rsqrt(d);
        double s = d * v;
        s = fma(0.5 * v, fma(-s, s, d), s);
        const double w = fma(v, fma(-s, v, 1.0), v);
        const double l = a[c] * w;
        a[c] = (lane & (kSB - 1)) == c ? s : l;
        if (lane == c) iv[k + c] = w;
        const double yc = __shfl_sync(0xffffffffu, t, c) * w;
        if ((lane & (kSB - 1)) == c) t = yc;
        else if ((lane & (kSB - 1)) > c) t = fma(-l, yc, t);
#pragma unroll
        for (int m = c + 1; m < kSB; ++m) {
          const double lm = __shfl_sync(0xffffffffu, l, m);
          a[m] = fma(-l, lm, a[m]);
        }
      }
      if (lane < kSB) {
#pragma unroll
        for (int c = 0; c < kSB; ++c) T[r][k + c] = a[c];
        ys[r] = t;
      }
    }
    __syncthreads();
    // rows below within the block
    const int r = k + kSB + tid;
    if (r < kT) {
      double x[kSB], t = ys[r];
#pragma unroll
      for (int c = 0; c < kSB; ++c) x[c] = T[r][k + c];
#pragma unroll
      for (int c = 0; c < kSB; ++c) {
        const double q = x[c] * iv[k + c];
        x[c] = fma(fma(-q, T[k + c][k + c], x[c]), iv[k + c], q);
        t = fma(-x[c], ys[k + c], t);
#pragma unroll
        for (int m = c + 1; m < kSB; ++m) x[m] = fma(-x[c], T[k + m][k + c], x[m]);
      }
#pragma unroll
      for (int c = 0; c < kSB; ++c) T[r][k + c] = x[c];
      ys[r] = t;
    }
    __syncthreads();
    // the rest's lower 16 x 16 blocks, an entry of each per thread: up to six
    // independent chains of 16 FMAs
    const int nb = (kT - k) / kSB - 1, ti = tid / kSB, tj = tid % kSB, o = k + kSB;
    double v[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int bi = q < 1 ? 0 : (q < 3 ? 1 : 2), bj = q - bi * (bi + 1) / 2;
      if (bi < nb) v[q] = T[o + bi * kSB + ti][o + bj * kSB + tj];
    }
#pragma unroll
    for (int c = 0; c < kSB; ++c)
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const int bi = q < 1 ? 0 : (q < 3 ? 1 : 2), bj = q - bi * (bi + 1) / 2;
        if (bi < nb) v[q] = fma(-T[o + bi * kSB + ti][k + c], T[o + bj * kSB + tj][k + c], v[q]);
      }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int bi = q < 1 ? 0 : (q < 3 ? 1 : 2), bj = q - bi * (bi + 1) / 2;
      if (bi < nb) T[o + bi * kSB + ti][o + bj * kSB + tj] = v[q];
    }
    __syncthreads();
  }
  if (tid < kT) {
    y[j0 + tid] = ys[tid];
    inv[j0 + tid] = iv[tid];
  }
  for (int e = tid; e < kT * kT; e += 256)
    if (e % kT <= e / kT) A[(size_t)(j0 + e / kT) * Mp + j0 + e % kT] = T[e / kT][e % kT];
}

// rows below the diagonal block: L[i][j0:j0+64] = A[i][j0:j0+64] L_jj^-T and
// b[i] -= L[i][j0:j0+64] y.  16 rows per CTA (a panel then spreads over the
// SMs); per 16 columns, the finished columns' products by all threads and a
// substitution by a row per lane, column by column so that its updates are
// independent (a whole row as one chain of 2016 FMAs took 141 us a panel of
// 1500 points).  Quotients are products with the reciprocal corrected once.
constexpr int kPR = 16;
__global__ void __launch_bounds__(256)
    k_chol_panel(int Mp, int j0, double *__restrict__ A, const double *__restrict__ inv,
                 const double *__restrict__ y, double *__restrict__ b) {
  __shared__ double L[kT][kT + 1];
  __shared__ double X[kPR][kT + 1];
  __shared__ double iv[kT], ys[kT];
  const int tid = threadIdx.x;
  const int i0 = j0 + kT + blockIdx.x * kPR;  // Mp is a multiple of 64: in range
  for (int e = tid; e < kT * kT; e += 256) {
    const int r = e / kT, c = e % kT;
    L[r][c] = c <= r ? A[(size_t)(j0 + r) * Mp + j0 + c] : 0.0;
  }
  for (int e = tid; e < kPR * kT; e += 256) X[e / kT][e % kT] = A[(size_t)(i0 + e / kT) * Mp + j0 + e % kT];
  if (tid < kT) {
    iv[tid] = inv[j0 + tid];
    ys[tid] = y[j0 + tid];
  }
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < kT; k += kSB) {
    {
      const int r = tid / kSB, c = k + tid % kSB;  // 16 x 16 entries
      double v = X[r][c];
      for (int q = 0; q < k; ++q) v = fma(-X[r][q], L[c][q], v);
      X[r][c] = v;
    }
    __syncthreads();
    if (tid < kPR) {
      double x[kSB];
#pragma unroll
      for (int c = 0; c < kSB; ++c) x[c] = X[tid][k + c];
#pragma unroll
      for (int c = 0; c < kSB; ++c) {
        const double q = x[c] * iv[k + c];
        x[c] = fma(fma(-q, L[k + c][k + c], x[c]), iv[k + c], q);
#pragma unroll
        for (int m = c + 1; m < kSB; ++m) x[m] = fma(-x[c], L[k + m][k + c], x[m]);
      }
#pragma unroll
      for (int c = 0; c < kSB; ++c) X[tid][k + c] = x[c];
    }
    __syncthreads();
  }
  for (int e = tid; e < kPR * kT; e += 256) A[(size_t)(i0 + e / kT) * Mp + j0 + e % kT] = X[e / kT][e % kT];
  if (tid < kPR) {
    double t = b[i0 + tid];
    for (int c = 0; c < kT; ++c) t = fma(-X[tid][c], ys[c], t);
    b[i0 + tid] = t;
  }
}

// trailing update: A[r][c] -= sum_{q < 64} L[r][j0+q] L[c][j0+q] for the
// lower tiles of rows / columns >= j0 + 64, in tiles of 32 x 32 (a 64 x 64
// tile is 68 us of one SM's FP64 pipe: 253 tiles on 152 SMs, or the few of the
// last steps, left most SMs waiting for it).  The first 64 columns (`rest`
// false: blockIdx.x = 2 row tile + column half), which the next diagonal block
// and panel wait for, or the other columns (blockIdx.x enumerates the pairs
// 2 <= column tile <= row tile), which run beside them on another stream.
constexpr int kUT = 32;
__global__ void __launch_bounds__(128)
    k_chol_update(int Mp, int j0, bool rest, double *__restrict__ A) {
  int t = blockIdx.x, rt = 0, ct = 0;
  if (rest) {
    // row tile rt + 2 holds rt + 1 of these column tiles
    rt = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((rt + 1) * (rt + 2) / 2 <= t) ++rt;
    while (rt * (rt + 1) / 2 > t) --rt;
    ct = t - rt * (rt + 1) / 2 + 2;
    rt += 2;
  } else {
    rt = t >> 1;
    ct = t & 1;
    if (ct > rt) return;
  }
  const int base = j0 + kT;
  const int rb = base + rt * kUT, cb = base + ct * kUT;
  __shared__ double Rs[kUT][kT + 1];
  __shared__ double Cs[kUT][kT + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int e = tid; e < kUT * kT; e += 128) {
    const int j = e / kT, q = e % kT;
    Rs[j][q] = A[(size_t)(rb + j) * Mp + j0 + q];
    Cs[j][q] = A[(size_t)(cb + j) * Mp + j0 + q];
  }
  __syncthreads();
  double acc[4][2] = {};
#pragma unroll 8
  for (int q = 0; q < kT; ++q) {
    double a[4], b[2];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = Rs[ty + 8 * u][q];
#pragma unroll
    for (int v = 0; v < 2; ++v) b[v] = Cs[tx + 16 * v][q];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int r = rb + ty + 8 * u, c = cb + tx + 16 * v;
      if (c <= r) A[(size_t)r * Mp + c] -= acc[u][v];
    }
}

// L^T c = y by blocks of 64 columns from the last one (the panels have already
// solved L y = b).  Every CTA substitutes within the block (a warp, by
// columns, its two rows per lane in registers), then takes the block's c out
// of 64 rows of y above it; CTA 0 writes c.  One launch per block spreads the
// reads of L over the SMs (one CTA for the whole solve read it at 0.03 TB/s:
// 10 ms at 1500 points with a serial substitution).
__global__ void __launch_bounds__(256)
    k_chol_back(int Mp, int j0, const double *__restrict__ A, double *y,
                const double *__restrict__ inv, double *__restrict__ c) {
  __shared__ double L[kT][kT + 1];
  __shared__ double cs[kT], iv[kT], part[4][kT];
  const int tid = threadIdx.x, cc = tid & 63, g = tid >> 6;
  for (int e = tid; e < kT * kT; e += 256) L[e / kT][e % kT] = A[(size_t)(j0 + e / kT) * Mp + j0 + e % kT];
  if (tid < kT) iv[tid] = inv[j0 + tid];
  // the rows' entries of this CTA's columns, loaded while the warp substitutes
  const int col = (int)blockIdx.x * kT + cc;
  double a[16];
#pragma unroll
  for (int q = 0; q < 16; ++q)
    a[q] = col < j0 ? A[(size_t)(j0 + 4 * q + g) * Mp + col] : 0.0;
  __syncthreads();
  if (tid < 32) {
    double v[2] = {y[j0 + tid], y[j0 + 32 + tid]};
#pragma unroll
    for (int h = 1; h >= 0; --h)
#pragma unroll 4
      for (int q = 31; q >= 0; --q) {
        const int r = 32 * h + q;
        double x = v[h] * iv[r];
        x = fma(fma(-x, L[r][r], v[h]), iv[r], x);
        x = __shfl_sync(0xffffffffu, x, q);
        if (tid == q) cs[r] = x;
        if (h == 1) {
          v[0] = fma(-L[r][tid], x, v[0]);
          if (tid < q) v[1] = fma(-L[r][32 + tid], x, v[1]);
        } else if (tid < q) {
          v[0] = fma(-L[r][tid], x, v[0]);
        }
      }
  }
  __syncthreads();
  if (blockIdx.x == 0 && tid < kT) c[j0 + tid] = cs[tid];
  double p = 0.0;
#pragma unroll
  for (int q = 0; q < 16; ++q) p = fma(a[q], cs[4 * q + g], p);
  part[g][cc] = p;
  __syncthreads();
  if (g == 0 && col < j0) y[col] -= ((part[0][cc] + part[1][cc]) + part[2][cc]) + part[3][cc];
}

template <typename T>
gapgb_status dev_alloc(T **p, size_t n) {
  if (cudaMalloc(p, n * sizeof(T)) != cudaSuccess) {
    set_last_error("cudaMalloc of " + std::to_string(n * sizeof(T)) + " bytes for the fit failed");
    return GAPGB_ERR_CUDA;
  }
  return GAPGB_OK;
}

}  // namespace

// Fits the coefficients from FP64 descriptors d_G[N][D] (structures by
// d_off, S + 1 offsets on the device), host energies[S] and, when forces is
// not null, host forces[N][3] (the neighbour list of the descriptors, built
// with capacity cap and slot count capS, must still be in the workspace);
// writes the M coefficients to host coeff.  Synchronises the stream.
gapgb_status fit_enqueue(gapgb_model *m, int S, int N, int cap, int capS, const int *d_off,
                         const double *d_G, const double *energy, const double *forces,
                         const double *stress, double sigma_e, double sigma_f, double sigma_s,
                         double jitter, double *coeff, cudaStream_t st) {
  const int M = m->host.M, D = m->host.D, Mp = (M + kT - 1) / kT * kT;
  const int R = forces ? 3 * N : 0;   // force rows
  const int RS = stress ? 6 * S : 0;  // stress rows
  const bool rowsFS = R > 0 || RS > 0;
  const int nt = Mp / kT, tiles = nt * (nt + 1) / 2;
  // slices of the rows of a normal-matrix product: several when the tiles
  // alone would leave most SMs idle
  auto slices = [&](int rows) { return std::max(1, std::min(2 * device_sms() / tiles, rows / 64)); };
  const int zmax = std::max(slices(S), std::max(slices(R), slices(RS)));
  // one allocation for everything (a dozen and a half of them, freed again at
  // the end, were a quarter of a small fit)
  gapgb_status s = GAPGB_OK;
  double *arena = nullptr;
  size_t need = 0;
  double **at[18];
  size_t off[18];
  int na = 0;
  auto want = [&](double **p, size_t n) {
    *p = nullptr;
    if (n == 0) return;
    at[na] = p;
    off[na++] = need;
    need += (n + 31) / 32 * 32;
  };
  double *phi, *A, *b, *y, *c, *inv, *w, *E, *Fk, *Sk, *Ek, *phif, *wf, *Fv, *phis, *ws6, *Sv, *gpart;
  want(&phi, (size_t)S * Mp), want(&A, (size_t)Mp * Mp), want(&b, Mp), want(&y, Mp), want(&c, Mp);
  want(&inv, Mp), want(&w, S), want(&E, S);
  want(&Fk, rowsFS ? (size_t)3 * N : 0), want(&Sk, rowsFS ? (size_t)6 * S : 0);
  want(&Ek, rowsFS ? S : 0);
  want(&phif, (size_t)R * Mp), want(&wf, R), want(&Fv, R);
  want(&phis, (size_t)RS * Mp), want(&ws6, RS), want(&Sv, RS);
  want(&gpart, zmax > 1 ? (size_t)zmax * Mp * Mp : 0);
  if ((s = dev_alloc(&arena, need))) return s;
  for (int q = 0; q < na; ++q) *at[q] = arena + off[q];
  auto tryc = [&](cudaError_t e) {
    if (e != cudaSuccess && s == GAPGB_OK) {
      set_last_error(std::string("fit: ") + cudaGetErrorString(e));
      s = GAPGB_ERR_CUDA;
    }
  };
  tryc(cudaMemcpyAsync(E, energy, sizeof(double) * S, cudaMemcpyHostToDevice, st));
  tryc(cudaMemsetAsync(A, 0, sizeof(double) * (size_t)Mp * Mp, st));
  tryc(cudaMemsetAsync(b, 0, sizeof(double) * (size_t)Mp, st));
  // Phi^T W Phi into A and Phi^T W y into b
  auto normal = [&](int rows, const double *ph, const double *wr, const double *yr) {
    const int z = slices(rows);
    k_fit_gram<<<dim3(nt, nt, z), 256, 0, st>>>(rows, M, Mp, ph, wr, A, z > 1 ? gpart : nullptr);
    if (z > 1)
      k_fit_gram_add<<<dim3((Mp + 255) / 256, Mp), 256, 0, st>>>(M, Mp, z, gpart, A);
    k_fit_rhs<<<Mp / 32, 1024, 0, st>>>(rows, Mp, ph, wr, yr, b);
  };
  // kernel values from the tensor cores where the model has their images
  if (!launch_kmm64(m, m->ws, Mp, A, st))
    k_fit_kmm<<<dim3(nt, (M + kRowsPerPass - 1) / kRowsPerPass), 256, 0, st>>>(M, Mp, D, m->d_mmt, A);
  k_fit_jitter<<<(M + 255) / 256, 256, 0, st>>>(M, Mp, jitter, A);
  k_fit_weights<<<(S + 255) / 256, 256, 0, st>>>(S, d_off, 1.0 / (sigma_e * sigma_e), w);
  if (!launch_phi64(m, m->ws, N, S, Mp, d_off, d_G, phi, st))
    k_fit_phi<<<dim3(nt, S), 256, 0, st>>>(M, Mp, D, d_off, d_G, m->d_invth, m->d_mmt, phi);
  normal(S, phi, w, E);
  if (R > 0 || RS > 0) {
    // force / stress rows: column k is the force field / stress of the unit
    // coefficient e_k, through the FP64 gradient kernel, the reverse-slot
    // gather and the structure sums
    Workspace &ws = m->ws;
    if (R > 0) {
      tryc(cudaMemcpyAsync(Fv, forces, sizeof(double) * R, cudaMemcpyHostToDevice, st));
      tryc(cudaMemsetAsync(phif, 0, sizeof(double) * (size_t)R * Mp, st));
      k_fit_fill<<<(R + 255) / 256, 256, 0, st>>>(R, 1.0 / (sigma_f * sigma_f), wf);
    }
    if (RS > 0) {
      tryc(cudaMemcpyAsync(Sv, stress, sizeof(double) * RS, cudaMemcpyHostToDevice, st));
      tryc(cudaMemsetAsync(phis, 0, sizeof(double) * (size_t)RS * Mp, st));
      k_fit_fill<<<(RS + 255) / 256, 256, 0, st>>>(RS, 1.0 / (sigma_s * sigma_s), ws6);
    }
    launch_reverse(ws, N, cap, st);
    // all sparse points from one pass over the pairs (the Jacobians), a chunk
    // of points at a time; a gradient pass per point where the Jacobians or
    // the batch's kernels are not to be had
    const size_t nj = (size_t)N * capS * 3;
    const int ld = std::min(M, std::max(kJK, (int)(((size_t)512 << 20) / (nj * 8)) / kJK * kJK));
    double *J = nullptr;
    bool jac = nj * D * 8 <= (size_t)16 << 30 &&
               cudaMalloc(&J, 8 * (nj * D + nj * ld + (size_t)N * 6 * ld)) == cudaSuccess;
    if (!jac) {
      J = nullptr;
      cudaGetLastError();
    }
    double *g = J + nj * D, *vir = g + nj * ld;
    jac = jac && launch_w64_jac(m, ws, N, cap, capS, J, st);
    if (jac) {
      const size_t smem = sizeof(double) * ((size_t)D * kJK + (size_t)kJR * (D + 1));
      kernel_smem((const void *)k_fit_jmul, (int)smem, true);
      for (int k0 = 0; k0 < M; k0 += ld) {
        const int n = std::min(ld, M - k0), by = (n + 127) / 128;
        k_fit_jmul<<<dim3(N, (n + kJK - 1) / kJK), 128, smem, st>>>(
            D, capS, M, k0, n, ws.nbr_cnt, d_G, m->d_invth, m->d_mmt, J, g);
        if (R > 0) {
          k_fit_jforce<<<dim3(N, by), 128, 0, st>>>(cap, capS, Mp, k0, n, ws.nbr_cnt, ws.nbr_j,
                                                    ws.nbr_rev, g, phif);
          k_fit_jorphans<<<by, 128, 0, st>>>(cap, capS, Mp, k0, n, ws.d_flags, ws.orphans,
                                             ws.orphan_cap, ws.nbr_j, g, phif);
        }
        if (RS > 0) {
          k_fit_jvirial<<<dim3(N, by), 128, 0, st>>>(cap, capS, n, ws.nbr_cnt, ws.nbr_xyz, ws.apos,
                                                     g, vir);
          k_fit_jstress<<<dim3(S, by, 6), 128, 0, st>>>(Mp, k0, n, ws.sinfo, vir, phis);
        }
      }
    }
    for (int k = 0; k < M && !jac; ++k) {
      k_fit_dedg_unit<<<(N + 3) / 4, 128, 0, st>>>(N, D, k, d_G, m->d_invth, m->d_mmt,
                                                   (double *)ws.dedg);
      launch_wacsf_bwd<double>(m, ws, N, cap, capS, Fk, st);
      if (R > 0) {
        launch_forces<double>(ws, N, cap, Fk, st);
        k_fit_col<<<(R + 255) / 256, 256, 0, st>>>(R, k, Mp, Fk, phif);
      }
      if (RS > 0) {
        launch_struct_reduce(ws, S, 1, Ek, Sk, nullptr, N, st);
        k_fit_col<<<(RS + 255) / 256, 256, 0, st>>>(RS, k, Mp, Sk, phis);
      }
    }
    if (jac) tryc(cudaStreamSynchronize(st));
    if (J) cudaFree(J);
    if (R > 0) normal(R, phif, wf, Fv);
    if (RS > 0) normal(RS, phis, ws6, Sv);
  }
  // right-looking Cholesky; the trailing update of step j beyond its first
  // tile column runs on the side stream, beside the diagonal block and panel
  // of step j + 1
  bool side = false;
  for (int j0 = 0; j0 < Mp; j0 += kT) {
    k_chol_diag<<<1, 256, 0, st>>>(Mp, j0, A, b, y, inv, m->ws.d_flags);
    const int nr = (Mp - j0 - kT) / kT;  // row tiles below
    if (nr == 0) break;
    k_chol_panel<<<nr * (kT / kPR), 256, 0, st>>>(Mp, j0, A, inv, y, b);
    if (side) cudaStreamWaitEvent(st, m->ev_join, 0);  // the previous step's update
    if (nr > 1) {
      cudaEventRecord(m->ev_fork, st);
      cudaStreamWaitEvent(m->side, m->ev_fork, 0);
      const int n32 = 2 * nr - 2;  // 32-row tiles past the first tile column
      k_chol_update<<<n32 * (n32 + 1) / 2, 128, 0, m->side>>>(Mp, j0, true, A);
      cudaEventRecord(m->ev_join, m->side);
    }
    side = nr > 1;
    k_chol_update<<<4 * nr, 128, 0, st>>>(Mp, j0, false, A);
  }
  if (side) cudaStreamWaitEvent(st, m->ev_join, 0);
  for (int j0 = Mp - kT; j0 >= 0; j0 -= kT)
    k_chol_back<<<std::max(1, j0 / kT), 256, 0, st>>>(Mp, j0, A, y, inv, c);
  tryc(cudaGetLastError());
  tryc(cudaMemcpyAsync(coeff, c, sizeof(double) * M, cudaMemcpyDeviceToHost, st));
  tryc(cudaStreamSynchronize(st));
  cudaFree(arena);
  return s;
}

}  // namespace gapgb
