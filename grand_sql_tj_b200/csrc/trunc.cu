// Reduced density matrices and the truncation operator on the device.
//
// Get_density_matrix_{sys,env}_new (code/tjsq/den_mat.f90:84-134) forms, per
// psi sector, rho = psi psi^T (system) or psi^T psi (environment) of the
// normalised wavefunction; Get_truncation_operator (den_mat.f90:141-383)
// diagonalises each rho (DSYEV), weighs the spectrum with the multiplet
// degeneracy 2S+1 for the entropies, sorts it, keeps kept_min..kept_max
// states by the discarded-weight rule and returns the kept eigenvectors.
//
// Here rho is one more grouped-GEMM pass (one cell per sector).  The
// eigen-decomposition follows the direct route of DSYEV's first stage and
// replaces its second: every sector is reduced to tridiagonal form by
// Householder reflections (one CTA per sector, or a thread-block cluster of
// 16 (8) CTAs for a large one), all eigenvalues come from
// Sturm-count multisection (one warp per eigenvalue), the host selects the
// kept states exactly as den_mat.f90 does, and only the kept eigenvectors
// are computed: inverse iteration on the tridiagonal matrix (one thread per
// vector), Gram-Schmidt orthonormalisation inside each kept block (by two
// matrix products for the vectors that inverse iteration left nearly
// orthogonal, vector by vector for the others), and the back-transformation by
// blocks of the stored reflectors, written straight into the truncation
// operator's layout, which stays on the device until the second call of the
// two-call protocol copies it out.  Everything is FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include <cooperative_groups.h>

#include "ctx.h"
#include "sturm.cuh"

namespace cg = cooperative_groups;

namespace tjb {

constexpr int EIG_THREADS = 512;
constexpr int EIG_MAX_N = 4096;
constexpr double EIG_EPS = 2.220446049250313e-16;        // 2^-52
constexpr double EIG_SAFMIN = 2.2250738585072014e-308;   // smallest normal FP64
constexpr int ORTH_THREADS = 512;
// A sector of up to TD_SMALL states is reduced in one CTA's shared memory (62
// states: 87 us, 133 from L2; with three rows a lane 96 would take 248 and 238,
// with five 160 720 and 558), one of up to TD_ONE states by one CTA from L2, one
// of at least TD_BIG by a whole cluster, and those between by either, whichever
// is done first for all sectors of a call (td_by_cluster).  Alone, 191 states
// take 0.85 ms in one CTA, 192 take 0.54 in a cluster and 0.84 in one CTA, 260
// 0.76 and 1.77, 319 0.96 and 3.0; but only seven clusters of 16 run at a time,
// so many equal sectors are done sooner side by side (14 of 180 states: 0.74 ms
// in one CTA each, 1.01 in clusters; 22 of 208: 1.03 and 2.32; 22 of 260: 1.78
// and 2.96).
constexpr int TD_SMALL = 64, TD_ONE = 191, TD_BIG = 320;

// Sum of the warps' partial sums r[0..nw-1] by every warp: lane w takes
// r[w] and a shuffle tree adds them, in the same order in every warp (a
// serial sum would chain 32 dependent shared-memory loads and adds).
__device__ __forceinline__ double warp_sum_slots(const double *r) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double s = lane < nw ? r[lane] : 0.0;
  for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  return s;
}

// Sum of one value per thread over the block, in a fixed order; every thread
// receives it.  red holds 32 doubles of shared memory.
__device__ __forceinline__ double block_sum(double x, double *red) {
  for (int k = 16; k > 0; k >>= 1) x += __shfl_xor_sync(0xffffffffu, x, k);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  return warp_sum_slots(red);
}

// Householder reduction of one symmetric sector matrix A (n x n,
// column-major, both triangles) to tridiagonal form T = Q^T A Q with
// Q = H_0 H_1 ... H_{n-2}, H_k = I - tau_k v_k v_k^T acting on the indices
// k+1..n-1 and v_k(k+1) = 1 (the lower-triangle scheme of LAPACK's dsytd2).
// v_k overwrites A(k+1:n, k); d and e receive the diagonal and the
// off-diagonal of T, info[4s..4s+3] its Gershgorin interval, max row sum and
// the Sturm-count pivot floor.  One CTA per sector (tridiag_small, tridiag_one)
// or one cluster per large sector (tridiag_coop).
// By all threads of one CTA: info, and the scaled diagonal ds and squared
// off-diagonal e2 that the Sturm counts read.  red: 48 doubles.
__device__ void tridiag_info(int s, int n, const double *d, const double *e, double *info, double *ds, double *e2,
                             double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double gl = 1e308, gu = -1e308, emax2 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double el = i > 0 ? fabs(e[i - 1]) : 0.0, er = i + 1 < n ? fabs(e[i]) : 0.0;
    gl = fmin(gl, d[i] - el - er);
    gu = fmax(gu, d[i] + el + er);
    if (i + 1 < n) emax2 = fmax(emax2, e[i] * e[i]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, o));
    gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, o));
    emax2 = fmax(emax2, __shfl_xor_sync(0xffffffffu, emax2, o));
  }
  __syncthreads();
  if (lane == 0) {
    red[warp] = gl;
    red[16 + warp] = gu;
    red[32 + warp] = emax2;
  }
  __syncthreads();
  for (int w = 0; w < nw; ++w) {
    gl = fmin(gl, red[w]);
    gu = fmax(gu, red[16 + w]);
    emax2 = fmax(emax2, red[32 + w]);
  }
  const double tnorm = fmax(fabs(gl), fabs(gu)), sc = tridiag_scale(tnorm);
  if (threadIdx.x == 0) {
    info[4 * s + 0] = gl;
    info[4 * s + 1] = gu;
    info[4 * s + 2] = tnorm;
    info[4 * s + 3] = EIG_SAFMIN * fmax(1.0, emax2);
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    ds[i] = d[i] * sc;
    const double es = i + 1 < n ? e[i] * sc : 0.0;
    e2[i] = es * es;
  }
}
static_assert(EIG_THREADS <= 512, "tridiag_info's scratch");

// One sector of up to 32 C states by one CTA, the matrix in shared memory.  Each
// warp keeps the whole reflector and the pending w, row lane + 32 c in register
// c of a lane, and owns the columns j = warp (mod NW): the rank-2 update of step
// k - 1, A <- A - v w^T - w v^T, is applied to them as they are read for
// p = A v of step k, whose entry j is (A being symmetric) the product of column
// j with v.  Every warp finds the reflector of column k and, from p, the new w
// for itself, so a step has one CTA barrier; the parts are a chain of three sums
// over a warp, a square root and a division, and the warps' instructions, most
// of them the same in each: NW = 8 of the CTA's 16 take part (62 states: 125 us
// with 4, 87 with 8, 96 with 16; the load of a column behind the store of the
// one before: 97).
template <int C, int NW>
__device__ void tridiag_small(int s, double *Aall, const int64_t *off, const int *dims, const int64_t *eoff,
                              double *dall, double *eall, double *tauall, double *info, double *dsall,
                              double *e2all, double *sm, double *red) {
  const int n = dims[s], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *A = Aall + off[s];
  double *d = dall + eoff[s], *e = eall + eoff[s], *tau = tauall + eoff[s];
  double *L = sm, *p = sm + n * n;   // p: two of n, by the parity of the step
  for (int x = tid; x < n * n; x += EIG_THREADS) L[x] = A[x];
  double vp[C], wp[C];
#pragma unroll
  for (int c = 0; c < C; ++c) vp[c] = wp[c] = 0.0;
  // entry j of a vector held as above
  auto at = [&](const double (&x)[C], int j) {
    double y = x[0];
#pragma unroll
    for (int c = 1; c < C; ++c) y = (j >> 5) == c ? x[c] : y;
    return __shfl_sync(0xffffffffu, y, j & 31);
  };
  auto wsum = [](double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  __syncthreads();
  for (int k = 0; k + 1 < n && warp < NW; ++k) {
    const int k1 = k + 1;
    const double wk = at(wp, k), vk = at(vp, k);
    double v[C], ss = 0.0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = lane + 32 * c;
      v[c] = i >= k && i < n ? L[k * n + i] - (vp[c] * wk + wp[c] * vk) : 0.0;
      if (i > k1) ss += v[c] * v[c];
    }
    ss = wsum(ss);
    const double dk = at(v, k), alpha = at(v, k1);
    double beta = alpha, t = 0.0, scl = 0.0;
    if (ss > 0.0) {
      const double nr = sqrt(alpha * alpha + ss);
      beta = alpha >= 0.0 ? -nr : nr;
      t = (beta - alpha) / beta;
      scl = 1.0 / (alpha - beta);
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = lane + 32 * c;
      v[c] = i > k1 ? v[c] * scl : i == k1 ? 1.0 : 0.0;
    }
    if (warp == k % NW) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int i = lane + 32 * c;
        if (i >= k1 && i < n) A[k * n + i] = v[c];
      }
      if (lane == 0) {
        d[k] = dk;
        e[k] = beta;
        tau[k] = t;
      }
    }
    double *pk = p + (k & 1) * n;
    for (int j0 = k1 + ((warp - k1) % NW + NW) % NW; j0 < n; j0 += 4 * NW) {
      // four columns' loads before their stores, which may alias them
      double acc[4], x[4][C];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double *Lj = L + (j0 + u * NW) * n + lane;
        const int top = j0 + u * NW < n ? n : 0;
#pragma unroll
        for (int c = 0; c < C; ++c) x[u][c] = lane + 32 * c >= k1 && lane + 32 * c < top ? Lj[32 * c] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = min(j0 + u * NW, n - 1);
        const double wj = at(wp, j), vj = at(vp, j);
        acc[u] = 0.0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          x[u][c] -= vp[c] * wj + wp[c] * vj;
          acc[u] += x[u][c] * v[c];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double *Lj = L + (j0 + u * NW) * n + lane;
        const int top = j0 + u * NW < n ? n : 0;
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (lane + 32 * c >= k1 && lane + 32 * c < top) Lj[32 * c] = x[u][c];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (lane == 0 && j0 + u * NW < n) pk[j0 + u * NW] = acc[u];
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
    double pv = 0.0, q[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = lane + 32 * c;
      q[c] = i >= k1 && i < n ? t * pk[i] : 0.0;
      pv += q[c] * v[c];
    }
    const double K = 0.5 * t * wsum(pv);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      wp[c] = q[c] - K * v[c];
      vp[c] = v[c];
    }
  }
  __syncthreads();
  if (tid == 0) {
    d[n - 1] = L[n * n - 1];   // the last reflector is none: nothing is pending
    tau[n - 1] = 0.0;
  }
  __syncthreads();
  tridiag_info(s, n, d, e, info, dsall + eoff[s], e2all + eoff[s], red);
}

// One sector too large for tridiag_small by one CTA, the matrix in L2: the
// rank-2 update of step k, A <- A - v w^T - w v^T, is applied inside the
// product p = A v of step k + 1, so each step reads and writes the trailing
// block once.
__device__ void tridiag_one(int s, double *Aall, const int64_t *off, const int *dims, const int64_t *eoff,
                            double *dall, double *eall, double *tauall, double *info, double *dsall, double *e2all,
                            double *sm, double *red, double &sh_tau, double &sh_scl) {
  const int n = dims[s], tid = threadIdx.x, nt = blockDim.x;
  double *A = Aall + off[s];
  double *d = dall + eoff[s], *e = eall + eoff[s], *tau = tauall + eoff[s];
  double *vp = sm, *wp = vp + n, *v = wp + n, *part = v + n;   // part: max(n, nt) entries
  if (n == 0) return;
  bool pending = false;
  for (int k = 0; k + 1 < n; ++k) {
    const int k1 = k + 1, m = n - k1;
    double *colk = A + (int64_t)k * n;
    // column k (rows k..n-1) with the pending update applied
    double ss = 0.0;
    for (int i = k + tid; i < n; i += nt) {
      double a = colk[i];
      if (pending) a -= vp[i] * wp[k] + wp[i] * vp[k];
      v[i] = a;
      if (i > k1) ss += a * a;
    }
    const double sigma2 = block_sum(ss, red);
    if (tid == 0) {
      d[k] = v[k];
      const double alpha = v[k1];
      double beta = alpha, t = 0.0, scl = 0.0;
      if (sigma2 > 0.0) {
        const double nr = sqrt(alpha * alpha + sigma2);
        beta = alpha >= 0.0 ? -nr : nr;
        t = (beta - alpha) / beta;
        scl = 1.0 / (alpha - beta);
      }
      e[k] = beta;
      tau[k] = t;
      sh_tau = t;
      sh_scl = scl;
    }
    __syncthreads();
    const double t = sh_tau, scl = sh_scl;
    for (int i = k1 + tid; i < n; i += nt) {
      const double x = i == k1 ? 1.0 : v[i] * scl;
      v[i] = x;
      colk[i] = x;
    }
    __syncthreads();
    // trailing block: apply the pending rank-2 update, p = A v
    const int R = min((m + 31) & ~31, nt), G = nt / R;
    const int g = tid / R, r = tid - g * R;
    if (g < G) {
      for (int ii = r; ii < m; ii += R) {
        const int i = k1 + ii;
        const double vpi = pending ? vp[i] : 0.0, wpi = pending ? wp[i] : 0.0;
        double acc = 0.0;
        double *a = A + (int64_t)(k1 + g) * n + i;
        const int64_t st = (int64_t)G * n;
        if (pending) {
          // eight loads issued before the eight stores: a store through a
          // may alias the next load, so loads and stores interleaved one
          // column at a time would wait out a full L2 round trip per column
          int jj = g;
          for (; jj + 7 * G < m; jj += 8 * G, a += 8 * st) {
            double x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = a[u * st];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int j = k1 + jj + u * G;
              x[u] -= vpi * wp[j] + wpi * vp[j];
              a[u * st] = x[u];
              acc += x[u] * v[j];
            }
          }
          for (; jj < m; jj += G, a += st) {
            const int j = k1 + jj;
            const double x = *a - (vpi * wp[j] + wpi * vp[j]);
            *a = x;
            acc += x * v[j];
          }
        } else {
#pragma unroll 4
          for (int jj = g; jj < m; jj += G, a += (int64_t)G * n) acc += *a * v[k1 + jj];
        }
        part[g * m + ii] = acc;
      }
    }
    __syncthreads();
    // p = tau A v, w = p - (tau/2)(p.v) v
    double pv = 0.0;
    for (int ii = tid; ii < m; ii += nt) {
      double p = 0.0;
      for (int q = 0; q < G; ++q) p += part[q * m + ii];
      p *= t;
      part[ii] = p;   // own entry only: q = 0 slot of the same ii
      pv += p * v[k1 + ii];
    }
    const double K = 0.5 * t * block_sum(pv, red);
    for (int ii = tid; ii < m; ii += nt) {
      const int i = k1 + ii;
      wp[i] = part[ii] - K * v[i];
      vp[i] = v[i];
    }
    pending = true;
    __syncthreads();
  }
  if (tid == 0) {
    d[n - 1] = A[(int64_t)(n - 1) * n + (n - 1)];
    if (n >= 1) tau[n - 1] = 0.0;
  }
  __syncthreads();
  tridiag_info(s, n, d, e, info, dsall + eoff[s], e2all + eoff[s], red);
}

// Sum of one value per thread over the block with one barrier: each warp's
// sum goes to its slot of red[2][32] (the half selected by the caller's
// alternating flag, so that the next sum does not overwrite a half still
// being read) and every thread adds the slots in the same order.
__device__ __forceinline__ double block_sum1(double x, double *red, int &half) {
  for (int k = 16; k > 0; k >>= 1) x += __shfl_xor_sync(0xffffffffu, x, k);
  double *r = red + 32 * half;
  half ^= 1;
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = x;
  __syncthreads();
  return warp_sum_slots(r);
}

// The same reduction of one large sector by the CL CTAs of a thread-block
// cluster, in panels of TD_NB reflectors as LAPACK's dsytrd does it: within a
// panel the trailing block A stays as it was at the panel's start and a step
// takes the rank-2 terms of the panel's earlier reflectors from the thin
// matrices V and W,
//   w = tau (A v - V (W^T v) - W (V^T v)) - (tau / 2) (p.v) v,
// and A <- A - V W^T - W V^T follows once per panel.  CTA c owns the columns
// (and the rows of V and W) j = c (mod CL).  As A is symmetric, entry j of A v
// is the product of owned column j with v, and entry j of the next column is an
// entry of owned column j.  A step has two exchanges:
//   1. the owned entries of column k (every CTA gets the whole column);
//   2. the CTA's parts of W^T a, V^T a and a.(A a), a the column below row
//      k + 1, and from the owner of column k + 1 its rows of V, W and A a, from
//      which every CTA finds that row's new w for itself.
// The reflector's scale is found by one warp while the others multiply, and
// enters the sums where they are read.
// A step is a chain of latencies (8 cycles an FP64 operation, 38 a level of a
// shuffle sum, 44 a CTA barrier; 48 doubles to each of 16 CTAs under a cluster
// barrier 2100, counted by the receiver's mbarrier 1380) and, with 16 warps, of
// instructions: so the exchanges are st.async, whole warps to consecutive
// places, and V, W, d, e and tau go to global memory at the panel's end only.
// The columns stay where they are between the panels' ends: as many of the
// last ones as fit live in the CTA's shared memory from the start, all of them
// from the first panel at which they fit; the others stream from L2.
// n = 857 on 16 CTAs: 8.6 us a step (7.3 ms) with the block read, updated and
// written in each and parts of A v exchanged under cluster barriers, 4.8 (4.1 ms)
// so; n = 320: 4.2 and 3.0.
constexpr int TD_NB = 16;              // reflectors of a panel
constexpr int TD_LD = 2 * TD_NB + 2;   // row of V and W in shared memory: V, W, pad
constexpr int TD_PT = 3 * TD_NB;       // a CTA's parts: W^T a, V^T a, a.(A a) by warp
constexpr double TD_CYCLES = 2e9;      // cycles a second, for the limit of the waits (tj_set_wait_limit)
constexpr int TD_PL = TD_PT + 1;       // their stride: odd, so that the CTAs' parts lie in different banks

// Doubles of shared memory besides the resident columns.
__host__ __device__ constexpr int td_coop_doubles(int n, int cl) {
  const int own = (n + cl - 1) / cl;
  return own * TD_LD + cl * (own | 1) + 2 * own + (cl + 1) * TD_PL + 2 * TD_LD + 3 * TD_NB + 8;
}

// acc[c] = column c . a, this lane's rows being i0, i0 + 32, ... below n; a is
// kept by owner (row i at (i mod CL) lc + i / CL).  dw and dv are summed over the
// warp with them if more.
template <int NC, int XS>
__device__ __forceinline__ void td_dots(const double *const (&p)[4], const double *x, int i0, int n, double (&acc)[4],
                                        bool more, double &dw, double &dv) {
#pragma unroll 4
  for (int i = i0; i < n; i += 32, x += XS) {
    const double a = *x;
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] += a * p[c][i];
  }
  if (more) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
      dw += __shfl_xor_sync(0xffffffffu, dw, o);
      dv += __shfl_xor_sync(0xffffffffu, dv, o);
    }
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  }
}

__device__ __forceinline__ uint32_t td_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// the shared-memory address of CTA r's copy of this CTA's place a
__device__ __forceinline__ uint32_t td_remote(uint32_t a, int r) {
  uint32_t o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(r));
  return o;
}
// v to another CTA's shared memory, counted there on the mbarrier bar
__device__ __forceinline__ void td_send(uint32_t dst, double v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void td_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of the given parity; false if it does not come within
// `limit` cycles (0: unless it has come already).
__device__ __forceinline__ bool td_wait(uint32_t bar, uint32_t parity, long long limit) {
  if (limit <= 0) {   // try_wait may block for a while, test_wait does not
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
  }
  const long long c0 = clock64();
  do {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  } while (clock64() - c0 < limit);
  return false;
}
__device__ __forceinline__ void td_dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int CL>
__device__ void tridiag_coop(cg::cluster_group &cl, int rank, int s, double *Aall, const int64_t *off,
                             const int *dims, const int64_t *eoff, double *dall, double *eall, double *tauall,
                             double *Wall, double *info, double *dsall, double *e2all, double *sm, int64_t smem_doubles,
                             double *red, uint64_t *mbar, int *status, long long limit) {
  constexpr int NB = TD_NB, NW = EIG_THREADS / 32, MW = NW - 1;   // MW warps multiply, the last finds the scale
  static_assert(NB == 16 && NW == 16 && CL <= NW, "the warps' shares below");
  const int n = dims[s], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *A = Aall + off[s], *Wg = Wall + NB * eoff[s];   // Wg: W, column-major
  double *d = dall + eoff[s], *e = eall + eoff[s], *tau = tauall + eoff[s];
  const int own = (n + CL - 1) / CL, lc = own | 1;        // an odd stride: no bank conflicts across owners
  const int nq = rank < n ? (n - 1 - rank) / CL + 1 : 0;  // owned columns rank + q CL
  auto own_from = [&](int i) { return i <= rank ? 0 : (i - rank + CL - 1) / CL; };  // first q with rank + q CL >= i
  double *vw = sm;                  // owned rows of V and W
  double *col = vw + own * TD_LD;   // column k: row i at (i % CL) lc + i / CL
  double *me = col + rank * lc;     // its owned entries
  double *ys = col + CL * lc;       // owned entries of A a (rows below k + 1 only)
  double *rk = ys + own;            // owned entries of row k + 1 of A
  double *part = rk + own;          // by CTA: its parts (TD_PT)
  double *stg = part + CL * TD_PL;  // the parts to send
  double *rb = stg + TD_PL;         // row k of V (NB), of W (NB), entries k of ys and rk
  double *cs = rb + TD_LD;          // W^T v, V^T v, a.(A a)
  double *de = cs + TD_LD;          // the panel's d, e, tau (NB each)
  double *sc = de + 3 * NB;         // scale and tau of the step
  double *sl = sc + 8;              // resident columns
  const int64_t cap = smem_doubles - td_coop_doubles(n, CL);
  // owned columns q >= qr are resident: row i of column q at sl[(q - qr) st + i - r0]
  int qr = nq - (int)min((int64_t)nq, max((int64_t)0, cap / n)), st = n, r0 = 0;
  auto res = [&](int q) -> double * { return sl + (int64_t)(q - qr) * st - r0; };
  auto glo = [&](int q) -> double * { return A + (int64_t)(rank + q * CL) * n; };
  for (int q = qr + warp; q < nq; q += NW)
    for (int i = lane; i < n; i += 32) res(q)[i] = glo(q)[i];
  // The exchanges: mbar[0] counts the bytes of column k, mbar[1] those of the
  // parts, one phase a step.  No buffer is doubled: a CTA sends its entries of
  // the next column once it has every CTA's parts, which each sends after its
  // last read of this column, and its next parts once it has every CTA's
  // entries, sent after the last read of the parts before.  (In the last
  // columns a CTA may own no row from k on: it sends no entries, the others may
  // be a step ahead of it, and their parts then count on its phase before and
  // overwrite parts that it has not summed.  It has no use for those sums, rows
  // of V and W to make being its only one, and over the phases the bytes are the
  // same.)
  const uint32_t bar0 = td_smem(mbar), bar1 = td_smem(mbar + 1);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // A wait that gives up leaves its phase open.  The thread that gave up neither
  // sends nor arrives nor waits any more; it only runs through the rest of the
  // steps, whose barriers the others count on, and the result is not used.  So
  // every store and every arrival is of a thread that has seen all earlier
  // phases complete, as the order above asks; and whoever misses the stores (or
  // its thread 0's arrival) gives up at its own next wait, so that no mbarrier
  // meets more than two steps' bytes.
  // (The thread's end of the owned columns to send says so, -1 once it gave up:
  // with a flag tested in front of the loop a step took 1 % longer.)
  int live = nq;
  auto wait = [&](uint32_t bar, uint32_t parity) {
    if (live >= 0 && !td_wait(bar, parity, limit)) live = -1;
  };
  int p = 0;   // the panel's first column
  // the panel's V (below each reflector's first row), d, e and tau to global memory
  auto flush = [&](int cols) {
    const int qp = own_from(p + 1);
    for (int x = tid; x < (nq - qp) * NB; x += EIG_THREADS) {
      const int q = qp + x / NB, l = x % NB, i = rank + q * CL;
      if (l < cols && i > p + l) A[(int64_t)(p + l) * n + i] = vw[q * TD_LD + l];
    }
    if (rank == 0 && tid < cols) {
      d[p + tid] = de[tid];
      e[p + tid] = de[NB + tid];
      tau[p + tid] = de[2 * NB + tid];
    }
  };
  cl.sync();
  for (int k = 0;; ++k) {
    // ---- v and w of step k - 1 (its panel column L), then the owned entries of column k
    const int q0 = own_from(k);
    const int grp = tid >> 3, h = tid & 7;
    bool fresh = k == p;   // column k is that of A itself
    if (!fresh) {
      const int L = k - 1 - p;
      const double scl = sc[0], t = sc[1];
      {
        const int dn = tid >> 4, r = tid & 15;
        double x = r < CL && (dn & 15) < L ? part[r * TD_PL + dn] : 0.0, y = 0.0;
        if (warp == MW) {
#pragma unroll
          for (int u = 0; u < CL / 2; ++u) y += part[(2 * u + (lane >> 4)) * TD_PL + 2 * NB + (lane & 15)];
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          x += __shfl_xor_sync(0xffffffffu, x, o);
          y += __shfl_xor_sync(0xffffffffu, y, o);
        }
        if (r == 0) cs[dn] = x * scl + ((dn & 15) < L ? rb[dn ^ 16] : 0.0);
        if (warp == MW) {
          y += __shfl_xor_sync(0xffffffffu, y, 16);
          if (lane == 0) cs[2 * NB] = y;
        }
      }
      __syncthreads();
      const bool last = L == NB - 1;
      // eight lanes a row: the row's sums, and those of row k with the totals
      // (cw: V(k) (W^T v) + W(k) (V^T v), ec: (W^T v).(V^T v))
      double cw = 0.0, ec = 0.0;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int l = h + 8 * u;
        if (l < L && q0 + 4 * warp < nq) {
          cw += rb[l] * cs[l] + rb[NB + l] * cs[NB + l];
          ec += cs[l] * cs[NB + l];
        }
      }
      // (a warp without rows has nothing to do: its instructions would only be in the others' way)
      const int qw = q0 + 4 * warp;
      for (int qb = qw; qb < nq; qb += EIG_THREADS / 8) {
        const int q = qb + (grp & 3);
        double P = 0.0, Q = 0.0;
        double *row = vw + q * TD_LD;
        if (q < nq) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int l = h + 8 * u;
            if (l < L) {
              const double v = row[l], w = row[NB + l];
              P += v * cs[l] + w * cs[NB + l];
              Q += v * rb[NB + l] + w * rb[l];
            }
          }
        }
        if (qb == qw) {
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            P += __shfl_xor_sync(0xffffffffu, P, o);
            Q += __shfl_xor_sync(0xffffffffu, Q, o);
            cw += __shfl_xor_sync(0xffffffffu, cw, o);
            ec += __shfl_xor_sync(0xffffffffu, ec, o);
          }
        } else {
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            P += __shfl_xor_sync(0xffffffffu, P, o);
            Q += __shfl_xor_sync(0xffffffffu, Q, o);
          }
        }
        // v_k = 1; v.(A v) from a.(A a), its row k and A's symmetry
        const double yk = rb[2 * NB] * scl + rb[2 * NB + 1];
        const double vy = scl * (scl * cs[2 * NB] + rb[2 * NB]) + yk;
        const double K = 0.5 * t * (t * (vy - 2.0 * ec));
        const double wk = t * (yk - cw) - K;
        if (q < nq && h == 0) {
          const double v = rank + q * CL == k ? 1.0 : me[q] * scl;
          const double w = t * (ys[q] * scl + rk[q] - P) - K * v;
          row[L] = v;
          row[NB + L] = w;
          me[q] = rk[q] - Q - (v * wk + w);   // not used at the panel's end
        }
      }
      __syncthreads();
      if (last) {
        // ---- the panel's rank-2 NB update of the owned columns from k on
        flush(NB);
        for (int x = tid; x < (nq - q0) * NB; x += EIG_THREADS) {
          const int q = q0 + x / NB, l = x % NB;
          Wg[(int64_t)l * n + rank + q * CL] = vw[q * TD_LD + NB + l];
        }
        cl.sync();
        // 8 x 8 tiles (owned columns x rows) by m8n8k4 products over [V | W]: a
        // warp holds the right-hand factors of 16 rows and takes the owned
        // columns past them (32 plain multiply-adds an entry would read their
        // factors from shared memory at 16 bytes a lane: four times as long)
        const int tr = lane >> 2, tk = lane & 3;
        for (int ib = k + 16 * warp; ib < n; ib += 16 * NW) {
          double bv[2][2 * NB / 4];
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int i = min(ib + 8 * g + tr, n - 1);   // a row past the end is not stored
            const double *Vp = A + (int64_t)p * n + i, *Wp = Wg + i;
#pragma unroll
            for (int u = 0; u < NB / 4; ++u) {
              bv[g][u] = __ldcg(Vp + (int64_t)(4 * u + tk) * n);
              bv[g][NB / 4 + u] = __ldcg(Wp + (int64_t)(4 * u + tk) * n);
            }
          }
          for (int q = q0; q < nq; q += 8) {
            const int qa = min(q + tr, nq - 1);   // nor a column past the last
            const double *row = vw + qa * TD_LD + tk;
            double *c0 = qa >= qr ? res(qa) : glo(qa);
            double c[2][2], av[2 * NB / 4];
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int i = ib + 8 * g + 2 * tk + u;
                c[g][u] = i < n ? c0[i] : 0.0;
              }
#pragma unroll
            for (int u = 0; u < NB / 4; ++u) {   // V of the rows meets W of the columns, and W V
              av[u] = -row[NB + 4 * u];
              av[NB / 4 + u] = -row[4 * u];
            }
#pragma unroll
            for (int u = 0; u < 2 * NB / 4; ++u)
#pragma unroll
              for (int g = 0; g < 2; ++g) td_dmma(c[g], av[u], bv[g][u]);
            if (q + tr < nq) {
#pragma unroll
              for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const int i = ib + 8 * g + 2 * tk + u;
                  if (i < n) c0[i] = c[g][u];
                }
            }
          }
        }
        __syncthreads();
        p = k;
        fresh = true;
        if (qr > q0 && (int64_t)(nq - q0) * (n - k) <= cap) {
          // all owned columns fit from here on
          for (int q = qr + warp; q < nq; q += NW)
            for (int i = k + lane; i < n; i += 32) glo(q)[i] = res(q)[i];
          __syncthreads();
          qr = q0;
          st = n - k;
          r0 = k;
          for (int q = qr + warp; q < nq; q += NW)
            for (int i = k + lane; i < n; i += 32) res(q)[i] = glo(q)[i];
          __syncthreads();
        }
      }
    }
    const int jc = k - p;   // the step's column of the panel
    if (fresh) {
      for (int q = q0 + tid; q < nq; q += EIG_THREADS) me[q] = q >= qr ? res(q)[k] : glo(q)[k];
      __syncthreads();
    }
    // warp w sends the owned entries to CTA w
    if (warp < CL && warp != rank) {
      const uint32_t o = td_remote(td_smem(me), warp), ob = td_remote(bar0, warp);
      for (int q = q0 + lane; q < live; q += 32) td_send(o + q * 8, me[q], ob);
    }
    if (live >= 0 && tid == 0) td_expect(bar0, (uint32_t)(n - k - (nq - q0)) * 8);
    wait(bar0, k & 1);
    if (rank == 0 && tid == 0) de[jc] = col[k % CL * lc + k / CL];
    if (k == n - 1) break;
    // ---- the reflector's scale; A a
    const int k1 = k + 1, q1 = own_from(k1);
    const int ia = k1 + 1 + lane;   // a starts at row k1 + 1
    const double *xa = col + ia % CL * lc + ia / CL;
    if (warp == MW) {
      const double alpha = col[k1 % CL * lc + k1 / CL];
      double s4[4] = {0.0, 0.0, 0.0, 0.0};
      const double *x = xa;
      int i = ia;
      for (; i + 96 < n; i += 128, x += 128 / CL) {
#pragma unroll
        for (int u = 0; u < 4; ++u) s4[u] += x[u * (32 / CL)] * x[u * (32 / CL)];
      }
      for (; i < n; i += 32, x += 32 / CL) s4[0] += *x * *x;
      double ss = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) {
        double beta = alpha, t = 0.0, scl = 0.0;
        if (ss > 0.0) {
          const double nr = sqrt(alpha * alpha + ss);
          beta = alpha >= 0.0 ? -nr : nr;
          t = (beta - alpha) / beta;
          scl = 1.0 / (alpha - beta);
        }
        sc[0] = scl;
        sc[1] = t;
        de[NB + jc] = beta;
        de[2 * NB + jc] = t;
        stg[2 * NB + MW] = 0.0;
      }
    } else {
      // parts of W^T a and V^T a: column l = warp
      double dw = 0.0, dv = 0.0, ya = 0.0;
      bool more = warp < jc;   // dw and dv are still to be summed
      if (warp < jc)
        for (int q = own_from(k1 + 1) + lane; q < nq; q += 32) {
          const double a = me[q];
          dw += a * vw[q * TD_LD + NB + warp];
          dv += a * vw[q * TD_LD + warp];
        }
      auto batch = [&](auto colptr, int qa, int qe) {
        for (int qb = qa + warp; qb < qe; qb += 4 * MW) {
          const double *cp[4];
          double f[4], acc[4] = {0.0, 0.0, 0.0, 0.0};
          const int nc = min(4, (qe - 1 - qb) / MW + 1);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            cp[c] = colptr(c < nc ? qb + c * MW : qb);
            f[c] = cp[c][k1];
          }
          switch (nc) {
            case 1: td_dots<1, 32 / CL>(cp, xa, ia, n, acc, more, dw, dv); break;
            case 2: td_dots<2, 32 / CL>(cp, xa, ia, n, acc, more, dw, dv); break;
            case 3: td_dots<3, 32 / CL>(cp, xa, ia, n, acc, more, dw, dv); break;
            default: td_dots<4, 32 / CL>(cp, xa, ia, n, acc, more, dw, dv); break;
          }
          more = false;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c >= nc) break;
            const int q = qb + c * MW;
            if (rank + q * CL != k1) ya += acc[c] * me[q];
            if (lane == 0) {
              ys[q] = acc[c];
              rk[q] = f[c];
            }
          }
        }
      };
      if (q1 < qr) batch([&](int q) -> const double * { return glo(q); }, q1, qr);
      batch([&](int q) -> const double * { return res(q); }, max(q1, qr), nq);
      if (more)
        for (int o = 16; o > 0; o >>= 1) {
          dw += __shfl_xor_sync(0xffffffffu, dw, o);
          dv += __shfl_xor_sync(0xffffffffu, dv, o);
        }
      if (lane == 0) {
        stg[warp] = dw;
        stg[NB + warp] = dv;
        stg[2 * NB + warp] = ya;
      }
    }
    __syncthreads();
    // warp w sends the parts, and the owner of row k1 its row, to CTA w
    if (live >= 0 && warp < CL) {
      const uint32_t o = td_remote(td_smem(part + rank * TD_PL), warp), ob = td_remote(bar1, warp);
      td_send(o + lane * 8, stg[lane], ob);
      if (lane < NB) td_send(o + (2 * NB + lane) * 8, stg[2 * NB + lane], ob);
      if (k1 % CL == rank) {
        const uint32_t b = td_remote(td_smem(rb), warp);
        td_send(b + lane * 8, vw[k1 / CL * TD_LD + lane], ob);
        if (lane < 2) td_send(b + (2 * NB + lane) * 8, (lane ? rk : ys)[k1 / CL], ob);
      }
    }
    if (live >= 0 && tid == 0) td_expect(bar1, (CL * TD_PT + TD_LD) * 8);
    wait(bar1, k & 1);
  }
  __syncthreads();
  flush(n - 1 - p);
  if (rank == 0 && tid == 0) {
    d[n - 1] = de[n - 1 - p];
    tau[n - 1] = 0.0;
  }
  const bool late = __syncthreads_or(live < 0);
  if (late && tid == 0) atomicOr(status, 4);
  __threadfence();
  cl.sync();   // every owner's writes are visible, and no CTA sends any more
  if (late) {
    // what this CTA did not wait for may still be on its way here: it does not leave at once
    const long long c0 = clock64();
    while (clock64() - c0 < 1000000) {
    }
  }
  if (rank == 0) tridiag_info(s, n, d, e, info, dsall + eoff[s], e2all + eoff[s], red);
}

// One cluster of CL CTAs per entry of the cluster list: a large sector
// shared by all of them (tbig), or up to CL small sectors, one per CTA
// (tsec[cluster * CL + rank], -1 for none).  Sectors largest first.  CL is
// 16 where the GPU can schedule clusters of 16 such CTAs (a non-portable
// size), else 8.
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(EIG_THREADS)
    tridiag_kernel(double *Aall, const int64_t *off, const int *dims, const int64_t *eoff, const int *tsec,
                   const int *tbig, double *dall, double *eall, double *tauall, double *Wall, double *info,
                   double *dsall, double *e2all, int64_t smem_doubles, int *status, long long limit) {
  extern __shared__ __align__(16) double td_sm[];
  __shared__ double red[48];
  __shared__ double sh_tau, sh_scl;
  __shared__ uint64_t mbar[2];
  cg::cluster_group cl = cg::this_cluster();
  const int b = blockIdx.x / CL, rank = (int)cl.block_rank();
  const int s = tsec[blockIdx.x];
  if (tbig[b]) {
    tridiag_coop<CL>(cl, rank, s, Aall, off, dims, eoff, dall, eall, tauall, Wall, info, dsall, e2all, td_sm, smem_doubles,
                     red, mbar, status, limit);
  } else if (s >= 0 && dims[s] > 0) {
    const int n = dims[s];
    if (n <= 32)
      tridiag_small<1, 8>(s, Aall, off, dims, eoff, dall, eall, tauall, info, dsall, e2all, td_sm, red);
    else if (n <= TD_SMALL)
      tridiag_small<TD_SMALL / 32, 8>(s, Aall, off, dims, eoff, dall, eall, tauall, info, dsall, e2all, td_sm, red);
    else
      tridiag_one(s, Aall, off, dims, eoff, dall, eall, tauall, info, dsall, e2all, td_sm, red, sh_tau, sh_scl);
  }
}

// Eigenvalue k (ascending) of every sector, one warp each: the interval
// [lo, hi) with count(lo) <= k < count(hi) starts at the Gershgorin bounds;
// per pass lane l counts the eigenvalues below lo + (l + 1) (hi - lo) / 33,
// and the interval becomes the 33rd between the last point at or below k
// and the first above it, until it is below 2 eps max(|lo|, |hi|) or
// eps ||T|| (the absolute accuracy of any backward-stable solver): about 11
// passes of one Sturm sequence per lane where bisection takes 52.
// The scaled minors instead of pivots (a division a step): 1577 -> 611 us on a
// 4x24 m = 2000 density matrix of 31 sectors of up to 857 states.
__global__ void bisect_kernel(const double *dsall, const double *e2all, const int64_t *eoff, const int *dims,
                              const double *info, const int *esec, int etot, double *evals) {
  const int idx = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (idx >= etot) return;   // uniform in a warp
  const int s = esec[idx], n = dims[s];
  const int k = (int)(idx - eoff[s]);
  const double *ds = dsall + eoff[s], *e2 = e2all + eoff[s];
  const double tnorm = info[4 * s + 2], pivmin = info[4 * s + 3];
  const double pad = 2.0 * EIG_EPS * tnorm + 2.0 * pivmin;
  const double sc = tridiag_scale(tnorm);
  double lo = info[4 * s + 0] - pad, hi = info[4 * s + 1] + pad;
  for (int it = 0; it < 40; ++it) {
    const double tol = fmax(fmax(2.0 * EIG_EPS * fmax(fabs(lo), fabs(hi)), EIG_EPS * tnorm), pivmin);
    if (hi - lo <= tol) break;
    const double h = (hi - lo) / 33.0;
    const int c = sturm1(ds, e2, n, (lo + (lane + 1) * h) * sc);
    const unsigned above = __ballot_sync(0xffffffffu, c > k);
    const int f = above ? __ffs(above) - 1 : 32;   // first point above eigenvalue k
    const double nlo = f == 0 ? lo : lo + f * h, nhi = f == 32 ? hi : lo + (f + 1) * h;
    if (nlo == lo && nhi == hi) break;   // the interval no longer shrinks in FP64
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) evals[idx] = 0.5 * (lo + hi);
}

// Pseudo-random start vector entry in [-1, 1) (splitmix64 of the indices).
__device__ __forceinline__ double start_entry(int s, int k, int i) {
  uint64_t z = ((uint64_t)(uint32_t)s << 40) ^ ((uint64_t)(uint32_t)k << 20) ^ (uint64_t)(uint32_t)i;
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  return (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// Eigenvector of T (sector job_sec[j]) for its eigenvalue job_k[j] by
// inverse iteration, one thread per vector: LU factorisation of T - lam I
// with partial pivoting (pivots below eps ||T|| raised to it, so that the
// nearly singular factor stays finite), three solves from a fixed
// pseudo-random start, each result rescaled.  The per-thread factors live in
// work[] with element i of job j at i * njobs + j (coalesced across a warp);
// the unit vector goes to Y[j * ldy + i].  status[0] bit 0: a non-finite
// value; the first such vector is described at status + 4 (six doubles).
__global__ void inverse_iter_kernel(const double *dall, const double *eall, const int64_t *eoff, const int *dims,
                                    const double *info, const double *evals, const int *job_sec, const int *job_k,
                                    int njobs, int nmax, double *work, unsigned char *piv, double *Y, int ldy,
                                    int *status) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= njobs) return;
  const int s = job_sec[j], k = job_k[j], n = dims[s];
  const double *__restrict__ d = dall + eoff[s];
  const double *__restrict__ e = eall + eoff[s];
  const double lam = evals[eoff[s] + k];
  const double pert = fmax(EIG_EPS * info[4 * s + 2], 1e-290);
  const size_t st = (size_t)njobs, pl = (size_t)nmax * st;
  // disjoint regions: the loads of the factors may run ahead of the stores to X
  double *__restrict__ U = work;
  double *__restrict__ DU = work + pl;
  double *__restrict__ DU2 = work + 2 * pl;
  double *__restrict__ DL = work + 3 * pl;
  double *__restrict__ X = work + 4 * pl;
#define AT(arr, i) arr[(size_t)(i) * st + j]
  // LU = P (T - lam I): row i of U is (1 / U_i, DU_i, DU2_i) at columns i, i+1,
  // i+2 (the reciprocal once, instead of a division in the chain of every row of
  // every solve)
  double di = d[0] - lam, dui = n > 1 ? e[0] : 0.0;
  for (int i = 0; i + 1 < n; ++i) {
    const double sub = e[i];
    double dn = d[i + 1] - lam, dun = i + 2 < n ? e[i + 1] : 0.0;
    if (fabs(di) >= fabs(sub) || fabs(sub) < pert) {
      const double r = 1.0 / (fabs(di) < pert ? copysign(pert, di) : di);
      const double l = sub * r;
      AT(U, i) = r;
      AT(DU, i) = dui;
      AT(DU2, i) = 0.0;
      AT(DL, i) = l;
      piv[(size_t)i * st + j] = 0;
      dn -= l * dui;
    } else {   // rows i and i+1 exchanged
      const double r = 1.0 / sub, l = di * r;
      AT(U, i) = r;
      AT(DU, i) = dn;
      AT(DU2, i) = dun;
      AT(DL, i) = l;
      piv[(size_t)i * st + j] = 1;
      dn = dui - l * dn;
      dun = -l * dun;
    }
    di = dn;
    dui = dun;
  }
  AT(U, n - 1) = 1.0 / (fabs(di) < pert ? copysign(pert, di) : di);
  AT(DU, n - 1) = 0.0;   // read (times zero) by the first back-substitution row
  AT(DU2, n - 1) = 0.0;
  if (n >= 2) AT(DU2, n - 2) = 0.0;
  for (int i = 0; i < n; ++i) AT(X, i) = start_entry(s, k, i);
  // Each sweep solves with X times `scale` (the previous sweep's rescale to
  // a largest entry of 1, applied where X is read) and keeps the largest
  // entry of its result as it goes.  Both passes read eight rows ahead of
  // their stores: X[i] is stored through the same pointer as the next row's
  // load, and a load the compiler must keep behind that store would wait out
  // an L2 round trip per row.
  bool bad = false;
  double scale = 1.0;
  for (int sweep = 0; sweep < 3; ++sweep) {
    // forward: P and L
    double cur = AT(X, 0) * scale;
    int i = 0;
    for (; i + 8 < n; i += 8) {   // rows i..i+7; their solves read X[i+1..i+8] as they were
      double l[8], nx[8];
      unsigned char pv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        l[u] = AT(DL, i + u);
        nx[u] = AT(X, i + u + 1) * scale;
        pv[u] = piv[(size_t)(i + u) * st + j];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (pv[u]) {   // rows i+u and i+u+1 exchanged
          AT(X, i + u) = nx[u];
          cur = cur - l[u] * nx[u];
        } else {
          AT(X, i + u) = cur;
          cur = nx[u] - l[u] * cur;
        }
      }
    }
    for (; i + 1 < n; ++i) {
      const double l = AT(DL, i), nxt = AT(X, i + 1) * scale;
      if (piv[(size_t)i * st + j]) {
        AT(X, i) = nxt;
        cur = cur - l * nxt;
      } else {
        AT(X, i) = cur;
        cur = nxt - l * cur;
      }
    }
    AT(X, n - 1) = cur;
    // backward: U, with a rescale of the whole vector if it nears overflow
    // (the rows loaded but not yet solved are rescaled in registers)
    double x1 = 0.0, x2 = 0.0, mx = 0.0;   // x_{i+1}, x_{i+2}, the largest |x| so far
    auto row = [&](double xv, double du, double du2, double uu, int at, double *ahead, int nahead) {
      double xi = (xv - du * x1 - du2 * x2) * uu;
      if (fabs(xi) > 1e250) {
        const double f = 1e-250;
        for (int q = 0; q < n; ++q) AT(X, q) *= f;
        for (int w = 0; w < nahead; ++w) ahead[w] *= f;
        xi *= f;
        x1 *= f;
        x2 *= f;
        mx *= f;
      }
      AT(X, at) = xi;
      mx = fmax(mx, fabs(xi));
      x2 = x1;
      x1 = xi;
    };
    i = n - 1;
    for (; i >= 7; i -= 8) {   // rows i, i-1, ..., i-7
      double xv[8], du[8], du2[8], uu[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        xv[u] = AT(X, i - u);
        du[u] = AT(DU, i - u);
        du2[u] = AT(DU2, i - u);
        uu[u] = AT(U, i - u);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) row(xv[u], du[u], du2[u], uu[u], i - u, xv + u + 1, 7 - u);
    }
    for (; i >= 0; --i) row(AT(X, i), AT(DU, i), AT(DU2, i), AT(U, i), i, nullptr, 0);
    if (!(mx > 0.0) || !isfinite(mx)) {
      bad = true;
      break;
    }
    scale = 1.0 / mx;
  }
  double nrm = 0.0;
  for (int i = 0; i < n; ++i) {
    const double x = AT(X, i) * scale;
    nrm += x * x;
  }
  if (bad || !(nrm > 0.0) || !isfinite(nrm)) {
    atomicOr(status, 1);
    // the first failing vector: sector, eigenvalue index, lam, pivot floor, n
    if (atomicCAS(status + 1, 0, j + 1) == 0) {
      double *diag = (double *)(status + 4);
      diag[0] = s;
      diag[1] = k;
      diag[2] = lam;
      diag[3] = pert;
      diag[4] = n;
      diag[5] = nrm;
    }
    nrm = 1.0;
    scale = 1.0;
  }
  const double inv = 1.0 / sqrt(nrm);
  double *y = Y + (size_t)j * ldy;
  for (int i = 0; i < n; ++i) y[i] = AT(X, i) * scale * inv;
  for (int i = n; i < nmax; ++i) y[i] = 0.0;
#undef AT
}

// Dots of y (rows 0..nr-1; shared or global memory) with the vectors zq(q),
// q = 0..nq-1, into out[q]: each warp takes eight vectors at a time so that
// their loads are in flight together (one vector at a time, every vector
// would wait out an L2 round trip: the store of a sum may alias the next
// vector's loads).  Each dot is summed as lane-strided parts and a shuffle
// tree, the same for every q.
template <class ZQ>
__device__ __forceinline__ void warp_dots8(ZQ zq, int nq, const double *y, int nr, double *out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int q0 = 8 * warp; q0 < nq; q0 += 8 * nw) {
    double acc[8];
    const double *z[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      acc[u] = 0.0;
      z[u] = zq(min(q0 + u, nq - 1));   // past nq: a repeat, discarded
    }
    for (int i = lane; i < nr; i += 32) {
      const double yi = y[i];
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] += z[u][i] * yi;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      double a = acc[u];
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane == 0 && q0 + u < nq) out[q0 + u] = a;
    }
  }
}

// y <- y - sum_q h[q] zq(q) over rows 0..nr-1, returning the thread's part
// of the new squared norm.  When the block's threads outnumber the rows, G
// groups of R threads split the vectors (group g takes q = g, g + G, ...) and
// their parts (gp: G * nr <= blockDim.x entries) are summed in group order;
// otherwise one thread per row runs over all of them.  Ends with the block's
// writes to y complete only for the writing thread (the caller's barrier
// follows).
template <class ZQ>
__device__ __forceinline__ double project_off(ZQ zq, int t, const double *h, double *y, int nr, double *gp) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int R = min(max((nr + 31) & ~31, 32), nt), G = nt / R;
  double ss = 0.0;
  if (G == 1) {
    for (int i = tid; i < nr; i += nt) {
      double acc = y[i];
      for (int q = 0; q < t; ++q) acc -= h[q] * zq(q)[i];
      y[i] = acc;
      ss += acc * acc;
    }
    return ss;
  }
  const int g = tid / R, r = tid - g * R;
  if (g < G && r < nr) {
    double acc = 0.0;
#pragma unroll 4
    for (int q = g; q < t; q += G) acc += h[q] * zq(q)[r];
    gp[g * nr + r] = acc;
  }
  __syncthreads();
  for (int i = tid; i < nr; i += nt) {
    double acc = 0.0;
    for (int c = 0; c < G; ++c) acc += gp[c * nr + i];
    const double yv = y[i] - acc;
    y[i] = yv;
    ss += yv * yv;
  }
  return ss;
}

// The vectors of a kept block that inverse iteration left nearly orthogonal,
// by two matrix products instead of a chain over the vectors.  G = Y^T Y holds
// every dot product; with E its deviation from I, Gram-Schmidt in descending
// eigenvalue order (vector j against the vectors q > j) is Y (I - L(E) -
// diag(E) / 2), L the strictly lower triangle, up to terms of the size of the
// products of E's columns.  These kernels turn each block's G (grp[b], at
// goff[b], leading dimension its count) into that factor R for the vectors
// whose column of E has a norm of at most 1e-8 (so those terms are below
// 1e-16) and so have all vectors above them; first[b] is the number of
// vectors this covers, and R leaves the others as they are, for
// orthonormalize_kernel.  Separated eigenvalues give columns of about
// eps ||T|| / gap: on a 4x24 m = 2000 density matrix (31 sectors of up to 857
// states) all blocks are covered, and the stage takes 0.11 ms, 2.77 ms vector
// by vector.
// (ortho_check_kernel: a warp per vector; first[b] starts at the count and ends
// at the index, in descending order, of the first vector not covered.)
__global__ void __launch_bounds__(256) ortho_check_kernel(const int *grp, const int64_t *goff, const double *Gall,
                                                          int *first) {
  const int b = blockIdx.x, cnt = grp[4 * b + 2], lane = threadIdx.x & 31;
  for (int j = blockIdx.y * 8 + (threadIdx.x >> 5); j < cnt; j += gridDim.y * 8) {
    const double *g = Gall + goff[b] + (int64_t)j * cnt;
    double ss = 0.0;
    for (int q = j + 1 + lane; q < cnt; q += 32) ss += g[q] * g[q];
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const bool fine = ss <= 1e-16 && fabs(g[j] - 1.0) <= 1e-8;   // false for a NaN
    if (lane == 0 && !fine) atomicMin(first + b, cnt - 1 - j);
  }
}
__global__ void __launch_bounds__(256) ortho_factor_kernel(const int *grp, const int64_t *goff, double *Gall,
                                                           const int *first) {
  const int b = blockIdx.x, cnt = grp[4 * b + 2], lane = threadIdx.x & 31, t0 = first[b];
  for (int j = blockIdx.y * 8 + (threadIdx.x >> 5); j < cnt; j += gridDim.y * 8) {
    double *g = Gall + goff[b] + (int64_t)j * cnt;
    const bool in = cnt - 1 - j < t0;
    const double c = in ? 1.0 - 0.5 * (g[j] - 1.0) : 1.0;   // 1 / the vector's norm
    __syncwarp();
    for (int q = lane; q < cnt; q += 32) g[q] = q == j ? c : q > j && in ? -g[q] : 0.0;
  }
}

// One kept block (grp = {sector, first job, count}), from vector t_first on
// (those before it are orthonormal already): classical Gram-Schmidt
// on its vectors in descending eigenvalue order, so that the dominant states
// are the least changed; inverse iteration leaves vectors of close
// eigenvalues only approximately orthogonal (to about eps ||T|| / gap).  The
// projection is repeated only when the first one removed more than half of
// the vector's squared norm ("twice is enough": after one pass that keeps
// the norm above 1/sqrt(2), the vector is orthogonal to working accuracy).
//
// A vector that loses more than 0.999 of its norm to the projection depends
// on the accepted ones.  That happens for a cluster of eigenvalues closer
// than the pivot floor eps ||T||, where inverse iteration amplifies one
// direction of the cluster far above the others -- in practice the null
// space of a rank-deficient density matrix (a sector with fewer environment
// than system states, or one of tiny weight), all of whose states the keep
// rule may keep.  When the vector's eigenvalue lies within 1e4 eps ||T|| of
// the sector's smallest, the cluster is the bottom of the spectrum, every
// eigenvector above it has been accepted (kept vectors are the largest of
// their sector), and the complement of the accepted vectors is the rest of
// the cluster: a pseudo-random vector projected off the accepted ones is then
// an eigenvector to working accuracy (residual <= the cluster's width), as
// good as any basis DSYEV returns for it.  Up to four such vectors are tried.
// status bit 1: a vector stayed dependent (or its cluster is not at the
// bottom of the spectrum).
__device__ void ortho_one(int blk, int t_first, const int *grp, const int *dims, const int64_t *eoff,
                          const double *evals, const double *info, const int *job_k, double *Y, int ldy, int *status,
                          double *h, double *red) {
  const int s = grp[4 * blk], j0 = grp[4 * blk + 1], cnt = grp[4 * blk + 2];
  const int n = dims[s], tid = threadIdx.x;
  const double lam_min = evals[eoff[s]], cluster = 1e4 * EIG_EPS * info[4 * s + 2];
  double *gp = h + cnt;   // project_off's group parts
  auto vec = [&](int q) -> const double * { return Y + (size_t)(j0 + cnt - 1 - q) * ldy; };
  for (int t = t_first; t < cnt; ++t) {
    const int jt = j0 + cnt - 1 - t;
    double *y = Y + (size_t)jt * ldy;
    bool ok = false;
    for (int attempt = 0; attempt < 5 && !ok; ++attempt) {
      if (attempt > 0) {   // a fresh pseudo-random unit vector (k + 4096 a never repeats a start)
        double ss = 0.0;
        for (int i = tid; i < n; i += blockDim.x) {
          const double v = start_entry(s, job_k[jt] + 4096 * attempt, i);
          y[i] = v;
          ss += v * v;
        }
        const double inv = 1.0 / sqrt(block_sum(ss, red));
        for (int i = tid; i < n; i += blockDim.x) y[i] *= inv;
        __syncthreads();
      }
      ok = true;
      for (int pass = 0; pass < 2; ++pass) {
        warp_dots8(vec, t, y, n, h);
        __syncthreads();
        const double ss = project_off(vec, t, h, y, n, gp);
        const double nrm = sqrt(block_sum(ss, red));   // the same value in every thread
        if (pass == 0 && !(nrm >= 1e-3)) {
          ok = false;
          break;
        }
        const double inv = 1.0 / nrm;
        for (int i = tid; i < n; i += blockDim.x) y[i] *= inv;
        __syncthreads();
        if (nrm > 0.7071067811865476) break;   // the vector entered with unit norm
      }
      if (!ok && attempt == 0 && !(evals[eoff[s] + job_k[jt]] - lam_min <= cluster)) break;
    }
    if (!ok && tid == 0) atomicOr(status, 2);
  }
}

// The same orthonormalisation of one large kept block by the CL CTAs of a
// cluster: CTA c owns a slice of rows of every vector.  Per projection pass
// each CTA forms its part of the dot products with the accepted vectors, the
// parts meet through distributed shared memory, every CTA sums them in rank
// order (so every CTA holds the same coefficients and takes the same
// decisions), subtracts on its own rows; the vector's squared norm travels
// with the dots, so that when the projection removes less than half of it
// (the common case: inverse iteration leaves the vectors nearly orthogonal)
// the new norm needs no second exchange; otherwise it is summed the same way
// after the subtraction.  Each exchange uses the buffer of its parity and ends with one
// cluster barrier; a buffer is written again only two exchanges later, after
// every CTA has passed the barrier that follows its reads.  A CTA reads and
// writes only its own rows of the vectors in global memory.
template <int CL>
__device__ void ortho_coop(cg::cluster_group &cl, int rank, int blk, int t_first, const int *grp, const int *dims,
                           const int64_t *eoff, const double *evals, const double *info, const int *job_k, double *Y,
                           int ldy, int *status, double *sm, double *red) {
  const int s = grp[4 * blk], j0 = grp[4 * blk + 1], cnt = grp[4 * blk + 2];
  const int n = dims[s], tid = threadIdx.x, nt = blockDim.x;
  const double lam_min = evals[eoff[s]], cluster = 1e4 * EIG_EPS * info[4 * s + 2];
  const int per = (n + CL - 1) / CL, r0 = min(n, rank * per), r1 = min(n, r0 + per), nr = r1 - r0;
  // hp: parts of the dots (2 x cnt), h: the dots (cnt), ys: own rows of the
  // vector (per), sl: parts of the squared norm (2), gp: project_off's group
  // parts (nt)
  double *hp = sm, *h = hp + 2 * cnt, *ys = h + cnt, *sl = ys + per, *gp = sl + 2;
  unsigned xch = 0;   // exchanges so far (buffer parity)
  int half = 0;       // block_sum1's alternating half of red
  auto cluster_sum = [&](double x) -> double {   // x: the CTA's value, the same in all its threads
    double *slot = sl + (xch & 1);
    if (tid == 0) *slot = x;
    cl.sync();
    ++xch;
    double tot = 0.0;
    for (int c = 0; c < CL; ++c) tot += *cl.map_shared_rank(slot, c);
    return tot;
  };
  auto vec = [&](int q) { return Y + (size_t)(j0 + cnt - 1 - q) * ldy; };   // q-th vector in descending order
  for (int t = t_first; t < cnt; ++t) {
    double *y = vec(t);
    const int jt = j0 + cnt - 1 - t;
    bool ok = false;
    for (int attempt = 0; attempt < 5 && !ok; ++attempt) {
      if (attempt == 0) {
        for (int i = tid; i < nr; i += nt) ys[i] = y[r0 + i];
        __syncthreads();
      } else {   // a fresh pseudo-random unit vector (see ortho_one)
        double ss = 0.0;
        for (int i = tid; i < nr; i += nt) {
          const double v = start_entry(s, job_k[jt] + 4096 * attempt, r0 + i);
          ys[i] = v;
          ss += v * v;
        }
        const double inv = 1.0 / sqrt(cluster_sum(block_sum1(ss, red, half)));
        for (int i = tid; i < nr; i += nt) ys[i] *= inv;
        __syncthreads();
      }
      ok = true;
      for (int pass = 0; pass < 2; ++pass) {
        // one exchange carries the dots with the accepted vectors and the
        // vector's own squared norm (slot t); when the projection removes
        // less than half of the squared norm, the new norm is yy - sum h^2
        // (accurate to rounding there), and no second exchange is needed
        double *hpw = hp + (xch & 1) * cnt;
        warp_dots8([&](int q) -> const double * { return q < t ? vec(q) + r0 : ys; }, t + 1, ys, nr, hpw);
        cl.sync();
        ++xch;
        double hh = 0.0;
        for (int q = tid; q <= t; q += nt) {
          double tot = 0.0;
          for (int c = 0; c < CL; ++c) tot += cl.map_shared_rank(hpw, c)[q];
          h[q] = tot;
          if (q < t) hh += tot * tot;
        }
        const double s2 = block_sum1(hh, red, half);   // also the barrier after h
        const double yy = h[t], rest = yy - s2;        // the same values in every CTA
        const bool fast = rest >= 0.5 * yy && rest > 0.0;
        const double ss = project_off([&](int q) -> const double * { return vec(q) + r0; }, t, h, ys, nr, gp);
        const double nrm = fast ? sqrt(rest) : sqrt(cluster_sum(block_sum1(ss, red, half)) / yy);
        if (pass == 0 && !(nrm >= 1e-3)) {
          ok = false;
          break;
        }
        const double inv = fast ? 1.0 / nrm : 1.0 / (nrm * sqrt(yy));
        for (int i = tid; i < nr; i += nt) ys[i] *= inv;
        __syncthreads();
        if (nrm > 0.7071067811865476) break;   // relative to the norm the vector entered with
      }
      if (!ok && attempt == 0 && !(evals[eoff[s] + job_k[jt]] - lam_min <= cluster)) break;
    }
    for (int i = tid; i < nr; i += nt) y[r0 + i] = ys[i];
    __syncthreads();
    if (!ok && rank == 0 && tid == 0) atomicOr(status, 2);
  }
  cl.sync();   // no CTA leaves while another may still read its buffers
}

// One cluster of CL CTAs per entry of the cluster list: a large kept block
// shared by all of them (obig), or up to CL small blocks, one per CTA
// (oblk[cluster * CL + rank], -1 for none); CL as for tridiag_kernel.
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(ORTH_THREADS, 1)
    orthonormalize_kernel(const int *oblk, const int *obig, const int *grp, const int *dims, const int64_t *eoff,
                          const double *evals, const double *info, const int *job_k, const int *first, double *Y,
                          int ldy, int *status) {
  extern __shared__ double sm[];
  __shared__ double red[64];
  cg::cluster_group cl = cg::this_cluster();
  const int b = blockIdx.x / CL, rank = (int)cl.block_rank();
  const int blk = oblk[blockIdx.x];
  if (obig[b])
    ortho_coop<CL>(cl, rank, blk, max(first[blk], 1), grp, dims, eoff, evals, info, job_k, Y, ldy, status, sm, red);
  else if (blk >= 0)
    ortho_one(blk, max(first[blk], 1), grp, dims, eoff, evals, info, job_k, Y, ldy, status, sm, red);
}

// Back-transformation of the kept vectors, one warp per vector and the
// vector in shared memory: y <- H_0 (H_1 (... H_{n-2} y)), reflector k read
// from A(k+1:n, k) of its sector.  The sign is fixed so that the entry of
// largest magnitude (the first of equal ones) is positive, and the column is
// written to the truncation operator at job_dst[j].  slab[2b], slab[2b+1]:
// the block (grp index) and its first column handled by CTA b.
__global__ void backtransform_kernel(const double *Aall, const int64_t *off, const double *tauall,
                                     const int64_t *eoff, const int *dims, const int *grp, const int *slab,
                                     const double *Y, int ldy, const int64_t *job_dst, double *out) {
  extern __shared__ double colsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = slab[2 * blockIdx.x], c = slab[2 * blockIdx.x + 1] + warp;
  const int s = grp[4 * g], j0 = grp[4 * g + 1], cnt = grp[4 * g + 2];
  if (c >= cnt) return;
  const int n = dims[s], j = j0 + c;
  const double *A = Aall + off[s], *tau = tauall + eoff[s];
  double *col = colsm + (size_t)warp * ldy;
  for (int i = lane; i < n; i += 32) col[i] = Y[(size_t)j * ldy + i];
  __syncwarp();
  for (int k = n - 2; k >= 0; --k) {
    const double t = tau[k];
    if (t == 0.0) continue;
    const double *v = A + (int64_t)k * n;
    double acc = 0.0;
    for (int i = k + 1 + lane; i < n; i += 32) acc += v[i] * col[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const double f = t * acc;
    for (int i = k + 1 + lane; i < n; i += 32) col[i] -= f * v[i];
    __syncwarp();
  }
  double best = -1.0;
  int bi = 0;
  for (int i = lane; i < n; i += 32)
    if (fabs(col[i]) > best) {
      best = fabs(col[i]);
      bi = i;
    }
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ob > best || (ob == best && oi < bi)) {
      best = ob;
      bi = oi;
    }
  }
  const double sg = col[bi] < 0.0 ? -1.0 : 1.0;
  double *dst = out + job_dst[j];
  for (int i = lane; i < n; i += 32) dst[i] = sg * col[i];
}

// The same back-transformation by matrix products, for sectors of up to
// 1536 states (a CTA's shared memory): BT_NB consecutive reflectors are one block reflector I - V T V^T
// (T upper triangular, by wy_t_kernel), applied to a CTA's 8 VT vectors of one
// kept block.  Vector by vector, each reflector is a dot product over the
// vector, a reduction across the warp and an update: a chain of some 300
// cycles for each of the sector's states (1.8 ms on the 4x24 m = 2000 density
// matrix with 857 states).  A block reflector has three barriers, and its
// products run on DMMA: 0.24 ms, and 0.05 ms for the T of all blocks.
//
// The vectors stay in registers as Y^T in accumulator layout: warp w holds the
// row tiles (8 rows) w, w + BT_WARPS, ..., lane (g, t) of tile j the entries
// (vector g, rows 2t and 2t + 1).  As the left operand of Y^T V an accumulator
// register is a fragment as it stands when the inner dimension is taken in the
// order rows 0, 2, 4, 6, then 1, 3, 5, 7; V is read to match.  Each warp keeps
// its own rows of the block's reflectors in shared memory, a tile's entry
// (row r, reflector q) at 8 q + (r with bit 2 flipped where q has bit 1).
constexpr int BT_WARPS = 16, BT_NB = 16;

// T of the block reflectors (LAPACK dlarft, forward and columnwise): block b of
// the grid makes T of reflectors [16 p, 16 p + 16) of sector s, pan[2b] = s,
// pan[2b + 1] = p, from the dot products of the reflectors.  Column-major.
__global__ void __launch_bounds__(256) wy_t_kernel(const double *Aall, const int64_t *off, const double *tauall,
                                                   const int64_t *eoff, const int *dims, const int *pan, double *Tall) {
  __shared__ double vs[BT_NB][65], G[BT_NB][BT_NB + 1], T[BT_NB][BT_NB + 1];
  const int s = pan[2 * blockIdx.x], k0 = pan[2 * blockIdx.x + 1] * BT_NB, n = dims[s], tid = threadIdx.x;
  const double *A = Aall + off[s], *tau = tauall + eoff[s];
  const int i = tid >> 4, j = tid & 15;
  double acc = 0.0;
  for (int r0 = (k0 + 1) & ~63; r0 < n; r0 += 64) {
    __syncthreads();
    for (int e = tid; e < BT_NB * 64; e += 256) {
      const int q = e >> 6, r = r0 + (e & 63), k = k0 + q;
      vs[q][e & 63] = k + 1 < n && r > k && r < n ? A[(int64_t)k * n + r] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int r = 0; r < 64; ++r) acc += vs[i][r] * vs[j][r];
  }
  G[i][j] = acc;
  T[i][j] = 0.0;
  __syncthreads();
  for (int c = 0; c < BT_NB; ++c) {
    const double t = k0 + c + 1 < n ? tau[k0 + c] : 0.0;
    if (tid < c) {
      double x = 0.0;
      for (int q = tid; q < c; ++q) x += T[tid][q] * G[q][c];
      T[tid][c] = -t * x;
    }
    if (tid == c) T[c][c] = t;
    __syncthreads();
  }
  Tall[(int64_t)blockIdx.x * (BT_NB * BT_NB) + j * BT_NB + i] = T[i][j];
}

__device__ __forceinline__ void bt_dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// shared memory of a CTA: the reflectors of a block, the warps' parts of Y^T V
// (later the largest entries), Y^T V, its product with T^T, and T
constexpr int bt_smem_doubles(int tiles, int vt) {
  return BT_WARPS * (tiles * 8 * BT_NB + 8 * vt * BT_NB) + 2 * 8 * vt * BT_NB + BT_NB * BT_NB;
}

// TILES: row tiles of a warp; pan0[s]: index of sector s's first T.
template <int TILES, int VT>
__global__ void __launch_bounds__(32 * BT_WARPS, 1)
    backtransform_wy_kernel(const double *Aall, const int64_t *off, const double *Tall, const int *pan0, const int *dims,
                            const int *grp, const int *slab, const double *Y, int ldy, const int64_t *job_dst,
                            double *out) {
  extern __shared__ double bsm[];
  constexpr int NV = 8 * VT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  double *vw = bsm + warp * (TILES * 8 * BT_NB);
  double *parts = bsm + BT_WARPS * TILES * 8 * BT_NB, *S = parts + BT_WARPS * NV * BT_NB, *Zt = S + NV * BT_NB,
         *T = Zt + NV * BT_NB;
  const int gi = slab[2 * blockIdx.x], c0 = slab[2 * blockIdx.x + 1];
  const int s = grp[4 * gi], j0 = grp[4 * gi + 1], cnt = grp[4 * gi + 2], n = dims[s];
  const double *A = Aall + off[s];
  double y[TILES][VT][2];
#pragma unroll
  for (int j = 0; j < TILES; ++j)
#pragma unroll
    for (int v = 0; v < VT; ++v)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + 8 * v + g, r = 8 * (warp + BT_WARPS * j) + 2 * t + e;
        y[j][v][e] = c < cnt && r < n ? Y[(int64_t)(j0 + c) * ldy + r] : 0.0;
      }
  const int np = (n - 1 + BT_NB - 1) / BT_NB;   // blocks of the n - 1 reflectors
  for (int p = np - 1; p >= 0; --p) {
    const int k0 = p * BT_NB;
    // the warp's rows of the reflectors: zero up to their own index; row tiles
    // that end above the block's first row are zero throughout
#pragma unroll
    for (int j = 0; j < TILES; ++j) {
      const int r0 = 8 * (warp + BT_WARPS * j), r = r0 + (lane & 7);
      if (r0 + 7 <= k0 || r0 >= n) continue;
#pragma unroll
      for (int u = 0; u < BT_NB / 4; ++u) {
        const int q = (lane >> 3) + 4 * u, k = k0 + q;
        vw[j * 8 * BT_NB + q * 8 + ((lane & 7) ^ ((q & 2) << 1))] =
            k + 1 < n && r > k && r < n ? A[(int64_t)k * n + r] : 0.0;
      }
    }
    if (tid < BT_NB * BT_NB) T[tid] = Tall[(int64_t)(pan0[s] + p) * (BT_NB * BT_NB) + tid];
    __syncwarp();
    // Y^T V of the warp's rows
    double w[VT][BT_NB / 8][2];
#pragma unroll
    for (int v = 0; v < VT; ++v)
#pragma unroll
      for (int h = 0; h < BT_NB / 8; ++h) w[v][h][0] = w[v][h][1] = 0.0;
#pragma unroll
    for (int j = 0; j < TILES; ++j) {
      const int r0 = 8 * (warp + BT_WARPS * j);
      if (r0 + 7 <= k0 || r0 >= n) continue;
#pragma unroll
      for (int h = 0; h < BT_NB / 8; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int q = 8 * h + g;
          const double b = vw[j * 8 * BT_NB + q * 8 + ((2 * t + e) ^ ((q & 2) << 1))];
#pragma unroll
          for (int v = 0; v < VT; ++v) bt_dmma(w[v][h], y[j][v][e], b);
        }
    }
#pragma unroll
    for (int v = 0; v < VT; ++v)
#pragma unroll
      for (int h = 0; h < BT_NB / 8; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) parts[warp * (NV * BT_NB) + (8 * v + g) * BT_NB + 8 * h + 2 * t + e] = w[v][h][e];
    __syncthreads();
    if (tid < NV * BT_NB) {
      double x = 0.0;
#pragma unroll
      for (int q = 0; q < BT_WARPS; ++q) x += parts[q * (NV * BT_NB) + tid];
      S[tid] = x;
    }
    __syncthreads();
    if (tid < NV * BT_NB) {   // (Y^T V T^T)[vector][q] = sum_i T[q][i] S[vector][i]
      const int v = tid / BT_NB, q = tid % BT_NB;
      double x = 0.0;
#pragma unroll
      for (int i = 0; i < BT_NB; ++i) x += T[i * BT_NB + q] * S[v * BT_NB + i];
      Zt[tid] = -x;
    }
    __syncthreads();
    // Y^T -= (Y^T V T^T) V^T
    double a[VT][BT_NB / 4];
#pragma unroll
    for (int v = 0; v < VT; ++v)
#pragma unroll
      for (int kk = 0; kk < BT_NB / 4; ++kk) a[v][kk] = Zt[(8 * v + g) * BT_NB + 4 * kk + t];
#pragma unroll
    for (int j = 0; j < TILES; ++j) {
      const int r0 = 8 * (warp + BT_WARPS * j);
      if (r0 + 7 <= k0 || r0 >= n) continue;
#pragma unroll
      for (int kk = 0; kk < BT_NB / 4; ++kk) {
        const int q = 4 * kk + t;
        const double b = vw[j * 8 * BT_NB + q * 8 + (g ^ ((q & 2) << 1))];
#pragma unroll
        for (int v = 0; v < VT; ++v) bt_dmma(y[j][v], a[v][kk], b);
      }
    }
    __syncwarp();   // the warp's reflectors are read
  }
  // the sign of each vector's entry of largest magnitude (the first of equal
  // ones), over the lane's rows, the four lanes of a vector, the warps
  __shared__ int bidx[BT_WARPS][NV];
#pragma unroll
  for (int v = 0; v < VT; ++v) {
    double best = 0.0;   // the entry itself
    int bi = 1 << 30;
#pragma unroll
    for (int j = 0; j < TILES; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 8 * (warp + BT_WARPS * j) + 2 * t + e;
        if (r < n && (fabs(y[j][v][e]) > fabs(best) || bi == 1 << 30)) {
          best = y[j][v][e];
          bi = r;
        }
      }
    for (int o = 1; o < 4; o <<= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (fabs(ob) > fabs(best) || (fabs(ob) == fabs(best) && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    if (t == 0) {
      parts[warp * NV + 8 * v + g] = best;
      bidx[warp][8 * v + g] = bi;
    }
  }
  __syncthreads();
  if (tid < NV) {
    double best = parts[tid];
    int bi = bidx[0][tid];
    for (int q = 1; q < BT_WARPS; ++q) {
      const double ob = parts[q * NV + tid];
      const int oi = bidx[q][tid];
      if (fabs(ob) > fabs(best) || (fabs(ob) == fabs(best) && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    S[tid] = best < 0.0 ? -1.0 : 1.0;
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < VT; ++v) {
    const int c = c0 + 8 * v + g;
    if (c < cnt) {
      const double sg = S[8 * v + g];
      double *dst = out + job_dst[j0 + c];
#pragma unroll
      for (int j = 0; j < TILES; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = 8 * (warp + BT_WARPS * j) + 2 * t + e;
          if (r < n) dst[r] = sg * y[j][v][e];
        }
    }
  }
}

// |psi|^2 from its block sums, and 1 / |psi|^2 as the coefficient of every task
// of the density matrix
__global__ void rho_scale_kernel(const double *part, int npart, Task *tasks, int ntasks, double *nrm2) {
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < npart; i += blockDim.x) s += part[i];
  s = block_sum(s, red);
  for (int i = threadIdx.x; i < ntasks; i += blockDim.x) tasks[i].coef = 1.0 / s;
  if (threadIdx.x == 0) *nrm2 = s;
}

}  // namespace tjb

using namespace tjb;

#define CKT(call)                                                                                        \
  do {                                                                                                   \
    cudaError_t e_ = (call);                                                                             \
    if (e_ != cudaSuccess) return set_err(TJ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

namespace {

struct TruncCache {
  bool valid = false;
  const double *data = nullptr;
  int64_t dim = 0;
  int side = 0, kept_min = 0, kept_max = 0;
  double trun_err = 0;
  uint64_t hash = 0;
  tj_trunc_result res{};
  std::vector<tj_block_sub> sub;
  // the operator stays on the device (trA of ctx) until the second call
  // copies it out: valid while ctx has computed no other truncation
  int64_t len = 0;
  const tj_ctx *ctx = nullptr;
  uint64_t seq = 0;
  const double *dev = nullptr;
};
thread_local TruncCache g_tc;

// Fingerprint of psi for the two-call cache: 4096 values spread over it
// (the second call of the protocol passes the same, unchanged psi; a full
// pass over psi would cost more than the rest of the second call).
uint64_t hash_data(const double *p, int64_t n) {
  uint64_t h = 1469598103934665603ull ^ (uint64_t)n;
  const int64_t k = n < 4096 ? n : 4096;
  for (int64_t i = 0; i < k; ++i) {
    const int64_t at = k > 1 ? i * (n - 1) / (k - 1) : 0;
    uint64_t u;
    std::memcpy(&u, p + at, 8);
    h = (h ^ u) * 1099511628211ull;
  }
  return h;
}

size_t al256(size_t x) { return (x + 255) / 256 * 256; }

// Host tables gathered into one buffer for one copy to the device, each at a
// 256-byte border; room() is device space behind them that nothing is copied
// into (so it comes last).
struct Tables {
  std::vector<char> buf;
  size_t extra = 0;
  size_t zeros(size_t bytes) {
    const size_t at = buf.size();
    buf.resize(at + al256(std::max<size_t>(bytes, 1)), 0);
    return at;
  }
  template <class T>
  size_t add(const std::vector<T> &v) {
    const size_t at = zeros(v.size() * sizeof(T));
    if (!v.empty()) std::memcpy(buf.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
  size_t room(size_t bytes) {
    const size_t at = size();
    extra += al256(std::max<size_t>(bytes, 1));
    return at;
  }
  size_t size() const { return buf.size() + extra; }
};

struct ClusterSize {
  size_t smem;
  int ctas;     // 16 (a non-portable size) or 8
  int active;   // clusters of 16 that run at a time
};
// Clusters of 16 CTAs where the GPU can schedule one with `threads` threads and
// `smem` bytes of dynamic shared memory per CTA; otherwise 8.  Asked once per
// kernel and shared-memory size.
template <typename K16>
ClusterSize cluster_size(K16 kernel16, int threads, size_t smem) {
  static thread_local std::vector<ClusterSize> seen;
  for (auto &x : seen)
    if (x.smem == smem) return x;
  ClusterSize c{smem, 8, 0};
  if (cudaFuncSetAttribute(kernel16, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
      cudaFuncSetAttribute(kernel16, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(16, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 16;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel16, &cfg) == cudaSuccess && n >= 1) {
      c.ctas = 16;
      c.active = n;
    }
  }
  cudaGetLastError();
  seen.push_back(c);
  return c;
}

// How many of the sectors (n: their states, largest first), the largest ones,
// are reduced by a cluster of 16 CTAs each, the others one to a CTA, 16 to a
// cluster: at least those of TD_BIG states, at most those above TD_ONE.  Where
// they do not all run at a time (`active` clusters do, started in this order),
// clusters give way to CTAs if the last sector is then done a tenth sooner.  The
// times (us) fit those of one sector to 8 % from 130 states on: by a cluster
// 0.54 ms (192 states), 0.96 (319), 1.27 (400), 4.1 (857), 12.1 (1400); by a CTA
// 0.57 (160), 0.84 (192), 1.45 (240), 2.6 (300), and with the shared memory that
// clusters ask for, which leaves it no L1, 1.12 (200), 1.65 (240), 2.9 (300).
int td_by_cluster(const std::vector<int> &n, int active) {
  const int ns = (int)n.size();
  int lo = 0;
  while (lo < ns && n[lo] >= TD_BIG) ++lo;
  int hi = lo;
  while (hi < ns && n[hi] > TD_ONE) ++hi;
  if (hi == lo || active < 1 || hi + (ns - hi + 15) / 16 <= active) return hi;
  auto done = [&](int b) {   // when the last cluster ends, b sectors having one each
    std::vector<double> end(active, 0.0);
    auto start = [&](double t) { *std::min_element(end.begin(), end.end()) += t; };
    for (int i = 0; i < b; ++i) start(n[i] * (2.7 + 2.85e-6 * n[i] * n[i]));
    for (int i = b; i < ns; i += 16) start(n[i] * ((b ? 2.45 : 1.45) + 7.95e-5 * n[i] * n[i]));
    return *std::max_element(end.begin(), end.end());
  };
  int best = hi;
  double t = 0.9 * done(hi);
  for (int b = hi - 1; b >= lo; --b) {
    const double tb = done(b);
    if (tb < t) {
      t = tb;
      best = b;
    }
  }
  return best;
}

}  // namespace

extern "C" int tj_truncation(tj_ctx *ctx, const tj_wave *wave, int side, int kept_min, int kept_max,
                             double trun_err, tj_trunc_result *out) {
  if (!ctx || !wave || !out) return set_err(TJ_ERR_ARG, "tj_truncation: null argument");
  if (side != 0 && side != 1) return set_err(TJ_ERR_ARG, "tj_truncation: side must be 0 (system) or 1 (environment)");
  if (wave->num < 1 || !wave->sub || !wave->data) return set_err(TJ_ERR_ARG, "tj_truncation: empty wavefunction");
  const int nsec = wave->num;
  const int64_t D = wave->dim;
  for (int i = 0; i < nsec; ++i) {
    const tj_wave_sub &w = wave->sub[i];
    if (w.sys_dim < 0 || w.env_dim < 0 || w.off < 0 || w.off + (int64_t)w.sys_dim * w.env_dim > D)
      return set_err(TJ_ERR_ARG, "tj_truncation: bad sector table");
    const int n = side == 0 ? w.sys_dim : w.env_dim;
    if (n > EIG_MAX_N) return set_err(TJ_ERR_LIMIT, "tj_truncation: a density-matrix sector exceeds 4096 states");
  }
  const uint64_t h = hash_data(wave->data, D);
  TruncCache &tc = g_tc;
  // The kept operator answers one pair of calls only, the second (with the
  // caller's arrays) after a first without them: the fingerprint is of samples,
  // and psi may have changed in place since.
  const bool second = out->sub && out->data;
  const bool hit = second && tc.valid && tc.data == wave->data && tc.dim == D && tc.side == side && tc.kept_min == kept_min &&
                   tc.kept_max == kept_max && tc.trun_err == trun_err && tc.hash == h && tc.ctx == ctx &&
                   tc.seq == ctx->trunc_seq;
  if (!hit) {
    CKT(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    const auto wall0 = std::chrono::steady_clock::now();
    tc.valid = false;   // until this computation completes
    tc.ctx = ctx;
    tc.seq = ++ctx->trunc_seq;
    tc.dev = nullptr;
    tc.len = 0;
    CKT(cudaEventRecord(ctx->tev[0], st));
    // psi on the device
    int rc;
    if ((rc = ctx->trA.reserve(sizeof(double) * (D + 4)))) return rc;
    double *psi = ctx->trA.d();
    CKT(upload(ctx, psi, wave->data, D, st));
    // rho per sector as one grouped-GEMM pass
    std::vector<Cell> cells;
    std::vector<Task> tasks;
    std::vector<Tile> tiles;
    std::vector<int64_t> roff(nsec), eoff(nsec);
    std::vector<int> dims(nsec), esec;
    int64_t rlen = 0, etot = 0;
    for (int i = 0; i < nsec; ++i) {
      const tj_wave_sub &w = wave->sub[i];
      const int n = side == 0 ? w.sys_dim : w.env_dim, K = side == 0 ? w.env_dim : w.sys_dim;
      dims[i] = n;
      roff[i] = rlen;
      eoff[i] = etot;
      rlen += ((int64_t)n * n + 31) / 32 * 32;
      etot += n;
      esec.insert(esec.end(), n, i);
      Cell c;
      std::memset(&c, 0, sizeof c);
      c.off = roff[i];
      c.ld = n;
      c.M = n;
      c.N = n;
      c.space = SP_SCR;
      c.t_begin = (int)tasks.size();
      Task t;
      std::memset(&t, 0, sizeof t);
      t.L.off = w.off;
      t.L.ld = w.sys_dim;
      t.L.space = SP_PSI;
      t.L.trans = (int8_t)(side == 0 ? 0 : 1);
      t.R = t.L;
      t.R.trans = (int8_t)(side == 0 ? 1 : 0);
      t.coef = 1.0;   // rho_scale_kernel sets 1 / |psi|^2
      t.K = K;
      if (n > 0 && K > 0) tasks.push_back(t);
      c.t_end = (int)tasks.size();
      cells.push_back(c);
    }
    // work items in order of weight (one sector of 857 states holds a fifth of
    // a density matrix's products)
    std::vector<Reduce> red;
    int64_t nslots = 0;
    split_tiles(cells, tasks, tiles, red, nslots, false);
    const int maxn = std::max(1, *std::max_element(dims.begin(), dims.end()));
    // sectors largest first for the one-CTA-per-sector reduction
    std::vector<int> order(nsec);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return dims[a] > dims[b]; });
    // trD: d, e, tau, eigenvalues, scaled d, scaled e^2 (etot each), then 4 per sector
    // trB: rho by sector, then the panel matrix W of each (TD_NB rows)
    if ((rc = ctx->trB.reserve(sizeof(double) * (rlen + TD_NB * etot + 4))) ||
        (rc = ctx->trD.reserve(sizeof(double) * (6 * etot + 4 * nsec + 8))))
      return rc;
    double *dd = ctx->trD.d(), *de = dd + etot, *dtau = de + etot, *dev = dtau + etot, *dds = dev + etot,
           *de2 = dds + etot, *dinfo = de2 + etot;
    // clusters of the tridiagonal reduction: one per large sector, then the
    // others tcl at a time (largest first)
    while (!order.empty() && dims[order.back()] == 0) order.pop_back();
    std::vector<int> sizes;
    for (int x : order) sizes.push_back(dims[x]);
    // shared memory: a small sector's matrix, a middle one's vectors; for one
    // reduced by a cluster as much as a CTA may have (its columns)
    auto td_smem_bytes = [&](int big) {
      size_t b = 0;
      for (size_t q = big; q < sizes.size(); ++q) {
        const size_t n = sizes[q];
        b = std::max(b, sizeof(double) * (n <= TD_SMALL ? n * (n + 2) : 3 * n + EIG_THREADS));
      }
      if (big) {
        b = std::max(b, sizeof(double) * (size_t)td_coop_doubles(maxn, 8));
        int optin = 0;
        cudaFuncAttributes fa;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, tridiag_kernel<16>) == cudaSuccess && optin > (int)fa.sharedSizeBytes + 1024)
          b = std::max(b, (size_t)(optin - (int)fa.sharedSizeBytes - 1024) / 256 * 256);
        cudaGetLastError();
      }
      return b;
    };
    int nbig = 0;
    while (nbig < (int)sizes.size() && sizes[nbig] > TD_ONE) ++nbig;
    size_t tsm = td_smem_bytes(nbig);
    ClusterSize tcs = cluster_size(tridiag_kernel<16>, EIG_THREADS, tsm);
    if (tcs.ctas == 16) {
      nbig = td_by_cluster(sizes, tcs.active);
      tsm = td_smem_bytes(nbig);
      tcs = cluster_size(tridiag_kernel<16>, EIG_THREADS, tsm);
    }
    const int tcl = tcs.ctas;
    std::vector<int> tsec, tbig;
    for (int q = 0; q < nbig; ++q) {
      tsec.insert(tsec.end(), tcl, order[q]);
      tbig.push_back(1);
    }
    for (size_t i = nbig; i < order.size(); i += tcl) {
      for (int r = 0; r < tcl; ++r) tsec.push_back(i + r < order.size() ? order[i + r] : -1);
      tbig.push_back(0);
    }
    const int nclus = (int)tbig.size();
    // the small tables in one buffer and one copy
    Tables tab;
    const size_t p_cells = tab.add(cells), p_tasks = tab.add(tasks), p_tiles = tab.add(tiles), p_red = tab.add(red);
    const size_t p_roff = tab.add(roff), p_eoff = tab.add(eoff), p_dims = tab.add(dims), p_tsec = tab.add(tsec);
    const size_t p_tbig = tab.add(tbig), p_esec = tab.add(esec), p_cnt = tab.zeros(256);
    const int ndot = dot_blocks(D);
    const size_t p_part = tab.room(sizeof(double) * ndot);   // partial sums of |psi|^2
    if ((rc = ctx->trE.reserve(tab.size())) || (rc = ctx->trC.reserve(sizeof(double) * (nslots * BM * BN + 4)))) return rc;
    char *tbase = (char *)ctx->trE.p;
    CKT(cudaMemcpyAsync(tbase, tab.buf.data(), tab.buf.size(), cudaMemcpyHostToDevice, st));
    const int64_t *d_roff = (const int64_t *)(tbase + p_roff), *d_eoff = (const int64_t *)(tbase + p_eoff);
    const int *d_dims = (const int *)(tbase + p_dims);
    int *d_status = (int *)(tbase + p_cnt + 16);
    double *d_nrm2 = (double *)(tbase + p_cnt + 8);   // |psi|^2, before the status words
    GemmParams g;
    std::memset(&g, 0, sizeof g);
    g.psi = psi;
    g.scr = ctx->trB.d();
    g.out = ctx->trB.d();
    g.cells = (const Cell *)(tbase + p_cells);
    g.tasks = (const Task *)(tbase + p_tasks);
    g.tiles = (const Tile *)(tbase + p_tiles);
    g.ntiles = (int)tiles.size();
    g.counter = (unsigned int *)(tbase + p_cnt);
    g.slots = ctx->trC.d();
    double *part = (double *)(tbase + p_part);
    launch_dot(psi, psi, D, part, ndot, st);
    rho_scale_kernel<<<1, 256, 0, st>>>(part, ndot, (Task *)(tbase + p_tasks), (int)tasks.size(), d_nrm2);
    launch_grouped_gemm(g, grouped_gemm_grid(g.ntiles), st);
    launch_reduce(g, (const Reduce *)(tbase + p_red), (int)red.size(), st);
    CKT(cudaGetLastError());
    CKT(cudaEventRecord(ctx->tev[1], st));
    // tridiagonal reduction, then all eigenvalues
    if (nclus) {
      const int *d_tsec = (const int *)(tbase + p_tsec), *d_tbig = (const int *)(tbase + p_tbig);
      const long long wait_cycles = (long long)(ctx->wait_s * TD_CYCLES);
      if (tcl == 16) {
        CKT(cudaFuncSetAttribute(tridiag_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm));
        tridiag_kernel<16><<<nclus * 16, EIG_THREADS, tsm, st>>>(ctx->trB.d(), d_roff, d_dims, d_eoff, d_tsec, d_tbig,
                                                                 dd, de, dtau, ctx->trB.d() + rlen, dinfo, dds, de2, (int64_t)(tsm / 8),
        d_status, wait_cycles);
      } else {
        CKT(cudaFuncSetAttribute(tridiag_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm));
        tridiag_kernel<8><<<nclus * 8, EIG_THREADS, tsm, st>>>(ctx->trB.d(), d_roff, d_dims, d_eoff, d_tsec, d_tbig,
                                                               dd, de, dtau, ctx->trB.d() + rlen, dinfo, dds, de2, (int64_t)(tsm / 8),
        d_status, wait_cycles);
      }
      CKT(cudaGetLastError());
    }
    CKT(cudaEventRecord(ctx->tev[2], st));
    if (etot) {
      bisect_kernel<<<(unsigned)((etot + 3) / 4), 128, 0, st>>>(dds, de2, d_eoff, d_dims, dinfo,
                                                                    (const int *)(tbase + p_esec), (int)etot, dev);
      CKT(cudaGetLastError());
    }
    std::vector<double> ev(etot);
    CKT(cudaMemcpyAsync(ctx->pinned, d_nrm2, 16, cudaMemcpyDeviceToHost, st));   // and the status word
    CKT(cudaMemcpyAsync(ev.data(), dev, sizeof(double) * etot, cudaMemcpyDeviceToHost, st));
    CKT(cudaEventRecord(ctx->tev[3], st));
    CKT(cudaStreamSynchronize(st));
    const double nrm2 = ctx->pinned[0];
    if (reinterpret_cast<const int *>(ctx->pinned + 1)[0] & 4)
      return set_err(TJ_ERR_TIMEOUT, "tj_truncation: a wait of the tridiagonal reduction gave up");
    if (!(nrm2 > 0) || !std::isfinite(nrm2)) return set_err(TJ_ERR_NUMERIC, "tj_truncation: zero or non-finite psi");
    const auto sel0 = std::chrono::steady_clock::now();
    float stage_ms[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int i = 0; i < 3; ++i) CKT(cudaEventElapsedTime(&stage_ms[i], ctx->tev[i], ctx->tev[i + 1]));
    double select_ms = 0;
    int max_kept = 0;

    // ---- selection (den_mat.f90:201-330) ----
    std::vector<int> qnu(nsec), qnd(nsec);
    for (int i = 0; i < nsec; ++i) {
      qnu[i] = side == 0 ? wave->sub[i].sys_num_up : wave->sub[i].env_num_up;
      qnd[i] = side == 0 ? wave->sub[i].sys_num_down : wave->sub[i].env_num_down;
    }
    // per sector, eigenvalue order (ascending, as DSYEV returns them)
    std::vector<std::vector<int>> asc(nsec);
    std::vector<double> val;
    std::vector<int> owner, mult;
    val.reserve(etot);
    for (int i = 0; i < nsec; ++i) {
      asc[i].resize(dims[i]);
      std::iota(asc[i].begin(), asc[i].end(), 0);
      const double *e = ev.data() + eoff[i];
      std::stable_sort(asc[i].begin(), asc[i].end(), [&](int a, int b) { return e[a] < e[b]; });
      for (int k = 0; k < dims[i]; ++k) {
        val.push_back(e[asc[i][k]]);
        owner.push_back(i);
        mult.push_back(qnd[i] + 1);
      }
    }
    const int total = (int)val.size();
    const double thr = (double)1.0e-15f;   // the reference compares against the literal 1.0E-15
    double tot_pm = 0;
    for (int i = 0; i < total; ++i) tot_pm += val[i] * mult[i];
    double ent1 = 0, ent2 = 0, ents = 0;
    for (int i = 0; i < total; ++i)
      if (val[i] >= thr) {
        const double v1 = val[i] / mult[i];
        ent1 -= v1 * std::log(v1) * mult[i];
      }
    for (int i = 0; i < total; ++i) {
      const double v = val[i] / tot_pm;
      if (v >= thr) ent2 -= v * std::log(v) * mult[i];
    }
    // descending order of the spectrum; ties keep the order of the sectors
    std::vector<int> ord(total);
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return val[a] > val[b]; });
    double sum = 0;
    for (int i = 0; i < total; ++i) sum += val[ord[i]];
    std::vector<double> w(total);
    for (int i = 0; i < total; ++i) w[i] = val[ord[i]] / sum;
    int num_state;
    double err = 0;
    if (total <= kept_min) {
      num_state = total;
    } else {
      for (int i = kept_min; i < total; ++i) err += w[i];
      num_state = kept_min;
      while (err > trun_err && num_state < total) {
        ++num_state;
        err -= w[num_state - 1];
        if (err <= trun_err || num_state >= kept_max) break;
      }
    }
    for (int i = 0; i < total; ++i)
      if (w[i] >= thr) ents -= w[i] * std::log(w[i]);
    std::vector<int> cnt(nsec, 0);
    for (int k = 0; k < num_state; ++k) ++cnt[owner[ord[k]]];
    // kept eigenvectors: the cnt largest of each sector, in ascending order
    std::vector<int> job_sec, job_k, grp, slab;
    std::vector<int64_t> job_dst;
    tc.sub.clear();
    int64_t dpos = 0;
    for (int i = 0; i < nsec; ++i) {
      if (cnt[i] == 0) continue;
      int x = 0;   // the reference copies from the first sector with the same labels
      while (x < nsec && !(qnu[x] == qnu[i] && qnd[x] == qnd[i])) ++x;
      const int row = dims[i], col = cnt[i];
      tj_block_sub sb;
      std::memset(&sb, 0, sizeof sb);
      sb.num_up = qnu[i];
      sb.num_down = qnd[i];
      sb.down_dif = 0;
      sb.row_dim = row;
      sb.sdim = col;
      sb.off = dpos;
      tc.sub.push_back(sb);
      grp.insert(grp.end(), {x, (int)job_sec.size(), col, 0});
      for (int c = 0; c < col; ++c) {
        job_sec.push_back(x);
        job_k.push_back(asc[x][dims[x] - col + c]);
        job_dst.push_back(dpos + (int64_t)c * row);
      }
      dpos += (int64_t)row * col;
    }
    tc.len = dpos;
    const int njobs = (int)job_sec.size(), ngrp = (int)grp.size() / 4;
    if (njobs > 0) {
      // back-transformation: blocks of reflectors on 16 vectors (8 for sectors
      // above 1024 states, whose rows would not fit the registers) a CTA, else
      // (above 1536) vector by vector in shared memory, W warps
      const bool bt_wy = maxn <= 1536;
      const int W = bt_wy ? (maxn <= 1024 ? 16 : 8) : std::max(1, std::min(32, (int)(196608 / (sizeof(double) * maxn))));
      std::vector<int> pan, pan0(nsec, 0);
      if (bt_wy)
        for (int b = 0; b < ngrp; ++b) {
          const int x = grp[4 * b];
          pan0[x] = (int)pan.size() / 2;
          for (int q = 0; q * BT_NB < dims[x] - 1; ++q) pan.insert(pan.end(), {x, q});
        }
      const int npan = (int)pan.size() / 2;
      for (int b = 0; b < ngrp; ++b)
        for (int c0 = 0; c0 < grp[4 * b + 2]; c0 += W) slab.insert(slab.end(), {b, c0});
      const int nslab = (int)slab.size() / 2;
      const int ldy = (maxn + 3) / 4 * 4;
      // trC: inverse-iteration factors and vectors; trA: tables and the operator
      const size_t wpl = (size_t)maxn * njobs;
      const size_t p_work = 0, p_y = p_work + al256(5 * wpl * 8), p_piv = p_y + al256((size_t)njobs * ldy * 8);
      // the two products of the orthonormalisation: G = Y^T Y of every block
      // (its lower triangle of tiles), and Z = Y R by column tiles, R lower
      // triangular
      std::vector<Cell> ocells;
      std::vector<Task> otasks;
      std::vector<Tile> gtiles, ztiles;
      std::vector<int64_t> goff(ngrp);
      int64_t glen = 0;
      {
        auto opnd = [&](int64_t off, int ld, int8_t space, int8_t trans) {
          Operand o;
          std::memset(&o, 0, sizeof o);
          o.off = off;
          o.ld = ld;
          o.space = space;
          o.trans = trans;
          return o;
        };
        auto cell = [&](int64_t off, int ld, int M, int N, const Operand &L, const Operand &R, int K) {
          Cell c;
          std::memset(&c, 0, sizeof c);
          c.off = off;
          c.ld = ld;
          c.M = M;
          c.N = N;
          c.t_begin = (int)otasks.size();
          Task t;
          std::memset(&t, 0, sizeof t);
          t.L = L;
          t.R = R;
          t.coef = 1.0;
          t.K = K;
          otasks.push_back(t);
          c.t_end = (int)otasks.size();
          ocells.push_back(c);
        };
        auto tile = [&](std::vector<Tile> &v, int r0, int c0) {
          const int ci = (int)ocells.size() - 1, t = ocells[ci].t_begin;
          v.push_back(Tile{ci, r0, c0, t, t + 1, t + 1, t + 1, -1});
        };
        for (int b = 0; b < ngrp; ++b) {
          const int n = dims[grp[4 * b]], cnt = grp[4 * b + 2];
          const int64_t y0 = (int64_t)grp[4 * b + 1] * ldy;
          goff[b] = glen;
          glen += ((int64_t)cnt * cnt + 3) / 4 * 4;
          cell(goff[b], cnt, cnt, cnt, opnd(y0, ldy, SP_PSI, 1), opnd(y0, ldy, SP_PSI, 0), n);
          for (int c0 = 0; c0 < cnt; c0 += BN)
            for (int r0 = c0 / BM * BM; r0 < cnt; r0 += BM) tile(gtiles, r0, c0);
          for (int c0 = 0; c0 < cnt; c0 += BN) {
            cell(y0 + (int64_t)c0 * ldy, ldy, n, std::min(BN, cnt - c0), opnd(y0 + (int64_t)c0 * ldy, ldy, SP_PSI, 0),
                 opnd(goff[b] + (int64_t)c0 * cnt + c0, cnt, SP_SCR, 0), cnt - c0);
            for (int r0 = 0; r0 < n; r0 += BM) tile(ztiles, r0, 0);
          }
        }
        // longest inner dimension first
        for (auto *v : {&gtiles, &ztiles})
          std::stable_sort(v->begin(), v->end(), [&](const Tile &a, const Tile &b) { return otasks[a.tb].K > otasks[b.tb].K; });
      }
      const size_t p_z = p_piv + al256(wpl), p_g = p_z + al256((size_t)njobs * ldy * 8);
      if ((rc = ctx->trC.reserve(p_g + al256((size_t)glen * 8)))) return rc;
      // clusters of the orthonormalisation: one per large kept block (cnt^2 n
      // above 3e7), then the other blocks ocl at a time, largest first
      const size_t osm = sizeof(double) * (3 * (size_t)maxn + (maxn + 7) / 8 + 8 + ORTH_THREADS);
      const int ocl = cluster_size(orthonormalize_kernel<16>, ORTH_THREADS, osm).ctas;
      std::vector<int> oblk, obig;
      {
        std::vector<int> bo(ngrp);
        std::iota(bo.begin(), bo.end(), 0);
        auto work = [&](int b) { return (double)grp[4 * b + 2] * grp[4 * b + 2] * dims[grp[4 * b]]; };
        std::stable_sort(bo.begin(), bo.end(), [&](int a, int b) { return work(a) > work(b); });
        size_t i = 0;
        for (; i < bo.size() && work(bo[i]) >= 3e7; ++i) {
          oblk.insert(oblk.end(), ocl, bo[i]);
          obig.push_back(1);
        }
        for (; i < bo.size(); i += ocl) {
          for (int r = 0; r < ocl; ++r) oblk.push_back(i + r < bo.size() ? bo[i + r] : -1);
          obig.push_back(0);
        }
      }
      const int nocl = (int)obig.size();
      Tables tab2;
      const size_t q_sec = tab2.add(job_sec), q_k = tab2.add(job_k), q_dst = tab2.add(job_dst), q_grp = tab2.add(grp);
      const size_t q_slab = tab2.add(slab), q_oblk = tab2.add(oblk), q_obig = tab2.add(obig), q_cells = tab2.add(ocells);
      const size_t q_tasks = tab2.add(otasks), q_gt = tab2.add(gtiles), q_zt = tab2.add(ztiles), q_goff = tab2.add(goff);
      const size_t q_pan = tab2.add(pan), q_pan0 = tab2.add(pan0);
      std::vector<int> first(ngrp);
      for (int b = 0; b < ngrp; ++b) first[b] = grp[4 * b + 2];
      const size_t q_cnt = tab2.zeros(256), q_first = tab2.add(first);
      const size_t q_wyt = tab2.room(sizeof(double) * BT_NB * BT_NB * npan), q_out = tab2.room((size_t)dpos * 8);
      if ((rc = ctx->trA.reserve(tab2.size()))) return rc;   // psi is no longer needed
      char *ab = (char *)ctx->trA.p, *cb = (char *)ctx->trC.p;
      CKT(cudaMemcpyAsync(ab, tab2.buf.data(), tab2.buf.size(), cudaMemcpyHostToDevice, st));
      double *Y = (double *)(cb + p_y), *Z = (double *)(cb + p_z), *d_out = (double *)(ab + q_out);
      tc.dev = d_out;
      for (int b = 0; b < ngrp; ++b) max_kept = std::max(max_kept, grp[4 * b + 2]);
      select_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - sel0).count();
      CKT(cudaEventRecord(ctx->tev[4], st));
      inverse_iter_kernel<<<(njobs + 63) / 64, 64, 0, st>>>(dd, de, d_eoff, d_dims, dinfo, dev,
                                                            (const int *)(ab + q_sec), (const int *)(ab + q_k), njobs,
                                                            maxn, (double *)(cb + p_work),
                                                            (unsigned char *)(cb + p_piv), Y, ldy, d_status);
      CKT(cudaGetLastError());
      CKT(cudaEventRecord(ctx->tev[5], st));
      {
        const int *d_oblk = (const int *)(ab + q_oblk), *d_obig = (const int *)(ab + q_obig);
        const int *d_grp = (const int *)(ab + q_grp), *d_k = (const int *)(ab + q_k);
        int *d_first = (int *)(ab + q_first);
        GemmParams g2;
        std::memset(&g2, 0, sizeof g2);
        g2.psi = Y;
        g2.scr = (double *)(cb + p_g);
        g2.out = (double *)(cb + p_g);
        g2.cells = (const Cell *)(ab + q_cells);
        g2.tasks = (const Task *)(ab + q_tasks);
        g2.tiles = (const Tile *)(ab + q_gt);
        g2.ntiles = (int)gtiles.size();
        g2.counter = (unsigned int *)(ab + q_cnt);
        launch_grouped_gemm(g2, grouped_gemm_grid(g2.ntiles), st);
        const dim3 ogrid(ngrp, std::max(1, std::min(32, (max_kept + 7) / 8)));
        ortho_check_kernel<<<ogrid, 256, 0, st>>>(d_grp, (const int64_t *)(ab + q_goff), (const double *)(cb + p_g), d_first);
        ortho_factor_kernel<<<ogrid, 256, 0, st>>>(d_grp, (const int64_t *)(ab + q_goff), (double *)(cb + p_g), d_first);
        g2.out = Z;
        g2.tiles = (const Tile *)(ab + q_zt);
        g2.ntiles = (int)ztiles.size();
        g2.counter = (unsigned int *)(ab + q_cnt) + 1;
        launch_grouped_gemm(g2, grouped_gemm_grid(g2.ntiles), st);
        if (ocl == 16) {
          CKT(cudaFuncSetAttribute(orthonormalize_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)osm));
          orthonormalize_kernel<16><<<nocl * 16, ORTH_THREADS, osm, st>>>(d_oblk, d_obig, d_grp, d_dims, d_eoff, dev,
                                                                          dinfo, d_k, d_first, Z, ldy, d_status);
        } else {
          CKT(cudaFuncSetAttribute(orthonormalize_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)osm));
          orthonormalize_kernel<8><<<nocl * 8, ORTH_THREADS, osm, st>>>(d_oblk, d_obig, d_grp, d_dims, d_eoff, dev,
                                                                        dinfo, d_k, d_first, Z, ldy, d_status);
        }
      }
      CKT(cudaGetLastError());
      CKT(cudaEventRecord(ctx->tev[6], st));
      if (bt_wy) {
        double *d_t = (double *)(ab + q_wyt);
        if (npan) wy_t_kernel<<<npan, 256, 0, st>>>(ctx->trB.d(), d_roff, dtau, d_eoff, d_dims, (const int *)(ab + q_pan), d_t);
        auto launch = [&](auto kern, int tiles, int vt) -> cudaError_t {
          const int bsm = (int)sizeof(double) * bt_smem_doubles(tiles, vt);
          cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bsm);
          if (e != cudaSuccess) return e;
          kern<<<nslab, 32 * BT_WARPS, bsm, st>>>(ctx->trB.d(), d_roff, d_t, (const int *)(ab + q_pan0), d_dims,
                                                  (const int *)(ab + q_grp), (const int *)(ab + q_slab), Z, ldy,
                                                  (const int64_t *)(ab + q_dst), d_out);
          return cudaGetLastError();
        };
        // 128 states per row tile of a warp
        if (maxn <= 128) CKT(launch(backtransform_wy_kernel<1, 2>, 1, 2));
        else if (maxn <= 256) CKT(launch(backtransform_wy_kernel<2, 2>, 2, 2));
        else if (maxn <= 512) CKT(launch(backtransform_wy_kernel<4, 2>, 4, 2));
        else if (maxn <= 768) CKT(launch(backtransform_wy_kernel<6, 2>, 6, 2));
        else if (maxn <= 1024) CKT(launch(backtransform_wy_kernel<8, 2>, 8, 2));
        else if (maxn <= 1280) CKT(launch(backtransform_wy_kernel<10, 1>, 10, 1));
        else CKT(launch(backtransform_wy_kernel<12, 1>, 12, 1));
      } else {
        const size_t bsm = sizeof(double) * (size_t)W * ldy;
        CKT(cudaFuncSetAttribute(backtransform_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsm));
        backtransform_kernel<<<nslab, 32 * W, bsm, st>>>(ctx->trB.d(), d_roff, dtau, d_eoff, d_dims,
                                                         (const int *)(ab + q_grp), (const int *)(ab + q_slab), Z,
                                                         ldy, (const int64_t *)(ab + q_dst), d_out);
        CKT(cudaGetLastError());
      }
      int status[16] = {0};
      CKT(cudaMemcpyAsync(status, d_status, sizeof status, cudaMemcpyDeviceToHost, st));
      CKT(cudaEventRecord(ctx->tev[7], st));
      CKT(cudaStreamSynchronize(st));
      for (int i = 4; i < 7; ++i) CKT(cudaEventElapsedTime(&stage_ms[i - 1], ctx->tev[i], ctx->tev[i + 1]));
      if (status[0] & 1) {
        double dg[6];
        std::memcpy(dg, status + 4, sizeof dg);
        char buf[256];
        std::snprintf(buf, sizeof buf,
                      "tj_truncation: inverse iteration produced a non-finite vector (sector %d, eigenvalue %d of "
                      "%d, lambda %.17g, pivot floor %.3g, norm %g)",
                      (int)dg[0], (int)dg[1], (int)dg[4], dg[2], dg[3], dg[5]);
        return set_err(TJ_ERR_NUMERIC, buf);
      }
      if (status[0] & 2)
        return set_err(TJ_ERR_NUMERIC,
                       "tj_truncation: inverse iteration gave linearly dependent eigenvectors for a cluster of "
                       "eigenvalues above the bottom of its sector's spectrum");
    }
    {
      tj_hpsi_stats &S = ctx->stats;
      S.trunc_ms_rho = stage_ms[0];
      S.trunc_ms_tridiag = stage_ms[1];
      S.trunc_ms_eig = stage_ms[2];
      S.trunc_ms_select = select_ms;
      S.trunc_ms_vec = stage_ms[3];
      S.trunc_ms_orth = stage_ms[4];
      S.trunc_ms_back = stage_ms[5];
      S.trunc_ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
      S.trunc_max_n = maxn;
      S.trunc_max_kept = max_kept;
    }
    std::memset(&tc.res, 0, sizeof tc.res);
    tc.res.num_state = num_state;
    tc.res.num = (int32_t)tc.sub.size();
    tc.res.data_len = dpos;
    tc.res.trunc_err = err;
    tc.res.entropy1 = ent1;
    tc.res.entropy2 = ent2;
    tc.res.entropys = ents;
    tc.valid = true;
    tc.data = wave->data;
    tc.dim = D;
    tc.side = side;
    tc.kept_min = kept_min;
    tc.kept_max = kept_max;
    tc.trun_err = trun_err;
    tc.hash = h;
  }
  tj_block_sub *usub = out->sub;
  double *udata = out->data;
  *out = tc.res;
  out->sub = usub;
  out->data = udata;
  if (usub && udata) {
    std::memcpy(usub, tc.sub.data(), sizeof(tj_block_sub) * tc.sub.size());
    if (tc.len > 0) {
      // straight from the device into the caller's array (the cache hit
      // above requires the device copy to be intact)
      CKT(cudaSetDevice(ctx->device));
      const int rc = download(ctx, udata, tc.dev, tc.len, ctx->stream);
      if (rc) return rc;
    }
    // the renormalisation of this step and the prediction of the next read
    // the operator again: with residency on, its device copy is kept (the
    // copy runs on the context's stream, ahead of anything that rewrites trA)
    if (tc.len > 0) {
      const int rc = res_keep(ctx, udata, tc.len, tc.dev, ctx->stream);
      if (rc) return rc;
    }
    tc.valid = false;
  }
  return TJ_OK;
}
