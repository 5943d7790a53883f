// Device kernels of the B200 tjsq hot path: grouped FP64 GEMM over psi cells,
// merged-operator sums (hmerge), and the Lanczos vector operations.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include <cooperative_groups.h>

#include "kernels.cuh"
#include "sturm.cuh"

namespace cg = cooperative_groups;

namespace tjb {

// ------------------------------------------------------------ grouped GEMM
// Persistent CTAs of four multiplying warps and two copying warps take 64x64
// tiles of cells, the first by their index and the others from a global
// counter, and accumulate sum_t coef_t * op(L_t) * op(R_t) over the cell's
// tasks with FP64 DMMA (mma.sync m8n8k4).
//
// All tiles of a CTA are one stream of steps of up to GEMM_BK inner-dimension
// entries, carried through GEMM_STAGES shared-memory stages.  A step takes
// whatever the next tasks of the tile give, each padded to groups of four
// entries with its own coefficient: half of the tasks of a superblock have an
// inner dimension of 13 and less, and a step per task left the cost of a step
// (its barriers and waits, some 400 cycles) larger than its products.  One
// copying warp fetches the L operands, the other the R operands, with
// cp.async, over task and tile borders; stages are handed over by named
// barriers (hardware barriers, no polling).  Sub-blocks have any leading
// dimension, so the copies are of single doubles.  A stage holds an operand
// as [k][i], i the row of op(L) or the column of op(R), at
// k * 64 + (i ^ f(k)) with f exchanging two bit pairs of k: copies along i,
// copies along k and fragment reads are all free of bank conflicts without
// padding.
//
// DMMA issues once per 16 cycles and sub-core and reaches 37 TFLOP/s from
// registers with one warp per sub-core, so a tile costs its DMMAs as long as
// nothing else is in the multiplying warps' way: the copies' address work is
// in warps of their own, the loop over a tile's steps is compiled for the
// warp's number of granules, and of the eight 8-row and eight 8-column
// granules of a tile only those inside the cell are copied and multiplied,
// with inner dimensions padded to 4 (the sub-blocks of a superblock fill
// 64x64x16 tiles to a half at m = 2000 and to a percent at m = 256).
// Granules go to the warps alternately, so that a part-filled tile still
// spreads over all four.  Two CTAs per SM, for the registers: held to 128 a
// thread for more of them, the accumulators are moved about and the kernel
// takes half as long again.
//
// Both launches of the FP64 H*psi of the 4x24 m = 2000 superblock together:
// 1355 -> 760 us (DMMA pipe 33 -> 60 % on products that count); grand-canonical
// 4x6 m = 300: 185 -> 80 us; 2x16 ladder m = 256: 55 -> 16 us; one 1024^3
// block: 18.7 -> 29.4 TFLOP/s.
constexpr int GEMM_MMA = 128, GEMM_COPY = 64;   // threads that multiply / copy
constexpr int GEMM_THREADS = GEMM_MMA + GEMM_COPY;
constexpr int GEMM_BK = 32;                      // inner-dimension entries of a step
constexpr int GEMM_STAGES = 3;
constexpr int GEMM_LAG = 1;                      // a step is handed over when this many later ones have been issued
constexpr int GEMM_STAGE_D = (BM + BN) * GEMM_BK;   // doubles of one stage
constexpr int GEMM_SMEM = GEMM_STAGES * GEMM_STAGE_D * 8;
constexpr int GEMM_CTAS = 2;                     // resident per SM
// named barriers (0 is __syncthreads): stage filled, stage read, next tile
constexpr int GEMM_FULL = 1, GEMM_EMPTY = GEMM_FULL + GEMM_STAGES, GEMM_NEXT = GEMM_EMPTY + GEMM_STAGES;

// what the multiplying warps learn with a stage
struct GemmStep {
  double coef[GEMM_BK / 4];   // of each group of four k
  int kn;                     // groups of four k
  int last;                   // 1: the tile's last step, 2: no more steps
  int nrow, ncol;             // of the tile
  int tile;                   // index of the tile (its partial sum in dot mode)
  int pad;
  Tile tl;                    // set at the last step
  Cell c;
};

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ const double *space_base(const GemmParams &p, int sp) {
  return sp == SP_OPS ? p.ops : (sp == SP_PSI ? p.psi : p.scr);
}

// the place of k in the swizzle of a stage: its low two bit pairs exchanged
__device__ __forceinline__ int gemm_f(int k) { return ((k & 3) << 2) | (k >> 2 & 3); }

// 8 bytes from global to shared memory; n = 0: zeros, src not read
__device__ __forceinline__ void cp_async8z(uint32_t dst, const double *src, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// One operand's k in [0, kv) into groups g, g + 1, ... of a stage, by one
// warp, element (i, k) at src[k * ld + i]: the lanes along i (2^LG < 32 of
// them: 32 >> LG k at a time).  Rows past n are left as they are (they meet
// only output rows past the cell); the last group is filled up with zeros.
template <int LG>
__device__ __forceinline__ void gemm_copy_i(uint32_t dst, const double *src, int ld, int n, int g, int kv) {
  constexpr int ST = 32 >> LG;   // k apart of a lane's copies
  const int lane = threadIdx.x & 31, i = lane & ((1 << LG) - 1), kb = lane >> LG;
  if (i >= n) return;
  const double *s = src + (int64_t)kb * ld + i;
  const int64_t st = (int64_t)ST * ld;
  const bool in2 = LG == 5 && i + 32 < n;
  uint32_t d = dst + (uint32_t)((4 * g + kb) * BM + (i ^ (kb << 2))) * 8u;
  int k = 0;
#pragma unroll 2
  for (; k + 4 <= kv; k += 4, ++g, d += 4 * BM * 8) {
    const uint32_t x = d ^ (uint32_t)((g & 3) * 8);
#pragma unroll
    for (int j = 0; j < 4; j += ST) {
      cp_async8((x ^ (uint32_t)(j * 32)) + j * BM * 8, s);
      if (in2) cp_async8((x ^ (uint32_t)(j * 32)) + j * BM * 8 + 256, s + 32);
      s += st;
    }
  }
  if (k < kv) {
    const uint32_t x = d ^ (uint32_t)((g & 3) * 8);
#pragma unroll
    for (int j = 0; j < 4; j += ST) {
      const int bytes = k + kb + j < kv ? 8 : 0;
      cp_async8z((x ^ (uint32_t)(j * 32)) + j * BM * 8, s, bytes);
      if (in2) cp_async8z((x ^ (uint32_t)(j * 32)) + j * BM * 8 + 256, s + 32, bytes);
      s += st;
    }
  }
}
// Element (i, k) at src[i * ld + k]: the lanes along k, 2^LK of them, 32 >> LK
// rows at a time.
template <int LK>
__device__ __forceinline__ void gemm_copy_k(uint32_t dst, const double *src, int ld, int n, int g, int kv) {
  constexpr int R = 32 >> LK;
  const int lane = threadIdx.x & 31, k = lane & ((1 << LK) - 1), ib = lane >> LK, at = 4 * g + k;
  if (k >= ((kv + 3) & ~3)) return;
  const double *s = src + (int64_t)ib * ld + k;
  const int64_t st = R * (int64_t)ld;
  const uint32_t d0 = dst + (uint32_t)(at * BM) * 8u;
  const uint32_t f = (uint32_t)gemm_f(at);
  const int bytes = k < kv ? 8 : 0;
#pragma unroll 4
  for (int i = ib; i < n; i += R, s += st) cp_async8z(d0 + ((uint32_t)i ^ f) * 8u, s, bytes);
}

// The warp's MM x NN granules of one step; la, lb: the lane's places in
// granule 0 of the two operands for each group kk of four k; the warp's
// granules are 16 entries apart.
template <int MM, int NN>
__device__ __forceinline__ void gemm_mma(double (&acc)[4][4][2], const double *st, const int (&la)[4],
                                         const int (&lb)[4], const double *coef, int kn) {
  auto load = [&](int kk, double (&a)[MM], double (&b)[NN]) {
    const double cf = coef[kk];
#pragma unroll
    for (int mi = 0; mi < MM; ++mi) a[mi] = cf * st[la[kk] + mi * 16];
#pragma unroll
    for (int ni = 0; ni < NN; ++ni) b[ni] = st[lb[kk] + ni * 16];
  };
  auto mul = [&](const double (&a)[MM], const double (&b)[NN]) {
#pragma unroll
    for (int mi = 0; mi < MM; ++mi)
#pragma unroll
      for (int ni = 0; ni < NN; ++ni) dmma_8x8x4(acc[mi][ni], a[mi], b[ni]);
  };
  // the next group's fragments are read under this group's products
  for (; kn >= 4; kn -= 4, st += 16 * BM, coef += 4) {
    double a[2][MM], b[2][NN];
    load(0, a[0], b[0]);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk < 3) load(kk + 1, a[(kk + 1) & 1], b[(kk + 1) & 1]);
      mul(a[kk & 1], b[kk & 1]);
    }
  }
#pragma unroll
  for (int kk = 0; kk < 3; ++kk) {
    if (kk >= kn) break;
    double a[MM], b[NN];
    load(kk, a, b);
    mul(a, b);
  }
}

// The steps of one tile for a warp that holds MM x NN of its granules, from
// the one in `stage` (filled) to the last, which is left to the caller.
template <int MM, int NN>
__device__ __forceinline__ void gemm_tile(double (&acc)[4][4][2], const double *gsm, const GemmStep *step, int &stage,
                                          const int (&la)[4], const int (&lb)[4]) {
  for (;;) {
    const GemmStep &s = step[stage];
    const int last = s.last, kn = s.kn;
    if (MM > 0) gemm_mma<MM == 0 ? 1 : MM, NN == 0 ? 1 : NN>(acc, gsm + stage * GEMM_STAGE_D, la, lb, s.coef, kn);
    if (last) return;
    bar_arrive(GEMM_EMPTY + stage, GEMM_THREADS);
    stage = stage == GEMM_STAGES - 1 ? 0 : stage + 1;
    bar_sync(GEMM_FULL + stage, GEMM_THREADS);
  }
}

// The copying warps: warp 0 of them the L operands and the steps' records,
// warp 1 the R operands.
__device__ __forceinline__ void gemm_copy_stream(const GemmParams &p, uint32_t sm0, GemmStep *step, int *s_next) {
  const int lane = threadIdx.x & 31;
  const bool left = threadIdx.x - GEMM_MMA < 32;
  int count = 0, stage = 0;   // steps issued, the next one's stage
  auto hand_over = [&](int n) {   // step n is in shared memory
    bar_arrive(GEMM_FULL + n % GEMM_STAGES, GEMM_THREADS);
  };
  auto acquire = [&]() {
    if (count >= GEMM_STAGES) bar_sync(GEMM_EMPTY + stage, GEMM_THREADS);
  };
  auto issued = [&]() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (count >= GEMM_LAG) {
      asm volatile("cp.async.wait_group %0;" ::"n"(GEMM_LAG) : "memory");
      hand_over(count - GEMM_LAG);
    }
    ++count;
    stage = stage == GEMM_STAGES - 1 ? 0 : stage + 1;
  };
  for (int t = blockIdx.x; t < p.ntiles;) {
    // the tile after this one; the CTAs fetch ntiles numbers in all, so the
    // counter has wrapped to 0 when the launch ends
    unsigned nxt = 0;
    if (left && lane == 0) nxt = atomicInc(p.counter, (unsigned)p.ntiles - 1u);
    const Tile tl = p.tiles[t];
    const Cell c = p.cells[tl.cell];
    const int nrow = min(BM, c.M - tl.row0), ncol = min(BN, c.N - tl.col0);
    const int n = left ? nrow : ncol, at = left ? tl.row0 : tl.col0;
    const int lg = n > 16 ? 5 : n > 8 ? 4 : 3;
    int g = GEMM_BK / 4;   // groups of the open stage in use; all: none is open
    bool open = false;
    auto begin = [&]() {
      acquire();
      g = 0;
      open = true;
    };
    auto finish = [&](int last) {
      if (left && lane == 0) {
        GemmStep &s = step[stage];
        s.kn = g;
        s.last = last;
        s.nrow = nrow;
        s.ncol = ncol;
        if (last) {
          s.tile = t;
          s.tl = tl;
          s.c = c;
        }
      }
      issued();
    };
    for (int tb = tl.tb; tb < tl.te; tb += 32) {
      // one task per lane, handed round by shuffles
      Operand op = Operand{0, 0, 0, 0, 0};
      double co = 0.0;
      int Kl = 0;
      if (tb + lane < tl.te) {
        const Task *tk = p.tasks + tb + lane;
        op = left ? tk->L : tk->R;
        co = tk->coef;
        Kl = tk->K;
      }
      const int nt = min(32, tl.te - tb);
      for (int q = 0; q < nt; ++q) {
        const int K = __shfl_sync(0xffffffffu, Kl, q), ld = __shfl_sync(0xffffffffu, op.ld, q);
        const int fl = __shfl_sync(0xffffffffu, (int)op.space | (int)op.trans << 8, q);
        const double *src = space_base(p, fl & 255) + __shfl_sync(0xffffffffu, op.off, q);
        const bool kmajor = left == (fl >> 8 != 0);   // k runs along the stored columns
        src += kmajor ? (int64_t)at * ld : at;
        const double coef = __shfl_sync(0xffffffffu, co, q);
        for (int k0 = 0; k0 < K;) {
          if (g == GEMM_BK / 4) {
            if (open) finish(0);
            begin();
          }
          const int kv = min(K - k0, GEMM_BK - 4 * g), kp = (kv + 3) & ~3;   // kp: in whole groups
          const uint32_t d = sm0 + (uint32_t)(stage * GEMM_STAGE_D + (left ? 0 : BM * GEMM_BK)) * 8u;
          if (kmajor) {
            if (kp > 16)
              gemm_copy_k<5>(d, src, ld, n, g, kv);
            else if (kp > 8)
              gemm_copy_k<4>(d, src, ld, n, g, kv);
            else if (kp > 4)
              gemm_copy_k<3>(d, src, ld, n, g, kv);
            else
              gemm_copy_k<2>(d, src, ld, n, g, kv);
          } else if (lg == 5)
            gemm_copy_i<5>(d, src, ld, n, g, kv);
          else if (lg == 4)
            gemm_copy_i<4>(d, src, ld, n, g, kv);
          else
            gemm_copy_i<3>(d, src, ld, n, g, kv);
          if (left && lane < kp >> 2) step[stage].coef[g + lane] = coef;
          src += kmajor ? kv : (int64_t)kv * ld;
          k0 += kv;
          g += kp >> 2;
        }
      }
    }
    if (!open) begin();   // no task: an empty step
    finish(1);
    if (left && lane == 0) *s_next = (int)(nxt + gridDim.x);
    bar_sync(GEMM_NEXT, GEMM_COPY);
    t = *s_next;
    bar_sync(GEMM_NEXT, GEMM_COPY);
  }
  acquire();
  if (left && lane == 0) step[stage].last = 2;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int n = count > GEMM_LAG ? count - GEMM_LAG : 0; n <= count; ++n) hand_over(n);
  // every barrier a stage's readers arrive at is completed before the exit
  for (int n = count >= GEMM_STAGES ? count - GEMM_STAGES + 1 : 0; n < count; ++n)
    bar_sync(GEMM_EMPTY + n % GEMM_STAGES, GEMM_THREADS);
}

__global__ void __launch_bounds__(GEMM_THREADS, GEMM_CTAS) grouped_gemm_f64(GemmParams p) {
  extern __shared__ __align__(128) double gsm[];
  __shared__ GemmStep step[GEMM_STAGES];
  __shared__ int s_next;
  __shared__ double s_red[GEMM_MMA / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  static_assert(BM == 64 && BN == 64 && GEMM_BK == 32, "layout of the stages");
  if (tid >= GEMM_MMA) {
    gemm_copy_stream(p, (uint32_t)__cvta_generic_to_shared(gsm), step, &s_next);
    return;
  }
  const int wr = warp >> 1, wc = warp & 1;
  int la[4], lb[4];   // gemm_mma's places within a stage
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    const int k = 4 * kk + (lane & 3);
    la[kk] = k * BM + ((wr * 8 + (lane >> 2)) ^ gemm_f(k));
    lb[kk] = BM * GEMM_BK + k * BN + ((wc * 8 + (lane >> 2)) ^ gemm_f(k));
  }
  // thread's entries of a tile: 16 mi + er, 16 ni + ec + e
  const int er = wr * 8 + (lane >> 2), ec = wc * 8 + 2 * (lane & 3);
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  for (int stage = 0;; stage = stage == GEMM_STAGES - 1 ? 0 : stage + 1) {
    bar_sync(GEMM_FULL + stage, GEMM_THREADS);
    if (step[stage].last == 2) break;
    const int nrow = step[stage].nrow, ncol = step[stage].ncol;
    // this warp's granules: rows wr, wr + 2, ..., columns wc, wc + 2, ...
    const int mym = (((nrow + 7) >> 3) + 1 - wr) >> 1, myn = (((ncol + 7) >> 3) + 1 - wc) >> 1;
#define GEMM_CASE(MM, NN) case MM * 8 + NN: gemm_tile<MM, NN>(acc, gsm, step, stage, la, lb); break
    switch (mym * 8 + myn) {
      GEMM_CASE(1, 1); GEMM_CASE(1, 2); GEMM_CASE(1, 3); GEMM_CASE(1, 4);
      GEMM_CASE(2, 1); GEMM_CASE(2, 2); GEMM_CASE(2, 3); GEMM_CASE(2, 4);
      GEMM_CASE(3, 1); GEMM_CASE(3, 2); GEMM_CASE(3, 3); GEMM_CASE(3, 4);
      GEMM_CASE(4, 1); GEMM_CASE(4, 2); GEMM_CASE(4, 3); GEMM_CASE(4, 4);
      default: gemm_tile<0, 0>(acc, gsm, step, stage, la, lb); break;   // no granule of the tile is this warp's
    }
#undef GEMM_CASE
    const GemmStep &sp = step[stage];
    const Tile tl = sp.tl;
    const int64_t c_off = sp.c.off;
    const int c_ld = sp.c.ld, tile = sp.tile;
    bar_arrive(GEMM_EMPTY + stage, GEMM_THREADS);
    for (int tj = tl.ab; tj < tl.ae; ++tj) {
      const Task ax = p.tasks[tj];
      const double *x = space_base(p, ax.L.space) + ax.L.off + (int64_t)(tl.col0 + ec) * ax.L.ld + tl.row0 + er;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double *xc = x + (int64_t)(ni * 16 + e) * ax.L.ld;
          if (ni * 16 + ec + e < ncol)
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
              if (mi * 16 + er < nrow) acc[mi][ni][e] += ax.coef * xc[mi * 16];
        }
    }
    const bool dot = p.dot_mode != 0, slot = !dot && tl.slot >= 0;
    const int64_t o0 = slot ? (int64_t)tl.slot * (BM * BN) + ec * BM + er
                            : c_off + (int64_t)(tl.col0 + ec) * c_ld + tl.row0 + er;
    const int old = slot ? BM : c_ld;
    double *o = (slot ? p.slots : p.out) + o0;   // dot mode: not written
    double local = 0.0;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (ni * 16 + ec + e < ncol) {
          const int64_t oc = (int64_t)(ni * 16 + e) * old;
#pragma unroll
          for (int mi = 0; mi < 4; ++mi)
            if (mi * 16 + er < nrow) {
              if (dot)
                local += acc[mi][ni][e] * p.dot_with[o0 + oc + mi * 16];
              else
                o[oc + mi * 16] = acc[mi][ni][e];
            }
        }
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) acc[mi][ni][e] = 0.0;
      }
    if (dot) {
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) local += __shfl_down_sync(0xffffffffu, local, s);
      if (lane == 0) s_red[warp] = local;
      bar_sync(GEMM_NEXT + 1, GEMM_MMA);
      if (tid == 0) {
        double tot = 0.0;
        for (int w = 0; w < GEMM_MMA / 32; ++w) tot += s_red[w];
        p.partials[tile] = tot;
      }
      bar_sync(GEMM_NEXT + 1, GEMM_MMA);
    }
  }
}

int grouped_gemm_grid(int ntiles, int ctas_per_sm) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int g = sms * std::min(GEMM_CTAS, std::max(1, ctas_per_sm));
  return ntiles < g ? (ntiles > 0 ? ntiles : 1) : g;
}

void launch_grouped_gemm(const GemmParams &p, int grid, cudaStream_t s) {
  if (p.ntiles <= 0) return;
  // the attribute belongs to the device's context: set at every launch
  cudaFuncSetAttribute(grouped_gemm_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM);
  grouped_gemm_f64<<<grid, GEMM_THREADS, GEMM_SMEM, s>>>(p);
}

// Four CTAs per split tile, 16 columns each, one row of four columns a thread:
// the slots are added in slot order, so the result does not depend on which
// items finished first; the slots of four columns are in flight together (one
// CTA per tile and one load at a time took 45 us of the 1.4 ms FP64 H*psi of
// the 4x24 m = 2000 superblock, 619 tiles).
__global__ void __launch_bounds__(256) reduce_slots_kernel(GemmParams p, const Reduce *red) {
  const Reduce rd = red[blockIdx.x];
  const Cell c = p.cells[rd.cell];
  const int rows = min(BM, c.M - rd.row0), cols = min(BN, c.N - rd.col0);
  const int r = threadIdx.x & (BM - 1), n0 = blockIdx.y * (BN / 4) + threadIdx.x / BM;
  constexpr int Q = BN / 16, DN = 256 / BM;   // columns of a thread, DN apart
  if (r >= rows || n0 >= cols) return;
  double v[Q];
  const double *s = p.slots + (int64_t)rd.slot0 * (BM * BN) + n0 * BM + r;
#pragma unroll
  for (int q = 0; q < Q; ++q) v[q] = 0.0;
#pragma unroll 4
  for (int k = 0; k < rd.nslot; ++k, s += BM * BN)
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (n0 + q * DN < cols) v[q] += s[q * DN * BM];
  for (int tj = rd.ab; tj < rd.ae; ++tj) {
    const Task ax = p.tasks[tj];
    const double *x = space_base(p, ax.L.space) + ax.L.off + (int64_t)(rd.col0 + n0) * ax.L.ld + rd.row0 + r;
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (n0 + q * DN < cols) v[q] += ax.coef * x[(int64_t)(q * DN) * ax.L.ld];
  }
  double *o = p.out + c.off + (int64_t)(rd.col0 + n0) * c.ld + rd.row0 + r;
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (n0 + q * DN < cols) o[(int64_t)(q * DN) * c.ld] = v[q];
}

void launch_reduce(const GemmParams &p, const Reduce *red, int nred, cudaStream_t s) {
  if (nred > 0) reduce_slots_kernel<<<dim3(nred, 4), 256, 0, s>>>(p, red);
}

// ------------------------------------------------------------------ merges
__global__ void merge_kernel(double *ops, const int64_t *dst, const int64_t *n, const int32_t *sb,
                             const int32_t *se, const int64_t *src, const double *coef) {
  const int r = blockIdx.x;
  const int64_t d = dst[r], len = n[r];
  const int b = sb[r], e = se[r];
  for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
    double acc = 0.0;
    for (int j = b; j < e; ++j) acc = acc + coef[j] * ops[src[j] + i];
    ops[d + i] = acc;
  }
}
void launch_merge(double *ops, const int64_t *dst, const int64_t *n, const int32_t *sb, const int32_t *se,
                  const int64_t *src, const double *coef, int nrec, cudaStream_t s) {
  if (nrec > 0) merge_kernel<<<nrec, 256, 0, s>>>(ops, dst, n, sb, se, src, coef);
}

// --------------------------------------------------------------- reductions
constexpr int VT = 256;   // threads of the vector kernels

__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double tot = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += sh[i];
  __syncthreads();
  return tot;   // valid in thread 0
}

int dot_blocks(int64_t n) {
  int64_t b = (n + VT * 8 - 1) / (VT * 8);
  if (b < 1) b = 1;
  if (b > 2048) b = 2048;
  return (int)b;
}

__global__ void dot_kernel(const double *__restrict__ x, const double *__restrict__ y, int64_t n,
                           double *partials) {
  __shared__ double sh[VT / 32];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += x[i] * y[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}
void launch_dot(const double *x, const double *y, int64_t n, double *partials, int nblk, cudaStream_t s) {
  dot_kernel<<<nblk, VT, 0, s>>>(x, y, n, partials);
}

__global__ void sum_kernel(const double *partials, int nblk, double *res, int sqrt_flag) {
  __shared__ double sh[VT / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < nblk; i += blockDim.x) s += partials[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) *res = sqrt_flag ? sqrt(s) : s;
}
void launch_sum(const double *partials, int nblk, double *res, int sqrt_flag, cudaStream_t s) {
  sum_kernel<<<1, VT, 0, s>>>(partials, nblk, res, sqrt_flag);
}

static int vgrid(int64_t n) {
  int64_t g = (n + VT - 1) / VT;
  if (g > 148 * 16) g = 148 * 16;
  if (g < 1) g = 1;
  return (int)g;
}
__global__ void scale_inv_kernel(double *x, const double *nrm, int64_t n) {
  const double d = *nrm;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = x[i] / d;
}
void launch_scale_inv(double *x, const double *nrm, int64_t n, cudaStream_t s) {
  scale_inv_kernel<<<vgrid(n), VT, 0, s>>>(x, nrm, n);
}

__global__ void combine_kernel(const double *__restrict__ V, int64_t ld, int k, const double *__restrict__ coef,
                               double *w, int64_t n) {
  __shared__ double c[128];
  for (int j = threadIdx.x; j < k && j < 128; j += blockDim.x) c[j] = coef[j];
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double t = 0.0;
    for (int j = 0; j < k; ++j) t = t + c[j] * V[(int64_t)j * ld + i];
    w[i] = t;
  }
}
void launch_combine(const double *V, int64_t ld, int k, const double *coef, double *w, int64_t n, cudaStream_t s) {
  combine_kernel<<<vgrid(n), VT, 0, s>>>(V, ld, k, coef, w, n);
}

// Ordered integer image of a double: monotone in the value, with +0 and -0
// both at 0, so that consecutive integers are adjacent doubles.
__device__ __forceinline__ int64_t ord_of(double x) {
  const int64_t bits = __double_as_longlong(x);
  return bits >= 0 ? bits : -(bits & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double val_of(int64_t k) {
  return k >= 0 ? __longlong_as_double(k) : __longlong_as_double((-k) | (int64_t)0x8000000000000000ULL);
}

constexpr int TRI_THREADS = 256;   // threads (multisection points) of the tridiagonal eigenvalue kernels

// Lowest eigenpair of a symmetric tridiagonal matrix (n <= 128): the lowest
// eigenvalue to full precision -- the pair of adjacent doubles where the
// Sturm count turns from 0 to 1 -- by multisection over the ordered integer
// images of the doubles (TRI_THREADS points per pass, one per thread, about
// eight bits per pass; the last pass places its points on consecutive
// doubles), then inverse iteration with a pivoted tridiagonal solve on one
// thread.  n is at most the Lanczos depth.  Runs on one block of TRI_THREADS
// threads; every thread returns the same bracket [lo, hi] of adjacent doubles.
// hint (if finite): an upper estimate of the eigenvalue, such as the lowest
// eigenvalue of the leading (n-1) x (n-1) matrix, which is never below it
// (Cauchy interlacing).  The first pass then places its points at
// geometrically growing distances below the hint (and one just above it), so
// that the bracket it leaves is a fraction of the eigenvalue's distance from
// the hint wide; the bracket at the end is the same either way.
__device__ void tridiag_min_bracket(const double *a, const double *b, int n, double hint, double &lo_out,
                                    double &hi_out) {
  // the matrix scaled to a largest row sum below one, its off-diagonal squared
  __shared__ double sa[128], sb2[128], slo[TRI_THREADS / 32], shi[TRI_THREADS / 32];
  __shared__ unsigned sv[TRI_THREADS / 32], su[TRI_THREADS / 32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  // the matrix to shared memory, and its Gershgorin bounds (a block-wide min
  // and max of a[i] -+ (|b[i-1]| + |b[i]|), exact in any order)
  double lo = INFINITY, hi = -INFINITY;
  for (int i = t; i < n; i += blockDim.x) {
    const double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + (i < n - 1 ? fabs(b[i]) : 0.0);
    lo = fmin(lo, a[i] - r);
    hi = fmax(hi, a[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    slo[w] = lo;
    shi[w] = hi;
  }
  __syncthreads();
  lo = slo[0];
  hi = shi[0];
  for (int q = 1; q < TRI_THREADS / 32; ++q) {
    lo = fmin(lo, slo[q]);
    hi = fmax(hi, shi[q]);
  }
  const double sc = tridiag_scale(fmax(fabs(lo), fabs(hi)));
  for (int i = t; i < n; i += blockDim.x) {
    const double bs = i < n - 1 ? b[i] * sc : 0.0;
    sa[i] = a[i] * sc;
    sb2[i] = bs * bs;
  }
  __syncthreads();
  // invariant: count(lo) = 0 < count(hi) (Gershgorin bounds)
  // images lie in (-2^63, 2^63), so their distance can exceed the int64
  // range: spans and offsets are taken modulo 2^64, where they are exact
  int64_t klo = ord_of(lo), khi = ord_of(hi);
  auto dist = [](int64_t kl, int64_t kh) -> uint64_t { return (uint64_t)kh - (uint64_t)kl; };
  auto point = [&](int j, int64_t kl, int64_t kh) -> int64_t {
    const uint64_t span = dist(kl, kh);
    if (span <= (uint64_t)TRI_THREADS + 1) return (int64_t)((uint64_t)kl + (uint64_t)(j + 1));
    return (int64_t)((uint64_t)kl +
                     (uint64_t)((double)span * ((double)(j + 1) / (double)(TRI_THREADS + 1))));
  };
  // first-pass points from the hint: point j = khint + 1 - (g - 1) with
  // g = below^((T-1-j)/(T-1)), below = khint + 1 - klo; non-decreasing in j,
  // the last one just above the hint
  const bool use_hint = isfinite(hint) && hint > lo && hint < hi;
  const int64_t khint = use_hint ? ord_of(hint) : 0;
  auto hint_point = [&](int j, int64_t kl) -> int64_t {
    const double below = (double)(dist(kl, khint) + 1);
    const double g = exp2((double)(TRI_THREADS - 1 - j) * log2(below) / (double)(TRI_THREADS - 1));
    const uint64_t off = g >= below ? dist(kl, khint) + 1 : (uint64_t)g;   // 1 .. below
    return (int64_t)((uint64_t)khint + 1 - (off - 1));
  };
  for (int pass = 0; pass < 64 && khi > klo && dist(klo, khi) > 1; ++pass) {
    const bool geo = use_hint && pass == 0;
    auto pt = [&](int j) { return geo ? hint_point(j, klo) : point(j, klo, khi); };
    const int64_t kx = pt(t);
    const bool valid = kx > klo && kx < khi;
    const bool up = valid && sturm1(sa, sb2, n, val_of(kx) * sc) >= 1;
    const unsigned vm = __ballot_sync(0xffffffffu, valid), um = __ballot_sync(0xffffffffu, up);
    if (lane == 0) {
      sv[w] = vm;
      su[w] = um;
    }
    __syncthreads();
    // f: the first point with a count of at least one; the new lo is the
    // highest valid point below it (all of them have a count of zero)
    int f = -1, g = -1;
    for (int q = 0; q < TRI_THREADS / 32 && f < 0; ++q)
      if (su[q]) f = q * 32 + __ffs(su[q]) - 1;
    const int lim = f < 0 ? TRI_THREADS : f;
    for (int q = (lim - 1) >> 5; q >= 0 && g < 0 && lim > 0; --q) {
      unsigned m = sv[q];
      const int top = lim - q * 32;
      if (top < 32) m &= (1u << top) - 1u;
      if (m) g = q * 32 + 31 - __clz(m);
    }
    const int64_t nlo = g >= 0 ? pt(g) : klo, nhi = f >= 0 ? pt(f) : khi;
    __syncthreads();
    if (nlo == klo && nhi == khi) break;   // no valid point: lo and hi are adjacent
    klo = nlo;
    khi = nhi;
  }
  lo_out = val_of(klo);
  hi_out = val_of(khi);
}

__device__ void tridiag_min_body(const double *a, const double *b, int n, double *lam, double *vec, int want_vec) {
  if (blockIdx.x != 0) return;
  double lo, hi;
  tridiag_min_bracket(a, b, n, __longlong_as_double(0x7FF8000000000000LL), lo, hi);
  const double l = 0.5 * (lo + hi);
  if (threadIdx.x != 0) return;
  *lam = l;
  if (!want_vec) return;
  // inverse iteration on (T - l I) with partial pivoting
  double x[128], dd[128], du[128], du2[128], dl[128];
  int piv[128];
  double scale = fabs(hi) + fabs(lo) + 1.0;
  for (int i = 0; i < n; ++i) x[i] = 1.0;
  for (int i = 0; i < n; ++i) {
    dd[i] = a[i] - l;
    du[i] = i < n - 1 ? b[i] : 0.0;
    dl[i] = i < n - 1 ? b[i] : 0.0;
    du2[i] = 0.0;
  }
  // LU with partial pivoting (dgttrf-like)
  for (int i = 0; i < n - 1; ++i) {
    if (fabs(dd[i]) >= fabs(dl[i])) {
      piv[i] = 0;
      if (dd[i] == 0.0) dd[i] = 1e-300 * scale + 1e-300;
      const double f = dl[i] / dd[i];
      dl[i] = f;
      dd[i + 1] -= f * du[i];
    } else {
      piv[i] = 1;
      const double f = dd[i] / dl[i];
      dd[i] = dl[i];
      dl[i] = f;
      const double t = du[i];
      du[i] = dd[i + 1];
      dd[i + 1] = t - f * dd[i + 1];
      if (i < n - 2) {
        du2[i] = du[i + 1];
        du[i + 1] = -f * du[i + 1];
      }
    }
  }
  if (dd[n - 1] == 0.0) dd[n - 1] = 1e-16 * scale;
  for (int iter = 0; iter < 3; ++iter) {
    // solve L U y = x
    for (int i = 0; i < n - 1; ++i) {
      if (piv[i] == 0) {
        x[i + 1] -= dl[i] * x[i];
      } else {
        const double t = x[i];
        x[i] = x[i + 1];
        x[i + 1] = t - dl[i] * x[i + 1];
      }
    }
    x[n - 1] /= dd[n - 1];
    if (n > 1) x[n - 2] = (x[n - 2] - du[n - 2] * x[n - 1]) / dd[n - 2];
    for (int i = n - 3; i >= 0; --i) x[i] = (x[i] - du[i] * x[i + 1] - du2[i] * x[i + 2]) / dd[i];
    double nr = 0.0;
    for (int i = 0; i < n; ++i) nr += x[i] * x[i];
    nr = sqrt(nr);
    for (int i = 0; i < n; ++i) x[i] /= nr;
  }
  // sign convention: first nonzero component positive
  double sgn = 1.0;
  for (int i = 0; i < n; ++i)
    if (x[i] != 0.0) { sgn = x[i] > 0 ? 1.0 : -1.0; break; }
  for (int i = 0; i < n; ++i) vec[i] = sgn * x[i];
}
__global__ void tridiag_min_kernel(const double *a, const double *b, int n, double *lam, double *vec, int want_vec) {
  tridiag_min_body(a, b, n, lam, vec, want_vec);
}
void launch_tridiag_min(const double *a, const double *b, int n, double *lam, double *vec, int want_vec,
                        cudaStream_t s) {
  tridiag_min_kernel<<<1, TRI_THREADS, 0, s>>>(a, b, n, lam, vec, want_vec);
}

// ---- one Lanczos iteration with its step read from device memory (*it), so
// that the same launches -- captured once as a CUDA graph -- serve every
// iteration.  S holds alpha (0..127), beta (128..255), uu (256..383), the
// Gram-Schmidt coefficients (384..511), the Ritz value (512) and a norm (513).
// Each norm or dot product is folded into the kernel that produces its
// vector (one pass over the vector instead of two, one launch instead of
// three): every block reduces its share of the squares or products, and the
// last block to finish adds the block partials in a fixed order, so the
// result does not depend on the order the blocks run in.
__device__ __forceinline__ double *lz_ptr(const LzRef &r) {
  return r.V + (int64_t)(*r.it + r.off - 1) * r.ld;
}

// The block partial s (valid in thread 0) to partials[blockIdx.x]; the last
// block to arrive (counted on *cnt, which it resets for the next kernel) adds
// the partials, thread i taking i, i + blockDim.x, ..., then the block tree,
// and stores the total (or its square root) at *res.
__device__ void lz_grid_sum(double s, double *partials, int *cnt, double *res, int sqrt_flag, double *sh) {
  __shared__ int last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(cnt, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) t += __ldcg(partials + i);
  t = block_sum(t, sh);
  if (threadIdx.x == 0) {
    *res = sqrt_flag ? sqrt(t) : t;
    *cnt = 0;
  }
}

// A long vector is cut into lz_slices equal slices of lz_slice(n) entries (the
// last may be short), one per block and two blocks per SM, so that every SM
// reads the same share of the vectors; at most LZ_SLICE entries, 64 KB.
constexpr int LZ_SLICE = 8192, LZ_THREADS = 512, LZ_PARTS = 4;
constexpr int LZ_KMAX = 128;
int lz_slices(int64_t n) {
  const int64_t w = 148 * 2;
  return (int)(w * std::max<int64_t>(1, (n + w * LZ_SLICE - 1) / (w * LZ_SLICE)));
}
static int lz_slice(int64_t n) {
  const int s = lz_slices(n);
  return (int)((n + s - 1) / s + 1) / 2 * 2;
}

// w = src - alpha(L) vec(L) - beta(L-1) vec(L-1), its square sum and its
// projections on vec(1..L): each block keeps its slice of w in shared memory
// and its warps take the L vectors' slices in quarters, so that no barrier
// stands between the reads (the kernel is bound by those: L vectors of n
// doubles).  1.4M entries, 23 vectors on average: 12 us for w and 54 for the
// projections when each was a kernel, the latter with a block-wide sum per
// vector; 54 for both now, 39 for the vectors alone at the copy bandwidth.
// Vectors have an even stride; what lies past n is masked.
__global__ void __launch_bounds__(LZ_THREADS, 2)
    lz_update_dots_kernel(const double *__restrict__ V, int64_t ld, const int *it, LzRef wr_,
                          const double *__restrict__ src, int64_t n, int per, const double *S, double *partials,
                          int kmax) {
  extern __shared__ double2 lz_w[];
  __shared__ double hp[LZ_KMAX][LZ_PARTS], sh[LZ_THREADS / 32];
  const int L = *it, tid = threadIdx.x, lane = tid & 31;
  const int k = min(L, kmax);
  const double av = S[L], bv = L >= 2 ? S[128 + L - 1] : 0.0;
  const int64_t r0 = min(n, (int64_t)blockIdx.x * per);
  const int nr = (int)min((int64_t)per, n - r0), np = (nr + 1) / 2;
  double2 *__restrict__ w = reinterpret_cast<double2 *>(lz_ptr(wr_) + r0);
  const double2 *__restrict__ y = reinterpret_cast<const double2 *>(src + r0);
  const double2 *__restrict__ p1 = reinterpret_cast<const double2 *>(V + (int64_t)(L - 1) * ld + r0);
  const double2 *__restrict__ p2 = L >= 2 ? p1 - ld / 2 : nullptr;
  double q = 0.0;
#pragma unroll 2
  for (int i = tid; i < np; i += LZ_THREADS) {
    const double2 a = y[i], b = p1[i];
    double2 x = make_double2(a.x - av * b.x, a.y - av * b.y);
    if (p2) {
      const double2 c = p2[i];
      x.x = x.x - bv * c.x;
      x.y = x.y - bv * c.y;
    }
    if (2 * i + 1 >= nr) x.y = 0.0;
    w[i] = x;
    lz_w[i] = x;
    q += x.x * x.x;
    q += x.y * x.y;
  }
  q = block_sum(q, sh);
  if (tid == 0) partials[(int64_t)blockIdx.x * (kmax + 1) + kmax] = q;
  const int pp = (np + LZ_PARTS - 1) / LZ_PARTS;
  for (int u = tid >> 5; u < k * LZ_PARTS; u += LZ_THREADS / 32) {
    const int j = u / LZ_PARTS, i0 = u % LZ_PARTS * pp, i1 = min(np, i0 + pp);
    const double2 *__restrict__ v = reinterpret_cast<const double2 *>(V + (int64_t)j * ld + r0);
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 8
    for (int i = i0 + lane; i < i1; i += 32) {
      const double2 x = v[i], y = lz_w[i];
      s0 += x.x * y.x;
      s1 += (2 * i + 1 < nr ? x.y : 0.0) * y.y;
    }
    s0 += s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s0 += __shfl_down_sync(0xffffffffu, s0, o);
    if (lane == 0) hp[j][u % LZ_PARTS] = s0;
  }
  __syncthreads();
  for (int j = tid; j < k; j += LZ_THREADS) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < LZ_PARTS; ++q) s += hp[j][q];
    partials[(int64_t)blockIdx.x * (kmax + 1) + j] = s;
  }
}

// beta(L) = |w| and coef(j) = (w . vec(j)) / beta(L) / uu(j), one block per vector
__global__ void lz_coef_kernel(const double *partials, int nblk, int kmax, const double *uu, double *coef, double *S,
                               const int *it) {
  __shared__ double sh[VT / 32];
  const int j = blockIdx.x, L = *it;
  if (j >= L) return;
  double s = 0.0, q = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    s += partials[(int64_t)b * (kmax + 1) + j];
    q += partials[(int64_t)b * (kmax + 1) + kmax];
  }
  s = block_sum(s, sh);
  q = block_sum(q, sh);
  if (threadIdx.x != 0) return;
  const double beta = sqrt(q);
  coef[j] = s / beta / uu[j];
  if (j == 0) S[128 + L] = beta;
}

// w = w / beta(L) - sum_j coef(j) vec(j); S[513] = |w|.  Bound by the reads of
// the vectors again (1.4M entries, 23 vectors: 54 us with one load in flight a
// thread, 50 with eight of 16 bytes).
__global__ void __launch_bounds__(LZ_THREADS, 2)
    lz_combine_norm_kernel(const double *__restrict__ V, int64_t ld, const int *it, const double *__restrict__ coef,
                           LzRef wr_, int64_t n, int per, double *S, double *partials, int *cnt) {
  __shared__ double c[LZ_KMAX];
  __shared__ double sh[32];
  const int k = min(*it, LZ_KMAX);
  for (int j = threadIdx.x; j < k; j += blockDim.x) c[j] = coef[j];
  __syncthreads();
  const int64_t r0 = min(n, (int64_t)blockIdx.x * per);
  const int nr = (int)min((int64_t)per, n - r0), np = (nr + 1) / 2;
  double2 *__restrict__ w = reinterpret_cast<double2 *>(lz_ptr(wr_) + r0);
  const double2 *__restrict__ v0 = reinterpret_cast<const double2 *>(V + r0);
  const int64_t ld2 = ld / 2;
  const double beta = S[128 + *it];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += LZ_THREADS) {
    double2 t = make_double2(0.0, 0.0), y = w[i];
    const double2 *x = v0 + i;
    int j = 0;
    for (; j + 8 <= k; j += 8, x += 8 * ld2) {   // eight loads in flight
      double2 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = x[u * ld2];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        t.x = t.x + c[j + u] * v[u].x;
        t.y = t.y + c[j + u] * v[u].y;
      }
    }
#pragma unroll 4
    for (; j < k; ++j, x += ld2) {
      const double2 v = *x;
      t.x = t.x + c[j] * v.x;
      t.y = t.y + c[j] * v.y;
    }
    y.x = y.x / beta - t.x;
    y.y = 2 * i + 1 < nr ? y.y / beta - t.y : 0.0;
    w[i] = y;
    s += y.x * y.x;
    s += y.y * y.y;
  }
  s = block_sum(s, sh);
  lz_grid_sum(s, partials, cnt, S + 513, 1, sh);
}

// w /= S[513], copied to x; uu(L+1) = w . w
__global__ void lz_scale_norm_kernel(LzRef wr_, double *__restrict__ x, int64_t n, double *S, const int *it,
                                     double *partials, int *cnt) {
  __shared__ double sh[VT / 32];
  const int L = *it;
  const double d = S[513];
  double *__restrict__ w = lz_ptr(wr_);
  double s = 0.0;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = w[i] / d;
    w[i] = v;
    x[i] = v;
    s += v * v;
  }
  s = block_sum(s, sh);
  lz_grid_sum(s, partials, cnt, S + 257 + L, 0, sh);
}

// alpha(L+1) = vec(L+1) . y
__global__ void lz_dot_kernel(LzRef xr, const double *__restrict__ y, int64_t n, double *S, const int *it,
                              double *partials, int *cnt) {
  __shared__ double sh[VT / 32];
  const int L = *it;
  const double *__restrict__ x = lz_ptr(xr);
  double s = 0.0;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += x[i] * y[i];
  s = block_sum(s, sh);
  lz_grid_sum(s, partials, cnt, S + 1 + L, 0, sh);
}

// The Ritz value of T(L+1); beta(L), the Ritz value and the split-precision
// kernels' error word to step L's place of the ring in page-locked host memory.
// By one block.
__device__ void lz_publish(double *S, int L, double flags, double *host) {
  double lo, hi;
  // from the second step on, S[512] holds the Ritz value of the step before
  tridiag_min_bracket(S + 1, S + 129, L + 1, L >= 2 ? S[512] : __longlong_as_double(0x7FF8000000000000LL), lo, hi);
  if (threadIdx.x != 0) return;
  S[512] = 0.5 * (lo + hi);
  host += LZ_HOST * (L % LZ_RING);
  host[0] = S[128 + L];
  host[1] = S[512];
  host[2] = flags;
  __threadfence_system();
}
__global__ void lz_tridiag_publish_kernel(double *S, int *it, const int *err, double *host) {
  const int L = *it;
  lz_publish(S, L, err ? (double)*err : 0.0, host);
  if (threadIdx.x == 0) *it = L + 1;
}
// the same of a given step, beside the next one's kernels
__global__ void lz_publish_short_kernel(double *S, int L, double *host) {
  lz_publish(S, L, S[LZ_FLAGS + L % LZ_RING], host);
}

// ---- the same steps for a short vector, by one thread-block cluster: the
// kernels above need a launch or two for each sum over the vector, and at the
// sizes of a ladder each of them is all latency (2x16 ladder m = 256, 23,140
// entries, 25 vectors on average: 42 us for recurrence, projections,
// combination and scaling as five kernels, 21 now; alpha 5).  CTA c of CL holds
// entries [c per, (c + 1) per) of the new vector in shared memory; sums meet
// through distributed shared memory and are added in rank order by everyone.
constexpr int LZC_THREADS = 512;
constexpr int LZC_MAX = 4096;   // entries of a CTA

// The sum over the cluster of x, one value per thread, in every thread; slot
// is used by no other sum of the kernel, red holds LZC_THREADS / 32 doubles.
template <int CL>
__device__ __forceinline__ double lz_cluster_sum(cg::cluster_group &cl, double x, double *slot, double *red) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if (lane == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
  if (threadIdx.x == 0) *slot = s;
  cl.sync();
  double p = lane < CL ? *cl.map_shared_rank(slot, lane < CL ? lane : 0) : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
  return p;
}

// vec(L+1) from H vec(L) in src: recurrence, beta(L), Gram-Schmidt against
// vec(1..L), normalisation; also to x, with uu(L+1).
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(LZC_THREADS, 1)
    lz_step_cluster_kernel(double *V, int64_t ld, const int *it, const double *__restrict__ src, double *__restrict__ x,
                           int64_t n, double *S) {
  __shared__ double w[LZC_MAX], hp[LZ_KMAX], cf[LZ_KMAX], slot[4], red[LZC_THREADS / 32];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int L = *it, k = min(L, LZ_KMAX);
  const int per = (int)((n + CL - 1) / CL);
  const int64_t r0 = min(n, (int64_t)rank * per);
  const int nr = (int)(min(n, r0 + per) - r0);
  const double av = S[L], bv = L >= 2 ? S[128 + L - 1] : 0.0;
  const double *p1 = V + (int64_t)(L - 1) * ld + r0, *p2 = L >= 2 ? p1 - ld : nullptr;
  double *out = V + (int64_t)L * ld + r0;
  double s = 0.0;
  for (int i = tid; i < nr; i += LZC_THREADS) {
    double v = src[r0 + i] - av * p1[i];
    if (p2) v = v - bv * p2[i];
    w[i] = v;
    s += v * v;
  }
  const double beta = sqrt(lz_cluster_sum<CL>(cl, s, slot, red));
  for (int i = tid; i < nr; i += LZC_THREADS) w[i] = w[i] / beta;
  __syncthreads();
  // the CTA's parts of the projections, a warp per vector
  for (int j = warp; j < k; j += LZC_THREADS / 32) {
    const double *v = V + (int64_t)j * ld + r0;
    double a = 0.0;
#pragma unroll 4
    for (int i = lane; i < nr; i += 32) a += v[i] * w[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) hp[j] = a;
  }
  cl.sync();
  if (tid < k) {
    double a = 0.0;
#pragma unroll
    for (int c = 0; c < CL; ++c) a += cl.map_shared_rank(hp, c)[tid];
    cf[tid] = a / S[257 + tid];
  }
  __syncthreads();
  s = 0.0;
  for (int i = tid; i < nr; i += LZC_THREADS) {
    double t = 0.0;
    const double *v = V + r0 + i;
#pragma unroll 4
    for (int j = 0; j < k; ++j) t = t + cf[j] * v[(int64_t)j * ld];
    const double y = w[i] - t;
    w[i] = y;
    s += y * y;
  }
  const double nrm = sqrt(lz_cluster_sum<CL>(cl, s, slot + 1, red));
  s = 0.0;
  for (int i = tid; i < nr; i += LZC_THREADS) {
    const double y = w[i] / nrm;
    out[i] = y;
    x[r0 + i] = y;
    s += y * y;
  }
  const double uu = lz_cluster_sum<CL>(cl, s, slot + 2, red);
  if (rank == 0 && tid == 0) {
    S[128 + L] = beta;
    S[513] = nrm;
    S[257 + L] = uu;
  }
  cl.sync();   // no CTA leaves while another may still read its shared memory
}

// alpha(L+1) = x . y; the error word to S; the step advances
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(LZC_THREADS, 1)
    lz_dot_cluster_kernel(const double *__restrict__ x, const double *__restrict__ y, int64_t n, double *S, int *it,
                          const int *err) {
  __shared__ double slot, red[LZC_THREADS / 32];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  double s = 0.0;
#pragma unroll 4
  for (int i = rank * LZC_THREADS + (int)threadIdx.x; i < n; i += CL * LZC_THREADS) s += x[i] * y[i];
  s = lz_cluster_sum<CL>(cl, s, &slot, red);
  if (rank == 0 && threadIdx.x == 0) {
    const int L = *it;
    S[1 + L] = s;
    S[LZ_FLAGS + L % LZ_RING] = err ? (double)*err : 0.0;
    *it = L + 1;
  }
  cl.sync();
}

// 16 CTAs where the device can place such a cluster (a non-portable size),
// else 8; asked once
static int lz_cluster_size() {
  static std::once_flag once;
  static int size = 8;
  std::call_once(once, [] {
    bool ok = true;
    auto fits = [&](auto kernel, int threads) {
      ok = ok && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(16, 1, 1);
      cfg.blockDim = dim3(threads, 1, 1);
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 16;
      attr.val.clusterDim.y = 1;
      attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int m = 0;
      ok = ok && cudaOccupancyMaxActiveClusters(&m, kernel, &cfg) == cudaSuccess && m >= 1;
    };
    fits(lz_step_cluster_kernel<16>, LZC_THREADS);
    fits(lz_dot_cluster_kernel<16>, LZC_THREADS);
    if (ok) size = 16;
    cudaGetLastError();
  });
  return size;
}
// Whether the cluster kernels take a vector of n entries.  A cluster reads the
// earlier vectors through its own 16 SMs only, so the grid-wide kernels win
// where those reads outweigh the launches (an iteration, cluster against
// grid: 5,628 entries 43 and 68 us, 23,140 57 and 77, 31,915 63 and 78, 45,315
// 72 and 81, 61,756 96 and 86).
bool lz_short(int64_t n) { return n <= 49152 && n <= (int64_t)lz_cluster_size() * LZC_MAX; }
void launch_lz_step_short(double *V, int64_t ld, const int *it, const double *src, double *x, int64_t n, double *S,
                          cudaStream_t s) {
  if (lz_cluster_size() == 16) {
    cudaFuncSetAttribute(lz_step_cluster_kernel<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    lz_step_cluster_kernel<16><<<16, LZC_THREADS, 0, s>>>(V, ld, it, src, x, n, S);
  } else {
    lz_step_cluster_kernel<8><<<8, LZC_THREADS, 0, s>>>(V, ld, it, src, x, n, S);
  }
}
void launch_lz_dot_short(const double *x, const double *y, int64_t n, double *S, int *it, const int *err,
                         cudaStream_t s) {
  if (lz_cluster_size() == 16) {
    cudaFuncSetAttribute(lz_dot_cluster_kernel<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    lz_dot_cluster_kernel<16><<<16, LZC_THREADS, 0, s>>>(x, y, n, S, it, err);
  } else {
    lz_dot_cluster_kernel<8><<<8, LZC_THREADS, 0, s>>>(x, y, n, S, it, err);
  }
}
void launch_lz_publish_short(double *S, int L, double *host, cudaStream_t s) {
  lz_publish_short_kernel<<<1, TRI_THREADS, 0, s>>>(S, L, host);
}

// partial sums a kernel may leave: the scaling and the dot product run on the
// grid of a dot product (fewer partials for the last block to add), the
// Gram-Schmidt kernels, which stream L vectors per element, on the slices
int lz_blocks(int64_t n) { return std::max(lz_slices(n), dot_blocks(n)); }
void launch_lz_update_gram_schmidt(const double *V, int64_t ld, const int *it, LzRef w, const double *src, int64_t n,
                                   double *S, double *mpartials, int kmax, const double *uu, double *coef,
                                   double *partials, int *cnt, cudaStream_t s) {
  const int ns = lz_slices(n), per = lz_slice(n);
  const int bytes = per * (int)sizeof(double);
  cudaFuncSetAttribute(lz_update_dots_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       LZ_SLICE * (int)sizeof(double));
  lz_update_dots_kernel<<<ns, LZ_THREADS, bytes, s>>>(V, ld, it, w, src, n, per, S, mpartials, kmax);
  lz_coef_kernel<<<kmax, VT, 0, s>>>(mpartials, ns, kmax, uu, coef, S, it);
  lz_combine_norm_kernel<<<ns, LZ_THREADS, 0, s>>>(V, ld, it, coef, w, n, per, S, partials, cnt);
}
void launch_lz_scale_norm(LzRef w, double *x, int64_t n, double *S, const int *it, double *partials, int *cnt,
                          cudaStream_t s) {
  lz_scale_norm_kernel<<<dot_blocks(n), VT, 0, s>>>(w, x, n, S, it, partials, cnt);
}
void launch_lz_dot(LzRef x, const double *y, int64_t n, double *S, const int *it, double *partials, int *cnt,
                   cudaStream_t s) {
  lz_dot_kernel<<<dot_blocks(n), VT, 0, s>>>(x, y, n, S, it, partials, cnt);
}
void launch_lz_tridiag_publish(double *S, int *it, const int *err, double *host, cudaStream_t s) {
  lz_tridiag_publish_kernel<<<1, TRI_THREADS, 0, s>>>(S, it, err, host);
}

}  // namespace tjb
