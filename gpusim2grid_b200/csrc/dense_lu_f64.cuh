// Dense FP64 LU (no pivoting) of one matrix by one CTA of 256 threads (or by
// the CTAs of a cluster), for the tail of the FP64 batched Newton–Raphson
// factorization: the FP64 arm, the FP64 re-solve of unconverged rows and
// the adjoint.  Device code only.  Crout order on 32-wide panels: step k0
// brings in everything the panel's columns and rows still owe,
//   1. C -= A B on the FP64 tensor pipe (mma.sync m8n8k4) for the panel's
//      column block (rows k0.., K = k0) and its row block (columns right of
//      it, K = k0), in 128 x 32 and 32 x 128 tiles: every element of the
//      matrix is read and written once for all updates before it (the
//      accumulators start from C and run over K in order), and the K loop is
//      long, fed by a 3-stage cp.async ring of 16-deep slabs;
//   2. the kb x kb diagonal block is copied to shared memory (identity
//      padded to 32 x 32) and factored there, a row over 8 lanes;
//   3. L21 = A21 U11^-1, one thread per row, and U12 = L11^-1 A12, one thread
//      per column, the row or column in registers, substitution against rows
//      read as broadcast double2.
// Why this shape: with two rows' matrices per SM in flight (2.1 MB each at
// n = 518) nothing stays in L2, so a right-looking update, which rewrites the
// trailing matrix for every panel, moves 24 MB per factorization through
// HBM; here 16 MB, almost all of it operand reads ahead of use.  mma.sync
// runs FP64 at the FMA pipe's rate (36.6 of 37 TFLOP/s measured, one
// accumulator chain per warp already at 31) with a fifth of the shared-memory
// reads of a 4 x 4 DFMA block, which bounded the update before.
// A is row-major in global memory with leading dimension ld, a multiple of
// 2 (rows 16-byte aligned); panels start at multiples of 32.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gs2g {
namespace dense64 {

constexpr int BS = 256;
constexpr int KP = 32;          // panel width
constexpr int SD = KP + 2;      // diagonal block stride (16-byte rows)
constexpr int KS = 16;          // slab depth of the update's operand ring
constexpr int NSTAGE = 3;
// operand strides = 4 mod 16 doubles: the fragment loads of a half-warp (4
// rows x 4 k) fall into 16 different banks
constexpr int SAK = KS + 4;
template <int TN>
__host__ __device__ constexpr int sbn() {
  return TN + 4;
}
template <int TM, int TN>
__host__ __device__ constexpr int stage_elems() {
  return TM * SAK + KS * sbn<TN>();
}

struct Smem {
  static constexpr int d_elems = KP * SD;
  static constexpr int r_elems = KP;  // reciprocal pivots
  static constexpr int stage = stage_elems<128, 32>() > stage_elems<32, 128>() ? stage_elems<128, 32>()
                                                                              : stage_elems<32, 128>();
  // outside the update the ring holds L11^T and a 32-row block per warp
  static constexpr int ring = NSTAGE * stage > 9 * d_elems ? NSTAGE * stage : 9 * d_elems;
  static constexpr int elems = d_elems + r_elems + ring;
  static constexpr int bytes = elems * 8;
};
__device__ __forceinline__ double clamp_piv(double piv, double floor_) {
  if (fabs(piv) < floor_) return piv < 0.0 ? -floor_ : floor_;
  return piv;
}

// Shared-memory loads issued in program order (asm volatile): the
// substitutions below hold 32 values per thread in registers, and letting
// the compiler hoist their broadcast loads ahead of the arithmetic would
// spill them.
__device__ __forceinline__ double2 lds2(const double* p) {
  double2 v;
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ double lds1(const double* p) {
  double v;
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(a));
  return v;
}

// This thread's share of a tile's operand slabs: PA 16-byte chunks of A (rows
// i0 + ra + i * RA) and PB of B (k rows kb + i * RB, columns j0 + n..), the
// same places in every slab, so the addresses only advance.  Rows past M and
// columns past N are zero-filled.
template <int TM, int TN>
struct Stager {
  static constexpr int PA = TM * KS / 2 / BS, RA = TM / PA, PB = TN * KS / 2 / BS, RB = KS / PB;
  static_assert(PA * RA == TM && PB * RB == KS && RA * (KS / 2) == BS && RB * (TN / 2) == BS, "whole chunks");
  const double* a;
  const double* b;
  int64_t lda, ldb, step_b;
  unsigned sa, sb;  // shared-memory byte offsets within a stage
  int arows, bbytes;
  __device__ __forceinline__ Stager(const double* A, const double* B, int ld, int M, int N, int i0, int j0) {
    const int tid = threadIdx.x;
    const int ra = tid / (KS / 2), ka = (tid % (KS / 2)) * 2;
    const int kb = tid / (TN / 2), n = (tid % (TN / 2)) * 2;
    arows = M - i0 - ra;  // chunk i is in range for i * RA < arows
    bbytes = (N - j0 - n) * 8;
    bbytes = bbytes < 0 ? 0 : (bbytes > 16 ? 16 : bbytes);
    a = A + (int64_t)(i0 + ra) * ld + ka;
    b = B + (int64_t)kb * ld + j0 + n;
    lda = (int64_t)RA * ld;
    ldb = (int64_t)RB * ld;
    step_b = (int64_t)KS * ld;
    sa = (unsigned)(ra * SAK + ka) * 8;
    sb = (unsigned)(TM * SAK + kb * sbn<TN>() + n) * 8;
  }
  // the next slab into the stage at shared-memory byte address st
  __device__ __forceinline__ void next(unsigned st) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int bytes = i * RA < arows ? 16 : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(st + sa + i * RA * SAK * 8),
                   "l"(bytes ? a + i * lda : a), "r"(bytes));
    }
#pragma unroll
    for (int i = 0; i < PB; ++i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(st + sb + i * RB * sbn<TN>() * 8),
                   "l"(b + i * ldb), "r"(bbytes));
    a += KS;
    b += step_b;
  }
};

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// C[i0.., j0..] -= A[i0.., 0..K) B[0..K, j0..) for one TM x TN tile of an
// M x N block (A, B, C parts of one matrix, leading dimension ld; K a
// positive multiple of KS).  8 warps as WM x WN, each a grid of 8 x 8 mma
// tiles.  An element's sum runs over K in order from C, whatever the tile
// shape, so every tiling gives the same bits.  Ends without a barrier; the
// ring may be refilled only after one.
template <int TM, int TN, int WM, int WN>
__device__ __noinline__ void update_tile(double* C, const double* A, const double* B, int ld, int M, int N, int K,
                                         int i0, int j0, double* ring) {
  constexpr int MT = TM / (8 * WM), NT = TN / (8 * WN);
  constexpr int SE = stage_elems<TM, TN>();
  static_assert(WM * WN * 32 == BS && MT > 0 && NT > 0, "8 warps tile TM x TN");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int wr = (warp / WN) * 8 * MT, wc = (warp % WN) * 8 * NT;
  const int nslab = K / KS;
  const unsigned sring = (unsigned)__cvta_generic_to_shared(ring);
  Stager<TM, TN> stager(A, B, ld, M, N, i0, j0);
#pragma unroll
  for (int s = 0; s < NSTAGE - 1; ++s) {
    if (s < nslab) stager.next(sring + s * SE * 8);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int cur = 0, fill = NSTAGE - 1;  // ring positions of slab t and of slab t + NSTAGE - 1
  double acc[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int r = i0 + wr + 8 * i + g;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int c = j0 + wc + 8 * j + 2 * q;
      double2 v = make_double2(0.0, 0.0);
      const double* src = C + (int64_t)r * ld + c;
      if (r < M && c + 1 < N) v = *reinterpret_cast<const double2*>(src);
      else if (r < M && c < N) v.x = *src;
      acc[i][j][0] = v.x;
      acc[i][j][1] = v.y;
    }
  }
  // a warp whose part lies past M or N only stages: the pipe is the others'
  // (296 CTAs with this and the 64 tiles of the remainders: n = 200 224 -> 190 us,
  // 518 1806 -> 1643, 1148 12768 -> 12358); in a cluster's 32 x 32 tiles the test
  // cost 5-15 %
  const bool idle = i0 + wr >= M || j0 + wc >= N;
  for (int t = 0; t < nslab; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NSTAGE - 2) : "memory");
    __syncthreads();  // slab t has landed; every warp is done with slab t - 1
    if (t + NSTAGE - 1 < nslab) stager.next(sring + fill * SE * 8);
    asm volatile("cp.async.commit_group;\n" ::);
    const double* sA = ring + cur * SE + (wr + g) * SAK + q;
    const double* sB = ring + cur * SE + TM * SAK + q * sbn<TN>() + wc + g;
    cur = cur + 1 < NSTAGE ? cur + 1 : 0;
    fill = fill + 1 < NSTAGE ? fill + 1 : 0;
    if (TM * TN > 32 * 32 && idle) continue;
#pragma unroll
    for (int k = 0; k < KS; k += 4) {
      double a[MT], b[NT];
#pragma unroll
      for (int i = 0; i < MT; ++i) a[i] = -sA[8 * i * SAK + k];
#pragma unroll
      for (int j = 0; j < NT; ++j) b[j] = sB[k * sbn<TN>() + 8 * j];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) mma884(acc[i][j], a[i], b[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int r = i0 + wr + 8 * i + g;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int c = j0 + wc + 8 * j + 2 * q;
      double* dst = C + (int64_t)r * ld + c;
      if (c + 1 < N) *reinterpret_cast<double2*>(dst) = make_double2(acc[i][j][0], acc[i][j][1]);
      else if (c < N) *dst = acc[i][j][0];
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Factor the identity-padded 32 x 32 block D (stride SD) in place, its first kb
// steps; rp gets the reciprocal pivots.  All 8 warps: thread (r, q) holds
// columns 4 q .. 4 q + 3 of row r in registers (a row is 8 lanes of one warp).
// Step j: row j's lanes clamp the pivot and publish the row and the pivot's
// reciprocal (two buffers, one barrier per step); the rows below take l = x_j
// rp (x_j from its lane by shuffle) and x_c -= l u_jc for c > j.  A step's
// chain is the division (85 cycles), a store, a barrier and a load: 0.19 k
// cycles against 0.36 k for one warp with a row per lane, whose 32 - j loads and
// products per lane were on it too.
__device__ __noinline__ void factor_diag(double* D, double* rp, double pfloor, int kb) {
  __shared__ __align__(16) double prow[2][KP];
  const int r = threadIdx.x >> 3, q = threadIdx.x & 7, lane = threadIdx.x & 31;
  double x[4];
  {
    const double2 v0 = *reinterpret_cast<const double2*>(D + r * SD + 4 * q);
    const double2 v1 = *reinterpret_cast<const double2*>(D + r * SD + 4 * q + 2);
    x[0] = v0.x;
    x[1] = v0.y;
    x[2] = v1.x;
    x[3] = v1.y;
  }
#pragma unroll
  for (int j = 0; j < KP; ++j) {
    if (j >= kb) break;  // the padding needs no step
    if (r == j) {
      if (q == j >> 2) {
        x[j & 3] = clamp_piv(x[j & 3], pfloor);
        rp[j] = 1.0 / x[j & 3];
      }
      *reinterpret_cast<double2*>(&prow[j & 1][4 * q]) = make_double2(x[0], x[1]);
      *reinterpret_cast<double2*>(&prow[j & 1][4 * q + 2]) = make_double2(x[2], x[3]);
    }
    __syncthreads();
    const double xj = __shfl_sync(0xffffffffu, x[j & 3], (lane & 24) | (j >> 2));
    if (r > j && q >= j >> 2) {
      const double l = xj * rp[j];
      const double2 u0 = *reinterpret_cast<const double2*>(&prow[j & 1][4 * q]);
      const double2 u1 = *reinterpret_cast<const double2*>(&prow[j & 1][4 * q + 2]);
      const double u[4] = {u0.x, u0.y, u1.x, u1.y};
      if (q > j >> 2) {
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = fma(-l, u[c], x[c]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (c > (j & 3)) x[c] = fma(-l, u[c], x[c]);
        x[j & 3] = l;
      }
    }
  }
  *reinterpret_cast<double2*>(D + r * SD + 4 * q) = make_double2(x[0], x[1]);
  *reinterpret_cast<double2*>(D + r * SD + 4 * q + 2) = make_double2(x[2], x[3]);
  __syncthreads();
}

// x <- x M^-1 for the 32 values x of one thread, M upper triangular given by
// its rows (stride SD) in shared memory: after x_p is final, x_q -= x_p M_pq
// for q > p.  SCALE: x_p is multiplied by rp[p] (1 / M_pp) first; else M has
// a unit diagonal.
template <bool SCALE>
__device__ __forceinline__ void subst32(double (&x)[KP], const double* M, const double* rp) {
#pragma unroll
  for (int p = 0; p < KP; ++p) {
    if (SCALE) x[p] *= lds1(rp + p);
    const double xp = x[p];
    const double* mp = M + p * SD;
    if ((p + 1) & 1)
      if (p + 1 < KP) x[p + 1] = fma(-xp, lds1(mp + p + 1), x[p + 1]);
#pragma unroll
    for (int q2 = ((p + 1) + 1) & ~1; q2 < KP; q2 += 2) {
      const double2 u = lds2(mp + q2);
      x[q2] = fma(-xp, u.x, x[q2]);
      x[q2 + 1] = fma(-xp, u.y, x[q2 + 1]);
    }
  }
}

// L21 = A21 U11^-1 (x U11 = a per row) for 32 rows (n of them valid) by one
// warp, a row per lane in registers.  The rows pass through the warp's block
// of shared memory (stride SD: conflict-free) so that global memory is read
// and written two whole rows at a time; with every lane on its own row a load
// touched 32 lines, and the substitution took 21 k cycles a panel instead of
// 9 k at n = 518.
__device__ __forceinline__ void trsm_rows32(double* A21, int ld, int n, const double* D, const double* rp,
                                            double* buf) {
  const int lane = threadIdx.x & 31, r2 = lane >> 4, c2 = (lane & 15) * 2;
#pragma unroll
  for (int h = 0; h < KP; h += 2)
    if (h + r2 < n)
      *reinterpret_cast<double2*>(buf + (h + r2) * SD + c2) =
          *reinterpret_cast<const double2*>(A21 + (int64_t)(h + r2) * ld + c2);
  __syncwarp();
  if (lane < n) {
    double x[KP];
#pragma unroll
    for (int q = 0; q < KP / 2; ++q) {
      const double2 v = lds2(buf + lane * SD + 2 * q);
      x[2 * q] = v.x;
      x[2 * q + 1] = v.y;
    }
    subst32<true>(x, D, rp);
#pragma unroll
    for (int q = 0; q < KP / 2; ++q)
      *reinterpret_cast<double2*>(buf + lane * SD + 2 * q) = make_double2(x[2 * q], x[2 * q + 1]);
  }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < KP; h += 2)
    if (h + r2 < n)
      *reinterpret_cast<double2*>(A21 + (int64_t)(h + r2) * ld + c2) =
          *reinterpret_cast<const double2*>(buf + (h + r2) * SD + c2);
  __syncwarp();
}

// U12 = L11^-1 A12 (per column: y^T L11^T = a^T, L11^T upper with unit
// diagonal, given by its rows LT), one column of A12 in registers.
__device__ __forceinline__ void trsm_col(double* colp, int ld, const double* LT) {
  double y[KP];
  const double* src = colp;
#pragma unroll
  for (int r = 0; r < KP; ++r, src += ld) {
    y[r] = *src;
    if ((r & 15) == 15) asm volatile("" ::: "memory");  // at most 16 loads in flight
  }
  subst32<false>(y, LT, nullptr);
  // the stores walk the column again from an opaque copy of ld, so the 32
  // load addresses are not kept alive across the substitution
  int ld2;
  asm volatile("mov.b32 %0, %1;\n" : "=r"(ld2) : "r"(ld));
  double* dst = colp;
#pragma unroll
  for (int r = 0; r < KP; ++r, dst += ld2) *dst = y[r];
}

// Both substitutions of a panel with m rows below and m columns to the right
// of its diagonal block, in groups of 32 rows or 32 columns taken by the
// warps of the `parts` CTAs (this one: part).  LT: L11^T, followed by a block
// per warp.
__device__ __noinline__ void trsm_panel(double* A21, double* A12, int ld, int m, const double* D, const double* rp,
                                        double* LT, int part, int parts) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ng = (m + 31) / 32;
  for (int t = part * (BS / 32) + warp; t < 2 * ng; t += parts * (BS / 32)) {
    if (t < ng) {
      trsm_rows32(A21 + (int64_t)t * 32 * ld, ld, min(32, m - 32 * t), D, rp, LT + Smem::d_elems * (1 + warp));
    } else {
      const int c = (t - ng) * 32 + lane;
      if (c < m) trsm_col(A12 + c, ld, LT);
    }
  }
}

// Load the kb x kb diagonal block at Akk into D (identity padded).
__device__ __forceinline__ void load_diag(double* D, const double* Akk, int ld, int kb) {
  for (int idx = threadIdx.x; idx < KP * KP; idx += BS) {
    const int r = idx / KP, c = idx % KP;
    D[r * SD + c] = (r < kb && c < kb) ? Akk[(int64_t)r * ld + c] : (r == c ? 1.0 : 0.0);
  }
}

// L11^T into LT (the idle tile staging area) for the column solves.
__device__ __forceinline__ void transpose_l11(double* LT, const double* D) {
  for (int idx = threadIdx.x; idx < KP * KP; idx += BS) {
    const int r = idx / KP, c = idx % KP;
    LT[c * SD + r] = r > c ? D[r * SD + c] : 0.0;
  }
}

// LU of A (n x n, leading dimension ld) in place.
__device__ void lu(double* A, int n, int ld, double* smem, double pfloor) {
  double* D = smem;
  double* rp = D + Smem::d_elems;
  double* ring = rp + Smem::r_elems;
  const int tid = threadIdx.x;
  for (int k0 = 0; k0 < n; k0 += KP) {
    const int kb = min(KP, n - k0);
    const int m = n - k0 - kb;  // > 0 only with kb == 32
    double* Akk = A + (int64_t)k0 * ld + k0;
    const double* Arow = A + (int64_t)k0 * ld;  // rows k0.. of the columns before the panel
    if (k0 > 0) {
      for (int i0 = 0; i0 < n - k0; i0 += 128) {
        if (n - k0 - i0 > 64)
          update_tile<128, 32, 8, 1>(Akk, Arow, A + k0, ld, n - k0, kb, k0, i0, 0, ring);
        else
          update_tile<64, 32, 8, 1>(Akk, Arow, A + k0, ld, n - k0, kb, k0, i0, 0, ring);
        __syncthreads();
      }
      for (int j0 = 0; j0 < m; j0 += 128) {
        if (m - j0 > 64)
          update_tile<32, 128, 1, 8>(Akk + kb, Arow, A + k0 + kb, ld, kb, m, k0, 0, j0, ring);
        else
          update_tile<32, 64, 2, 4>(Akk + kb, Arow, A + k0 + kb, ld, kb, m, k0, 0, j0, ring);
        __syncthreads();
      }
    }
    load_diag(D, Akk, ld, kb);
    __syncthreads();
    factor_diag(D, rp, pfloor, kb);
    for (int idx = tid; idx < kb * kb; idx += BS) {
      const int r = idx / kb, c = idx % kb;
      Akk[(int64_t)r * ld + c] = D[r * SD + c];
    }
    if (m > 0) {
      double* LT = ring;
      transpose_l11(LT, D);
      __syncthreads();
      trsm_panel(A + (int64_t)(k0 + kb) * ld + k0, Akk + kb, ld, m, D, rp, LT, 0, 1);
    }
    __syncthreads();  // L21, U12 and the diagonal block complete
  }
}

// Barrier over every thread of every CTA of the cluster, ordering the
// memory accesses before it (global and distributed shared) before those
// after it.  Block-uniform calls only.
__device__ __forceinline__ void cluster_sync_all() {
  __threadfence();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// The same LU as lu(), by the `parts` CTAs of a cluster together (this CTA
// has rank `part`); A in global memory, every CTA with its own scratch.  The
// update's blocks are split into 32 x 32 tiles by rank (its critical path is
// the K loop of one tile), each CTA factors the diagonal block itself (every
// CTA needs it in its own shared memory), the substitutions are split by rank,
// and three cluster barriers per panel order the stages.  Every element goes
// through the same operations in the same order as in lu(), so the factor is
// bit-identical.  Every CTA of the cluster must call it with the same n.
__device__ void lu_cluster(double* A, int n, int ld, double* smem, double pfloor, int part, int parts) {
  double* D = smem;
  double* rp = D + Smem::d_elems;
  double* ring = rp + Smem::r_elems;
  const int tid = threadIdx.x;
  for (int k0 = 0; k0 < n; k0 += KP) {
    const int kb = min(KP, n - k0);
    const int m = n - k0 - kb;
    double* Akk = A + (int64_t)k0 * ld + k0;
    const double* Arow = A + (int64_t)k0 * ld;
    if (k0 > 0) {
      const int nc = (n - k0 + 31) / 32, nr = (m + 31) / 32;
      for (int t = part; t < nc + nr; t += parts) {
        if (t < nc)
          update_tile<32, 32, 4, 2>(Akk, Arow, A + k0, ld, n - k0, kb, k0, 32 * t, 0, ring);
        else
          update_tile<32, 32, 4, 2>(Akk + kb, Arow, A + k0 + kb, ld, kb, m, k0, 0, 32 * (t - nc), ring);
        __syncthreads();
      }
      cluster_sync_all();  // the panel's blocks complete
    }
    load_diag(D, Akk, ld, kb);
    __syncthreads();
    factor_diag(D, rp, pfloor, kb);
    cluster_sync_all();  // every CTA holds the block: rank 0 may write it back below
    if (m > 0) {
      double* LT = ring;
      transpose_l11(LT, D);
      __syncthreads();
      trsm_panel(A + (int64_t)(k0 + kb) * ld + k0, Akk + kb, ld, m, D, rp, LT, part, parts);
    }
    if (part == 0)
      for (int idx = tid; idx < kb * kb; idx += BS) {
        const int r = idx / kb, c = idx % kb;
        Akk[(int64_t)r * ld + c] = D[r * SD + c];
      }
    cluster_sync_all();  // L21, U12 and the diagonal block complete
  }
}

}  // namespace dense64
}  // namespace gs2g
