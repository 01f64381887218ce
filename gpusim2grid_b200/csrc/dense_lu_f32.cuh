// Dense FP32 LU (no pivoting) of one matrix by one CTA of 256 threads (or by
// the CTAs of a cluster), for the tail of the mixed-precision batched
// Newton–Raphson factorization.  Device code only.
//
// The Crout order and stages of dense_lu_f64.cuh on 32-wide panels, with the
// update's products as FP32 FMAs (tcgen05 and mma.sync take FP32 operands only
// as TF32, below the FP32 held here): per panel the column block and the row
// block take all earlier panels' products at once, on tiles up to 256 high
// (column block) or wide (row block), fed by a cp.async ring of 32-deep slabs;
// then the diagonal block is factored by the whole CTA and the rows and columns
// are solved against it, a row or column per lane.
// What bounds it: few matrices, the chain of panels (about 14 us each beside
// the update); one matrix per CTA on every SM, the update.  Against a
// right-looking form with 64-wide panels, whose trailing update writes and
// reads the whole matrix once per panel (us per factorization):
//   n     one CTA       296 CTAs        cluster of 8   cluster of 16
//   42      27 -> 20        28 -> 23        27 -> 23        29 -> 23
//   133    130 -> 75       149 -> 81       142 -> 67       142 -> 73
//   518   1042 -> 815     1811 -> 1283     513 -> 350      475 -> 328
//   1148  6229 -> 5413   10638 -> 9018    1511 -> 1424    1225 -> 1080
// (296 CTAs: 33 TFLOP/s at n = 1148.)  The same order with the products on the
// FP64 tensor pipe (operands widened) took 1668 and 11559 us for 296 CTAs at
// n = 518 and 1148, 308 and 1080 us on clusters of 16.  Largest error against
// an FP64 factorization at n = 518: 3.7e-4 -> 2.8e-4.
// A is row-major in global memory with leading dimension ld, a multiple of
// 4 (rows 16-byte aligned); panels start at multiples of 32.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gs2g {
namespace dense32 {

constexpr int BS = 256;
constexpr int KP = 32;          // panel width
constexpr int SD = KP + 4;      // diagonal block stride (16-byte rows)
constexpr int KS = 32;          // slab depth of the update's operand ring
// operand strides: A's 4 mod 32 words, so that the 4 rows a warp reads at once
// lie in different banks (its 8 column groups of B are consecutive)
constexpr int SAK = KS + 4;
template <int TN>
__host__ __device__ constexpr int sbn() {
  return TN + 8;
}
template <int TM, int TN>
__host__ __device__ constexpr int stage_elems() {
  return TM * SAK + KS * sbn<TN>();
}

// ring depth: three slabs of the 128-wide and smaller tiles, two of the 256-wide
template <int TM, int TN>
__host__ __device__ constexpr int n_stage() {
  return TM * TN > 128 * 32 ? 2 : 3;
}
template <int TM, int TN>
__host__ __device__ constexpr int ring_elems() {
  return n_stage<TM, TN>() * stage_elems<TM, TN>();
}
constexpr int max_of(int a, int b) { return a > b ? a : b; }

struct Smem {
  static constexpr int d_elems = KP * SD;
  static constexpr int r_elems = KP;  // reciprocal pivots
  // outside the update the ring holds L11^T and a 32-row block per warp
  static constexpr int ring = max_of(max_of(max_of(ring_elems<128, 32>(), ring_elems<32, 128>()),
                                            max_of(ring_elems<256, 32>(), ring_elems<32, 256>())),
                                     9 * d_elems);
  static constexpr int elems = d_elems + r_elems + ring;
  static constexpr int bytes = elems * 4;
};
__device__ __forceinline__ float clamp_piv(float piv, double floor_) {
  const float f = (float)floor_;
  if (fabsf(piv) < f) return piv < 0.f ? -f : f;
  return piv;
}

// Shared-memory loads issued in program order (asm volatile): the
// substitutions below hold 32 values per thread in registers, and letting
// the compiler hoist their broadcast loads ahead of the arithmetic would
// spill them.
__device__ __forceinline__ float4 lds4(const float* p) {
  float4 v;
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float lds1(const float* p) {
  float v;
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(a));
  return v;
}

// This thread's share of a tile's operand slabs: PA 16-byte chunks of A (rows
// i0 + ra + i * RA) and PB of B (k rows kb + i * RB, columns j0 + n..), the
// same places in every slab, so the addresses only advance.  Rows past M and
// columns past N are zero-filled.
template <int TM, int TN>
struct Stager {
  static constexpr int PA = TM * KS / 4 / BS, RA = TM / PA, PB = TN * KS / 4 / BS, RB = KS / PB;
  static_assert(PA * RA == TM && PB * RB == KS && RA * (KS / 4) == BS && RB * (TN / 4) == BS, "whole chunks");
  const float* a;
  const float* b;
  int64_t lda, ldb, step_b;
  unsigned sa, sb;  // shared-memory byte offsets within a stage
  int arows, bbytes;
  __device__ __forceinline__ Stager(const float* A, const float* B, int ld, int M, int N, int i0, int j0) {
    const int tid = threadIdx.x;
    const int ra = tid / (KS / 4), ka = (tid % (KS / 4)) * 4;
    const int kb = tid / (TN / 4), n = (tid % (TN / 4)) * 4;
    arows = M - i0 - ra;  // chunk i is in range for i * RA < arows
    bbytes = (N - j0 - n) * 4;
    bbytes = bbytes < 0 ? 0 : (bbytes > 16 ? 16 : bbytes);
    a = A + (int64_t)(i0 + ra) * ld + ka;
    b = B + (int64_t)kb * ld + j0 + n;
    lda = (int64_t)RA * ld;
    ldb = (int64_t)RB * ld;
    step_b = (int64_t)KS * ld;
    sa = (unsigned)(ra * SAK + ka) * 4;
    sb = (unsigned)(TM * SAK + kb * sbn<TN>() + n) * 4;
  }
  // the next slab into the stage at shared-memory byte address st
  __device__ __forceinline__ void next(unsigned st) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int bytes = i * RA < arows ? 16 : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(st + sa + i * RA * SAK * 4),
                   "l"(bytes ? a + i * lda : a), "r"(bytes));
    }
#pragma unroll
    for (int i = 0; i < PB; ++i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(st + sb + i * RB * sbn<TN>() * 4),
                   "l"(b + i * ldb), "r"(bbytes));
    a += KS;
    b += step_b;
  }
};

// C[i0.., j0..] -= A[i0.., 0..K) B[0..K, j0..) for one TM x TN tile of an
// M x N block (A, B, C parts of one matrix, leading dimension ld; K a
// positive multiple of KS).  8 warps as WM x WN; a lane has R rows (4 apart)
// of 4 columns, so that a k step of 4 takes R + 4 16-byte loads, each of few
// distinct addresses, for 16 R products.  An element's products are summed
// slab by slab, each slab from zero (as many roundings at the size of the
// result as K has slabs, not as many as K), in the same order whatever the
// tile shape, so every tiling gives the same bits.  Ends without a barrier;
// the ring may be refilled only after one.
template <int TM, int TN, int WM, int WN>
__device__ __noinline__ void update_tile(float* C, const float* A, const float* B, int ld, int M, int N, int K,
                                         int i0, int j0, float* ring) {
  constexpr int R = TM / (4 * WM);
  constexpr int SE = stage_elems<TM, TN>(), NSTAGE = n_stage<TM, TN>();
  static_assert(WM * WN * 32 == BS && R > 0 && TN == 32 * WN, "8 warps tile TM x TN");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wr = (warp / WN) * 4 * R + (lane >> 3), wc = (warp % WN) * 32 + (lane & 7) * 4;
  const int nslab = K / KS;
  const unsigned sring = (unsigned)__cvta_generic_to_shared(ring);
  Stager<TM, TN> stager(A, B, ld, M, N, i0, j0);
#pragma unroll
  for (int s = 0; s < NSTAGE - 1; ++s) {
    if (s < nslab) stager.next(sring + s * SE * 4);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int cur = 0, fill = NSTAGE - 1;  // ring positions of slab t and of slab t + NSTAGE - 1
  float acc[R][4];
  const int c = j0 + wc;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = i0 + wr + 4 * i;
    const float* src = C + (int64_t)r * ld + c;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < M && c + 3 < N) {
      v = *reinterpret_cast<const float4*>(src);
    } else if (r < M) {
      if (c < N) v.x = src[0];
      if (c + 1 < N) v.y = src[1];
      if (c + 2 < N) v.z = src[2];
    }
    acc[i][0] = v.x;
    acc[i][1] = v.y;
    acc[i][2] = v.z;
    acc[i][3] = v.w;
  }
  // a warp of a last tile whose part lies past M or N only stages (296 CTAs at
  // n = 200: 173 -> 159 us); in the 256 tiles the test cost 20 %
  const bool idle = i0 + wr - (lane >> 3) >= M || j0 + (warp % WN) * 32 >= N;
  for (int t = 0; t < nslab; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NSTAGE - 2) : "memory");
    __syncthreads();  // slab t has landed; every warp is done with slab t - 1
    if (t + NSTAGE - 1 < nslab) stager.next(sring + fill * SE * 4);
    asm volatile("cp.async.commit_group;\n" ::);
    const float* sA = ring + cur * SE + wr * SAK;
    const float* sB = ring + cur * SE + TM * SAK + wc;
    cur = cur + 1 < NSTAGE ? cur + 1 : 0;
    fill = fill + 1 < NSTAGE ? fill + 1 : 0;
    if (TM * TN == 128 * 32 && idle) continue;
    float p[R][4];
#pragma unroll
    for (int i = 0; i < R; ++i) p[i][0] = p[i][1] = p[i][2] = p[i][3] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; k += 4) {
      float4 b[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) b[h] = *reinterpret_cast<const float4*>(sB + (k + h) * sbn<TN>());
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 av = *reinterpret_cast<const float4*>(sA + 4 * i * SAK + k);
        const float a[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          p[i][0] = fmaf(a[h], b[h].x, p[i][0]);
          p[i][1] = fmaf(a[h], b[h].y, p[i][1]);
          p[i][2] = fmaf(a[h], b[h].z, p[i][2]);
          p[i][3] = fmaf(a[h], b[h].w, p[i][3]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] -= p[i][e];
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = i0 + wr + 4 * i;
    if (r >= M) continue;
    float* dst = C + (int64_t)r * ld + c;
    if (c + 3 < N) {
      *reinterpret_cast<float4*>(dst) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
      if (c < N) dst[0] = acc[i][0];
      if (c + 1 < N) dst[1] = acc[i][1];
      if (c + 2 < N) dst[2] = acc[i][2];
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Factor the identity-padded 32 x 32 block D (stride SD) in place, its first kb
// steps; rp gets the reciprocal pivots (see dense_lu_f64.cuh).
__device__ __noinline__ void factor_diag(float* D, float* rp, double pfloor, int kb) {
  __shared__ __align__(16) float prow[2][KP];
  const int r = threadIdx.x >> 3, q = threadIdx.x & 7, lane = threadIdx.x & 31;
  float x[4];
  {
    const float4 v = *reinterpret_cast<const float4*>(D + r * SD + 4 * q);
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
  }
#pragma unroll
  for (int j = 0; j < KP; ++j) {
    if (j >= kb) break;  // the padding needs no step
    if (r == j) {
      if (q == j >> 2) {
        x[j & 3] = clamp_piv(x[j & 3], pfloor);
        rp[j] = 1.f / x[j & 3];
      }
      *reinterpret_cast<float4*>(&prow[j & 1][4 * q]) = make_float4(x[0], x[1], x[2], x[3]);
    }
    __syncthreads();
    const float xj = __shfl_sync(0xffffffffu, x[j & 3], (lane & 24) | (j >> 2));
    if (r > j && q >= j >> 2) {
      const float l = xj * rp[j];
      const float4 uv = *reinterpret_cast<const float4*>(&prow[j & 1][4 * q]);
      const float u[4] = {uv.x, uv.y, uv.z, uv.w};
      if (q > j >> 2) {
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = fmaf(-l, u[c], x[c]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (c > (j & 3)) x[c] = fmaf(-l, u[c], x[c]);
        x[j & 3] = l;
      }
    }
  }
  *reinterpret_cast<float4*>(D + r * SD + 4 * q) = make_float4(x[0], x[1], x[2], x[3]);
  __syncthreads();
}

// x <- x M^-1 for the 32 values x of one thread, M upper triangular given by
// its rows (stride SD) in shared memory: after x_p is final, x_q -= x_p M_pq
// for q > p.  SCALE: x_p is multiplied by rp[p] (1 / M_pp) first; else M has
// a unit diagonal.
template <bool SCALE>
__device__ __forceinline__ void subst32(float (&x)[KP], const float* M, const float* rp) {
#pragma unroll
  for (int p = 0; p < KP; ++p) {
    if (SCALE) x[p] *= lds1(rp + p);
    const float xp = x[p];
    const float* mp = M + p * SD;
#pragma unroll
    for (int q4 = (p + 1) & ~3; q4 < KP; q4 += 4) {
      const float4 u = lds4(mp + q4);
      if (q4 > p) x[q4] = fmaf(-xp, u.x, x[q4]);
      if (q4 + 1 > p) x[q4 + 1] = fmaf(-xp, u.y, x[q4 + 1]);
      if (q4 + 2 > p) x[q4 + 2] = fmaf(-xp, u.z, x[q4 + 2]);
      if (q4 + 3 > p) x[q4 + 3] = fmaf(-xp, u.w, x[q4 + 3]);
    }
  }
}

// L21 = A21 U11^-1 (x U11 = a per row) for 32 rows (n of them valid) by one
// warp, a row per lane in registers.  The rows pass through the warp's block
// of shared memory (stride SD: conflict-free) so that global memory is read
// and written four whole rows at a time.
__device__ __forceinline__ void trsm_rows32(float* A21, int ld, int n, const float* D, const float* rp, float* buf) {
  const int lane = threadIdx.x & 31, r4 = lane >> 3, c4 = (lane & 7) * 4;
#pragma unroll
  for (int h = 0; h < KP; h += 4)
    if (h + r4 < n)
      *reinterpret_cast<float4*>(buf + (h + r4) * SD + c4) =
          *reinterpret_cast<const float4*>(A21 + (int64_t)(h + r4) * ld + c4);
  __syncwarp();
  if (lane < n) {
    float x[KP];
#pragma unroll
    for (int q = 0; q < KP; q += 4) {
      const float4 v = lds4(buf + lane * SD + q);
      x[q] = v.x;
      x[q + 1] = v.y;
      x[q + 2] = v.z;
      x[q + 3] = v.w;
    }
    subst32<true>(x, D, rp);
#pragma unroll
    for (int q = 0; q < KP; q += 4)
      *reinterpret_cast<float4*>(buf + lane * SD + q) = make_float4(x[q], x[q + 1], x[q + 2], x[q + 3]);
  }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < KP; h += 4)
    if (h + r4 < n)
      *reinterpret_cast<float4*>(A21 + (int64_t)(h + r4) * ld + c4) =
          *reinterpret_cast<const float4*>(buf + (h + r4) * SD + c4);
  __syncwarp();
}

// U12 = L11^-1 A12 (per column: y^T L11^T = a^T, L11^T upper with unit
// diagonal, given by its rows LT), one column of A12 in registers.
__device__ __forceinline__ void trsm_col(float* colp, int ld, const float* LT) {
  float y[KP];
#pragma unroll
  for (int r = 0; r < KP; ++r) y[r] = colp[(int64_t)r * ld];
  subst32<false>(y, LT, nullptr);
#pragma unroll
  for (int r = 0; r < KP; ++r) colp[(int64_t)r * ld] = y[r];
}

// Both substitutions of a panel with m rows below and m columns to the right
// of its diagonal block, in groups of 32 rows or 32 columns taken by the
// warps of the `parts` CTAs (this one: part).  LT: L11^T, followed by a block
// per warp.
__device__ __noinline__ void trsm_panel(float* A21, float* A12, int ld, int m, const float* D, const float* rp,
                                        float* LT, int part, int parts) {
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
__device__ __forceinline__ void load_diag(float* D, const float* Akk, int ld, int kb) {
  for (int idx = threadIdx.x; idx < KP * KP; idx += BS) {
    const int r = idx / KP, c = idx % KP;
    D[r * SD + c] = (r < kb && c < kb) ? Akk[(int64_t)r * ld + c] : (r == c ? 1.f : 0.f);
  }
}

// L11^T into LT (the idle tile staging area) for the column solves.
__device__ __forceinline__ void transpose_l11(float* LT, const float* D) {
  for (int idx = threadIdx.x; idx < KP * KP; idx += BS) {
    const int r = idx / KP, c = idx % KP;
    LT[c * SD + r] = r > c ? D[r * SD + c] : 0.f;
  }
}

// LU of A (n x n, leading dimension ld) in place.
__device__ void lu(float* A, int n, int ld, float* smem, double pfloor) {
  float* D = smem;
  float* rp = D + Smem::d_elems;
  float* ring = rp + Smem::r_elems;
  const int tid = threadIdx.x;
  for (int k0 = 0; k0 < n; k0 += KP) {
    const int kb = min(KP, n - k0);
    const int m = n - k0 - kb;  // > 0 only with kb == 32
    float* Akk = A + (int64_t)k0 * ld + k0;
    const float* Arow = A + (int64_t)k0 * ld;  // rows k0.. of the columns before the panel
    if (k0 > 0) {
      int i0 = 0, j0 = 0;
      for (; n - k0 - i0 > 128; i0 += 256) {
        update_tile<256, 32, 8, 1>(Akk, Arow, A + k0, ld, n - k0, kb, k0, i0, 0, ring);
        __syncthreads();
      }
      if (i0 < n - k0) {
        update_tile<128, 32, 8, 1>(Akk, Arow, A + k0, ld, n - k0, kb, k0, i0, 0, ring);
        __syncthreads();
      }
      for (; m - j0 > 128; j0 += 256) {
        update_tile<32, 256, 1, 8>(Akk + kb, Arow, A + k0 + kb, ld, kb, m, k0, 0, j0, ring);
        __syncthreads();
      }
      if (j0 < m) {
        update_tile<32, 128, 2, 4>(Akk + kb, Arow, A + k0 + kb, ld, kb, m, k0, 0, j0, ring);
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
      float* LT = ring;
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

// Height of the tiles a cluster splits a panel's update into: the column block
// has mc rows, the row block mr columns, and a k step of a 32-, 64- or 128-high
// tile takes about 5, 6 and 9 units (its loads from shared memory, then its
// products, bound it), so the fewest units over the rounds.
__device__ __forceinline__ int tile_height(int mc, int mr, int parts) {
  int best = 32, cost = 1 << 30;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int h = 32 << i, tiles = (mc + h - 1) / h + (mr + h - 1) / h;
    const int c = (tiles + parts - 1) / parts * (i == 0 ? 5 : i == 1 ? 6 : 9);
    if (c < cost) {
      cost = c;
      best = h;
    }
  }
  return best;
}

// This CTA's tiles (H x 32 of the column block, 32 x H of the row block) of
// panel k0's update.  WM x WN: the warps of a row-block tile.
template <int H, int WM, int WN>
__device__ __forceinline__ void cluster_update(float* A, int n, int ld, int k0, int kb, float* ring, int part,
                                               int parts) {
  const int m = n - k0 - kb;
  float* Akk = A + (int64_t)k0 * ld + k0;
  const float* Arow = A + (int64_t)k0 * ld;
  const int nc = (n - k0 + H - 1) / H, nr = (m + H - 1) / H;
  for (int t = part; t < nc + nr; t += parts) {
    if (t < nc)
      update_tile<H, 32, 8, 1>(Akk, Arow, A + k0, ld, n - k0, kb, k0, H * t, 0, ring);
    else
      update_tile<32, H, WM, WN>(Akk + kb, Arow, A + k0 + kb, ld, kb, m, k0, 0, H * (t - nc), ring);
    __syncthreads();
  }
}

// The same LU as lu(), by the `parts` CTAs of a cluster together (this CTA
// has rank `part`); A in global memory, every CTA with its own scratch.  The
// update's blocks are split into tiles by rank, each CTA factors the diagonal block itself (every
// CTA needs it in its own shared memory), the substitutions are split by rank,
// and three cluster barriers per panel order the stages.  Every element goes
// through the same operations in the same order as in lu(), so the factor is
// bit-identical.  Every CTA of the cluster must call it with the same n.
__device__ void lu_cluster(float* A, int n, int ld, float* smem, double pfloor, int part, int parts) {
  float* D = smem;
  float* rp = D + Smem::d_elems;
  float* ring = rp + Smem::r_elems;
  const int tid = threadIdx.x;
  for (int k0 = 0; k0 < n; k0 += KP) {
    const int kb = min(KP, n - k0);
    const int m = n - k0 - kb;
    float* Akk = A + (int64_t)k0 * ld + k0;
    if (k0 > 0) {
      const int h = tile_height(n - k0, m, parts);
      if (h == 128)
        cluster_update<128, 2, 4>(A, n, ld, k0, kb, ring, part, parts);
      else if (h == 64)
        cluster_update<64, 4, 2>(A, n, ld, k0, kb, ring, part, parts);
      else
        cluster_update<32, 8, 1>(A, n, ld, k0, kb, ring, part, parts);
      cluster_sync_all();  // the panel's blocks complete
    }
    load_diag(D, Akk, ld, kb);
    __syncthreads();
    factor_diag(D, rp, pfloor, kb);
    cluster_sync_all();  // every CTA holds the block: rank 0 may write it back below
    if (m > 0) {
      float* LT = ring;
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

}  // namespace dense32
}  // namespace gs2g
