// BF16 GEMM of the warm-start network on the 5th-generation tensor cores:
//   C[M x N] = A . B^T summed over K in fp32, then an epilogue per element,
// with each operand either K-major (row i holds K contiguous: X[i][k]) or
// MN-major (row k holds the M or N index contiguous: X[k][i]); the backward
// pass's products over the batch and over the weights' rows take their
// operands as they lie in memory, without transposes.
//
// One persistent CTA per SM, 10 warps: warp 0 streams 64-deep operand slabs
// into a 4-stage ring by TMA (128-byte swizzle; 128 x 64 of A, BN x 64 of B);
// one thread of warp 1 issues tcgen05.mma.kind::f16 (M = 128, N = BN) into one
// of two tensor-memory accumulators; warps 2..9 empty the other one through a
// padded shared-memory block each, so that global memory sees 128-byte rows,
// and apply the epilogue there while the next tile's products run.
// BN = 256 takes 3/4 of the operand bytes per product of 128 x 128 tiles, and
// those bytes bound the kernel (64 bytes a cycle into an SM); BN = 128 and a split
// of K into partial planes (summed in order by finish_kernel with the same
// epilogue) serve shapes with fewer tiles than SMs.  gemm_plan picks both by
// the waves they take.
// Every mbarrier wait is bounded (2 s): on timeout the kernel sets *err, waits
// (bounded) for its copies and MMAs in flight, frees its tensor memory and
// returns.
#pragma once

#include <cuda.h>  // CUtensorMap (types only; the encoder comes from the runtime)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace gs2g {
namespace mlp {

constexpr int GT = 128;  // tile rows; M and N are multiples of it
constexpr int GK = 64;   // K per stage
constexpr int STAGES = 4;
constexpr int EPI_WARPS = 8;
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
constexpr int A_BYTES = GT * GK * 2;
constexpr int EPI_LD = 33;  // floats per row of a warp's 32 x 32 block
template <int BN>
__host__ __device__ constexpr int stage_bytes() {
  return A_BYTES + BN * GK * 2;
}
template <int BN>
constexpr int gemm_smem() {
  return STAGES * stage_bytes<BN>() + EPI_WARPS * 32 * EPI_LD * 4 + 1024;
}
static_assert(gemm_smem<256>() <= 232448 - 256, "ring and epilogue blocks within a CTA's shared memory");
constexpr uint64_t WAIT_NS = 2000000000ull;  // bound of one mbarrier wait (2 s)
constexpr int MAX_SPLIT = 8;

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

// What happens to a finished sum v of element (r, c).
enum EpiOp : int {
  EPI_STORE = 0,  // D = v (+ D with accumulate)
  EPI_BIAS,       // D = v + bias[c]
  EPI_GELU,       // z = v + bias[c]; D = z unless null; act = bf16(gelu(z))
  EPI_GELU_BWD,   // act = bf16(v * gelu'(D)), D the layer's stored z
};
struct Epilogue {
  int op;
  int accumulate;
  float* D;
  int ldd;
  const float* bias;
  __nv_bfloat16* act;
  int lda;
};

// The epilogue of column c, rows r0, r0 + 1, ..: OP the operation at compile
// time, or EPI_ANY to look at it per element.  (With the operation looked up and
// the addresses formed per element, the GELU epilogue took longer than the
// products of a K = 1024 layer.)
constexpr int EPI_ANY = -1;
template <int OP>
struct ColumnEpilogue {
  const int op;
  const int accumulate;
  const float bias;
  float* d;
  __nv_bfloat16* act;
  const int64_t ldd, lda;
  __device__ __forceinline__ ColumnEpilogue(const Epilogue& e, int r0, int c)
      : op(OP == EPI_ANY ? e.op : OP),
        accumulate(e.accumulate),
        bias(op == EPI_BIAS || op == EPI_GELU ? e.bias[c] : 0.f),
        d(e.D != nullptr ? e.D + (int64_t)r0 * e.ldd + c : nullptr),
        act(op >= EPI_GELU ? e.act + (int64_t)r0 * e.lda + c : nullptr),
        ldd(e.ldd),
        lda(e.lda) {}
  __device__ __forceinline__ void row(int q, float v) const {
    float* dq = d + q * ldd;
    if (op == EPI_STORE) {
      *dq = accumulate ? v + *dq : v;
    } else if (op == EPI_BIAS) {
      *dq = v + bias;
    } else if (op == EPI_GELU) {
      const float z = v + bias;
      if (d != nullptr) *dq = z;
      act[q * lda] = __float2bfloat16(gelu_f(z));
    } else {
      act[q * lda] = __float2bfloat16(v * gelu_grad_f(*dq));
    }
  }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor, 128-byte swizzle.  K-major: 8-row groups
// 1024 bytes apart (lbo unused).  MN-major: 8-k groups 1024 bytes apart, blocks
// of 64 rows lbo bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 | (uint64_t)(1024 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// Instruction descriptor: kind::f16, A = B = bf16, D = f32.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait for the phase with the given parity; false after WAIT_NS, or as
// soon as another wait of the CTA has failed (*fail, nullptr: not looked at).
// The timer is first read after 64 tries: reading it on every wait took longer
// than a 64-deep step's products.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  uint64_t t0 = 0;
  for (uint32_t i = 0;; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 63) == 63) {
      if (fail != nullptr && *fail) return false;
      const uint64_t now = global_ns();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > WAIT_NS) {
        if (fail != nullptr) *fail = 1;
        return false;
      }
    }
  }
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// tiles: tiles_m x tiles_n x splits (n fastest, then m); split s takes
// k-tiles [s * kt_split, min(KT, (s + 1) * kt_split)) and, with splits > 1,
// stores its sum into plane s of part ([splits][M][N] fp32).
struct GemmShape {
  int M, N, KT, tiles_m, tiles_n, splits, kt_split;
  float* part;
};

template <int BN, bool A_MN, bool B_MN, int OP>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const GemmShape g, const Epilogue e, int* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], tfull[2], tempty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_fail, s_loads, s_mmas;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ring = (smem_u32(smem) + 1023) & ~1023u;
  float* epi_smem = reinterpret_cast<float*>(smem + (ring - smem_u32(smem)) + STAGES * stage_bytes<BN>());
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    s_fail = 0;
    s_loads = s_mmas = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(2 * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  const uint32_t tmem = tmem_base_s;
  volatile int* fail = &s_fail;
  const int n_tiles = g.tiles_m * g.tiles_n * g.splits;
  auto k_range = [&](int t, int& k0, int& k1) {
    const int s = t / (g.tiles_m * g.tiles_n);
    k0 = s * g.kt_split;
    k1 = min(g.KT, k0 + g.kt_split);
  };

  if (warp == 0 && lane == 0) {
    // ---- producer
    int it = 0;
    for (int t = blockIdx.x; t < n_tiles && !*fail; t += gridDim.x) {
      const int mn = t % (g.tiles_m * g.tiles_n);
      const int m0 = (mn / g.tiles_n) * GT, n0 = (mn % g.tiles_n) * BN;
      int k0, k1;
      k_range(t, k0, k1);
      for (int kt = k0; kt < k1; ++kt, ++it) {
        const int s = it % STAGES;
        if (it >= STAGES && !mbar_wait(smem_u32(&empty[s]), (uint32_t)((it / STAGES - 1) & 1), fail)) break;
        const uint32_t bar = smem_u32(&full[s]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(stage_bytes<BN>())
                     : "memory");
        const uint32_t a = ring + (uint32_t)(s * stage_bytes<BN>()), b = a + A_BYTES;
        if (A_MN) {
#pragma unroll
          for (int h = 0; h < GT / 64; ++h) tma_load(a + h * 8192, &map_a, m0 + 64 * h, kt * GK, bar);
        } else {
          tma_load(a, &map_a, kt * GK, m0, bar);
        }
        if (B_MN) {
#pragma unroll
          for (int h = 0; h < BN / 64; ++h) tma_load(b + h * 8192, &map_b, n0 + 64 * h, kt * GK, bar);
        } else {
          tma_load(b, &map_b, kt * GK, n0, bar);
        }
        s_loads = it + 1;
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    constexpr uint32_t idesc = umma_idesc_bf16(GT, BN, A_MN, B_MN);
    int it = 0, n = 0;
    for (int t = blockIdx.x; t < n_tiles && !*fail; t += gridDim.x, ++n) {
      int k0, k1;
      k_range(t, k0, k1);
      const int acc = n & 1;
      if (n >= 2 && !mbar_wait(smem_u32(&tempty[acc]), (uint32_t)((n / 2 - 1) & 1), fail)) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
      const uint32_t d = tmem + (uint32_t)(acc * BN);
      bool ok = true;
      for (int kt = k0; kt < k1; ++kt, ++it) {
        const int s = it % STAGES;
        ok = mbar_wait(smem_u32(&full[s]), (uint32_t)((it / STAGES) & 1), fail);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
        const uint32_t a = ring + (uint32_t)(s * stage_bytes<BN>()), b = a + A_BYTES;
#pragma unroll
        for (int j = 0; j < GK / 16; ++j) {
          // 16 k further: 32 bytes along a swizzled K-major row, two 8-k
          // groups of an MN-major block
          const uint64_t ad = umma_desc(a + j * (A_MN ? 2048 : 32), A_MN ? 8192 : 16);
          const uint64_t bd = umma_desc(b + j * (B_MN ? 2048 : 32), B_MN ? 8192 : 16);
          const uint32_t en = (kt > k0 || j > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d),
              "l"(ad), "l"(bd), "r"(idesc), "r"(en), "r"(0), "r"(0), "r"(0), "r"(0));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
            smem_u32(&empty[s])));
        s_mmas = it + 1;
      }
      if (!ok) break;
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
          smem_u32(&tfull[acc])));
    }
  } else if (warp >= 2) {
    // ---- epilogue: tensor-memory lanes 32 (warp % 4).. (the only ones a warp
    // reaches), half of the columns, 32 at a time
    const int ew = warp - 2, quad = warp & 3, half = ew >> 2;
    float* buf = epi_smem + ew * 32 * EPI_LD;
    int n = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++n) {
      const int s = t / (g.tiles_m * g.tiles_n), mn = t % (g.tiles_m * g.tiles_n);
      const int m0 = (mn / g.tiles_n) * GT, n0 = (mn % g.tiles_n) * BN;
      const int acc = n & 1;
      // the whole warp goes on or gives up: lanes whose waits end differently
      // (one sees the flag, another the barrier) must not part ahead of the
      // .aligned loads; a tile that is full when the flag goes up is finished
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&tfull[acc]), (uint32_t)((n / 2) & 1), fail))) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
#pragma unroll 1
      for (int cc = 0; cc < BN / 2; cc += 32) {
        const int c0 = half * (BN / 2) + cc;
        uint32_t v[32];
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * BN + c0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,"
            "%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
              "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
              "=r"(v[30]), "=r"(v[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (cc + 32 == BN / 2) {
          // this warp has read its part of the accumulator
          asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[acc]);
        }
#pragma unroll
        for (int q = 0; q < 32; ++q) buf[lane * EPI_LD + q] = __uint_as_float(v[q]);
        __syncwarp();
        const int c = n0 + c0 + lane;
        if (c < g.N) {
          const int r0 = m0 + 32 * quad;
          if (g.splits > 1) {
            float* p = g.part + ((int64_t)s * g.M + r0) * g.N + c;
#pragma unroll 8
            for (int q = 0; q < 32; ++q) p[(int64_t)q * g.N] = buf[q * EPI_LD + lane];
          } else {
            const ColumnEpilogue<OP> ep(e, r0, c);
#pragma unroll 8
            for (int q = 0; q < 32; ++q) ep.row(q, buf[q * EPI_LD + lane]);
          }
        }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  if (*fail && tid == 0) {
    atomicExch(err, 1);
    // copies in flight land, MMAs in flight finish (or their waits run out too)
    // before the shared and tensor memory are given up
    for (int it = max(0, s_loads - STAGES); it < s_loads; ++it)
      mbar_wait(smem_u32(&full[it % STAGES]), (uint32_t)((it / STAGES) & 1), nullptr);
    if (s_mmas > 0) mbar_wait(smem_u32(&empty[(s_mmas - 1) % STAGES]), (uint32_t)(((s_mmas - 1) / STAGES) & 1), nullptr);
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(2 * BN));
  }
}

// Sums the partial planes of a split product in order and applies the epilogue.
template <int OP>
__global__ void __launch_bounds__(256) finish_kernel(const GemmShape g, const Epilogue e) {
  const int64_t plane = (int64_t)g.M * g.N;
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= g.N) return;
  for (int r = blockIdx.y; r < g.M; r += gridDim.y) {
    const float* p = g.part + (int64_t)r * g.N + c;
    float x[MAX_SPLIT];
#pragma unroll
    for (int s = 0; s < MAX_SPLIT; ++s) x[s] = s < g.splits ? p[s * plane] : 0.f;
    float v = x[0];
#pragma unroll
    for (int s = 1; s < MAX_SPLIT; ++s)
      if (s < g.splits) v += x[s];
    ColumnEpilogue<OP>(e, r, c).row(0, v);
  }
}

// Tile width and K split of an M x N x K product on n_sm SMs: the pair that
// takes the fewest cycles in whole waves.  A 64-deep step brings 48 KB (128 x 256
// tile) or 32 KB (128 x 128) into the SM, and that, not the tensor pipe (540 or
// 270 cycles), sets its time: about 850 and 700 cycles measured.  A tile costs
// about 3000 more (filling the ring, the last epilogue).  A split adds a launch
// and a pass over its planes: K = 7232 on 2944 x 1024 took 51 us whole and 63 in
// three, on 1024 x 1024 44 us in two and 35 in four; K = 3712 on 1024 x 1024 43
// us whole, 30 in two.
struct GemmPlan {
  int bn, splits, kt_split;
};
inline GemmPlan gemm_plan(int M, int N, int K, int n_sm, bool may_split) {
  const int KT = K / GK;
  GemmPlan best{256, 1, KT};
  double best_cost = 1e300;
  for (int bn : {256, 128}) {
    const int64_t tiles = (int64_t)(M / GT) * ((N + bn - 1) / bn);
    for (int s = 1; s <= (may_split ? MAX_SPLIT : 1); ++s) {
      if (s > 1 && (s > KT || tiles * s > 2 * n_sm)) break;
      const int kts = (KT + s - 1) / s;
      if ((s - 1) * kts >= KT) continue;  // an empty split
      const double waves = (double)((tiles * s + n_sm - 1) / n_sm);
      double cost = waves * (kts * (bn == 256 ? 850.0 : 700.0) + 3000.0);
      if (s > 1) cost += 6000.0 + (double)M * N * 4.0 * (s + 1) / 2000.0;  // the finishing launch
      if (cost < best_cost) {
        best_cost = cost;
        best = {bn, s, kts};
      }
    }
  }
  return best;
}

}  // namespace mlp
}  // namespace gs2g
