// Kernels of the warm-start MLP: the launches of its BF16 GEMM on the
// 5th-generation tensor cores (mlp_gemm.cuh) and the pieces around it: the
// first layer of outage rows, the loss gradient, bias gradients, the Adam step
// and the start voltages.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/gs2g.h"
#include "mlp_gemm.cuh"

namespace gs2g {
namespace mlp {

// ------------------------------------------------------------ elementwise
// Two-dimensional kernels: a thread owns one column and walks over rows.
// pre[r][c] += bias[c]; act[r][c] = bf16(gelu(pre)) (or bf16(pre) when !gelu)
__global__ void bias_act_kernel(float* pre, int ldp, const float* bias, __nv_bfloat16* act, int lda, int rows,
                                int cols, int gelu) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const float b = bias[c];
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const float v = pre[(int64_t)r * ldp + c] + b;
    pre[(int64_t)r * ldp + c] = v;
    if (act) act[(int64_t)r * lda + c] = __float2bfloat16(gelu ? gelu_f(v) : v);
  }
}

// dpre = dact * gelu'(pre) (fp32 in, bf16 out)
__global__ void gelu_bwd_kernel(const float* dact, int ldg, const float* pre, int ldp, __nv_bfloat16* dpre, int ldo,
                                int rows, int cols) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  for (int r = blockIdx.y; r < rows; r += gridDim.y)
    dpre[(int64_t)r * ldo + c] = __float2bfloat16(dact[(int64_t)r * ldg + c] * gelu_grad_f(pre[(int64_t)r * ldp + c]));
}

// dy = scale * (y - t) over the first `cols_valid` columns (0 elsewhere),
// bf16; loss += sum (y - t)^2 over valid entries, one atomic per block (one
// per warp of a grid-stride pass serialised on the loss).
__global__ void __launch_bounds__(256) mse_grad_kernel(const float* y, const float* t, int ld, __nv_bfloat16* dy,
                                                       int rows, int cols, int cols_valid, float scale, float* loss) {
  __shared__ float s_sum[8];
  const int c = blockIdx.x * 256 + threadIdx.x;
  float acc = 0.f;
  if (c < cols)
#pragma unroll 4
    for (int r = blockIdx.y; r < rows; r += gridDim.y) {
      const int64_t i = (int64_t)r * ld + c;
      float g = 0.f;
      if (c < cols_valid) {
        const float d = y[i] - t[i];
        acc += d * d;
        g = scale * d;
      }
      dy[i] = __float2bfloat16(g);
    }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0 && loss) {
    for (int w = 1; w < 8; ++w) acc += s_sum[w];
    atomicAdd(loss, acc);
  }
}

// column sums of a bf16 matrix: out[c] += sum_r x[r][c]; block (128 columns)
// x (a chunk of COLSUM_ROWS rows), one atomicAdd per column and chunk
constexpr int COLSUM_ROWS = 64;
__global__ void colsum_bf16_kernel(const __nv_bfloat16* x, int ld, int rows, int cols, float* out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  const int r0 = blockIdx.y * COLSUM_ROWS;
  const int r1 = min(rows, r0 + COLSUM_ROWS);
  float s = 0.f;
#pragma unroll 16
  for (int r = r0; r < r1; ++r) s += __bfloat162float(x[(int64_t)r * ld + c]);
  atomicAdd(out + c, s);
}

// out[c][r] = in[r][c] (bf16), 32x32 tiles through shared memory
__global__ void transpose_bf16_kernel(const __nv_bfloat16* in, int ldi, __nv_bfloat16* out, int ldo, int rows,
                                      int cols) {
  __shared__ __nv_bfloat16 t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = r0 + k, c = c0 + threadIdx.x;
    t[k][threadIdx.x] = (r < rows && c < cols) ? in[(int64_t)r * ldi + c] : __float2bfloat16(0.f);
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int c = c0 + k, r = r0 + threadIdx.x;
    if (c < cols && r < rows) out[(int64_t)c * ldo + r] = t[threadIdx.x][k];
  }
}

__global__ void f32_to_bf16_kernel(const float* in, __nv_bfloat16* out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(in[i]);
}

// Adam on fp32 master weights; writes the bf16 copy used by the GEMMs.
__global__ void adam_kernel(float* w, const float* g, float* m, float* v, __nv_bfloat16* wb, int64_t n, float lr,
                            float b1, float b2, float eps, float c1, float c2, float wd) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i] + wd * w[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16(wi);
  }
}

// Start voltages from predicted, standardised unknowns: for bus b of row r,
// Va = y[r][ia[b]] * std + mean when b is a pv/pq bus (ia[b] >= 0), else the
// angle of vinit[b]; Vm = y[r][im[b]] * std + mean when b is a pq bus
// (im[b] >= 0), else |vinit[b]|; V0 = Vm e^{j Va} (FP64).
__global__ void start_voltages_kernel(const float* y, int ldy, const float* ymean, const float* ystd, const int* ia,
                                      const int* im, const double2* vinit, int n_bus, double2* v0, int rows) {
  const int64_t n = (int64_t)rows * n_bus;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / n_bus), b = (int)(i % n_bus);
    const double2 v = vinit[b];
    double va = atan2(v.y, v.x), vm = hypot(v.x, v.y);
    const int a = ia[b], m = im[b];
    if (a >= 0) va = (double)y[(int64_t)r * ldy + a] * ystd[a] + ymean[a];
    if (m >= 0) vm = (double)y[(int64_t)r * ldy + m] * ystd[m] + ymean[m];
    double s, c;
    sincos(va, &s, &c);
    v0[i] = make_double2(vm * c, vm * s);
  }
}

// Standardised bf16 network inputs of the rows, in one pass (one CTA per
// row of the padded input block X [rows_pad x ldx]):
//   column c < n_pvpq:            Re(S_r - S_base) at bus pvpq[c]
//   column n_pvpq + c', c' < n_pq: Im(S_r - S_base) at bus pq[c']
//   (0 without injection rows)
//   plus, for every branch the row trips, the four contributions
//   br_val[4 b + k] at column br_col[4 b + k] (columns >= n_in dropped)
// then (x - mean) / std for c < n_in, 0 in the padding.  At most
// FEAT_MAX_TERMS trip contributions per row are held; more are read back
// from global memory per column.
constexpr int FEAT_MAX_TERMS = 256;
__global__ void features_kernel(const double2* __restrict__ sbus_rows, const double2* __restrict__ sbus_base,
                                const int* __restrict__ pvpq, int n_pvpq, const int* __restrict__ pq, int n_pq,
                                const int* __restrict__ trip_ptr, const int* __restrict__ trip_ids,
                                const int* __restrict__ br_col, const float* __restrict__ br_val,
                                const float* __restrict__ x_mean, const float* __restrict__ x_std, int n_in,
                                __nv_bfloat16* __restrict__ X, int ldx, int rows, int n_bus) {
  __shared__ int s_c[FEAT_MAX_TERMS];
  __shared__ float s_v[FEAT_MAX_TERMS];
  __shared__ int s_n;
  const int r = blockIdx.x;
  __nv_bfloat16* xr = X + (int64_t)r * ldx;
  if (r >= rows) {
    for (int c = threadIdx.x; c < ldx; c += blockDim.x) xr[c] = __float2bfloat16(0.f);
    return;
  }
  const int q0 = trip_ptr != nullptr ? trip_ptr[r] : 0, q1 = trip_ptr != nullptr ? trip_ptr[r + 1] : 0;
  if (threadIdx.x == 0) {
    int n = 0;
    for (int q = q0; q < q1 && n + 4 <= FEAT_MAX_TERMS; ++q) {
      const int b = trip_ids[q];
      for (int k = 0; k < 4; ++k) {
        const int c = br_col[4 * b + k];
        if (c >= 0 && c < n_in) {
          s_c[n] = c;
          s_v[n] = br_val[4 * b + k];
          ++n;
        }
      }
    }
    s_n = n;
  }
  __syncthreads();
  const int n_terms = s_n;
  const bool overflow = (q1 - q0) * 4 > FEAT_MAX_TERMS;
  const double2* sr = sbus_rows != nullptr ? sbus_rows + (int64_t)r * n_bus : nullptr;
  const int dim = n_pvpq + n_pq;
  for (int c = threadIdx.x; c < ldx; c += blockDim.x) {
    float v = 0.f;
    if (c < n_in) {
      if (sr != nullptr && c < dim) {
        const int b = c < n_pvpq ? pvpq[c] : pq[c - n_pvpq];
        v = c < n_pvpq ? (float)(sr[b].x - sbus_base[b].x) : (float)(sr[b].y - sbus_base[b].y);
      }
      if (!overflow) {
        for (int e = 0; e < n_terms; ++e)
          if (s_c[e] == c) v += s_v[e];
      } else {
        for (int q = q0; q < q1; ++q)
          for (int k = 0; k < 4; ++k)
            if (br_col[4 * trip_ids[q] + k] == c) v += br_val[4 * trip_ids[q] + k];
      }
      v = (v - x_mean[c]) / x_std[c];
    }
    xr[c] = __float2bfloat16(v);
  }
}

// First layer of the network for rows whose inputs have no injection part
// (sbus_rows NULL in features_kernel: outage rows at the base injections).
// Such a row's standardised input differs from the constant row
// xb_c = bf16((0 - mean_c) / std_c) only in the columns its tripped branches
// reach, so X W0^T = base + sum over those columns of
// (bf16(xs_c) - xb_c) W0[:, c], with base = xb W0^T (first_layer_base_kernel,
// once per set of weights) and W0T = W0^T [k0 x h] (coalesced over the
// outputs).  The column values are summed as features_kernel sums them.  A
// row with more than FEAT_MAX_TERMS contributions computes its full input
// row in shared memory and the whole dot product instead.  pre [rows_pad x
// ldp] fp32 (0 in the padding rows, as the GEMM of zero rows gives).
__global__ void sparse_first_layer_kernel(const float* __restrict__ base, const __nv_bfloat16* __restrict__ w0t,
                                          int h, const int* __restrict__ trip_ptr, const int* __restrict__ trip_ids,
                                          const int* __restrict__ br_col, const float* __restrict__ br_val,
                                          const float* __restrict__ x_mean, const float* __restrict__ x_std,
                                          int n_in, float* __restrict__ pre, int ldp, int rows) {
  extern __shared__ float s_x[];  // [n_in]: overflow rows only
  __shared__ int s_c[FEAT_MAX_TERMS];
  __shared__ float s_d[FEAT_MAX_TERMS];
  __shared__ int s_n;
  const int r = blockIdx.x;
  float* pr = pre + (int64_t)r * ldp;
  if (r >= rows) {
    for (int n = threadIdx.x; n < h; n += blockDim.x) pr[n] = 0.f;
    return;
  }
  const int q0 = trip_ptr[r], q1 = trip_ptr[r + 1];
  const bool overflow = (q1 - q0) * 4 > FEAT_MAX_TERMS;
  if (overflow) {
    // the row's full standardised input (features_kernel's overflow form)
    for (int c = threadIdx.x; c < n_in; c += blockDim.x) {
      float v = 0.f;
      for (int q = q0; q < q1; ++q)
        for (int k = 0; k < 4; ++k)
          if (br_col[4 * trip_ids[q] + k] == c) v += br_val[4 * trip_ids[q] + k];
      s_x[c] = __bfloat162float(__float2bfloat16((v - x_mean[c]) / x_std[c]));
    }
    __syncthreads();
    for (int n = threadIdx.x; n < h; n += blockDim.x) {
      float acc = 0.f;
      for (int c = 0; c < n_in; ++c) acc = fmaf(s_x[c], __bfloat162float(w0t[(int64_t)c * h + n]), acc);
      pr[n] = acc;
    }
    return;
  }
  if (threadIdx.x == 0) {
    int n = 0;
    for (int q = q0; q < q1; ++q) {
      const int b = trip_ids[q];
      for (int k = 0; k < 4; ++k) {
        const int c = br_col[4 * b + k];
        if (c < 0 || c >= n_in) continue;
        int e = 0;
        while (e < n && s_c[e] != c) ++e;
        if (e == n) {
          s_c[n] = c;
          s_d[n] = 0.f;
          ++n;
        }
        s_d[e] += br_val[4 * b + k];
      }
    }
    for (int e = 0; e < n; ++e) {
      const int c = s_c[e];
      const float xs = __bfloat162float(__float2bfloat16((s_d[e] - x_mean[c]) / x_std[c]));
      const float xb = __bfloat162float(__float2bfloat16((0.f - x_mean[c]) / x_std[c]));
      s_d[e] = xs - xb;
    }
    s_n = n;
  }
  __syncthreads();
  const int nt = s_n;
  for (int n = threadIdx.x; n < h; n += blockDim.x) {
    float acc = base[n];
    for (int e = 0; e < nt; ++e) acc = fmaf(s_d[e], __bfloat162float(w0t[(int64_t)s_c[e] * h + n]), acc);
    pr[n] = acc;
  }
}

// base[n] = sum_c bf16((0 - mean_c) / std_c) W0T[c][n] over the n_in input
// columns (one thread per output, fp32).
__global__ void first_layer_base_kernel(const __nv_bfloat16* __restrict__ w0t, int h,
                                        const float* __restrict__ x_mean, const float* __restrict__ x_std, int n_in,
                                        float* __restrict__ base) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= h) return;
  float acc = 0.f;
  for (int c = 0; c < n_in; ++c)
    acc = fmaf(__bfloat162float(__float2bfloat16((0.f - x_mean[c]) / x_std[c])),
               __bfloat162float(w0t[(int64_t)c * h + n]), acc);
  base[n] = acc;
}

inline int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 148 * 32) b = 148 * 32;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace mlp
}  // namespace gs2g

// ------------------------------------------------------------ C-ABI
// Status: 0 ok, 1 invalid argument, 3 CUDA error (see include/gs2g.h).
namespace gs2g {
void set_last_error(const char* msg);  // session.cpp
}
namespace {
using namespace gs2g::mlp;
int status_of(cudaError_t e) {
  if (e == cudaSuccess) return 0;
  gs2g::set_last_error(cudaGetErrorString(e));
  return e == cudaErrorInvalidValue ? 1 : 3;
}
int invalid(const char* what) {
  gs2g::set_last_error(what);
  return 1;
}

// 256 columns per block, rows over at most 148 * 8 blocks in all
dim3 col_grid(int rows, int cols) {
  const int gx = (cols + 255) / 256;
  int gy = (148 * 8 + gx - 1) / gx;
  if (gy > rows) gy = rows;
  return dim3(gx, gy < 1 ? 1 : gy);
}

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 148;
  return n > 0 ? n : 148;
}

// The tensor map of one GEMM operand with `rows` M or N indices: K-major
// X[i][k] in boxes of 64 k x box rows, MN-major X[k][i] in boxes of 64 i x 64 k;
// what lies past the matrix reads as zero.
bool operand_map(CUtensorMap* map, const void* p, int ld, bool mn, int rows, int K, int box) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Encode>(f);
  }();
  if (encode == nullptr) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)(mn ? rows : K), (cuuint64_t)(mn ? K : rows)};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t boxes[2] = {64u, (cuuint32_t)(mn ? 64 : box)}, ones[2] = {1u, 1u};
  const auto run = [&] {
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, boxes, ones,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = run();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // a thread's first CUDA call: the runtime binds its context with its first
    // launch or here, the driver's encoder does not
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = run();
  }
  return r == CUDA_SUCCESS;
}

template <int BN, bool A_MN, bool B_MN, int OP>
cudaError_t launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, const GemmShape& g, const Epilogue& e, int* err,
                        void* stream) {
  cudaError_t rc = cudaFuncSetAttribute(gemm_bf16_kernel<BN, A_MN, B_MN, OP>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem<BN>());
  if (rc != cudaSuccess) return rc;
  const int tiles = g.tiles_m * g.tiles_n * g.splits, n_sm = sm_count();
  gemm_bf16_kernel<BN, A_MN, B_MN, OP><<<tiles < n_sm ? tiles : n_sm, GEMM_THREADS, gemm_smem<BN>(),
                                         (cudaStream_t)stream>>>(ma, mb, g, e, err);
  return cudaGetLastError();
}

// The network's own combinations of layout and epilogue have kernels of their
// own; any other pair runs with the operation looked up per element.
template <int BN>
cudaError_t launch_gemm_any(bool a_mn, bool b_mn, const CUtensorMap& ma, const CUtensorMap& mb, const GemmShape& g,
                            const Epilogue& e, int* err, void* stream) {
  if (!a_mn && !b_mn && e.op == EPI_GELU) return launch_gemm<BN, false, false, EPI_GELU>(ma, mb, g, e, err, stream);
  if (!a_mn && !b_mn && e.op == EPI_BIAS) return launch_gemm<BN, false, false, EPI_BIAS>(ma, mb, g, e, err, stream);
  if (!a_mn && !b_mn && e.op == EPI_STORE) return launch_gemm<BN, false, false, EPI_STORE>(ma, mb, g, e, err, stream);
  if (a_mn && b_mn && e.op == EPI_STORE) return launch_gemm<BN, true, true, EPI_STORE>(ma, mb, g, e, err, stream);
  if (!a_mn && b_mn && e.op == EPI_GELU_BWD)
    return launch_gemm<BN, false, true, EPI_GELU_BWD>(ma, mb, g, e, err, stream);
  if (a_mn)
    return b_mn ? launch_gemm<BN, true, true, EPI_ANY>(ma, mb, g, e, err, stream)
                : launch_gemm<BN, true, false, EPI_ANY>(ma, mb, g, e, err, stream);
  return b_mn ? launch_gemm<BN, false, true, EPI_ANY>(ma, mb, g, e, err, stream)
              : launch_gemm<BN, false, false, EPI_ANY>(ma, mb, g, e, err, stream);
}
}  // namespace

extern "C" {

int64_t gs2g_mlp_gemm_part(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || M % GT || N % GT || K % GK) return 0;
  const GemmPlan p = gemm_plan(M, N, K, sm_count(), true);
  return p.splits > 1 ? (int64_t)p.splits * M * N : 0;
}

int gs2g_mlp_gemm(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, int M, int N, int K, int op,
                  int accumulate, float* D, int ldd, const float* bias, void* act_bf16, int ld_act, float* part,
                  int64_t part_elems, int* err, void* stream) {
  if (M % GT || N % GT || K % GK || M <= 0 || N <= 0 || K <= 0)
    return invalid("gemm: M, N must be positive multiples of 128 and K of 64");
  if (lda % 8 || ldb % 8 || lda < (a_mn ? M : K) || ldb < (b_mn ? N : K) || !err)
    return invalid("gemm: leading dimensions must cover the rows and be 16-byte multiples");
  if (((uintptr_t)A | (uintptr_t)B) & 15) return invalid("gemm: operands must be 16-byte aligned");
  if (op < EPI_STORE || op > EPI_GELU_BWD || (!D && op != EPI_GELU) || (D && ldd < N) ||
      ((op == EPI_BIAS || op == EPI_GELU) && !bias) || ((op == EPI_GELU || op == EPI_GELU_BWD) && (!act_bf16 || ld_act < N)))
    return invalid("gemm: the epilogue's buffers are missing or too narrow");
  GemmPlan p = gemm_plan(M, N, K, sm_count(), part != nullptr);
  if (p.splits > 1 && part_elems < (int64_t)p.splits * M * N) p = gemm_plan(M, N, K, sm_count(), false);
  GemmShape g{M, N, K / GK, M / GT, (N + p.bn - 1) / p.bn, p.splits, p.kt_split, part};
  const Epilogue e{op, accumulate, D, ldd, bias, (__nv_bfloat16*)act_bf16, ld_act};
  CUtensorMap ma, mb;
  if (!operand_map(&ma, A, lda, a_mn, M, K, GT) || !operand_map(&mb, B, ldb, b_mn, N, K, p.bn)) {
    gs2g::set_last_error("gemm: the driver rejected a tensor map");
    return 3;
  }
  cudaError_t rc = p.bn == 256 ? launch_gemm_any<256>(a_mn != 0, b_mn != 0, ma, mb, g, e, err, stream)
                               : launch_gemm_any<128>(a_mn != 0, b_mn != 0, ma, mb, g, e, err, stream);
  if (rc == cudaSuccess && g.splits > 1) {
    const dim3 grid((N + 255) / 256, M < 512 ? M : 512);
    cudaStream_t st = (cudaStream_t)stream;
    if (op == EPI_GELU) finish_kernel<EPI_GELU><<<grid, 256, 0, st>>>(g, e);
    else if (op == EPI_GELU_BWD) finish_kernel<EPI_GELU_BWD><<<grid, 256, 0, st>>>(g, e);
    else finish_kernel<EPI_ANY><<<grid, 256, 0, st>>>(g, e);
    rc = cudaGetLastError();
  }
  return status_of(rc);
}

int gs2g_mlp_gemm_tn_bf16(const void* A, int lda, const void* B, int ldb, float* D, int ldd, int M, int N, int K,
                          int accumulate, int* err, void* stream) {
  if (ldd % 4 || ((uintptr_t)D & 15)) return invalid("gemm_tn_bf16: D must be 16-byte aligned with 16-byte row steps");
  return gs2g_mlp_gemm(A, lda, 0, B, ldb, 0, M, N, K, EPI_STORE, accumulate, D, ldd, nullptr, nullptr, 0, nullptr, 0,
                       err, stream);
}

int gs2g_mlp_bias_act(float* pre, int ldp, const float* bias, void* act_bf16, int lda, int rows, int cols, int gelu,
                      void* stream) {
  const int64_t n = (int64_t)rows * cols;
  if (n <= 0) return n < 0 ? invalid("bias_act: negative size") : 0;
  bias_act_kernel<<<col_grid(rows, cols), 256, 0, (cudaStream_t)stream>>>(pre, ldp, bias, (__nv_bfloat16*)act_bf16,
                                                                          lda, rows, cols, gelu);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_gelu_bwd(const float* dact, int ldg, const float* pre, int ldp, void* dpre_bf16, int ldo, int rows,
                      int cols, void* stream) {
  const int64_t n = (int64_t)rows * cols;
  if (n <= 0) return n < 0 ? invalid("gelu_bwd: negative size") : 0;
  gelu_bwd_kernel<<<col_grid(rows, cols), 256, 0, (cudaStream_t)stream>>>(dact, ldg, pre, ldp,
                                                                          (__nv_bfloat16*)dpre_bf16, ldo, rows, cols);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_mse_grad(const float* y, const float* t, int ld, void* dy_bf16, int rows, int cols, int cols_valid,
                      float scale, float* loss, void* stream) {
  const int64_t n = (int64_t)rows * cols;
  if (n == 0) return 0;
  if (n < 0 || ld != cols || cols_valid > cols) return invalid("mse_grad: ld must equal cols >= cols_valid");
  mse_grad_kernel<<<col_grid(rows, cols), 256, 0, (cudaStream_t)stream>>>(y, t, ld, (__nv_bfloat16*)dy_bf16, rows,
                                                                          cols, cols_valid, scale, loss);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_colsum_bf16(const void* x, int ld, int rows, int cols, float* out, void* stream) {
  if (cols == 0) return 0;
  if (cols < 0 || rows < 0) return invalid("colsum: negative size");
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(float) * (size_t)cols, (cudaStream_t)stream);
  if (e != cudaSuccess || rows == 0) return status_of(e);
  dim3 grid((cols + 127) / 128, (rows + COLSUM_ROWS - 1) / COLSUM_ROWS);
  colsum_bf16_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, ld, rows, cols, out);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_transpose_bf16(const void* in, int ldi, void* out, int ldo, int rows, int cols, void* stream) {
  if (rows < 0 || cols < 0) return invalid("transpose: negative size");
  if (rows == 0 || cols == 0) return 0;
  dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
  transpose_bf16_kernel<<<grid, block, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, ldi, (__nv_bfloat16*)out,
                                                                  ldo, rows, cols);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_to_bf16(const float* in, void* out, int64_t n, void* stream) {
  if (n <= 0) return n < 0 ? invalid("to_bf16: negative size") : 0;
  f32_to_bf16_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(in, (__nv_bfloat16*)out, n);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_adam(float* w, const float* g, float* m, float* v, void* w_bf16, int64_t n, float lr, float beta1,
                  float beta2, float eps, int step, float weight_decay, void* stream) {
  if (n == 0) return 0;
  if (n < 0 || step < 1) return invalid("adam: negative size or step < 1");
  float c1 = 1.f, c2 = 1.f;
  for (int i = 0; i < step; ++i) {
    c1 *= beta1;
    c2 *= beta2;
  }
  adam_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, (__nv_bfloat16*)w_bf16, n, lr, beta1,
                                                                  beta2, eps, 1.f - c1, 1.f - c2, weight_decay);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_features(const double* sbus_rows, const double* sbus_base, const int* pvpq, int n_pvpq, const int* pq,
                      int n_pq, const int* trip_ptr, const int* trip_ids, const int* br_col, const float* br_val,
                      const float* x_mean, const float* x_std, int n_in, void* x_bf16, int ldx, int rows,
                      int rows_pad, int n_bus, void* stream) {
  if (rows < 0 || rows_pad < rows || n_in < 0 || ldx < n_in || n_bus <= 0 || n_pvpq < 0 || n_pq < 0 || !x_bf16 ||
      !x_mean || !x_std || !sbus_base || (trip_ptr && (!trip_ids || !br_col || !br_val)))
    return invalid("features: bad arguments");
  if (rows_pad == 0) return 0;
  gs2g::mlp::features_kernel<<<rows_pad, 256, 0, (cudaStream_t)stream>>>(
      (const double2*)sbus_rows, (const double2*)sbus_base, pvpq, n_pvpq, pq, n_pq, trip_ptr, trip_ids, br_col,
      br_val, x_mean, x_std, n_in, (__nv_bfloat16*)x_bf16, ldx, rows, n_bus);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_first_layer_base(const void* w0t_bf16, int h, const float* x_mean, const float* x_std, int n_in,
                              float* base, void* stream) {
  if (h <= 0 || n_in < 0 || !w0t_bf16 || !x_mean || !x_std || !base) return invalid("first_layer_base: bad arguments");
  gs2g::mlp::first_layer_base_kernel<<<(h + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)w0t_bf16, h, x_mean, x_std, n_in, base);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_sparse_first_layer(const float* base, const void* w0t_bf16, int h, const int* trip_ptr,
                                const int* trip_ids, const int* br_col, const float* br_val, const float* x_mean,
                                const float* x_std, int n_in, float* pre, int ldp, int rows, int rows_pad,
                                void* stream) {
  if (h <= 0 || ldp < h || rows < 0 || rows_pad < rows || n_in < 0 || !base || !w0t_bf16 || !trip_ptr ||
      !trip_ids || !br_col || !br_val || !x_mean || !x_std || !pre)
    return invalid("sparse_first_layer: bad arguments");
  if (rows_pad == 0) return 0;
  const int smem = n_in * (int)sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(gs2g::mlp::sparse_first_layer_kernel,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return status_of(e);
  }
  gs2g::mlp::sparse_first_layer_kernel<<<rows_pad, 256, smem, (cudaStream_t)stream>>>(
      base, (const __nv_bfloat16*)w0t_bf16, h, trip_ptr, trip_ids, br_col, br_val, x_mean, x_std, n_in, pre, ldp,
      rows);
  return status_of(cudaGetLastError());
}

int gs2g_mlp_start_voltages(const float* y, int ldy, const float* y_mean, const float* y_std, const int* va_index,
                            const int* vm_index, const double* vinit, int n_bus, double* v0, int rows, void* stream) {
  if (rows < 0 || n_bus <= 0) return invalid("start_voltages: bad sizes");
  const int64_t n = (int64_t)rows * n_bus;
  if (n == 0) return 0;
  start_voltages_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
      y, ldy, y_mean, y_std, va_index, vm_index, (const double2*)vinit, n_bus, (double2*)v0, rows);
  return status_of(cudaGetLastError());
}

// ---- whole passes of the network, one call each

static int net_ok(const gs2g_mlp_net* n, const char* what) {
  if (!n || n->layers < 1 || n->rows <= 0 || n->rows % GT || n->k0 % GT || n->h % GT || n->o % GT || !n->w_off ||
      !n->b_off || !n->wb || !n->master || !n->act || !n->y || !n->err)
    return invalid(what);
  return 0;
}

int gs2g_mlp_net_forward(const gs2g_mlp_net* n, int first, void* stream) {
  if (int rc = net_ok(n, "net_forward: bad network")) return rc;
  const size_t bh = (size_t)n->rows * n->h;
  for (int l = first; l <= n->layers; ++l) {
    const int in = l == 0 ? n->k0 : n->h, out = l == n->layers ? n->o : n->h;
    const void* a = l == 0 ? n->x : (const void*)((const __nv_bfloat16*)n->act + (l - 1) * bh);
    const void* w = (const __nv_bfloat16*)n->wb + n->w_off[l];
    const float* b = n->master + n->b_off[l];
    const bool last = l == n->layers;
    const int rc = gs2g_mlp_gemm(a, l == 0 ? n->ldx : in, 0, w, in, 0, n->rows, out, in, last ? EPI_BIAS : EPI_GELU, 0,
                                 last ? n->y : (n->pre && (l == 0 || n->dy) ? n->pre + l * bh : nullptr), out, b,
                                 last ? nullptr : (void*)((__nv_bfloat16*)n->act + l * bh), out, n->part,
                                 n->part_elems, n->err, stream);
    if (rc) return rc;
  }
  return 0;
}

int gs2g_mlp_net_backward(const gs2g_mlp_net* n, const float* t, int n_out, float scale, void* stream) {
  if (int rc = net_ok(n, "net_backward: bad network")) return rc;
  if (!n->pre || !n->grad || !n->dy || !n->g || !t || !n->loss) return invalid("net_backward: training buffers missing");
  const size_t bh = (size_t)n->rows * n->h;
  int rc = gs2g_mlp_mse_grad(n->y, t, n->o, n->dy, n->rows, n->o, n_out, scale, n->loss, stream);
  const __nv_bfloat16* g = (const __nv_bfloat16*)n->dy;
  for (int l = n->layers; l >= 0 && !rc; --l) {
    const int in = l == 0 ? n->k0 : n->h, out = l == n->layers ? n->o : n->h;
    const void* a = l == 0 ? n->x : (const void*)((const __nv_bfloat16*)n->act + (l - 1) * bh);
    // dW = g^T a over the batch rows, both operands as they lie
    rc = gs2g_mlp_gemm(g, out, 1, a, l == 0 ? n->ldx : in, 1, out, in, n->rows, EPI_STORE, 0, n->grad + n->w_off[l], in,
                       nullptr, nullptr, 0, n->part, n->part_elems, n->err, stream);
    if (!rc) rc = gs2g_mlp_colsum_bf16(g, out, n->rows, out, n->grad + n->b_off[l], stream);
    if (l > 0 && !rc) {
      // the layer below's g = (g W) gelu', into the buffer g is not in
      __nv_bfloat16* nxt = (__nv_bfloat16*)n->g + ((l - 1) & 1) * bh;
      rc = gs2g_mlp_gemm(g, out, 0, (const __nv_bfloat16*)n->wb + n->w_off[l], in, 1, n->rows, in, out, EPI_GELU_BWD, 0,
                         n->pre + (l - 1) * bh, in, nullptr, nxt, in, n->part, n->part_elems, n->err, stream);
      g = nxt;
    }
  }
  return rc;
}

}  // extern "C"
