// C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores with float32 accumulation.
//
// This is the matrix product of the true 32-bit path (no tensor-core mode of any
// kind) and the any-size product of the bfloat16 path (sizes the tcgen05 kernel
// refuses).  Every element of C accumulates k = 0..K-1 in the same order for any M,
// so a row's result does not depend on what else is in the batch.  The reference's
// float32 product (kernel/Gemm/Gemm_f32.h:18-141) reads past M and needs K % 16 == 0;
// this one guards every access and takes any M, N, K.
#include "common.cuh"
#include "warp_mma.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, THREADS = 256;

template <typename T, int VEC>
__device__ __forceinline__ void load_k(const T* __restrict__ row, int k, int K, bool row_ok, float (&v)[4]) {
  if (VEC == 4) {
    if (row_ok && k + 3 < K) {
      if (sizeof(T) == 4) {
        const float4 f = *reinterpret_cast<const float4*>(row + k);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
        const uint2 u = *reinterpret_cast<const uint2*>(row + k);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x);
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
        v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
      }
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (row_ok && k + i < K) ? to_f32(row[k + i]) : 0.f;
}

template <typename T, typename TC, int VEC>
__global__ void __launch_bounds__(THREADS)
gemm_simt_kernel(const T* __restrict__ A, const T* __restrict__ W, TC* __restrict__ C, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, long long a_batch, long long w_batch, long long c_batch,
                 const T* __restrict__ gate, long long gate_stride) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  pdl_launch_dependents();      // let the next kernel start its own prologue now
  pdl_wait();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // blockIdx.z: one of several products of the same sizes (the heads of a per-head projection)
  A += (size_t)blockIdx.z * a_batch;
  W += (size_t)blockIdx.z * w_batch;
  C += (size_t)blockIdx.z * c_batch;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;
  const int ty = tid >> 4, tx = tid & 15;
  const bool a_ok = m0 + lrow < M, w_ok = n0 + lrow < N;
  const T* a_row = A + (size_t)(a_ok ? m0 + lrow : 0) * lda;
  const T* w_row = W + (size_t)(w_ok ? n0 + lrow : 0) * ldw;

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    float av[4], wv[4];
    load_k<T, VEC>(a_row, k0 + lk, K, a_ok, av);
    load_k<T, VEC>(w_row, k0 + lk, K, w_ok, wv);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      As[lk + i][lrow] = av[i];
      Ws[lk + i][lrow] = wv[i];
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][ty * TM]);
      const float4 w4 = *reinterpret_cast<const float4*>(&Ws[kk][tx * TN]);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w};
      const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
    // a gate per (row, product): the row's results are multiplied by sigmoid(gate[m, z])
    const float g = gate ? 1.f / (1.f + expf(-to_f32(gate[(size_t)m * gate_stride + blockIdx.z]))) : 1.f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(gate ? acc[i][j] * g : acc[i][j]);
    }
  }
}

// Products too small for the tiles above to fill the chip (float32, 16-byte pieces): tiles of 16 x 32, the whole of K (in blocks of 128, two of
// them in flight) asked for at once instead of 16 k at a time behind two barriers.  Each element is one chain of multiply-adds over k = 0..K-1,
// as above, so that a product's bits do not depend on which of the two kernels made it.  The weights of the first blocks are asked for
// before the kernel waits.  Both are bound by latency at these sizes, and a 64 x 64 tile on one SM also takes 4 us of multiply-adds at K = 256:
// in the steps of a model of width 96 (feed-forward 256, up to 100 rows) a launch took 8.2 us with the large tiles, 3.0 us with these.
constexpr int SBM = 16, SBN = 32, SBK = 128, SPITCH = SBK + 4;

__global__ void __launch_bounds__(128)
gemm_simt_small_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, long long lda,
                       long long ldw, long long ldc, long long a_batch, long long w_batch, long long c_batch,
                       const float* __restrict__ gate, long long gate_stride) {
  extern __shared__ __align__(16) float tiles[];          // [2][SBM + SBN][SPITCH]
  pdl_launch_dependents();
  const int tid = threadIdx.x, m0 = blockIdx.y * SBM, n0 = blockIdx.x * SBN;
  A += (size_t)blockIdx.z * a_batch;
  W += (size_t)blockIdx.z * w_batch;
  C += (size_t)blockIdx.z * c_batch;
  // a thread copies its 16 bytes (four k) of every fourth row; rows past the end give results that nobody stores
  const int copy_k = (tid & 31) * 4, copy_row = tid >> 5;
  auto copy = [&](int block, const float* src, long long ld, int rows, int row0, int first, int last) {
    const int k = block * SBK + copy_k;
    if (k >= K) return;
    float* dst = tiles + ((size_t)(block & 1) * (SBM + SBN) + first) * SPITCH + copy_k;
    for (int r = copy_row; r < last; r += 4)
      if (row0 + r < rows) cp_async16(dst + r * SPITCH, src + (size_t)(row0 + r) * ld + k);
  };
  auto commit = []() { asm volatile("cp.async.commit_group;" ::: "memory"); };
  const int blocks = (K + SBK - 1) / SBK;
  copy(0, W, ldw, N, n0, SBM, SBN);
  if (blocks > 1) copy(1, W, ldw, N, n0, SBM, SBN);
  pdl_wait();
  copy(0, A, lda, M, m0, 0, SBM);
  commit();
  if (blocks > 1) copy(1, A, lda, M, m0, 0, SBM);
  commit();
  const int m = (tid >> 4) * 2, n = tid & 15;              // this thread's elements: rows m, m + 1, columns n, n + 16
  float acc[2][2] = {};
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float* a = tiles + ((size_t)(b & 1) * (SBM + SBN) + m) * SPITCH;
    const float* w = tiles + ((size_t)(b & 1) * (SBM + SBN) + SBM + n) * SPITCH;
    const int here = min(SBK, K - b * SBK);
#pragma unroll 4
    for (int k = 0; k < here; k += 4) {
      float x[2][4], y[2][4];
      Vec4<float>::load(a + k, x[0]); Vec4<float>::load(a + SPITCH + k, x[1]);
      Vec4<float>::load(w + k, y[0]); Vec4<float>::load(w + 16 * SPITCH + k, y[1]);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) acc[i][j] = fmaf(x[i][kk], y[j][kk], acc[i][j]);
    }
    if (b + 2 < blocks) {
      __syncthreads();
      copy(b + 2, W, ldw, N, n0, SBM, SBN);
      copy(b + 2, A, lda, M, m0, 0, SBM);
    }
    commit();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (m0 + m + i >= M) continue;
    const float g = gate ? 1.f / (1.f + expf(-gate[(size_t)(m0 + m + i) * gate_stride + blockIdx.z])) : 1.f;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (n0 + n + 16 * j < N) C[(size_t)(m0 + m + i) * ldc + n0 + n + 16 * j] = gate ? acc[i][j] * g : acc[i][j];
  }
}

template <typename T, typename TC>
int launch(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw,
           long long ldc, cudaStream_t stream, int batches = 1, long long a_batch = 0, long long w_batch = 0,
           long long c_batch = 0, const void* gate = nullptr, long long gate_stride = 0) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batches);
  const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && (a_batch % 4 == 0) && (w_batch % 4 == 0) &&
                   ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
  if constexpr (sizeof(T) == 4 && sizeof(TC) == 4) {
    // the small tiles while the large ones would leave more than half of the SMs idle
    if (vec && (long long)grid.x * grid.y * grid.z * 2 <= llmk_sm_count()) {
      const size_t smem = 2 * (SBM + SBN) * SPITCH * sizeof(float);
      cudaError_t e = cudaFuncSetAttribute(gemm_simt_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return llmk_fail((int)e, "gemm_simt: %s", cudaGetErrorString(e));
      launch_kernel(gemm_simt_small_kernel, dim3((N + SBN - 1) / SBN, (M + SBM - 1) / SBM, batches), dim3(128), smem, stream, (const float*)A,
                    (const float*)W, (float*)C, M, N, K, lda, ldw, ldc, a_batch, w_batch, c_batch, (const float*)gate, gate_stride);
      LLMK_LAUNCH_CHECK("gemm_simt_small");
    }
  }
  if (vec)
    launch_kernel(gemm_simt_kernel<T, TC, 4>, grid, dim3(THREADS), 0, stream, (const T*)A, (const T*)W, (TC*)C, M, N, K, lda, ldw, ldc,
                  a_batch, w_batch, c_batch, (const T*)gate, gate_stride);
  else
    launch_kernel(gemm_simt_kernel<T, TC, 1>, grid, dim3(THREADS), 0, stream, (const T*)A, (const T*)W, (TC*)C, M, N, K, lda, ldw, ldc,
                  a_batch, w_batch, c_batch, (const T*)gate, gate_stride);
  LLMK_LAUNCH_CHECK("gemm_simt");
}

// Few rows (a decode step): one warp per (product, output column).  The warp keeps its weight row in
// registers (lane l holds k = l, l + 32, ...), dots every row of A with it and sums over the lanes in a
// fixed order; the weights are read once, as a stream.  K up to 32 * PER_LANE, which is 4, 8 or GEMV_PER_LANE.
constexpr int GEMV_PER_LANE = 20, GEMV_WARPS = 4;

template <typename T, int PER_LANE>
__global__ void __launch_bounds__(GEMV_WARPS * 32)
gemv_batched_kernel(const T* __restrict__ A, const T* __restrict__ W, T* __restrict__ C, int M, int N, int K, long long lda,
                    long long ldw, long long ldc, long long a_batch, long long w_batch, long long c_batch,
                    const T* __restrict__ gate, long long gate_stride) {
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * GEMV_WARPS + warp, z = blockIdx.y;
  if (n >= N) return;
  const T* w_row = W + (size_t)z * w_batch + (size_t)n * ldw;
  float wr[PER_LANE];
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int k = lane + 32 * i;
    wr[i] = k < K ? to_f32(w_row[k]) : 0.f;          // the weights do not depend on the kernel before
  }
  pdl_wait();
  for (int m = 0; m < M; ++m) {
    const T* a_row = A + (size_t)m * lda + (size_t)z * a_batch;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int k = lane + 32 * i;
      if (k < K) s = fmaf(to_f32(a_row[k]), wr[i], s);
    }
    s = warp_sum(s);
    if (lane == 0) {
      if (gate) s *= 1.f / (1.f + expf(-to_f32(gate[(size_t)m * gate_stride + z])));
      C[(size_t)m * ldc + (size_t)z * c_batch + n] = from_f32<T>(s);
    }
  }
}

// The same on warp-level MMAs, for K and rows on the 8-grid: a warp makes 8 columns of 16 rows, the weights (8 rows of W) asked for before
// the wait, then all of the rows' 128 columns in one go.  The four lanes of a group take 8 neighbouring k each, of rows and weights alike:
// 16 bytes a load, two MMAs a load, which permutes the sum's terms and nothing else.  A row after the other, as above, is a chain of a
// load, products and five shuffles per row: 16 heads of 128 x 128, 16 rows, inside a decode step 10.6 us a launch, this way 3.6 us.
constexpr int HEADS_WARPS = 4, HEADS_GROUPS = 4;

__global__ void __launch_bounds__(HEADS_WARPS * 32)
heads_mma_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ C, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, long long a_batch, long long w_batch, long long c_batch,
                 const __nv_bfloat16* __restrict__ gate, long long gate_stride) {
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, quad = lane & 3;
  const int n0 = (blockIdx.x * HEADS_WARPS + warp) * 8, z = blockIdx.y, m0 = blockIdx.z * 16 + row, m1 = m0 + 8;
  const bool has_n = n0 + row < N;
  const __nv_bfloat16* w_row = W + (size_t)z * w_batch + (size_t)(has_n ? n0 + row : 0) * ldw;
  const __nv_bfloat16* a0 = A + (size_t)min(m0, M - 1) * lda + (size_t)z * a_batch;
  const __nv_bfloat16* a1 = A + (size_t)min(m1, M - 1) * lda + (size_t)z * a_batch;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 w[HEADS_GROUPS];
  auto load_w = [&](int k0) {
#pragma unroll
    for (int j = 0; j < HEADS_GROUPS; ++j) {
      const int k = k0 + 32 * j + 8 * quad;
      w[j] = has_n && k < K ? *reinterpret_cast<const uint4*>(w_row + k) : zero;
    }
  };
  load_w(0);
  pdl_wait();
  float c[2][4] = {};
  for (int k0 = 0; k0 < K; k0 += 32 * HEADS_GROUPS) {
    if (k0) load_w(k0);
    uint4 x[HEADS_GROUPS], y[HEADS_GROUPS];
#pragma unroll
    for (int j = 0; j < HEADS_GROUPS; ++j) {
      const int k = k0 + 32 * j + 8 * quad;
      x[j] = m0 < M && k < K ? *reinterpret_cast<const uint4*>(a0 + k) : zero;
      y[j] = m1 < M && k < K ? *reinterpret_cast<const uint4*>(a1 + k) : zero;
    }
#pragma unroll
    for (int j = 0; j < HEADS_GROUPS; ++j) {
      const uint32_t lo[4] = {x[j].x, y[j].x, x[j].y, y[j].y}, hi[4] = {x[j].z, y[j].z, x[j].w, y[j].w};
      mma(c[0], lo, w[j].x, w[j].y);
      mma(c[1], hi, w[j].z, w[j].w);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int m = h ? m1 : m0;
    if (m >= M) continue;
    const float g = gate ? 1.f / (1.f + expf(-to_f32(gate[(size_t)m * gate_stride + z]))) : 1.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int n = n0 + quad * 2 + i;
      if (n < N) C[(size_t)m * ldc + (size_t)z * c_batch + n] = from_f32<__nv_bfloat16>((c[0][2 * h + i] + c[1][2 * h + i]) * g);
    }
  }
}

}  // namespace

// in_dtype: element kind of A and W; out_dtype: element kind of C (float32 or the same as in_dtype).
LLMK_API int llmk_gemm_simt(const void* A, const void* W, void* C, int M, int N, int K, long long lda,
                            long long ldw, long long ldc, int in_dtype, int out_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  LLMK_REQUIRE(K > 0 && lda >= K && ldw >= K && ldc >= N, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
  LLMK_REQUIRE((M + BM - 1) / BM <= 65535, "gemm_simt: M=%d exceeds the grid limit", M);
  if (in_dtype == LLMK_F32 && out_dtype == LLMK_F32) return launch<float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (in_dtype == LLMK_BF16 && out_dtype == LLMK_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (in_dtype == LLMK_BF16 && out_dtype == LLMK_F32)
    return launch<__nv_bfloat16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  return llmk_fail(-1, "gemm_simt: unsupported element kinds in=%d out=%d", in_dtype, out_dtype);
}

// `batches` products of the same sizes in one launch: product z reads A + z * a_batch, W + z * w_batch
// and writes C + z * c_batch (strides in elements).  With a gate ([M, gate_stride] of the input kind),
// row m of product z is multiplied by sigmoid(gate[m, z]).  The per-head projections of a latent
// attention are such a batch: the columns of one head in, the columns of one head out.
LLMK_API int llmk_gemm_simt_batched(const void* A, const void* W, void* C, int M, int N, int K, long long lda,
                                    long long ldw, long long ldc, int batches, long long a_batch, long long w_batch,
                                    long long c_batch, const void* gate, long long gate_stride, int dtype,
                                    cudaStream_t stream) {
  if (M == 0 || N == 0 || batches == 0) return 0;
  LLMK_REQUIRE(K > 0 && lda >= K && ldw >= K && ldc >= N, "gemm_simt_batched: bad sizes M=%d N=%d K=%d", M, N, K);
  LLMK_REQUIRE((M + BM - 1) / BM <= 65535 && batches <= 65535, "gemm_simt_batched: M=%d or %d batches exceed the grid limit", M, batches);
  if (dtype == LLMK_F32) return launch<float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream, batches, a_batch, w_batch, c_batch, gate, gate_stride);
  if (dtype == LLMK_BF16 && M <= 24 && K <= 32 * GEMV_PER_LANE) {
    // a decode step in bfloat16: the weights as a stream, one warp per output column (float32 keeps the tiled
    // kernel at every row count, so that its sums never depend on how many rows a step brings)
    using T = __nv_bfloat16;
    if (K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && a_batch % 8 == 0 && w_batch % 8 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0) {
      launch_kernel(heads_mma_kernel, dim3((N + 8 * HEADS_WARPS - 1) / (8 * HEADS_WARPS), batches, (M + 15) / 16), dim3(HEADS_WARPS * 32), 0, stream,
                    (const T*)A, (const T*)W, (T*)C, M, N, K, lda, ldw, ldc, a_batch, w_batch, c_batch, (const T*)gate, gate_stride);
      LLMK_LAUNCH_CHECK("heads_mma");
    }
    auto kern = K <= 128 ? gemv_batched_kernel<T, 4> : K <= 256 ? gemv_batched_kernel<T, 8> : gemv_batched_kernel<T, GEMV_PER_LANE>;
    launch_kernel(kern, dim3((N + GEMV_WARPS - 1) / GEMV_WARPS, batches), dim3(GEMV_WARPS * 32), 0, stream,
                  (const T*)A, (const T*)W, (T*)C, M, N, K, lda, ldw, ldc, a_batch, w_batch, c_batch, (const T*)gate, gate_stride);
    LLMK_LAUNCH_CHECK("gemv_batched");
  }
  if (dtype == LLMK_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16>(A, W, C, M, N, K, lda, ldw, ldc, stream, batches, a_batch, w_batch, c_batch, gate, gate_stride);
  return llmk_fail(-1, "gemm_simt_batched: unsupported element kind %d", dtype);
}
