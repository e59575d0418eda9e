// Plain tiled matrix product on the CUDA cores with 32-bit accumulation:
//   C[m][n] (=|+=) sum_k A[m][k] * W[n][k]        A: [M][K], W: [N][K] (row-major, "out x in")
// It is the matrix product of the true 32-bit path and the reference beside the tensor-core
// kernels.  The order of an output element's sum depends on N and K only, so a row's result does
// not depend on which other rows are in the batch.  Two kernels: 32-bit operands whose rows start
// on 16-byte boundaries go to gemm_f32_kernel, all else to gemm_simt_kernel (a sum over k in
// ascending order).
#include "common.cuh"

#include <cooperative_groups.h>

namespace {
// ---- 32-bit operands.
// Bound by the multiply-adds (a step of 211 rows through Qwen3-0.6B's matrices has 100 of them per
// weight byte that is read).  What this form does about it, against the tile of 64 x 64 with 4 x 4
// sums per thread and scalar loads that took it before (211 rows, N x K 4,096 x 1,024 / 1,024 x 2,048 /
// 6,144 x 1,024 / 1,024 x 3,072: 680 us a layer -> 225 us, 26 to 29 TFLOP/s with the padding of the last
// tile; 512 x 6,144 x 1,024 at 38 TFLOP/s, the multiply-add pipe half busy with eight warps to an SM,
// the most that the registers allow):
//   * 8 x 8 sums per thread, made as pairs: the two halves of a packed multiply-add
//     (fma.rn.f32x2) are the sums over the even and the odd k, so both operands are read from
//     shared memory as they lie in memory (no transposing, no duplicating) and 16 16-byte reads
//     feed 128 packed instructions;
//   * rows of 16 k plus a pad of 4 floats: the eight lanes that a 16-byte read serves together
//     hit different banks; four such tiles are in flight by cp.async;
//   * K is cut over the CTAs of a cluster where a matrix has few rows (1,024 rows of weights are 8
//     tiles for 148 SMs), and the parts are added through distributed shared memory in ascending
//     order.  How often it is cut depends on the weights' shape alone (f32_splits), never on the
//     rows of X, so that a row keeps its bits whatever else is in the batch.
// Rows of X: tiles of 32 to 64, whichever pads least (211 rows are four of 56, not of 64), of 16 for
// up to 16 rows (then the weights' bytes bound the product).
constexpr int F_BK = 16, F_LD = F_BK + 4, F_STAGES = 4;

__device__ __forceinline__ void f32_copy16(float* smem, const float* gmem, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(there ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// WM x WN warps; a warp is 4 x 8 lanes with TM x 8 sums each
template <int WM, int WN, int TM>
__global__ void __launch_bounds__(WM * WN * 32, 2)
    gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                    int lda, int ldw, int ldc, int k_part, int accumulate, int wide_out) {
  constexpr int THREADS = WM * WN * 32, BM_ = WM * 4 * TM, BN_ = WN * 64, ROWS = BM_ + BN_, OUT_LD = BN_ + 4;
  constexpr int STAGE = ROWS * F_LD;
  extern __shared__ __align__(16) float f_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN_;
  const int k_first = blockIdx.z * k_part, k_end = min(K, k_first + k_part);
  const int steps = k_end > k_first ? (k_end - k_first + F_BK - 1) / F_BK : 0;
  // Four threads bring a row's 16 k; a thread has the rows r + i * RPI of both operands.  Rows that do
  // not exist are cleared once in all stages and never copied, so that a copy costs a pointer's step.
  constexpr int RPI = THREADS / 4, A_IT = (BM_ + RPI - 1) / RPI, W_IT = BN_ / RPI;
  const int r = tid >> 2, kq = (tid & 3) * 4;
  int k_next = k_first + kq;
  const float* a_ptr = A + (size_t)(m0 + r) * lda + k_next;      // (formed, not read, where there is no row)
  const float* w_ptr = W + (size_t)(n0 + r) * ldw + k_next;
  const size_t a_step = (size_t)RPI * lda, w_step = (size_t)RPI * ldw;
  const int a_rows = min(M - m0, BM_) - r, w_rows = min(N - n0, BN_) - r;      // i * RPI below: there
  for (int i = 0; i < A_IT; ++i)
    if (i * RPI >= a_rows && r + i * RPI < BM_)
      for (int st = 0; st < F_STAGES; ++st)
        *reinterpret_cast<float4*>(f_smem + st * STAGE + (r + i * RPI) * F_LD + kq) = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = 0; i < W_IT; ++i)
    if (i * RPI >= w_rows)
      for (int st = 0; st < F_STAGES; ++st)
        *reinterpret_cast<float4*>(f_smem + st * STAGE + (BM_ + r + i * RPI) * F_LD + kq) = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](int step) {
    if (step < steps) {
      float* st = f_smem + (step % F_STAGES) * STAGE + r * F_LD + kq;
      const bool there = k_next < k_end;      // (else the last columns of a last step: zeros)
#pragma unroll
      for (int i = 0; i < A_IT; ++i)
        if (i * RPI < a_rows) f32_copy16(st + i * RPI * F_LD, there ? a_ptr + i * a_step : A, there);
#pragma unroll
      for (int i = 0; i < W_IT; ++i)
        if (i * RPI < w_rows) f32_copy16(st + (BM_ + i * RPI) * F_LD, there ? w_ptr + i * w_step : W, there);
      a_ptr += F_BK, w_ptr += F_BK, k_next += F_BK;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < F_STAGES - 1; ++s) fetch(s);
  const int ty = lane >> 3, tx = lane & 7, wm = warp / WN, wn = warp % WN;
  const int a_row = wm * 4 * TM + ty, w_row = wn * 64 + tx;       // this lane's rows: a_row + 4 i, w_row + 8 j
  unsigned long long acc[TM][8];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;       // (the bits of two zeros)
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(F_STAGES - 2) : "memory");
    __syncthreads();
    fetch(step + F_STAGES - 1);       // into the stage that every thread has left before the barrier
    const float* as = f_smem + (step % F_STAGES) * STAGE + a_row * F_LD;
    const float* ws = f_smem + (step % F_STAGES) * STAGE + (BM_ + w_row) * F_LD;
#pragma unroll
    for (int kk = 0; kk < F_BK; kk += 4) {
      ulonglong2 w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * F_LD + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + 4 * i * F_LD + kk);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fma_pair(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fma_pair(a.y, w[j].y, acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // the tile leaves through shared memory: whole rows to the output, or to the cluster's sum
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      f_smem[(a_row + 4 * i) * OUT_LD + w_row + 8 * j] =
          __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int parts = gridDim.z, part = blockIdx.z;
  if (parts > 1) cluster.sync();
  else __syncthreads();
  const int rows_here = BM_ / parts;      // this CTA finishes so many of the tile's rows (parts: 1, 2, 4 or 8)
  for (int idx = tid; idx < rows_here * (BN_ / 4); idx += THREADS) {
    const int tr = part * rows_here + idx / (BN_ / 4), c = (idx % (BN_ / 4)) * 4;
    const int m = m0 + tr, n = n0 + c;
    if (m >= M || n >= N) continue;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p = 0; p < parts; ++p) {
      const float* from = parts > 1 ? cluster.map_shared_rank(f_smem, p) : f_smem;
      const float4 v = *reinterpret_cast<const float4*>(from + tr * OUT_LD + c);
      if (p == 0) sum = v;
      else sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
    }
    float* dst = C + (size_t)m * ldc + n;
    if (wide_out && n + 3 < N) {
      if (accumulate) {
        const float4 old = *reinterpret_cast<const float4*>(dst);
        sum.x += old.x, sum.y += old.y, sum.z += old.z, sum.w += old.w;
      }
      *reinterpret_cast<float4*>(dst) = sum;
    } else {
      const float s[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n + e < N) dst[e] = accumulate ? dst[e] + s[e] : s[e];
    }
  }
  if (parts > 1) cluster.sync();      // (no CTA leaves while another reads its sums)
}

// CTAs along K: until the weights alone make some 128 tiles, with at least 128 of K each
int f32_splits(int N, int K) {
  const int tiles = (N + 127) / 128;
  int s = 1;
  while (s < 8 && tiles * s < 128 && K / (2 * s) >= 128) s *= 2;
  return s;
}

template <int WM, int WN, int TM>
int launch_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate,
               cudaStream_t stream) {
  constexpr int BM_ = WM * 4 * TM, BN_ = WN * 64;
  constexpr int SMEM = F_STAGES * (BM_ + BN_) * F_LD * 4;
  static_assert(SMEM >= BM_ * (BN_ + 4) * 4, "the tile of sums reuses the stages");
  static_assert(BM_ % 8 == 0, "up to eight CTAs share a tile's rows");
  const int splits = f32_splits(N, K);
  const int k_part = ((K + splits - 1) / splits + F_BK - 1) / F_BK * F_BK;
  auto kernel = gemm_f32_kernel<WM, WN, TM>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_, splits);
  cfg.blockDim = dim3(WM * WN * 32);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = splits;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int wide_out = ((uintptr_t)C & 15) == 0 && ldc % 4 == 0;
  return (int)cudaLaunchKernelEx(&cfg, kernel, A, W, C, M, N, K, lda, ldw, ldc, k_part, accumulate, wide_out);
}

// whether the operands can be read in 16-byte pieces
bool f32_wide(const void* A, const void* W, int K, int lda, int ldw) {
  return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
}

int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate,
             cudaStream_t stream) {
  if (M <= 16) return launch_f32<1, 2, 4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream);
  // the tile with the least padding, the higher one among equals; a tile's height costs as much
  // as its rows and about eight more (what it reads of the weights)
  int best = 8;
  for (int tm = 7; tm >= 4; --tm) {
    auto cost = [&](int t) { return (M + 8 * t - 1) / (8 * t) * (t + 1); };
    if (cost(tm) < cost(best)) best = tm;
  }
  switch (best) {
    case 4: return launch_f32<2, 2, 4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream);
    case 5: return launch_f32<2, 2, 5>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream);
    case 6: return launch_f32<2, 2, 6>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream);
    case 7: return launch_f32<2, 2, 7>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream);
    default: return launch_f32<2, 2, 8>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream);
  }
}

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TA, typename TW, typename TC, bool ACCUMULATE>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                        TC* __restrict__ C, int M, int N, int K,
                                                        int lda, int ldw, int ldc, long long a_batch,
                                                        long long w_batch, long long c_batch) {
  // blockIdx.z: one of several independent products (a head of a per-head map), operands a
  // fixed number of elements apart
  A += (size_t)blockIdx.z * a_batch, W += (size_t)blockIdx.z * w_batch, C += (size_t)blockIdx.z * c_batch;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  // each thread loads 4 elements of each tile per k-step: row = tid / 4, k = (tid % 4) * 4 ..
  const int lrow = tid / 4, lk = (tid % 4) * 4;
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + lk + i;
      const int m = m0 + lrow, n = n0 + lrow;
      As[lk + i][lrow] = (m < M && k < K) ? to_f32(A[(size_t)m * lda + k]) : 0.f;
      Ws[lk + i][lrow] = (n < N && k < K) ? to_f32(W[(size_t)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = Ws[k][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n >= N) continue;
      TC* c = C + (size_t)m * ldc + n;
      if (ACCUMULATE)
        *c = from_f32<TC>(to_f32(*c) + acc[i][j]);
      else
        *c = from_f32<TC>(acc[i][j]);
    }
  }
}

template <typename TA, typename TW, typename TC>
int launch(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc,
           int accumulate, cudaStream_t s, int batch = 1, long long a_batch = 0, long long w_batch = 0,
           long long c_batch = 0) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
  if (accumulate)
    gemm_simt_kernel<TA, TW, TC, true><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw,
                                                            ldc, a_batch, w_batch, c_batch);
  else
    gemm_simt_kernel<TA, TW, TC, false><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw,
                                                             ldc, a_batch, w_batch, c_batch);
  return launch_status();
}
}  // namespace

// dtypes: a, w in {f32, bf16}; c in {f32, bf16}.  accumulate: C += A W^T (C must be f32).
LLM_EXPORT int llm_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* C,
                             int c_dtype, int M, int N, int K, int lda, int ldw, int ldc,
                             int accumulate, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return LLM_ERR_ARGUMENT;
  if (accumulate && c_dtype != LLM_F32) return LLM_ERR_UNSUPPORTED;
#define GO(TA, TW, TC) return launch<TA, TW, TC>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, stream)
  if (a_dtype == LLM_F32 && w_dtype == LLM_F32 && c_dtype == LLM_F32) {
    if (f32_wide(A, W, K, lda, ldw))
      return gemm_f32((const float*)A, (const float*)W, (float*)C, M, N, K, lda, ldw, ldc, accumulate, stream);
    GO(float, float, float);
  }
  if (a_dtype == LLM_BF16 && w_dtype == LLM_BF16 && c_dtype == LLM_F32) GO(bf16, bf16, float);
  if (a_dtype == LLM_BF16 && w_dtype == LLM_BF16 && c_dtype == LLM_BF16) GO(bf16, bf16, bf16);
  if (a_dtype == LLM_BF16 && w_dtype == LLM_F32 && c_dtype == LLM_F32) GO(bf16, float, float);
  if (a_dtype == LLM_BF16 && w_dtype == LLM_F32 && c_dtype == LLM_BF16) GO(bf16, float, bf16);
  if (a_dtype == LLM_F32 && w_dtype == LLM_BF16 && c_dtype == LLM_F32) GO(float, bf16, float);
#undef GO
  return LLM_ERR_UNSUPPORTED;
}

// `batch` independent products of the same sizes in one launch: product b reads A + b * a_batch
// and W + b * w_batch and writes C + b * c_batch (elements).  Operands and result of one type.
LLM_EXPORT int llm_gemm_simt_batched(const void* A, const void* W, void* C, int dtype, int c_dtype, int M, int N,
                                     int K, int lda, int ldw, int ldc, int batch, long long a_batch,
                                     long long w_batch, long long c_batch, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K <= 0 || batch > 65535) return LLM_ERR_ARGUMENT;
#define GO(TA, TW, TC) \
  return launch<TA, TW, TC>(A, W, C, M, N, K, lda, ldw, ldc, 0, stream, batch, a_batch, w_batch, c_batch)
  if (dtype == LLM_F32 && c_dtype == LLM_F32) GO(float, float, float);
  if (dtype == LLM_BF16 && c_dtype == LLM_F32) GO(bf16, bf16, float);
  if (dtype == LLM_BF16 && c_dtype == LLM_BF16) GO(bf16, bf16, bf16);
#undef GO
  return LLM_ERR_UNSUPPORTED;
}
