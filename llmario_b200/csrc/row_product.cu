// Products of one to four rows with a small weight matrix (a step of few requests through a small
// model):  out[r][n] (=|+=) sum_k h[r][k] * W[n][k],  bfloat16 W, 32-bit sums, in which h is given in
// bfloat16 or is the RMS norm of 32-bit rows (made here: no kernel of its own), and a gated form
// silu(gate) * up with gate and up rows interleaved in blocks of 16.
//
// What bounds such a step is not its bytes (Qwen3-0.6B sizes: 31 MB a layer, 5 us) but its chain
// of kernels, each of which waits for the one before it.  On tcgen05 (gemm_tcgen05.cu) a link is a
// TMA load of the rows, MMAs, the accumulator's way through tensor memory and shared memory, and a
// TMA reduction into the output: 3.5 to 6.5 us, with 2 us for the norm in front.  Here the matrix is
// cut into one slice of rows per SM, which is in shared memory, brought by bulk copies, before the
// wait on the kernel ahead ends; what is left behind that wait is to read the rows of h (a few KB
// that every warp keeps in registers, so that no barrier follows), the dot products from shared
// memory, five shuffles and a store: 2.6 to 4.5 us with the norm inside, a decode step of one request
// (28 layers of Qwen3-0.6B sizes) 935 -> 698 us.  No atomics: an output is one warp's sum.
// Limits: K up to 3,072 for one row and up to 2,048 for two, so that the rows fit a warp's registers
// beside a second CTA, and slices of at most 100 KB, so that the slices of two kernels of the chain fit
// an SM and the next one's copies overlap this one's work.  All else, up to four rows of up to 4,096,
// keeps h in shared memory, a warp per row making it, behind one barrier: a step of three or four
// requests (14 layers) 507 -> 478 us.  So does the norm of two rows, which every warp would make for
// both.  Links of a chain K -> K, in shared memory -> in registers, K 512 / 1,024 / 1,536 / 2,048 / 2,560: one
// row's norm 2.9 / 3.5 / 5.0 / 5.8 / 8.2 -> 2.3 / 2.9 / 3.7 / 4.3 / 5.7 us, one row 1.9 / 2.5 / 4.5 / 5.0 / 7.2
// -> 1.3 / 1.6 / 2.5 / 3.0 / 4.0, two rows' norm 2.8 / 3.2 / 4.8 / 5.3 / 8.3 -> 3.0 / 3.8 / 5.5 / 9.1 / -, two rows
// - / 2.5 / - / 4.9 / - -> - / 1.9 / - / 3.4 / -.  With room for eight rows the dot products took longer than the
// chain saved (six or eight requests: 511 -> 631 us), so those stay on tcgen05.
#include "common.cuh"

namespace {
constexpr int RP_WARPS = 8, RP_ROWS = 4;       // warps; weight rows a warp multiplies at a time
// most bytes of a slice; of a slice and h, so that two CTAs fit an SM (two rows of up to 2,048: 16 KB beside
// any slice)
constexpr int RP_SLICE = 100 * 1024, RP_SHARED = 112 * 1024, RP_SHARED_2 = RP_SLICE + 16 * 1024;
constexpr int RP_MAX = 4;                      // rows
enum RowMode : int { ROW_STORE = 0, ROW_ADD = 1, ROW_GATED = 2 };

__device__ __forceinline__ void bulk_load(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem)),
               "l"(gmem), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// The halves of a pair as 32-bit numbers.  (volatile: otherwise the compiler unpacks all of h once in
// front of the loop over the outputs, which takes twice the registers)
__device__ __forceinline__ float low_half(uint32_t v) {
  uint32_t r;
  asm volatile("shl.b32 %0, %1, 16;" : "=r"(r) : "r"(v));
  return __uint_as_float(r);
}
__device__ __forceinline__ float high_half(uint32_t v) {
  uint32_t r;
  asm volatile("and.b32 %0, %1, 0xffff0000;" : "=r"(r) : "r"(v));
  return __uint_as_float(r);
}

// KC: K / 256; R: rows; NORM: h is the norm of 32-bit rows.  A CTA has the `per` outputs from
// per * blockIdx.x on.
template <int KC, int R, int MODE, bool NORM>
__global__ void __launch_bounds__(RP_WARPS * 32, 2)
    row_product_kernel(const void* __restrict__ x, int ldx, const float* __restrict__ norm_w, float eps,
                       const bf16* __restrict__ W, void* __restrict__ out, int ldc, int N, int per,
                       int* __restrict__ status) {
  constexpr int K = KC * 256;
  extern __shared__ __align__(128) uint8_t rp_raw[];
  bf16* w_s = reinterpret_cast<bf16*>(rp_raw);
  __shared__ __align__(8) uint64_t full;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * per, cnt = min(per, N - n0);
  if (tid == 0) {
    mbar_init(&full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();
  if (tid == 0 && cnt > 0) {
    // the weights do not depend on earlier kernels
    mbar_expect_tx(&full, (uint32_t)cnt * (MODE == ROW_GATED ? 2 : 1) * K * 2);
    if (MODE != ROW_GATED) {
      bulk_load(w_s, W + (size_t)n0 * K, (uint32_t)cnt * K * 2, &full);
    } else {
      for (int f = 0; f < cnt;) {      // runs inside a block of 16 features: gate rows first, then up rows
        const int at = n0 + f, run = min(16 - (at & 15), cnt - f);
        const bf16* gate = W + (size_t)((at >> 4) * 32 + (at & 15)) * K;
        bulk_load(w_s + (size_t)f * K, gate, (uint32_t)run * K * 2, &full);
        bulk_load(w_s + (size_t)(cnt + f) * K, gate + (size_t)16 * K, (uint32_t)run * K * 2, &full);
        f += run;
      }
    }
  }
  pdl_wait();
  if (cnt <= 0) return;
  // ---- the rows, pairs of bfloat16: lane values k = 256 c + 8 lane + e (128 registers a thread, so
  // that a CTA of the next kernel finds room beside this one)
  uint32_t h[R][KC][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (NORM) {
      const float* xr = (const float*)x + (size_t)r * ldx + lane * 8;
      float ss = 0.f;
#pragma unroll
      for (int c = 0; c < KC; ++c) {
        const float4 a = *reinterpret_cast<const float4*>(xr + c * 256);
        const float4 b = *reinterpret_cast<const float4*>(xr + c * 256 + 4);
        ss = fmaf(a.x, a.x, ss), ss = fmaf(a.y, a.y, ss), ss = fmaf(a.z, a.z, ss), ss = fmaf(a.w, a.w, ss);
        ss = fmaf(b.x, b.x, ss), ss = fmaf(b.y, b.y, ss), ss = fmaf(b.z, b.z, ss), ss = fmaf(b.w, b.w, ss);
      }
      const float scale = 1.0f / sqrtf(warp_sum(ss) / (float)K + eps);
#pragma unroll
      for (int c = 0; c < KC; ++c) {
        float v[8], w[8];
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(xr + c * 256);
        *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(xr + c * 256 + 4);
        *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(norm_w + c * 256 + lane * 8);
        *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(norm_w + c * 256 + lane * 8 + 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 two = __floats2bfloat162_rn(v[2 * e] * scale * w[2 * e], v[2 * e + 1] * scale * w[2 * e + 1]);
          h[r][c][e] = *reinterpret_cast<const uint32_t*>(&two);
        }
      }
    } else {
      const bf16* xr = (const bf16*)x + (size_t)r * ldx + lane * 8;
#pragma unroll
      for (int c = 0; c < KC; ++c) {
        const uint4 a = *reinterpret_cast<const uint4*>(xr + c * 256);
        h[r][c][0] = a.x, h[r][c][1] = a.y, h[r][c][2] = a.z, h[r][c][3] = a.w;
      }
    }
  }
  // (the wait for the copies is bounded; a warp that gives up leaves, nothing waits for it)
  if (!mbar_wait(&full, 0)) {
    if (lane == 0) atomicExch(status, 7);
    return;
  }
  // ---- the outputs: a warp takes RP_ROWS weight rows at a time (gated: two features)
  constexpr int OUTS = MODE == ROW_GATED ? RP_ROWS / 2 : RP_ROWS;
  for (int i0 = warp * OUTS; i0 < cnt; i0 += RP_WARPS * OUTS) {
    // lane r * OUTS + o finishes row r of output o
    const int my_o = i0 + (lane & (OUTS - 1)), my_r = lane / OUTS;
    const bool mine = my_o < cnt && my_r < R;
    float old = 0.f;
    if (MODE == ROW_ADD && mine) old = ((const float*)out)[(size_t)my_r * ldc + n0 + my_o];
    const uint4* wr[RP_ROWS];
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      const int o = min(i0 + (j % OUTS), cnt - 1) + (j / OUTS) * cnt;      // (gated: the up rows behind the gate rows)
      wr[j] = reinterpret_cast<const uint4*>(w_s + (size_t)o * K) + lane;
    }
    float acc[RP_ROWS][R];
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[j][r] = 0.f;
#pragma unroll
    for (int c = 0; c < KC; ++c) {
      uint4 v[RP_ROWS];
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j) v[j] = wr[j][c * 32];
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float h_lo = low_half(h[r][c][e]), h_hi = high_half(h[r][c][e]);
#pragma unroll
          for (int j = 0; j < RP_ROWS; ++j) {
            const uint32_t u = e == 0 ? v[j].x : e == 1 ? v[j].y : e == 2 ? v[j].z : v[j].w;
            acc[j][r] = fmaf(h_lo, __uint_as_float(u << 16), acc[j][r]);
            acc[j][r] = fmaf(h_hi, __uint_as_float(u & 0xffff0000u), acc[j][r]);
          }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[j][r] += __shfl_xor_sync(0xffffffffu, acc[j][r], o);
    float val = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int o = 0; o < OUTS; ++o)
        if (lane == r * OUTS + o) {
          if (MODE == ROW_GATED) {
            const float g = acc[o][r], u = acc[OUTS + o < RP_ROWS ? OUTS + o : 0][r];
            val = __fdividef(g, 1.0f + __expf(-g)) * u;
          } else {
            val = acc[o][r];
          }
        }
    if (mine) {
      if (MODE == ROW_GATED) ((bf16*)out)[(size_t)my_r * ldc + n0 + my_o] = from_f32<bf16>(val);
      else ((float*)out)[(size_t)my_r * ldc + n0 + my_o] = MODE == ROW_ADD ? old + val : val;
    }
  }
}

// The same for more values of h: the rows lie in shared memory, up to RP_MAX of them (those that are
// not there are summed from whatever lies there and not written).
template <int MODE, bool NORM>
__global__ void __launch_bounds__(RP_WARPS * 32, 2)
    row_product_shared_kernel(const void* __restrict__ x, int ldx, const float* __restrict__ norm_w, float eps,
                              const bf16* __restrict__ W, void* __restrict__ out, int ldc, int rows, int N, int K, int per,
                              int* __restrict__ status) {
  constexpr int R = RP_MAX;
  extern __shared__ __align__(128) uint8_t rp_raw[];
  bf16* h_s = reinterpret_cast<bf16*>(rp_raw);            // [R][K]
  bf16* w_s = h_s + (size_t)R * K;
  __shared__ __align__(8) uint64_t full;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * per, cnt = min(per, N - n0), chunks = K >> 8;
  if (tid == 0) {
    mbar_init(&full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();
  if (tid == 0 && cnt > 0) {
    mbar_expect_tx(&full, (uint32_t)cnt * (MODE == ROW_GATED ? 2 : 1) * K * 2);
    if (MODE != ROW_GATED) {
      bulk_load(w_s, W + (size_t)n0 * K, (uint32_t)cnt * K * 2, &full);
    } else {
      for (int f = 0; f < cnt;) {
        const int at = n0 + f, run = min(16 - (at & 15), cnt - f);
        const bf16* gate = W + (size_t)((at >> 4) * 32 + (at & 15)) * K;
        bulk_load(w_s + (size_t)f * K, gate, (uint32_t)run * K * 2, &full);
        bulk_load(w_s + (size_t)(cnt + f) * K, gate + (size_t)16 * K, (uint32_t)run * K * 2, &full);
        f += run;
      }
    }
  }
  pdl_wait();
  if (cnt <= 0) return;
  // a warp makes a row
  if (warp < rows) {
    uint4* dst = reinterpret_cast<uint4*>(h_s + (size_t)warp * K) + lane;
    if (NORM) {
      const float* xr = (const float*)x + (size_t)warp * ldx + lane * 8;
      float ss = 0.f;
#pragma unroll 4
      for (int c = 0; c < chunks; ++c) {
        const float4 a = *reinterpret_cast<const float4*>(xr + c * 256);
        const float4 b = *reinterpret_cast<const float4*>(xr + c * 256 + 4);
        ss = fmaf(a.x, a.x, ss), ss = fmaf(a.y, a.y, ss), ss = fmaf(a.z, a.z, ss), ss = fmaf(a.w, a.w, ss);
        ss = fmaf(b.x, b.x, ss), ss = fmaf(b.y, b.y, ss), ss = fmaf(b.z, b.z, ss), ss = fmaf(b.w, b.w, ss);
      }
      const float scale = 1.0f / sqrtf(warp_sum(ss) / (float)K + eps);
#pragma unroll 4
      for (int c = 0; c < chunks; ++c) {
        float v[8], w[8];
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(xr + c * 256);
        *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(xr + c * 256 + 4);
        *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(norm_w + c * 256 + lane * 8);
        *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(norm_w + c * 256 + lane * 8 + 4);
        uint32_t two[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * e] * scale * w[2 * e], v[2 * e + 1] * scale * w[2 * e + 1]);
          two[e] = *reinterpret_cast<const uint32_t*>(&t);
        }
        dst[c * 32] = make_uint4(two[0], two[1], two[2], two[3]);
      }
    } else {
      const uint4* src = reinterpret_cast<const uint4*>((const bf16*)x + (size_t)warp * ldx) + lane;
#pragma unroll 4
      for (int c = 0; c < chunks; ++c) dst[c * 32] = src[c * 32];
    }
  }
  __syncthreads();
  if (!mbar_wait(&full, 0)) {
    if (lane == 0) atomicExch(status, 7);
    return;
  }
  constexpr int OUTS = MODE == ROW_GATED ? RP_ROWS / 2 : RP_ROWS, VALUES = RP_ROWS * R;
  const uint4* hr = reinterpret_cast<const uint4*>(h_s) + lane;
  for (int i0 = warp * OUTS; i0 < cnt; i0 += RP_WARPS * OUTS) {
    // value j * R + r, weight row j with row r, ends up in the lane of that number
    const int my_v = lane & (VALUES - 1), my_j = my_v / R, my_r = my_v % R, my_o = i0 + my_j;
    const bool mine = lane < OUTS * R && my_o < cnt && my_r < rows;
    float old = 0.f;
    if (MODE == ROW_ADD && mine) old = ((const float*)out)[(size_t)my_r * ldc + n0 + my_o];
    const uint4* wr[RP_ROWS];
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      const int o = min(i0 + (j % OUTS), cnt - 1) + (j / OUTS) * cnt;
      wr[j] = reinterpret_cast<const uint4*>(w_s + (size_t)o * K) + lane;
    }
    float acc[VALUES];
#pragma unroll
    for (int i = 0; i < VALUES; ++i) acc[i] = 0.f;
    for (int c = 0; c < chunks; ++c) {
      float w[RP_ROWS][8];
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j) {
        const uint4 v = wr[j][c * 32];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) w[j][2 * e] = __uint_as_float(u[e] << 16), w[j][2 * e + 1] = __uint_as_float(u[e] & 0xffff0000u);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint4 v = hr[(size_t)r * (K / 8) + c * 32];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float lo = __uint_as_float(u[e] << 16), hi = __uint_as_float(u[e] & 0xffff0000u);
#pragma unroll
          for (int j = 0; j < RP_ROWS; ++j) {
            acc[j * R + r] = fmaf(lo, w[j][2 * e], acc[j * R + r]);
            acc[j * R + r] = fmaf(hi, w[j][2 * e + 1], acc[j * R + r]);
          }
        }
      }
    }
    static_assert(VALUES == 16, "the two halves of a warp are summed first");
#pragma unroll
    for (int i = 0; i < VALUES; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
#pragma unroll
    for (int half = VALUES / 2; half > 0; half >>= 1) {
      const bool hi = (lane & half) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float send = hi ? acc[i] : acc[i + half], keep = hi ? acc[i + half] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
      }
    }
    float val = acc[0];
    if (MODE == ROW_GATED) {
      const float up = __shfl_down_sync(0xffffffffu, val, OUTS * R);
      val = __fdividef(val, 1.0f + __expf(-val)) * up;
    }
    if (mine) {
      if (MODE == ROW_GATED) ((bf16*)out)[(size_t)my_r * ldc + n0 + my_o] = from_f32<bf16>(val);
      else ((float*)out)[(size_t)my_r * ldc + n0 + my_o] = MODE == ROW_ADD ? old + val : val;
    }
  }
}

int rp_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    n = v > 0 ? v : 148;
  }
  return n;
}

template <int KC, int R, int MODE, bool NORM>
int rp_launch(const void* x, int ldx, const float* norm_w, float eps, const void* W, void* out, int ldc, int N, int per,
              int* status, cudaStream_t stream) {
  auto kernel = row_product_kernel<KC, R, MODE, NORM>;
  const int smem = per * (MODE == ROW_GATED ? 2 : 1) * KC * 256 * 2;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RP_SLICE);
  if (e != cudaSuccess) return (int)e;
  return launch_pdl(kernel, (N + per - 1) / per, RP_WARPS * 32, smem, stream, x, ldx, norm_w, eps, (const bf16*)W, out,
                    ldc, N, per, status);
}

template <int KC, int R>
int rp_mode(const void* x, int ldx, const float* norm_w, float eps, const void* W, void* out, int ldc, int N, int per,
            int mode, int* status, cudaStream_t stream) {
#define RP(M)                                                                                                       \
  do {                                                                                                              \
    if (!norm_w) return rp_launch<KC, R, M, false>(x, ldx, norm_w, eps, W, out, ldc, N, per, status, stream);       \
    if constexpr (R == 1) return rp_launch<KC, R, M, true>(x, ldx, norm_w, eps, W, out, ldc, N, per, status, stream); \
    return LLM_ERR_UNSUPPORTED;                                                                                     \
  } while (0)
  if (mode == ROW_STORE) RP(ROW_STORE);
  if (mode == ROW_ADD) RP(ROW_ADD);
  RP(ROW_GATED);
#undef RP
}
int rp_shared(const void* x, int ldx, const float* norm_w, float eps, const void* W, void* out, int ldc, int rows, int N,
              int K, int per, int mode, int* status, cudaStream_t stream) {
  const int smem = (RP_MAX * K + per * (mode == ROW_GATED ? 2 : 1) * K) * 2;
  auto go = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RP_SHARED_2);
    if (e != cudaSuccess) return (int)e;
    return launch_pdl(kernel, (N + per - 1) / per, RP_WARPS * 32, smem, stream, x, ldx, norm_w, eps, (const bf16*)W, out,
                      ldc, rows, N, K, per, status);
  };
  if (mode == ROW_STORE) return norm_w ? go(row_product_shared_kernel<ROW_STORE, true>) : go(row_product_shared_kernel<ROW_STORE, false>);
  if (mode == ROW_ADD) return norm_w ? go(row_product_shared_kernel<ROW_ADD, true>) : go(row_product_shared_kernel<ROW_ADD, false>);
  return norm_w ? go(row_product_shared_kernel<ROW_GATED, true>) : go(row_product_shared_kernel<ROW_GATED, false>);
}

// whether the rows go to a warp's registers
bool rp_in_registers(int rows, int K, bool norm) { return (rows == 1 && K <= 3072) || (rows == 2 && K <= 2048 && !norm); }
}  // namespace

// Whether llm_row_product takes these sizes: rows x K values of h in registers or in shared memory, N
// (gated: features) outputs whose weights fit the SMs' slices.
LLM_EXPORT int llm_row_product_ok(int rows, int N, int K, int gated) {
  if (rows < 1 || rows > RP_MAX || N < 1 || K < 256 || K > 4096 || K % 256) return 0;
  const int per = (N + rp_sm_count() - 1) / rp_sm_count();
  const long long slice = (long long)per * (gated ? 2 : 1) * K * 2;
  if (slice > RP_SLICE) return 0;
  return rp_in_registers(rows, K, false) || slice + RP_MAX * K * 2 <= RP_SHARED;
}

// mode 0: out f32 = h W^T; 1: out f32 += h W^T; 2: out bf16 = silu(gate) * up, W interleaved, N features
// (a multiple of 16).  norm_w null: x is h in bfloat16; else x is 32-bit and h its RMS norm, rounded to
// bfloat16.  W [N (gated: 2 N)][K] without gaps; x, W and norm_w on 16-byte boundaries.
LLM_EXPORT int llm_row_product(const void* x, int ldx, const float* norm_w, float eps, const void* W, void* out, int ldc,
                               int rows, int N, int K, int mode, int* status, cudaStream_t stream) {
  if (rows <= 0 || N <= 0) return 0;
  if (mode < 0 || mode > 2) return LLM_ERR_ARGUMENT;
  if (!llm_row_product_ok(rows, N, K, mode == ROW_GATED) || (mode == ROW_GATED && N % 16)) return LLM_ERR_UNSUPPORTED;
  if ((((uintptr_t)x | (uintptr_t)W | (uintptr_t)norm_w) & 15) || ldx % (norm_w ? 4 : 8)) return LLM_ERR_UNSUPPORTED;
  const int per = (N + rp_sm_count() - 1) / rp_sm_count();
  if (!rp_in_registers(rows, K, norm_w != nullptr))
    return rp_shared(x, ldx, norm_w, eps, W, out, ldc, rows, N, K, per, mode, status, stream);
#define RP_GO(KC, R) return rp_mode<KC, R>(x, ldx, norm_w, eps, W, out, ldc, N, per, mode, status, stream)
#define RP_ROWS_1(KC) case KC * 8 + 1: RP_GO(KC, 1);
#define RP_ROWS_2(KC) case KC * 8 + 1: RP_GO(KC, 1); case KC * 8 + 2: RP_GO(KC, 2);
  switch (K / 256 * 8 + rows) {
    RP_ROWS_2(1) RP_ROWS_2(2) RP_ROWS_2(3) RP_ROWS_2(4) RP_ROWS_2(5) RP_ROWS_2(6) RP_ROWS_2(7) RP_ROWS_2(8)
    RP_ROWS_1(9) RP_ROWS_1(10) RP_ROWS_1(11) RP_ROWS_1(12)
  }
#undef RP_ROWS_1
#undef RP_ROWS_2
#undef RP_GO
  return LLM_ERR_UNSUPPORTED;
}
