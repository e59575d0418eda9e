// Shared helpers of the kernels: element types, conversions, warp and block reductions, and the
// status convention of the C interface (0 = launched, otherwise a cudaError_t or a negative code
// of this library).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define LLM_EXPORT extern "C" __attribute__((visibility("default")))

// negative status codes of this library (positive ones are cudaError_t values)
#define LLM_ERR_UNSUPPORTED (-1)   // a size or dtype the kernel refuses
#define LLM_ERR_ARGUMENT (-2)      // inconsistent arguments

enum LlmDtype : int { LLM_F32 = 0, LLM_BF16 = 1 };

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f32<bf16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over a block of up to 1024 threads; every thread gets the result.  `scratch` holds 33 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nwarps ? scratch[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

// The lowest key position that a query at position p sees, for the one integer by which every
// attention kernel is told its mask.  window > 0: the last `window` keys (sliding window).
// window < 0: the keys of the query's own chunk of -window positions, chunks counted from
// position 0 of the sequence.  window == 0: every earlier key.  Non-decreasing in p.
__host__ __device__ __forceinline__ int first_key(int p, int window) {
  if (window > 0) return p + 1 > window ? p + 1 - window : 0;
  if (window < 0) return p - p % (-window);
  return 0;
}

// ---- mbarriers (shared by the kernels that move data with the TMA unit)
constexpr long long WAIT_CYCLES = 4000000000LL;   // bound of every wait: about two seconds

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// Bounded wait for the phase with the given parity.  mbarrier.try_wait parks the thread until the
// phase completes or a hardware time limit passes, so waking up costs no polling delay; the loop
// around it gives up after WAIT_CYCLES clock cycles (about two seconds).  Returns false then.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit = WAIT_CYCLES) {
  const uint32_t addr = smem_u32(bar);
  long long start = 0;
  for (uint32_t i = 0;; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (i == 0) start = clock64();
    else if (clock64() - start > limit) return false;
  }
}
static inline int launch_status() { return (int)cudaGetLastError(); }

// Programmatic dependent launch.  A kernel that starts with pdl_trigger() lets the next kernel
// of the stream be scheduled as soon as all of its own blocks have started; that next kernel may
// do work that does not depend on earlier kernels (fetching weights, setting up barriers) and
// must call pdl_wait() before it touches anything an earlier kernel wrote or still reads.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

extern int g_llm_pdl;   // 1: launch with the programmatic-serialization attribute (llm_set_pdl)
// 1: the last kernel this library launched was the rotation kernel (rope_kv.cu).  The product on
// CTA pairs honours it: it is then launched without the programmatic attribute, i.e. only after
// the rotation kernel has finished.  A measurement once ran the sequence "rotation kernel of 2,048
// rows, then directly the CTA-pair product as its programmatic dependent" (no model has it: the
// attention kernel always comes between them) and it stopped making progress in two of three
// tries, with no bounded wait having given up; reading the kernels did not show why.  The
// sequence is therefore not launched that way by anyone, a part registered by a user included.
extern int g_llm_after_rotation;

// What the rotation kernel does for the reason above, for any kernel of many blocks that stands
// directly in front of a product of many rows: called behind its launch, it makes a CTA-pair
// product that follows wait for the kernel's end instead of starting as its programmatic
// dependent.  (The chains of the first models are proven as they are and do not call it.)
static inline int launched_many_blocks(int rc, long long blocks) {
  if (blocks >= 512) g_llm_after_rotation = 1;
  return rc;
}

// 1: the next launch starts in plain stream order, whatever g_llm_pdl says (then 0 again).  A
// kernel that is launched as a programmatic dependent becomes resident as soon as the kernel before
// it allows it and waits there for that kernel's end.  Behind a kernel that runs for a millisecond
// with fewer than two warps per scheduler (the walk of a recurrence over a prompt) the waiting
// blocks cost the walk half of its rate (measured: 1,345 us against 607 us for the delta rule over
// 2,048 tokens), so such a kernel asks for a plain launch of whatever follows it.
extern int g_llm_next_plain;
static inline void next_launch_plain() { g_llm_next_plain = 1; }

// Launch a kernel that calls pdl_wait() itself.
template <typename... KArgs, typename... Args>
static inline int launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, Args... args) {
  g_llm_after_rotation = 0;
  const int plain = g_llm_next_plain;
  g_llm_next_plain = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_llm_pdl && !plain ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// The walk of a thread over [rows][n4] pieces of four columns, a stride of the whole grid at a time:
// f(piece, column piece).  The column is carried along: the remainder of a 64-bit index by a width that
// is known at run time costs more than a pass over 32-bit values has time for.
template <typename F>
__device__ __forceinline__ void for_each_piece(unsigned total4, unsigned n4, F f) {
  const unsigned stride = gridDim.x * blockDim.x, wrap = stride % n4;
  unsigned i = blockIdx.x * blockDim.x + threadIdx.x, c = i % n4;
  for (; i < total4; i += stride) {
    f(i, c);
    c += wrap;
    if (c >= n4) c -= n4;
  }
}
// whether a contiguous matrix of `total` values, n to a row, goes by pieces of four
static inline bool in_pieces(long long total, int n, const void* a, const void* b) {
  return n % 4 == 0 && (((uintptr_t)a | (uintptr_t)b) & 15) == 0 && total / 4 < (1LL << 31);
}
static inline int piece_blocks(long long total) {
  const long long want = (total / 4 + 255) / 256;
  return (int)(want < 148 * 8 ? want : 148 * 8);
}
