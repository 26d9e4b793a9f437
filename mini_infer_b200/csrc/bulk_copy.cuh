// Bulk copies into rings of shared memory: mbarriers with bounded waits, TMA loads with an L2 policy, tensor maps.  For
// libraries whose blocks are fed by the copy engine.
#pragma once

#include "common.cuh"

#include <cuda.h>

#define SPIN_LIMIT (1 << 22)

static __device__ int g_own_status;
// Where a give-up is reported: this library's own word above, or a word the host shares among
// its kernel libraries (mi_set_status_word) so that one small copy per step tells it about all.
static __device__ int* g_status_word;
#define MI_MAX_DEVICES 64
static int* g_status_word_host[MI_MAX_DEVICES];
__device__ __forceinline__ void report_give_up() { atomicExch(g_status_word ? g_status_word : &g_own_status, 1); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* give_up, int limit = SPIN_LIMIT) {
  for (int it = 0; it < limit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 1023) == 1023 && *give_up) return false;   // another role of this block gave up
  }
  report_give_up();
  *give_up = 1;
  return false;
}

// After a wait that ran out: whether the copy lands all the same within some ms.
__device__ __forceinline__ bool mbar_drain(uint64_t* bar, uint32_t parity) {
  uint32_t landed = 0;
  for (int it = 0; it < (1 << 18) && !landed; ++it)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(landed)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
  return landed != 0;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// The same loads with an L2 eviction policy.  Weights are read once per step and are far larger
// than the L2, so they are marked to be evicted first: what the step's kernels hand to one another
// (activations, the residual stream, partial tiles) then stays resident between them.
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ void tma_load_2d_hint(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, "
      "%4}], [%2], %5;\n" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_hint(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, "
      "%4, %5}], [%2], %6;\n" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}

// Report give-ups of this library's kernels on the current device into `device_word` (an int in device memory that the caller
// owns and keeps alive; null: back to the library's own word); NAME(reset): non-zero when a block gave up a bounded wait since
// the last reset (synchronises the device).
#define MI_DEFINE_STATUS_API(NAME)                                                                                    \
  extern "C" int mi_set_status_word(int* device_word) {                                                               \
    int dev = -1;                                                                                                     \
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MI_MAX_DEVICES) MI_REFUSE("status word: bad device"); \
    cudaError_t e = cudaMemcpyToSymbol(g_status_word, &device_word, sizeof(int*));                                    \
    if (e != cudaSuccess) return (int)e;                                                                              \
    g_status_word_host[dev] = device_word;                                                                            \
    return 0;                                                                                                         \
  }                                                                                                                   \
  extern "C" int NAME(int reset) {                                                                                    \
    int dev = -1, v = 0;                                                                                              \
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MI_MAX_DEVICES) return -1;                            \
    int* word = g_status_word_host[dev];                                                                              \
    if (!word && cudaGetSymbolAddress((void**)&word, g_own_status) != cudaSuccess) return -1;                         \
    if (cudaMemcpy(&v, word, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;                          \
    if (reset && v) cudaMemset(word, 0, sizeof(int));                                                                 \
    return v;                                                                                                         \
  }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}
