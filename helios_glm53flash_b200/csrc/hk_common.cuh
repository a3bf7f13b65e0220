// Shared host/device helpers of libhelios_b200 (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <utility>

#include "../../include/helios_b200.h"

#if defined(__CUDA_ARCH__) && !defined(__CUDA_ARCH_FEAT_SM100_ALL)
#error "libhelios_b200 is written for sm_100a only (compile with -gencode arch=compute_100a,code=sm_100a)"
#endif

#define HK_API extern "C" __attribute__((visibility("default")))

#define HK_REQUIRE(cond)                    \
  do {                                      \
    if (!(cond)) return HK_ERR_INVALID;     \
  } while (0)

#define HK_LAUNCH_CHECK()                                        \
  do {                                                           \
    if (cudaPeekAtLastError() != cudaSuccess) return HK_ERR_CUDA; \
  } while (0)

namespace hk {

constexpr int LATENT = 512;     // MLA latent width (ckv row, absorbed query row)
constexpr int IDX_DIM = 128;    // indexer head dim
constexpr int POOL = 4;         // tokens per pooled indexer key

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

inline int device_index() {
  int dev = 0;
  cudaGetDevice(&dev);
  return dev < 0 || dev >= 64 ? 0 : dev;
}
inline int sm_count(int dev = device_index()) {
  static int cached[64] = {0};
  if (!cached[dev]) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cached[dev] = n > 0 ? n : 148;
  }
  return cached[dev];
}

// ---- programmatic dependent launch ----
// The small kernels of a decode step take 2-10 us each, and a plain launch behind a running kernel adds 1-2 us to each.  They
// are launched with programmatic stream serialisation and wait (pdl_wait) before their first access to memory that an earlier
// kernel may have written or may still read: the launch itself is over when the kernel before them ends.  EVERY kernel
// launched this way executes pdl_wait() in every CTA: the wait covers the grid before it only, and the chain of waits is what
// orders a kernel behind all earlier ones.
// The small kernels of a chain (one-token prologue, cache append, layer norm, pooled keys, top-k, the merge of partials) release
// their dependents at entry (pdl_release), whatever their grid: the next kernel's CTAs are placed, set up their barriers and tensor
// memory and ask for their weights in L2 while the small one runs.  Ahead of its wait a kernel may do no more than that: it may
// not load or store anything.  MLA layer at 5,001 tokens in a graph, nothing released -> released: 1 token 35.0 -> 32.3 us, 8
// 49.7 -> 44.4, 32 65.0 -> 60.5, 256 129.5 -> 126.7; 45-layer decode at 262,144 618 -> 572 (with limits of 16 to 32 CTAs on some
// of them, 9 to 256 tokens took 1.1-1.9 us more).
// The absorbed projections of ONE row do so too (absorb_tc.cu).
// The other kernels do not: CTAs placed beside a running grid land where it left room, not evenly - the per-token KDA kernel
// behind the convolution took twice as long, scorer and attention releasing theirs cost the decode chains what the others gain, and
// KDA decode layers behind one another took 4.2 us instead of 3.9.
// Launches of many waves are plain: as programmatic dependents the convolution of 32K tokens took 495 us instead of 362.
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// cluster: CTAs of a thread-block cluster along x
template <class... P, class... A>
inline cudaError_t pdl_launch_cluster(unsigned cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  const int64_t ctas = (int64_t)grid.x * grid.y * grid.z;
  attr[0].val.programmaticStreamSerializationAllowed = ctas <= 128 || ctas <= 8 * sm_count() ? 1 : 0;   // (no part of a B200 has fewer than 16 SMs)
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <class... P, class... A>
inline cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  return pdl_launch_cluster(1, kernel, grid, block, smem, s, std::forward<A>(args)...);
}

// device word (per device) where kernels record that a bounded wait gave up; see hk_read_device_status
int* device_status_ptr(int dev = device_index());

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float bf16_bits_to_f(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ float bf16lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// packed pairs of fp32 values: two products or sums per instruction
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// 16-byte read-only load that does not allocate in L1 (streaming data touched once)
__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

}  // namespace hk
