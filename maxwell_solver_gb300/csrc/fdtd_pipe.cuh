/*
 * fdtd_pipe.cuh -- the shared pieces of the TMA pipelines (fdtd_tma.cu,
 * fdtd_fused.cu): mbarrier operations with bounded waits, bulk and tensor
 * copies into shared memory, and the host-side tensor-map encoding.
 */
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fdtd_internal.h"

namespace fdtd_pipe {

// Bounded mbarrier waits give up after kWaitNs of the global timer (2 s),
// whatever a poll costs on the GPU at hand; a poll of a phase that has not
// completed suspends the thread for a few us, so the timer is read every
// 32 polls, and a backstop of kSpinLimit polls (about 4 s at 3.8 us a
// poll, measured on GB300) ends the wait even if the timer stood still.
constexpr unsigned long long kWaitNs = 2000000000ull;
constexpr unsigned kSpinLimit = 1u << 20;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void proxy_fence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase with the given parity at most limit_ns of the global
// timer (and at most kSpinLimit polls); false when it gave up.
__device__ __forceinline__ bool mbar_wait_for(uint64_t *bar, uint32_t parity,
                                              unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
#pragma unroll 1
  for (unsigned it = 1; it < kSpinLimit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 31u) == 0u && global_ns() - t0 > limit_ns) return false;
  }
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  return mbar_wait_for(bar, parity, kWaitNs);
}

// Plain bulk copy global -> shared (16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int x, int y, int z, int c) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(c), "r"(smem_u32(bar))
      : "memory");
}

// ------------------------------------------------------------------ host

inline PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

inline int encode(CUtensorMap *out, void *base, CUtensorMapDataType dt, int esize, const fdtd_dev *d,
           int boxw, int boxh) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encoder();
  if (!enc) return (int)cudaErrorNotSupported;
  const cuuint64_t gdim[3] = {(cuuint64_t)d->I, (cuuint64_t)d->J, (cuuint64_t)d->K};
  const cuuint64_t gstride[2] = {(cuuint64_t)d->Ip * esize, (cuuint64_t)d->plane * esize};
  const cuuint32_t box[3] = {(cuuint32_t)boxw, (cuuint32_t)boxh, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(out, dt, 3, base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

// Three field arrays `stride` elements apart as one 4-D map: a box holds the
// three components' tiles one after the other.
inline int encode3(CUtensorMap *out, void *base, const fdtd_dev *d, int64_t stride, int boxw,
                   int boxh) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encoder();
  if (!enc) return (int)cudaErrorNotSupported;
  const cuuint64_t gdim[4] = {(cuuint64_t)d->I, (cuuint64_t)d->J, (cuuint64_t)d->K, 3};
  const cuuint64_t gstride[3] = {(cuuint64_t)d->Ip * 4, (cuuint64_t)d->plane * 4,
                                 (cuuint64_t)stride * 4};
  const cuuint32_t box[4] = {(cuuint32_t)boxw, (cuuint32_t)boxh, 1, 3};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, gdim, gstride, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

}  // namespace fdtd_pipe
