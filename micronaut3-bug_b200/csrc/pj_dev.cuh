/*
 * pj_dev.cuh — device primitives every kernel of the library uses: warp and block scans, the look-back words, bulk
 * asynchronous copies between global and shared memory (cp.async.bulk, the untiled TMA form) and their mbarriers.
 */
#ifndef PJ_DEV_CUH
#define PJ_DEV_CUH

#include <cuda_runtime.h>
#include <stdint.h>

namespace pj {

/* ---- scans ------------------------------------------------------------------------------------------ */
template <class T>
__device__ __forceinline__ T warp_incl_scan(T v) {
  const unsigned lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    T u = __shfl_up_sync(0xFFFFFFFFu, v, d);
    if (lane >= (unsigned)d) v += u;
  }
  return v;
}
/* Exclusive prefix of v over the block (any multiple of 32 threads up to 1024); *total = block sum.
 * `sh` needs 33 entries. Safe to call repeatedly. */
template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T* total, T* sh) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  T inc = warp_incl_scan(v);
  __syncthreads(); /* protect sh from the previous call */
  if (lane == 31) sh[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nwarps ? sh[lane] : T(0);
    T wi = warp_incl_scan(w);
    if (lane < nwarps) sh[lane] = wi - w;
    if (lane == nwarps - 1) sh[32] = wi;
  }
  __syncthreads();
  *total = sh[32];
  return sh[warp] + inc - v;
}

/* ---- words other blocks read while this kernel runs: 32-bit values next to a valid bit, written once --------------- */
static constexpr unsigned long long TS_VALID = 1ull << 63;
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

/* ---- bulk asynchronous copy (TMA, untiled form) global -> shared, completion on an mbarrier ------------ */
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
/* dst and src 16-byte aligned, bytes a multiple of 16; no multicast: the copy lands in this block's own shared memory */
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)), "l"(src),
               "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
/* bounded: false when the copy has not landed after limit_ns */
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, uint32_t parity, unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (;;) {
    if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) return false;
    __nanosleep(64);
  }
}

/* bulk asynchronous copy shared -> global (same alignment rules); the issuing thread waits until shared memory
 * has been read before the block may leave */
__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_s2g_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
/* makes this thread's earlier writes to shared memory visible to the asynchronous proxy (the bulk copy engine) */
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

}  // namespace pj
#endif
