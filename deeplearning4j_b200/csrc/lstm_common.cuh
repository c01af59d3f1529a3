// Device helpers shared by the LSTM sequence kernels (lstm_seq.cu, lstm_split.cu): fast cell non-linearities, bounded waits on
// counters in global memory and on mbarriers that other CTAs of a cluster arrive on, timeline stamps.
#pragma once
#include "common.cuh"

namespace dl4j {

constexpr int LS_UNITS = 16;                 // hidden units per CTA
constexpr int LS_BK = 64;                    // K elements per k-block (128 bytes, SWIZZLE_128B)

// Named barrier over the four epilogue warps (barrier 0 is __syncthreads).
__device__ __forceinline__ void epilogue_bar_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Acquire loads: once the target is seen, the other CTAs' stores that preceded their arrivals (released) are visible to this thread;
// no separate fence is needed after the wait.
__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add(unsigned int* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ bool wait_counter(const unsigned int* counter, unsigned int target, int* status) {
  if (ld_acquire_gpu(counter) >= target) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (ld_acquire_gpu(counter) < target) {
    if ((++spins & 0xff) == 0 && (clock64() - t0 > 4000000000LL || *((volatile int*)status) != 0)) {
      atomicCAS(status, 0, DL4J_ERR_TIMEOUT_PEER);
      return false;
    }
  }
  return true;
}

// Timeline of one CTA: slot `i` of step `s` receives this SM's clock.  Slots: 0 producer saw the step's grid barrier open,
// 1 producer issued the step's last load, 2..17 MMA thread saw k-block (slot - 2) land (first 16 k-blocks), 18 MMA thread
// committed the accumulator, 19 epilogue saw the accumulator, 20 after the TMEM loads, 21 after the global stores, 22 after the
// fences, 23 after the barrier arrive.
__device__ __forceinline__ void ls_stamp(long long* trace, int s, int slot) {
  if (trace != nullptr && blockIdx.x == gridDim.x / 2) trace[s * 32 + slot] = clock64();
}

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// sigmoid(x) = 0.5 tanh(x / 2) + 0.5: one special-function instruction
__device__ __forceinline__ float sigm_fast(float x) { return fmaf(0.5f, tanh_fast(0.5f * x), 0.5f); }

__device__ __forceinline__ void unpack8(const uint4& u, float* o) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
}
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return u;
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_cluster(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// release at cluster scope: the stores above are visible to the peer thread that observes this arrival with an acquire
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t remote_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (!mbar_try_wait_cluster(bar, parity)) {
    if ((++spins & 0x3ff) == 0 && (clock64() - t0 > 4000000000LL || *((volatile int*)status) != 0)) {
      atomicCAS(status, 0, code);
      return false;
    }
  }
  return true;
}
// shared memory of this CTA -> shared memory of a CTA of the cluster; the bytes are counted on that CTA's mbarrier
__device__ __forceinline__ void bulk_copy_to_cluster(uint32_t dst_cluster, uint32_t src_cta, uint32_t bytes, uint32_t bar_cluster) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster), "r"(src_cta),
               "r"(bytes), "r"(bar_cluster)
               : "memory");
}
// every thread of every CTA of the cluster
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace dl4j
