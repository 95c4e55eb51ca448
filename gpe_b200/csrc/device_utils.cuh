// device_utils.cuh -- PTX wrappers (mbarrier, TMA tile loads), complex pair
// loads/stores and block reductions used by the GPE stage kernels.
//
// TMA: plain tile loads only (cp.async.bulk.tensor ... .tile), never the
// cluster-multicast form; every load's source is this GPU's own memory.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace gpe {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(count)
               : "memory");
}

// Make barrier initialisation visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Order earlier generic-proxy shared-memory accesses before later TMA writes
// into the same buffer.
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar,
                                                      uint32_t bytes) {
  asm volatile(
      "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
          smem_u32(bar)),
      "r"(bytes)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
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

// First statement of a kernel that is launched with launch_overlapped, by every
// thread: waits until the kernel before it has completed and its memory is
// visible, and lets the kernel behind it set up its blocks in turn.  In this
// order: a trigger before the wait would let a third kernel start while the first
// still runs, and its wait covers the second only (steps then read ghosts that
// are not filled yet).  Without the launch attribute both are no-ops.
// Such a kernel runs while the one before it still writes, so no pointer it is
// given to memory of the step (read or written) is __restrict__: the qualifier
// lets the compiler take a load for invariant and move it above this wait, which
// a memory clobber does not forbid.  Only tables that are constant since the
// context was created keep it.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// Barrier among the first `nthreads` threads (a multiple of 32) of the CTA.
__device__ __forceinline__ void named_barrier_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// try_wait that may suspend the warp for up to `hint_ns` before it gives up:
// a warp that waits long leaves its issue slots to its siblings.
__device__ __forceinline__ bool mbar_try_wait_for(uint64_t* bar, uint32_t parity,
                                                  uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}

// Wait for phase `parity` of an mbarrier, giving up after limit_ns.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar,
                                                  uint32_t parity,
                                                  uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  while (true) {
    if (mbar_try_wait_for(bar, parity, 20000u)) return true;
    if (global_timer_ns() - t0 > limit_ns) return false;
  }
}

// 3-D tiled TMA load global -> shared, completion counted on `bar`.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map,
                                            uint64_t* bar, int c0, int c1,
                                            int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::"
      "complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2),
      "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(
                   reinterpret_cast<uint64_t>(map))
               : "memory");
}

// ---------------------------------------------------------------------------
// Two consecutive complex values along x (re0, im0, re1, im1).

template <typename T>
struct Pair {
  T r0, i0, r1, i1;
};

template <typename T>
__device__ __forceinline__ Pair<T> ld_pair(const T* p);
template <>
__device__ __forceinline__ Pair<float> ld_pair<float>(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return {v.x, v.y, v.z, v.w};
}
template <>
__device__ __forceinline__ Pair<double> ld_pair<double>(const double* p) {
  const double2 a = reinterpret_cast<const double2*>(p)[0];
  const double2 b = reinterpret_cast<const double2*>(p)[1];
  return {a.x, a.y, b.x, b.y};
}

template <typename T>
__device__ __forceinline__ void st_pair(T* p, const Pair<T>& v);
template <>
__device__ __forceinline__ void st_pair<float>(float* p, const Pair<float>& v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.r0, v.i0, v.r1, v.i1);
}
template <>
__device__ __forceinline__ void st_pair<double>(double* p,
                                                const Pair<double>& v) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v.r0, v.i0);
  reinterpret_cast<double2*>(p)[1] = make_double2(v.r1, v.i1);
}

template <typename T>
__device__ __forceinline__ void st_one(T* p, T re, T im) {
  p[0] = re;
  p[1] = im;
}
template <>
__device__ __forceinline__ void st_one<float>(float* p, float re, float im) {
  *reinterpret_cast<float2*>(p) = make_float2(re, im);
}
template <>
__device__ __forceinline__ void st_one<double>(double* p, double re,
                                               double im) {
  *reinterpret_cast<double2*>(p) = make_double2(re, im);
}

template <typename TO, typename TI>
__device__ __forceinline__ Pair<TO> cvt_pair(const Pair<TI>& a) {
  return {static_cast<TO>(a.r0), static_cast<TO>(a.i0),
          static_cast<TO>(a.r1), static_cast<TO>(a.i1)};
}

// ---------------------------------------------------------------------------
// Block reductions in FP64 (fixed order => deterministic).

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Ghost layers on each side of each axis of a field that is stepped two stages at
// a time: two stages of an order-4 stencil reach 4 sites, which pair_kernel.cuh
// evaluates in one launch (the one-stage kernels read and fill the inner 2, and
// fields that only they step have 2).
constexpr int GH = 4;

// Ghost targets of interior index i along an axis of n points: the ghost
// positions within `depth` of the ends whose value is a copy of point i.
// Periodic (bcs 1): ghost g holds f(g mod n).  Reflective (bcs 2): mirror about
// the end nodes, f(-g) = f(g), f(n-1+g) = f(n-1-g).  At most two for n >= 6.
constexpr int NO_GHOST = -1000000;
__device__ __forceinline__ void ghost_targets(int i, int n, int bcs, int depth, int& g0, int& g1) {
  const int lo = bcs == 1 ? i - n : -i;              // image below 0
  const int hi = bcs == 1 ? i + n : 2 * (n - 1) - i;  // image above n - 1
  g0 = (lo < 0 && lo >= -depth && i >= 0 && i < n) ? lo : NO_GHOST;
  g1 = (hi >= n && hi < n + depth && i >= 0 && i < n) ? hi : NO_GHOST;
}

// Interior index whose value position g (-n < g < 2 n - 1) holds.
__device__ __forceinline__ int ghost_source(int g, int n, int bcs) {
  if (bcs == 1) return g < 0 ? g + n : g >= n ? g - n : g;
  return g < 0 ? -g : g >= n ? 2 * (n - 1) - g : g;
}

}  // namespace gpe
