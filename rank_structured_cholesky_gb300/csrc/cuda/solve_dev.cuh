// Device helpers shared by the single-vector and batched solves and the fused
// Cholesky: warp reductions and bounded inter-block waits.
#pragma once
#include <cuda_runtime.h>

namespace rschol {
namespace solvedev {

constexpr unsigned FULL = 0xffffffffu;

template <class V>
__device__ __forceinline__ V warp_sum(V v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

constexpr int SPIN_LIMIT = 1 << 22;   // polls (with a short sleep) before a wait gives up

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }

// Warp-uniform bounded wait for *p >= target.  Returns false when the wait
// gave up (after `limit` polls, or as soon as another block reported an
// error); the error word is then set.
__device__ __forceinline__ bool wait_geq(const int* p, int target, int* err, int limit = SPIN_LIMIT) {
  if (__all_sync(FULL, ld_acquire(p) >= target)) return true;
  for (int it = 1; it <= limit; ++it) {
    __nanosleep(64);
    if (__all_sync(FULL, ld_acquire(p) >= target)) return true;
    if ((it & 63) == 0 && __any_sync(FULL, ld_volatile(err) != 0)) return false;
  }
  if ((threadIdx.x & 31) == 0) atomicExch(err, 1);
  return false;
}

// Same, with the poll limit read from *limitP only once the first poll has
// failed (the fast path adds no dependent load to the caller's critical path).
__device__ __forceinline__ bool wait_geq_lim(const int* p, int target, int* err, const int* limitP) {
  if (__all_sync(FULL, ld_acquire(p) >= target)) return true;
  return wait_geq(p, target, err, __ldcg(limitP));
}

}  // namespace solvedev
}  // namespace rschol
