// Device side of the apply engine shared by the single-vector and the batched
// kernels: 16-byte vectors, barriers and bulk copies, the producer warp.
#pragma once
#include <cuda_runtime.h>

#include "solve.cuh"
#include "solve_dev.cuh"
#include "stage_order.h"

namespace rschol {
namespace solvedev {

// 16-byte vectors of the factor's type.
template <class T> struct Vec16;
template <> struct Vec16<float> {
  using type = float4;
  static constexpr int V = 4;
};
template <> struct Vec16<double> {
  using type = double2;
  static constexpr int V = 2;
};
__device__ __forceinline__ float vdot(float4 a, float4 b, float s) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}
__device__ __forceinline__ double vdot(double2 a, double2 b, double s) { return fma(a.y, b.y, fma(a.x, b.x, s)); }
__device__ __forceinline__ void vaxpy(float4& acc, float4 a, float x) {
  acc.x = fmaf(a.x, x, acc.x);
  acc.y = fmaf(a.y, x, acc.y);
  acc.z = fmaf(a.z, x, acc.z);
  acc.w = fmaf(a.w, x, acc.w);
}
__device__ __forceinline__ void vaxpy(double2& acc, double2 a, double x) {
  acc.x = fma(a.x, x, acc.x);
  acc.y = fma(a.y, x, acc.y);
}
__device__ __forceinline__ void vadd(float4& a, float4 b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
  a.w += b.w;
}
__device__ __forceinline__ void vadd(double2& a, double2 b) {
  a.x += b.x;
  a.y += b.y;
}
__device__ __forceinline__ float4 vzero(float) { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ double2 vzero(double) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ void vshfl_add(float4& v, int o) {
  v.x += __shfl_xor_sync(FULL, v.x, o);
  v.y += __shfl_xor_sync(FULL, v.y, o);
  v.z += __shfl_xor_sync(FULL, v.z, o);
  v.w += __shfl_xor_sync(FULL, v.w, o);
}
__device__ __forceinline__ void vshfl_add(double2& v, int o) {
  v.x += __shfl_xor_sync(FULL, v.x, o);
  v.y += __shfl_xor_sync(FULL, v.y, o);
}

// ---------------------------------------------------------------------------
// The apply engine: one persistent launch runs a whole preconditioner
// application as a list of work items (ApplyItem) in a topological order.
//
// Roles: a CTA is one producer warp and two groups of four consumer warps.  The
// producer takes the next item from a ticket counter and bulk-copies
// (cp.async.bulk, completion on an mbarrier) its descriptor and its piece of
// the factor into one of three shared-memory stages, running ahead of the
// consumers: the factor does not depend on the right-hand side, so its bytes
// arrive while earlier items still wait or compute.  The groups take the items
// in turn: a group waits (bounded) until the counters the item names have
// reached their targets, gathers the vector entries, forms the products from
// shared memory, stores, and one thread releases the item's own counter.  An
// item is about 3 us of dependent steps whatever its bytes, so what counts is
// the bytes being worked on at once: six groups an SM.
//
// Every item waits only on items earlier in the list (checked when the list is
// built) and a group works its tickets in order, so the smallest unfinished
// ticket can always proceed, whatever else shares the GPU.  The next kernel
// (clear_counters / convert_out_kernel) zeroes ticket and counters, so the
// launch needs no host state and replays inside a CUDA graph.
//
// Bound: a chain of hand-overs (release, poll, gather, product: ~3 us each, one
// or two a tree level and direction), then the factor's bytes.  The products with X
// lie off that chain and fill its gaps.  Measured, one
// application (before: a triangular solve per supernode on the chain, two
// ticketed launches for the interior and eight launches per compressed level):
// 3D 64^3 FP32 0.914 -> 0.397 ms (616 MB, 0.091 ms at the copy rate), 3D 96^3
// FP32 2.23 -> 1.21 ms, 2D 193 x 187 FP64 0.632 -> 0.178 ms, 2D 40 x 37 FP64
// 0.159 -> 0.077 ms.  Two groups of four warps against one of eight (half the
// items in work at once): 3D 64^3 0.400 against 0.494 ms.

constexpr int ST_DATA = 16384, ST_DESC = 3584, ST_BYTES = ST_DATA + ST_DESC;
constexpr int GT = 128, GW = GT / 32;   // threads and warps of a consumer group
constexpr int IW_N = 32, IW_M = 128;     // members of a group item: n <= IW_N, m <= IW_M
constexpr int GRP = 8;                   // most members of a group
constexpr int GH = 10;                   // header words of a member
constexpr int SHALLOW = 1;               // phases of up to this many items a group (in all CTAs) draw tickets singly
constexpr int ROWS8 = 8 * GW;            // most rows of W or V in an item (eight a warp)
// columns of f that a chunk item of the single-vector apply holds at a time: three
// CTAs an SM then fit whatever the widest supernode is
template <class T> constexpr int F_TILE = 4096 / (int)sizeof(T);

enum ItemKind : int { IT_FGRP = 0, IT_FWD, IT_CF, IT_CU, IT_Y, IT_XT, IT_CS, IT_CX, IT_BGRP, IT_BWD, IT_CR, IT_BR, IT_END };

// tile of X of the Y = X f items (rows x columns) and of the t = X^T y items
constexpr int Y_ROWS = 16, T_COLS = 64;
template <class T> constexpr int Y_COLS = ST_DATA / Y_ROWS / (int)sizeof(T);
template <class T> constexpr int T_ROWS = ST_DATA / T_COLS / (int)sizeof(T);

// barrier of the caller's consumer group (bar.sync wants whole warps)
__device__ __forceinline__ void cbar() {
  __syncwarp();
  asm volatile("bar.sync %0, 128;" ::"r"(1 + (int)(threadIdx.x / GT)) : "memory");
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Warp-wide wait for a phase: lane 0 polls, for at most about four seconds;
// false when it gave up.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0 && !mbar_test(bar, parity)) {
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int it = 1; !mbar_test(bar, parity); ++it) {
      if (it > 64) __nanosleep(20);
      if ((it & 255) == 0) {
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t - t0 > 4000000000ull) {
          ok = 0;
          break;
        }
      }
    }
  }
  ok = __shfl_sync(FULL, ok, 0);
  __syncwarp();   // what lane 0 has seen complete, the others may read
  return ok != 0;
}
// A consumer's wait for its item k (stage_order.h); bars: the full, then the empty barriers.
__device__ __forceinline__ bool wait_stage(int k, unsigned bars) {
  return stage_landed(
      k, [&](int s, unsigned parity) { return mbar_wait(bars + 8 * s, parity); },
      [&](int s, unsigned parity) { return mbar_wait(bars + 8 * (NSTAGE + s), parity); });
}
// global -> shared, 16-byte aligned addresses and size, completion on bar
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, int bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Warp-wide bounded wait until every listed counter has reached its target
// (pairs of counter index and target).
__device__ __forceinline__ void wait_list(const int* pairs, int count, const int* sync, int* err) {
  const int lane = threadIdx.x & 31;
  for (int c0 = 0; c0 < count; c0 += 32) {
    const bool have = c0 + lane < count;
    const int idx = have ? pairs[2 * (c0 + lane)] : 0, target = have ? pairs[2 * (c0 + lane) + 1] : 0;
    for (int it = 0;; ++it) {
      const bool ok = !have || ld_acquire(sync + idx) >= target;
      if (__all_sync(FULL, ok)) break;
      if (it >= SPIN_LIMIT) {
        if (lane == 0) atomicExch(err, 1);
        return;
      }
      if ((it & 63) == 63 && __any_sync(FULL, ld_volatile(err) != 0)) return;
      if (it) __nanosleep(20);
    }
  }
}

template <class T>
struct ApplyArgs {
  const ApplyItem* items;
  int nItems;
  const int* blob;
  int* sync;        // [0] error word, [1] ticket, then the counters
  int* err;         // the error word (of the first slice of columns)
  T* w;             // permuted vector, in place
  T* t;             // y = X f of the interior columns
  T* wu;            // update vectors
  T* zp;            // partials of z = W^T f
  T* sp;            // partials of s = V^T x_R
  T* yp;            // partials of X f
  T* xp;            // partials of X^T y
  T* ip;            // partials of X^T y - G^T x_R
  int work;         // elements of a group's work area in shared memory
};

// The producer warp: draws tickets, stages the items' pieces, marks the end for
// every group.
template <class T>
__device__ __forceinline__ void apply_producer(const ApplyArgs<T>& A, unsigned char* apsm, ApplyItem* sItem,
                                               unsigned full0, unsigned empty0) {
  const int lane = threadIdx.x & 31;
  int* const err = A.err;
  // Tickets are drawn in pairs (one latency for two items) as far ahead as
  // there are stages -- except in a phase of few items (ApplyItem::shallow),
  // where a CTA that holds more than a group's worth keeps items from idle
  // CTAs: there the next single ticket waits for the last item but one
  // (c2 apply: 0.39 ms in pairs throughout, 0.376 ms so).
  int have = 0, ends = 0;   // items read ahead (0 ... 2)
  bool more = true;
  ApplyItem cur, nxt;
  for (int k = 0;; ++k) {
    const int s = k % NSTAGE, use = k / NSTAGE;
    if (have == 0 && more) {
      const int want = k > 0 && cur.shallow ? 1 : 2;
      if (want == 1 && k > 1) mbar_wait(empty0 + 8 * ((k - 2) % NSTAGE), ((k - 2) / NSTAGE) & 1);
      int tk = 0;
      if (lane == 0) tk = atomicAdd(A.sync + 1, want);
      tk = __shfl_sync(FULL, tk, 0);
      if (tk < A.nItems) {
        nxt = A.items[tk];
        have = 1;
      }
      more = tk + want <= A.nItems;
      if (want == 2 && tk + 1 < A.nItems) {
        cur = nxt;
        nxt = A.items[tk + 1];
        have = 2;
      } else {
        cur = nxt;
      }
    } else if (have == 1) {
      cur = nxt;
    }
    const bool end = have == 0;
    if (!end) --have;
    bool ok = true;
    if (use > 0) ok = mbar_wait(empty0 + 8 * s, (use - 1) & 1);
    if (!ok && lane == 0) atomicExch(err, 4);
    if (end || !ok) {   // one end mark per group
      if (lane == 0) {
        sItem[s].kind = IT_END;
        mbar_arrive(full0 + 8 * s);
      }
      more = false;
      have = 0;
      if (++ends == NGRP) break;
      continue;
    }
    const ApplyItem& it = cur;
    unsigned char* st = apsm + (size_t)s * ST_BYTES;
    if (lane == 0) {
      sItem[s] = it;
      const int total = it.descBytes + it.desc2Bytes + it.bytes0 + it.bytes1;
      mbar_expect(full0 + 8 * s, total);
      if (it.descBytes) bulk_copy(st + ST_DATA, A.blob + it.desc, it.descBytes, full0 + 8 * s);
      if (it.desc2Bytes) bulk_copy(st + ST_DATA + it.descBytes, A.blob + it.desc2, it.desc2Bytes, full0 + 8 * s);
    }
    __syncwarp();
    if (lane == 0) {
      if (it.bytes0) bulk_copy(st, it.g0, it.bytes0, full0 + 8 * s);
      if (it.bytes1) bulk_copy(st + it.bytes0, it.g1, it.bytes1, full0 + 8 * s);
    }
  }
}

}  // namespace solvedev
}  // namespace rschol
