#include <algorithm>
#include <climits>
#include <mutex>
#include <cstdlib>
#include <type_traits>

#include "apply_dev.cuh"
#include "solve.cuh"
#include "solve_dev.cuh"

namespace rschol {

namespace {

using namespace solvedev;

// v[i] + the pull list [b[i], e[i]) of wu entries, in order, for N targets at
// once: the loads of a round (two entries a target) are all in flight together.
template <class T, int N>
__device__ __forceinline__ void pull_sums(T (&v)[N], const int* const (&ent)[N], int (&b)[N], const int (&e)[N],
                                          const T* wu) {
  bool more = true;
  while (more) {
    T x[N], y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = b[i] < e[i] ? __ldcg(wu + ent[i][b[i]]) : T(0);
      y[i] = b[i] + 1 < e[i] ? __ldcg(wu + ent[i][b[i] + 1]) : T(0);
    }
    more = false;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      v[i] = (v[i] + x[i]) + y[i];
      b[i] += 2;
      more = more || b[i] < e[i];
    }
  }
}

// zs[k] = the sum of `parts` partial rows (row stride rp, 16-byte aligned) over
// the columns [k0, k0 + GT vectors), in a fixed order: groups of threads take
// every ng-th row, the groups are added in order.
template <class T>
__device__ __forceinline__ void sum_parts(const T* __restrict__ part, int rp, int cols, int k0, int parts, T* zs,
                                          T* redT) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  Vt* red = reinterpret_cast<Vt*>(redT);
  const int tid = threadIdx.x % GT;
  const int nv = min(GT, (cols - k0 + V - 1) / V);
  int ng = GT / nv;
  if (ng > parts) ng = parts;
  const int g = tid / nv, c = tid - g * nv;
  const Vt* p = reinterpret_cast<const Vt*>(part + k0) + c;
  const size_t stride = rp / V;
  if (g < ng) {
    Vt a0 = vzero(T(0));
    for (int i = g; i < parts; i += 8 * ng) {
      Vt v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = i + q * ng < parts ? __ldcg(p + (size_t)(i + q * ng) * stride) : vzero(T(0));
#pragma unroll
      for (int q = 0; q < 8; ++q) vadd(a0, v[q]);
    }
    red[g * nv + c] = a0;
  }
  cbar();
  for (int k = tid; k < nv * V; k += GT) {
    T s = T(0);
    for (int q = 0; q < ng; ++q) s += redT[q * nv * V + k];
    zs[k] = s;
  }
  cbar();
}

// out[k] = sum_{i < h} M[i][k] v[i], k < r (and zeros up to whole sectors), M in
// shared or global memory (row stride r): 2^g-wide column groups, rows split over the remaining threads and
// the parts added in a fixed order.
template <class T>
__device__ __forceinline__ void cols_gemv(const T* M, int r, int h, const T* v, T* out, T* red) {
  const int tid = threadIdx.x % GT;
  int wd = 32;
  while (wd < r && wd < GT) wd <<= 1;
  const int ng = GT / wd, g = tid / wd, c = tid & (wd - 1);
  for (int k0 = 0; k0 < r; k0 += wd) {
    T s = T(0);
    if (k0 + c < r) {
#pragma unroll 8
      for (int i = g; i < h; i += ng) s += M[(size_t)i * r + k0 + c] * v[i];
    }
    if (ng == 1) {
      if (k0 + c < ((r + 7) & ~7)) out[k0 + c] = s;
    } else {
      red[tid] = s;
      cbar();
      if (tid < wd && k0 + tid < ((r + 7) & ~7)) {
        T z = T(0);
        for (int q = 0; q < ng; ++q) z += red[q * wd + tid];
        out[k0 + tid] = z;
      }
      cbar();
    }
  }
}

// A group of small interior supernodes, forward: u = (children's rows) - G f
// and y = X f; a warp a member, or several when there are fewer members.  FP32:
// lanes along the rows, partial sums by shuffles.  FP64 adds run at 1/64 of the
// FP32 rate, so there a lane forms a whole row (the odd row stride in 16-byte
// units keeps that free of bank conflicts).
template <class T>
__device__ __forceinline__ void item_fgrp(const ApplyArgs<T>& A, const int* hdr0, const int* d, int cnt, const T* data,
                                          T* wk) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % GW;
  const int wpn = cnt <= 1 ? GW : cnt <= GW / 2 ? GW / (GW / 2) : 1;
  T* f = wk + warp * (IW_N + IW_M);
  T* ub = f + IW_N;
  const int part = warp % wpn;
  for (int q = warp / wpn; q < cnt; q += GW / wpn) {
    const int* h = hdr0 + GH * q;
    const int n = h[0], m = h[1], c0 = h[2], nv = h[7] / V;
    const Vt* G = reinterpret_cast<const Vt*>(data + h[4]);
    const Vt* X = reinterpret_cast<const Vt*>(data + h[5]);
    const int* ps = h[6] ? d + h[6] : nullptr;
    const int* ent = ps + n + m + 1;
    const int mp = ((m + wpn - 1) / wpn + 7) & ~7, aLo = part * mp, aHi = min(m, aLo + mp);
    T* u = A.wu + h[3];
    T* t = A.t + h[8];
    __syncwarp();
    T v[1 + IW_M / 32];   // the lane's column, then its rows
    int b[1 + IW_M / 32], e[1 + IW_M / 32];
    v[0] = lane < n ? __ldcg(A.w + c0 + lane) : T(0);
    b[0] = ps && lane < n ? ps[lane] : 0;
    e[0] = ps && lane < n ? ps[lane + 1] : 0;
#pragma unroll
    for (int i = 1; i <= IW_M / 32; ++i) {
      const int a = aLo + lane + 32 * (i - 1);
      const bool in = ps && a < aHi;
      v[i] = T(0);
      b[i] = in ? ps[n + a] : 0;
      e[i] = in ? ps[n + a + 1] : 0;
    }
    if (ps) {
      const int* const lists[1 + IW_M / 32] = {ent, ent, ent, ent, ent};
      pull_sums(v, lists, b, e, A.wu);
    }
#pragma unroll
    for (int i = 1; i <= IW_M / 32; ++i)
      if (aLo + lane + 32 * (i - 1) < aHi) ub[aLo + lane + 32 * (i - 1)] = v[i];
    f[lane] = v[0];
    __syncwarp();
    if constexpr (sizeof(T) == 8) {
      const int rows = max(0, aHi - aLo), sp = ((n + wpn - 1) / wpn + 7) & ~7, sLo = part * sp, sRows = max(0, min(n, sLo + sp) - sLo);
      const Vt* fs = reinterpret_cast<const Vt*>(f);
      const int nq = (n + V - 1) / V;
      for (int i = lane; i < rows + sRows; i += 32) {   // rows of G, then of X
        const Vt* row = i < rows ? G + (aLo + i) * nv : X + (sLo + i - rows) * nv;
        T v0 = T(0), v1 = T(0);
        int c = 0;
        for (; c + 1 < nq; c += 2) {
          v0 = vdot(row[c], fs[c], v0);
          v1 = vdot(row[c + 1], fs[c + 1], v1);
        }
        if (c < nq) v0 = vdot(row[c], fs[c], v0);
        if (i < rows) u[aLo + i] = ub[aLo + i] - (v0 + v1);
        else t[sLo + i - rows] = v0 + v1;
      }
    } else {
      const int lg = nv <= 4 ? 2 : 3;   // lanes per row: 2^lg
      const int c = lane & ((1 << lg) - 1), g = lane >> lg, rpl = 32 >> lg;
      const Vt fc = c < nv ? reinterpret_cast<const Vt*>(f)[c] : vzero(T(0));
#pragma unroll 4
      for (int a0 = aLo; a0 < aHi; a0 += rpl) {
        const int a = a0 + g;
        T v = (a < aHi && c < nv) ? vdot(G[a * nv + c], fc, T(0)) : T(0);
        for (int o = 1; o < (1 << lg); o <<= 1) v += __shfl_xor_sync(FULL, v, o);
        if (c == 0 && a < aHi) u[a] = ub[a] - v;
      }
      for (int i0 = part * rpl; i0 < n; i0 += rpl * wpn) {
        const int i = i0 + g;
        T v = (i < n && c < nv) ? vdot(X[i * nv + c], fc, T(0)) : T(0);
        for (int o = 1; o < (1 << lg); o <<= 1) v += __shfl_xor_sync(FULL, v, o);
        if (c == 0 && i < n) t[i] = v;
      }
    }
    // the last sectors whole
    if (part == wpn - 1) {
      if (m + lane < ((m + 7) & ~7)) u[m + lane] = T(0);
      if (n + lane < ((n + 7) & ~7)) t[n + lane] = T(0);
    }
  }
}

// A group, backward: x = X^T y - G^T x_R; a warp a member.
template <class T>
__device__ __forceinline__ void item_bgrp(const ApplyArgs<T>& A, const int* hdr0, const int* d, int cnt, const T* data,
                                          T* wk) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % GW;
  T* xr = wk + warp * (IW_N + IW_M);   // -x_R, then y
  for (int q = warp; q < cnt; q += GW) {
    const int* h = hdr0 + GH * q;
    const int n = h[0], m = h[1], c0 = h[2], nv = h[7] / V, nq = (n + V - 1) / V;
    const Vt* G = reinterpret_cast<const Vt*>(data + h[4]);
    const Vt* X = reinterpret_cast<const Vt*>(data + h[5]);
    const int* rw = d + h[6];
    __syncwarp();
    if (lane < n) xr[m + lane] = __ldcg(A.t + h[8] + lane);
#pragma unroll 4
    for (int a = lane; a < m; a += 32) xr[a] = -__ldcg(A.w + rw[a]);
    __syncwarp();
    const int lg = nq <= 4 ? 2 : nq <= 8 ? 3 : 4;
    const int c = lane & ((1 << lg) - 1), g = lane >> lg, rpl = 32 >> lg;
    Vt acc = vzero(T(0));
    if (c < nq) {
#pragma unroll 4
      for (int a = g; a < m; a += rpl) vaxpy(acc, G[a * nv + c], xr[a]);
#pragma unroll 4
      for (int a = g; a < n; a += rpl) vaxpy(acc, X[a * nv + c], xr[m + a]);
    }
    for (int o = 1 << lg; o < 32; o <<= 1) vshfl_add(acc, o);
    __syncwarp();
    if (g == 0 && c < nq) reinterpret_cast<Vt*>(xr)[c] = acc;
    __syncwarp();
    if (lane < n) A.w[c0 + lane] = xr[lane];
  }
}

// One chunk of a larger interior supernode, forward.
// hdr: n, rows, c0, u offset (of the chunk's first row), s0, sRows, list, ldk, t offset, whole sectors
template <class T>
__device__ __forceinline__ void item_fwd(const ApplyArgs<T>& A, const int* h, const int* d, const int* d2, const T* Gd,
                                         const T* Xd, T* f, T* ub) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  const int tid = threadIdx.x % GT;
  const int n = h[0], rows = h[1], c0 = h[2], nv = h[7] / V;
  // pull lists: the chunk's rows' (rows + 1 offsets, entries) in the descriptor,
  // the columns' (n + 1 offsets, entries) in the part that the chunks share
  const bool pull = h[6] != 0;
  const int* ps = d + h[6];
  const int* ent = ps + rows + 1;
  const int* ent2 = d2 + n + 1;
  const Vt* fs = reinterpret_cast<const Vt*>(f);
  const int R = rows + h[5];   // rows of G, then the chunk's rows of X
  int lt = 1;                  // threads of a row: 2^lt
  while (lt < 5 && R << (lt + 1) <= GT) ++lt;
  const int sub = tid & ((1 << lt) - 1);
  // f in tiles (a supernode of several is read in place, at most 32 rows an item: one
  // sweep of them, its sums kept in acc); a thread's order along a row is that of one tile
  T acc = T(0);
  for (int j0 = 0; j0 < nv * V; j0 += F_TILE<T>) {
    const int jn = min(F_TILE<T>, nv * V - j0);
    if (j0 > 0) cbar();   // every thread is done with the last tile
    for (int t0 = 0; t0 < jn; t0 += 2 * GT) {   // two columns and (first pass) one row a thread
      T v[3];
      int b[3], e[3];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = j0 + t0 + tid + i * GT;
        const bool in = t0 + tid + i * GT < jn && t < n;
        v[i] = in ? __ldcg(A.w + c0 + t) : T(0);
        b[i] = pull && in ? d2[t] : 0;
        e[i] = pull && in ? d2[t + 1] : 0;
      }
      const bool in = j0 == 0 && t0 == 0 && tid < rows;
      v[2] = T(0);
      b[2] = pull && in ? ps[tid] : 0;
      e[2] = pull && in ? ps[tid + 1] : 0;
      if (pull) {
        const int* const lists[3] = {ent2, ent2, ent};
        pull_sums(v, lists, b, e, A.wu);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (t0 + tid + i * GT < jn) f[t0 + tid + i * GT] = v[i];
      if (in) ub[tid] = v[2];
    }
    cbar();
    const bool last = j0 + jn >= nv * V;
    for (int r0 = 0; r0 < R; r0 += GT >> lt) {
      const int row = r0 + (tid >> lt);
      T v = acc;
      if (row < R) {
        const Vt* m =
            reinterpret_cast<const Vt*>(row < rows ? Gd : Xd) + (size_t)(row < rows ? row : row - rows) * nv + j0 / V;
#pragma unroll 4
        for (int c = sub; c < jn / V; c += 1 << lt) v = vdot(m[c], fs[c], v);
      }
      if (!last) {
        acc = v;
        continue;
      }
      for (int o = 1; o < (1 << lt); o <<= 1) v += __shfl_xor_sync(FULL, v, o);
      if (sub == 0 && row < R) {
        if (row < rows) A.wu[h[3] + row] = ub[row] - v;
        else A.t[h[8] + h[4] + row - rows] = v;
      }
    }
  }
  if (h[9]) {   // chunks of whole sectors: the last ones to their ends
    constexpr int SE = 32 / (int)sizeof(T);
    if (tid < (SE - rows % SE) % SE) A.wu[h[3] + rows + tid] = T(0);
    if (tid < (SE - h[5] % SE) % SE) A.t[h[8] + h[4] + h[5] + tid] = T(0);
  }
}

// One chunk of a larger interior supernode, backward: its part of X^T y - G^T x_R,
// which is x when there is no other chunk (several: item BR).
// hdr: n, rows of G, c0, ipOff, chunk, chunks, rows list, ldk, ip stride, y offset (of
// the chunk's first row of X), rows of X
template <class T>
__device__ __forceinline__ void item_bwd(const ApplyArgs<T>& A, const int* h, const int* d, const T* Gd, const T* Xd,
                                         T* xr, T* red) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  const int tid = threadIdx.x % GT, lane = tid & 31, warp = tid >> 5;
  const int n = h[0], rows = h[1], c0 = h[2], nch = h[5], nv = h[7] / V, R = rows + h[10];
  if (tid < R) xr[tid] = tid < rows ? -__ldcg(A.w + d[h[6] + tid]) : __ldcg(A.t + h[9] + tid - rows);
  cbar();
  // 2^lg threads along a row (4 ... 128), the others on further rows
  int lg = 2;
  while ((1 << lg) < nv && lg < 7) ++lg;
  const int wd = 1 << lg, c = tid & (wd - 1), g = tid >> lg, ng = GT >> lg;
  const Vt* G = reinterpret_cast<const Vt*>(Gd);
  const Vt* X = reinterpret_cast<const Vt*>(Xd) - (size_t)rows * nv;   // row a >= rows at a * nv
  Vt* rv = reinterpret_cast<Vt*>(red);
  for (int v0 = 0; v0 < nv; v0 += GT) {
    Vt acc = vzero(T(0));
    if (v0 + c < nv) {
#pragma unroll 4
      for (int a = g; a < R; a += ng) vaxpy(acc, (a < rows ? G : X)[(size_t)a * nv + v0 + c], xr[a]);
    }
    for (int o = wd; o < 32; o <<= 1) vshfl_add(acc, o);
    const int parts = lg <= 5 ? GW : ng;
    if (lg > 5) rv[g * wd + c] = acc;
    else if (lane < wd) rv[warp * wd + lane] = acc;
    cbar();
    for (int q = tid; q < max(wd * V, 8); q += GT) {
      const int j = v0 * V + q;
      T s = T(0);
      if (j < n)
        for (int p = 0; p < parts; ++p) s += red[p * wd * V + q];
      if (nch > 1) {
        if (j < h[8]) A.ip[h[3] + (size_t)h[4] * h[8] + j] = s;
      } else if (j < n) {
        A.w[c0 + j] = s;
      }
    }
    cbar();
  }
}

// Compressed supernode, up: f of a block of columns (added into w) and the
// block's part of z = W^T f.
// hdr: c (first column's vector index), h (columns), r, zp row offset, list
template <class T>
__device__ __forceinline__ void item_cf(const ApplyArgs<T>& A, const int* h, const int* d, const T* Wd, T* fb, T* red) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % GW;
  const int c0 = h[0], cols = h[1], r = h[2];
  const int* ps = d + h[4];
  const int* ent = ps + cols + 1;
  // a warp per eight rows, lanes along the rows' contribution lists
  int b[8], e[8];
  T acc[8], wv[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int i = warp + GW * q;
    const bool in = i < cols;
    b[q] = in ? ps[i] + lane : 0;
    e[q] = in ? ps[i + 1] : 0;
    wv[q] = (in && lane == 0) ? __ldcg(A.w + c0 + i) : T(0);
    acc[q] = T(0);
  }
  bool more = true;
  while (more) {
    T v[8], x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      v[q] = b[q] < e[q] ? __ldcg(A.wu + ent[b[q]]) : T(0);
      x[q] = b[q] + 32 < e[q] ? __ldcg(A.wu + ent[b[q] + 32]) : T(0);
    }
    more = false;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      acc[q] = (acc[q] + v[q]) + x[q];
      b[q] += 64;
      more = more || b[q] - lane < e[q];
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int i = warp + GW * q;
    if (i >= cols) break;
    const T s = warp_sum(acc[q]);
    if (lane == 0) {
      const T v = wv[q] + s;
      A.w[c0 + i] = v;
      fb[i] = v;
    }
  }
  cbar();
  if (r > 0) cols_gemv<T>(Wd, r, cols, fb, A.zp + h[3], red);
}

// acc = the product of this warp's rows (i = warp, warp + GW, ...) of M (row
// stride r) with the sum of the partial rows.
template <class T>
__device__ __forceinline__ void rows_times_parts(const T* M, int r, int rows, const T* part, int parts, T (&acc)[8],
                                                 T* zs, T* red) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % GW;
  constexpr int KT = GT * Vec16<T>::V;
  const int rp = (r + 7) & ~7;
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = T(0);
  for (int k0 = 0; k0 < r; k0 += KT) {
    sum_parts<T>(part, rp, rp, k0, parts, zs, red);
    const int kn = min(KT, r - k0);
    const T* m = M + (size_t)warp * r + k0;
#pragma unroll 2
    for (int k = lane; k < kn; k += 32) {
      const T z = zs[k];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (warp + GW * q < rows) acc[q] += m[(size_t)GW * q * r + k] * z;
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = warp_sum(acc[q]);
}

template <class T>
__global__ void __launch_bounds__(NGRP * GT + 32, 3) apply_kernel(ApplyArgs<T> A) {
  extern __shared__ __align__(128) unsigned char apsm[];
  __shared__ __align__(8) unsigned long long bars[2 * NSTAGE];
  __shared__ __align__(16) ApplyItem sItem[NSTAGE];
  const int lane = threadIdx.x & 31;
  int* const err = A.err;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(smem_u32(&bars[s]), 1);              // full: the producer's arrival and its bytes
      mbar_init(smem_u32(&bars[NSTAGE + s]), 1);     // empty: one consumer thread
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (threadIdx.x >= NGRP * GT) {   // ---- producer
    apply_producer<T>(A, apsm, sItem, smem_u32(&bars[0]), smem_u32(&bars[NSTAGE]));
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    return;
  }

  // ---- consumers
  const int grp = threadIdx.x / GT, tid = threadIdx.x % GT, warp = tid >> 5;
  T* const red = reinterpret_cast<T*>(apsm + NSTAGE * ST_BYTES) + grp * A.work;   // GT vectors (a group item: its buffers)
  T* const zs = red + GT * Vec16<T>::V;                                           // GT vectors
  T* const f = zs + GT * Vec16<T>::V;                                             // the widest chunk item's columns
  for (int k = grp;; k += NGRP) {
    const int s = k % NSTAGE;
    if (!wait_stage(k, smem_u32(&bars[0]))) {   // cannot happen while the producer runs
      if (tid == 0) atomicExch(err, 3);
      break;
    }
    const ApplyItem& it = sItem[s];
    const int kind = it.kind;
    if (kind == IT_END) break;
    const unsigned char* st = apsm + (size_t)s * ST_BYTES;
    const T* data = reinterpret_cast<const T*>(st);
    const int* d = it.descBytes ? reinterpret_cast<const int*>(st + ST_DATA) : A.blob + it.desc;
    const int* h = d + 2 * it.waits;
    const int* d2 = it.desc2Bytes ? reinterpret_cast<const int*>(st + ST_DATA + it.descBytes) : A.blob + it.desc2;
    // (The early waits follow from the others, where there are any.  The products with X
    // between the two, as the batched kernel has them, in phases of few items in FP64: 2D
    // 40 x 37 95 against 100 us a call, but 193 x 187 193 against 190.)
    const int beg = it.early < it.waits ? it.early : 0;
    if (warp == 0) wait_list(d + 2 * beg, it.waits - beg, A.sync, err);
    cbar();
    // pieces too wide for a stage are read where they are
    const T* g0 = it.bytes0 ? data : reinterpret_cast<const T*>(it.g0);
    const T* g1 = it.bytes1 ? data + it.bytes0 / sizeof(T) : reinterpret_cast<const T*>(it.g1);
    switch (kind) {
      case IT_FGRP: item_fgrp<T>(A, h, d, it.count, data, red); break;
      case IT_BGRP: item_bgrp<T>(A, h, d, it.count, data, red); break;
      case IT_FWD: item_fwd<T>(A, h, d, d2, g0, g1, f, zs); break;
      case IT_BWD: item_bwd<T>(A, h, d, g0, g1, zs, red); break;
      case IT_BR: {   // hdr: n, c0, ipOff, parts, ip stride: x = the parts of X^T y - G^T x_R, added in order
        for (int k0 = 0; k0 < h[0]; k0 += GT * Vec16<T>::V) {
          const int kn = min(GT * Vec16<T>::V, h[0] - k0);
          sum_parts<T>(A.ip + h[2], h[4], h[0], k0, h[3], zs, red);
          for (int q = tid; q < kn; q += GT) A.w[h[1] + k0 + q] = zs[q];
          cbar();
        }
        break;
      }
      case IT_CF: item_cf<T>(A, h, d, g0, zs, red); break;
      case IT_CU: {   // hdr: rows, r, zp offset, parts, u offset
        T acc[8];
        rows_times_parts<T>(g0, h[1], h[0], A.zp + h[2], h[3], acc, zs, red);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (lane == 0 && warp + GW * q < ((h[0] + 7) & ~7)) A.wu[h[4] + warp + GW * q] = -acc[q];   // (acc: 0 past the rows)
        break;
      }
      case IT_Y: {   // hdr: c0 + j0, columns, rows, yp offset (block jb, row i0)
        for (int j = tid; j < Y_COLS<T>; j += GT) red[j] = j < h[1] ? __ldcg(A.w + h[0] + j) : T(0);
        cbar();
        T v[Y_ROWS / GW];
#pragma unroll
        for (int q = 0; q < Y_ROWS / GW; ++q) v[q] = T(0);
        for (int j = lane; j < h[1]; j += 32) {
          const T fj = red[j];
#pragma unroll
          for (int q = 0; q < Y_ROWS / GW; ++q)
            if (warp + GW * q < h[2]) v[q] += data[(warp + GW * q) * Y_COLS<T> + j] * fj;
        }
#pragma unroll
        for (int q = 0; q < Y_ROWS / GW; ++q) {
          const T y = warp_sum(v[q]);
          if (lane == 0 && warp + GW * q < ((h[2] + 7) & ~7)) A.yp[h[3] + warp + GW * q] = y;
        }
        break;
      }
      case IT_XT: {   // hdr: rows, columns, yp offset (row i0), yp stride, i0, xp offset (block ib, column j0), column blocks
        using Vt = typename Vec16<T>::type;
        constexpr int V = Vec16<T>::V, TR = T_ROWS<T>, TPR = GT / TR, NV = T_COLS / V, NG = GT / NV;
        {   // TPR threads a row add its partials of y (fixed order)
          const int i = tid / TPR, sub = tid - i * TPR;
          T y = T(0);
          if (i < h[0]) {
            const int nj = min(h[6], ((h[4] + i) / Y_ROWS * Y_ROWS + Y_ROWS - 1) / Y_COLS<T> + 1);
#pragma unroll 4
            for (int jb = sub; jb < nj; jb += TPR) y += __ldcg(A.yp + h[2] + (size_t)jb * h[3] + i);
          }
#pragma unroll
          for (int o = 1; o < TPR; o <<= 1) y += __shfl_xor_sync(FULL, y, o);
          if (sub == 0) zs[i] = y;
        }
        cbar();
        const int g = tid / NV, c = tid - g * NV;
        Vt acc = vzero(T(0));
        if (g < NG && c * V < h[1])
          for (int i = g; i < h[0]; i += NG) vaxpy(acc, reinterpret_cast<const Vt*>(data)[i * NV + c], zs[i]);
        if (g < NG) reinterpret_cast<Vt*>(red)[g * NV + c] = acc;
        cbar();
        if (tid < ((h[1] + 7) & ~7)) {
          T x = T(0);
#pragma unroll
          for (int q = 0; q < NG; ++q) x += red[q * T_COLS + tid];
          A.xp[h[5] + tid] = x;
        }
        break;
      }
      case IT_CR: {   // hdr: partials' offset (first column), parts, row stride, columns, offset of the sums, 1: of s
        using Vt = typename Vec16<T>::type;
        constexpr int V = Vec16<T>::V;
        T* const base = h[5] ? A.sp : A.zp;
        const int nv = h[3] / V, ng = GT / nv, g = tid / nv, c = tid - g * nv;
        const Vt* p = reinterpret_cast<const Vt*>(base + h[0]) + c;
        const size_t stride = h[2] / V;
        Vt acc = vzero(T(0));
        if (g < ng) {
          for (int i = g; i < h[1]; i += 8 * ng) {
            Vt v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = i + q * ng < h[1] ? __ldcg(p + (size_t)(i + q * ng) * stride) : vzero(T(0));
#pragma unroll
            for (int q = 0; q < 8; ++q) vadd(acc, v[q]);
          }
          reinterpret_cast<Vt*>(red)[g * nv + c] = acc;
        }
        cbar();
        if (tid < h[3]) {
          T x = T(0);
          for (int q = 0; q < ng; ++q) x += red[q * h[3] + tid];
          base[h[4] + tid] = x;
        }
        break;
      }
      case IT_CS: {   // hdr: rows, r, sp offset, rows list
        if (tid < h[0]) zs[tid] = __ldcg(A.w + d[h[3] + tid]);
        cbar();
        cols_gemv<T>(g0, h[1], h[0], zs, A.sp + h[2], red);
        break;
      }
      default: {   // IT_CX; hdr: c, columns, r, sp offset, parts, xp offset (first column), xp stride, j0, first row block, row blocks
        // t of a column: its tiles' partials from the diagonal down, a lane a
        // column, the warps' sums added in order
        const int cols = h[1], ib0 = (h[7] + lane) / T_COLS * T_COLS / T_ROWS<T>;
        T t = T(0), acc[8];
#pragma unroll 8
        for (int ib = h[8] + warp; ib < h[9]; ib += GW)
          t += (lane < cols && ib >= ib0) ? __ldcg(A.xp + h[5] + (size_t)ib * h[6] + lane) : T(0);
        if (h[4] > 0) {
          rows_times_parts<T>(g0, h[2], cols, A.sp + h[3], h[4], acc, zs, red);
        } else {
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[q] = T(0);
        }
        cbar();
        red[warp * 32 + lane] = t;
        T own = T(0);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (lane == q) own = acc[q];
        cbar();
        const int j = warp + GW * lane;
        if (lane < 8 && j < cols) {
          T x = T(0);
#pragma unroll
          for (int q = 0; q < GW; ++q) x += red[q * 32 + j];
          A.w[h[0] + j] = x - own;
        }
        break;
      }
    }
    const int sig = it.sig;
    cbar();   // every consumer has stored and is done with the stage
    if (tid == GT - 32) {   // not the warp that polls for the next item
      mbar_arrive(smem_u32(&bars[NSTAGE + s]));
      __threadfence();
      atomicAdd(A.sync + sig, 1);
    }
  }
}

// The tiles of X = L11^{-1} that the items read, each packed into one stage's
// bytes (zeros outside the matrix), so that one bulk copy brings it: a copy per
// row of a 64 x 64 tile costs its producer 64 issues of about 15 ns.  A block a
// tile; bound by HBM (X read, and written once per tile shape).
template <class T>
__global__ void __launch_bounds__(256) pack_tiles_kernel(const SNode<T>* __restrict__ nodes,
                                                         const PackTile* __restrict__ tiles, T* __restrict__ out) {
  const PackTile p = tiles[blockIdx.x];
  const SNode<T>& nd = nodes[p.node];
  T* o = out + (size_t)blockIdx.x * (ST_DATA / sizeof(T));
  const int lg = 31 - __clz(p.cols);   // columns: a power of two
#pragma unroll 4
  for (int e = threadIdx.x; e < ST_DATA / (int)sizeof(T); e += 256) {
    const int i = p.i0 + (e >> lg), j = p.j0 + (e & (p.cols - 1));
    o[e] = (i < nd.n && j < nd.n) ? nd.X[(size_t)i * nd.ldx + j] : T(0);
  }
}

// G = L21 X of an interior supernode of up to 64 columns, X = L11^{-1}.  A block per
// 64 rows; a thread per (row, NQ of the 4 NQ columns); X's zeros above the diagonal
// are skipped in steps of four.  Latency-bound: the products of all supernodes are a
// few GFLOP.
template <class T, int NQ>
__global__ void __launch_bounds__(256) interior_ops_kernel(const SNode<T>* __restrict__ nodes,
                                                           const RowBlock* __restrict__ work) {
  constexpr int W = 4 * NQ, P = W + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  T (*Xs)[P] = reinterpret_cast<T (*)[P]>(smraw);
  T (*Rs)[P] = reinterpret_cast<T (*)[P]>(smraw + sizeof(T) * W * P);
  const RowBlock wk = work[blockIdx.x];
  const SNode<T>& nd = nodes[wk.node];
  const int n = nd.n, m = nd.m, r0 = wk.b * 64;
  for (int idx = threadIdx.x; idx < W * W; idx += 256) {
    const int i = idx / W, j = idx - i * W;
    Xs[i][j] = (i < n && j <= i) ? nd.X[(size_t)i * nd.ldx + j] : T(0);
  }
  for (int idx = threadIdx.x; idx < 64 * W; idx += 256) {
    const int i = idx / W, k = idx - i * W, row = r0 + i;
    Rs[i][k] = (k < n && row < m) ? nd.L[(size_t)(n + row) * nd.ld + k] : T(0);
  }
  __syncthreads();
  const int i = threadIdx.x >> 2, cg = threadIdx.x & 3;
  T acc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) acc[q] = T(0);
  for (int kb = 0; kb < NQ && 4 * kb < n; ++kb) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const T l = Rs[i][4 * kb + kk];
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q <= kb) acc[q] += l * Xs[4 * kb + kk][cg + 4 * q];
    }
  }
  if (r0 + i < m) {
    T* out = nd.G + (size_t)(r0 + i) * nd.ldk;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (cg + 4 * q < n) out[cg + 4 * q] = acc[q];
  }
}

// Inverse of each lower-triangular diagonal block (column c by thread c,
// forward substitution), written as pad x pad (row-major, row stride ldD)
// with zeros outside the h x h lower triangle.  The columns are formed in
// shared memory (Xs[i][c], conflict-free across threads) and stored once, in
// rows: the substitution's reads of earlier entries never go to global memory
// (writing and re-reading D instead: c2 factorisation 21.64 vs 21.52 ms).
// Dynamic shared memory: two SOLVE_RB x (SOLVE_RB + 1) tiles of T.
template <class T>
__global__ void __launch_bounds__(64) invert_diag_blocks(const DinvTask<T>* __restrict__ tasks) {
  extern __shared__ __align__(16) unsigned char idb_smem[];
  T (*Ls)[SOLVE_RB + 1] = reinterpret_cast<T (*)[SOLVE_RB + 1]>(idb_smem);
  T (*Xs)[SOLVE_RB + 1] = reinterpret_cast<T (*)[SOLVE_RB + 1]>(idb_smem + sizeof(T) * SOLVE_RB * (SOLVE_RB + 1));
  const DinvTask<T> t = tasks[blockIdx.x];
  const int h = t.h, pad = t.pad, ldD = t.ldD, c = threadIdx.x;
  for (int idx = threadIdx.x; idx < h * h; idx += blockDim.x) {
    const int i = idx / h, j = idx - i * h;
    Ls[i][j] = (j <= i) ? t.L[(size_t)i * t.ld + j] : T(0);
  }
  for (int i = 0; i < SOLVE_RB; ++i) Xs[i][c] = T(0);
  __syncthreads();
  if (c < h) {
    for (int i = c; i < h; ++i) {
      T s = (i == c) ? T(1) : T(0);
      for (int k = c; k < i; ++k) s -= Ls[i][k] * Xs[k][c];
      Xs[i][c] = s / Ls[i][i];
    }
  }
  __syncthreads();
  T* D = t.D;
  if (c < pad)
    for (int i = 0; i < pad; ++i) D[(size_t)i * ldD + c] = (i < h && c < h) ? Xs[i][c] : T(0);
}

template <class A, class B>
__global__ void convert_kernel(const A* __restrict__ src, B* __restrict__ dst, int n) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (B)src[i];
}

// Zero the ticket and the items' counters after their last reader (the apply
// kernel), grid-stride.
__device__ __forceinline__ void clear_piece(int* c, int count) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) c[i] = 0;
}

__global__ void clear_counters(int* __restrict__ c, int count) {
  pdl_enter();
  clear_piece(c, count);
}

// last kernel of a mixed-precision apply: w64 = (double) w and the counters cleared
template <class T>
__global__ void convert_out_kernel(const T* __restrict__ src, double* __restrict__ dst, int n, int* __restrict__ c,
                                   int count) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (double)src[i];
  clear_piece(c, count);
}

}  // namespace

template <class T>
SolveEngine<T>::SolveEngine(FactorEngine<T>& F) : F_(F) {
  const char* e = std::getenv("RSCHOL_AUTOTUNE");
  autotune_ = e && e[0] == '1';
}

template <class T>
void SolveEngine<T>::plan() {
  PlanClock clk("solve plan");
  const Symbolic& S = F_.S;
  const int nn = (int)S.nodes.size();
  nodes_.assign(nn, SNode<T>{});
  std::vector<int> rel;
  // the single-vector apply's u and t of a supernode, each on whole 32-byte
  // sectors: a sector has one writer and is written whole (words stored into
  // part of a sector long evicted cost its reader a fill from DRAM)
  long long uCur = 0, tCur = 0;
  auto take = [](long long& cur, int len) {
    const long long at = cur;
    cur += (len + 7) & ~7;
    if (cur > INT_MAX) throw std::runtime_error("solve plan: a work vector has more than 2^31 entries");
    return (int)at;
  };
  long long xCur = 0, xiCur = 0, gCur = 0, wCur = 0;
  std::vector<long long> xOff(nn, 0), gOff(nn, 0), wOff(nn, -1);
  bytesPerApply_ = 0;
  std::vector<int> pos(S.n, -1);
  std::vector<DinvTask<T>> dinvTasks;
  std::vector<RowBlock> dinvOf;   // a task's supernode and block
  // X = L11^{-1} (n x ldx, upper triangle zero): the inverted 64 x 64 diagonal
  // blocks go in place
  auto plan_x = [&](int s) {
    SNode<T>& sn = nodes_[s];
    for (int b = 0; b * SOLVE_RB < sn.n; ++b) {
      DinvTask<T> t{};
      t.L = sn.L + (size_t)b * SOLVE_RB * sn.ld + (size_t)b * SOLVE_RB;
      t.ld = sn.ld;
      t.h = std::min(SOLVE_RB, sn.n - b * SOLVE_RB);
      t.pad = t.h;
      t.ldD = sn.ldx;
      dinvTasks.push_back(t);
      dinvOf.push_back(RowBlock{s, b});
    }
  };
  for (int s = 0; s < nn; ++s) {
    const Node& nd = S.nodes[s];
    SNode<T>& sn = nodes_[s];
    sn.ld = F_.ld[s];
    sn.n = nd.n;
    sn.m = nd.m();
    sn.c0 = nd.c0;
    sn.uOff = take(uCur, nd.m());
    sn.tOff = nd.compressed ? 0 : take(tCur, nd.n);
    if (!nd.compressed) {
      sn.L = F_.interior() + F_.frontOff[s];
      sn.r = 0;
      // FP64: an odd row stride in 16-byte units, so that a lane a row reads
      // shared memory without bank conflicts
      sn.ldk = (nd.n + 3) & ~3;
      if (sizeof(T) == 8 && (sn.ldk = (nd.n + 1) & ~1) % 4 == 0) sn.ldk += 2;
      sn.ldx = sn.ldk;
      bytesPerApply_ += 2.0 * sizeof(T) * ((double)nd.n + nd.m()) * nd.n;
    } else {
      sn.L = F_.compressed() + F_.frontOff[s];
      sn.r = F_.rank[s];
      sn.V = sn.r ? F_.vu() + F_.vOff[s] : nullptr;
      sn.U = sn.r ? F_.vu() + F_.uOff[s] : nullptr;
      wOff[s] = wCur;
      wCur = (wCur + (long long)nd.n * sn.r + 3) & ~3LL;
      sn.ldx = (nd.n + 3) & ~3;
      xOff[s] = xCur;
      xCur += (long long)nd.n * sn.ldx;
      bytesPerApply_ += 2.0 * sizeof(T) * ((double)nd.n * (nd.n + 1) / 2 + (double)sn.r * (nd.m() + nd.n));
    }
    plan_x(s);
  }
  // G and X of the interior supernodes, in the order of the levels (the members
  // of a work item are neighbours)
  for (auto& lv : F_.interiorLevels)
    for (int pass = 0; pass < 2; ++pass)
      for (int s : lv)
        if (group_member(s) == (pass == 0)) {
          gOff[s] = gCur;
          gCur += (long long)nodes_[s].m * nodes_[s].ldk;
          xOff[s] = xiCur;
          xiCur += (long long)nodes_[s].n * nodes_[s].ldk;
        }
  // rel maps (target index of each interior child's row in the parent front)
  for (int s = 0; s < nn; ++s) {
    const Node& nd = S.nodes[s];
    if (nd.compressed) continue;
    for (int a = 0; a < nd.m(); ++a) pos[nd.rows[a]] = a;
    for (int c : S.children[s]) {
      const Node& cn = S.nodes[c];
      nodes_[c].relOff = (long long)rel.size();
      for (int a = 0; a < cn.m(); ++a) {
        int g = cn.rows[a];
        rel.push_back(g <= nd.c1 ? g - nd.c0 : nd.n + pos[g]);
      }
    }
    for (int a = 0; a < nd.m(); ++a) pos[nd.rows[a]] = -1;
  }
  // contribution sources of compressed supernodes: interior roots' update
  // vectors first, then compressed descendants' V z
  std::vector<std::vector<SPull>> pl(nn);
  for (int c = 0; c < nn; ++c) {
    const Node& cn = S.nodes[c];
    bool isRoot = !cn.compressed && (cn.parent < 0 || S.nodes[cn.parent].compressed);
    if (!cn.compressed && !isRoot) continue;
    for (size_t q = 0; q < cn.interNode.size(); ++q)
      pl[cn.interNode[q]].push_back(SPull{c, cn.interStart[q], cn.interStart[q + 1], cn.compressed ? 1 : 0});
  }
  for (int s = 0; s < nn; ++s)
    if (S.nodes[s].compressed)
      std::stable_sort(pl[s].begin(), pl[s].end(), [](const SPull& a, const SPull& b) { return a.kind < b.kind; });
  // G of the supernodes of up to 64 columns: 64-row blocks of it, by column class
  // (<= 16, <= 32, <= 64)
  std::vector<RowBlock> opsWork;
  for (int cls = 0; cls < 3; ++cls) {
    const int lo = cls == 0 ? 0 : 8 << cls, hi = 16 << cls;
    opsClass_[cls].first = (long long)opsWork.size();
    for (int s = 0; s < nn; ++s)
      if (!S.nodes[s].compressed && S.nodes[s].n > lo && S.nodes[s].n <= hi)
        for (int b = 0; b * 64 < S.nodes[s].m(); ++b) opsWork.push_back(RowBlock{s, b});
    opsClass_[cls].second = (int)(opsWork.size() - opsClass_[cls].first);
  }
  clk.mark("layout");
  cudaStream_t st = F_.stream;
  auto up = [&](DevBuf& b, const void* src, size_t bytes) {
    b.alloc(bytes);
    if (bytes) RSCHOL_CUDA(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, st));
  };
  dT_.alloc(sizeof(T) * std::max(8LL, tCur));
  dX_.alloc(sizeof(T) * xCur);   // (what a factor does not have is not allocated)
  if (xCur > 0) RSCHOL_CUDA(cudaMemsetAsync(dX_.p, 0, sizeof(T) * xCur, st));   // upper triangles and padding stay zero
  dG_.alloc(sizeof(T) * std::max(1LL, gCur));
  dXi_.alloc(sizeof(T) * std::max(1LL, xiCur));
  RSCHOL_CUDA(cudaMemsetAsync(dG_.p, 0, dG_.bytes, st));   // the row padding stays zero
  RSCHOL_CUDA(cudaMemsetAsync(dXi_.p, 0, dXi_.bytes, st));
  dWc_.alloc(sizeof(T) * wCur);
  for (int s = 0; s < nn; ++s) {
    SNode<T>& sn = nodes_[s];
    sn.X = (S.nodes[s].compressed ? dX_ : dXi_).template as<T>() + xOff[s];
    if (S.nodes[s].compressed) sn.W = dWc_.as<T>() + wOff[s];
    else sn.G = dG_.as<T>() + gOff[s];
  }
  for (size_t q = 0; q < dinvTasks.size(); ++q) {
    const SNode<T>& sn = nodes_[dinvOf[q].node];
    dinvTasks[q].D = sn.X + (size_t)dinvOf[q].b * SOLVE_RB * (sn.ldx + 1);
  }
  nDinv_ = (int)dinvTasks.size();
  clk.mark("arenas");
  plan_inverse();
  clk.mark("inverse");
  // per-row contribution lists of the compressed supernodes (in source order)
  std::vector<long long> cstart;
  std::vector<int> ents;   // offsets into the update-vector arena
  {
    for (int s = 0; s < nn; ++s) {
      const Node& nd = S.nodes[s];
      if (!nd.compressed) continue;
      std::vector<int> cnt(nd.n + 1, 0);
      for (const SPull& P : pl[s])
        for (int a = P.a0; a < P.a1; ++a) cnt[S.nodes[P.src].rows[a] - nd.c0 + 1]++;
      for (int t = 0; t < nd.n; ++t) cnt[t + 1] += cnt[t];
      const long long base = (long long)ents.size();
      nodes_[s].cOff = (long long)cstart.size();
      for (int t = 0; t <= nd.n; ++t) cstart.push_back(base + cnt[t]);
      ents.resize(ents.size() + cnt[nd.n]);
      std::vector<int> fill(cnt.begin(), cnt.end() - 1);
      for (const SPull& P : pl[s]) {
        const SNode<T>& src = nodes_[P.src];
        for (int a = P.a0; a < P.a1; ++a) {
          ents[base + fill[S.nodes[P.src].rows[a] - nd.c0]++] = src.uOff + a;
        }
      }
    }
  }
  dWu_.alloc(sizeof(T) * std::max(8LL, uCur));
  RSCHOL_CUDA(cudaMemsetAsync(dWu_.p, 0, dWu_.bytes, st));
  clk.mark("lists");
  plan_items(rel, cstart, ents);
  clk.mark("items");
  up(dNodes_, nodes_.data(), nodes_.size() * sizeof(SNode<T>));
  up(dOpsWork_, opsWork.data(), opsWork.size() * sizeof(RowBlock));
  kAllocB_ = 0;   // the batched apply's buffers follow the new plan
  dSyncB_.release();
  ++batchGen_;
  up(dDinvTasks_, dinvTasks.data(), dinvTasks.size() * sizeof(DinvTask<T>));
  if (!std::is_same<T, double>::value) dW_.alloc(sizeof(T) * std::max(1, S.n));
  RSCHOL_CUDA(cudaStreamSynchronize(st));
  clk.mark("upload");
  launchesPerApply_ = 1 + (std::is_same<T, double>::value ? 1 : 2);
  bytesPerApply_ += 8.0 * 4 * S.n;
}

// Whether an interior supernode joins a group item: at most a warp's lanes of
// columns and its X and G within one stage.
template <class T>
bool SolveEngine<T>::group_member(int s) const {
  const SNode<T>& sn = nodes_[s];
  return sn.n <= IW_N && sn.m <= IW_M && (long long)(sn.n + sn.m) * sn.ldk * (long long)sizeof(T) <= ST_DATA;
}

// The work items of one application, in ticket order, with their descriptors.
// rel: target index of each row in the parent front (interior children);
// cstart / ents: contribution lists of the compressed columns.
template <class T>
void SolveEngine<T>::plan_items(const std::vector<int>& rel, const std::vector<long long>& cstart,
                                const std::vector<int>& ents) {
  const Symbolic& S = F_.S;
  const int nn = (int)S.nodes.size();
  cudaStream_t st = F_.stream;
  std::vector<ApplyItem> items;
  std::vector<int> blob(4, 0), phaseOf;
  int phase = 0;
  const int E = (int)sizeof(T);
  struct Done {   // "finished" of a supernode in one direction: a counter and its target
    int ctr = -1, target = 0;
  };
  std::vector<Done> up(nn), zDone(nn), solved(nn), tDone(nn), sDone(nn), fDone(nn);
  std::vector<int> upCount(nn, 0);
  int nCtr = 2;   // [0] error word, [1] ticket
  std::vector<int> produced(2, 0);
  auto counter = [&]() {
    produced.push_back(0);
    return nCtr++;
  };
  auto pairs_of = [&](std::vector<int>& w, const Done& d) {
    for (size_t q = 0; q + 1 < w.size(); q += 2)
      if (w[q] == d.ctr) {
        w[q + 1] = std::max(w[q + 1], d.target);
        return;
      }
    w.push_back(d.ctr);
    w.push_back(d.target);
  };
  auto i32 = [](long long v) {
    if (v < 0 || v > INT_MAX) throw std::runtime_error("solve plan: a work vector has more than 2^31 entries");
    return (int)v;
  };
  auto bytes16 = [](long long b) { return (int)((b + 15) & ~15LL); };
  auto open_part = [&]() {   // the blob's next 16-byte boundary
    blob.resize((blob.size() + 3) & ~(size_t)3, 0);
    return i32((long long)blob.size());
  };
  // Append an item.  Its descriptor is written straight into the blob: begin
  // (the waits), then the header and the lists, then end; an offset of a list
  // in the descriptor is the blob's size then minus it.desc.
  auto begin = [&](ApplyItem& it, const std::vector<int>& waits) {
    it.waits = (int)waits.size() / 2;
    for (size_t q = 0; q < waits.size(); q += 2)   // every wait must be met by earlier items
      if (produced[waits[q]] < waits[q + 1]) throw std::runtime_error("solve plan: an item waits on a later one");
    it.desc = open_part();
    blob.insert(blob.end(), waits.begin(), waits.end());
  };
  auto off16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 != 0; };
  auto end = [&](ApplyItem& it) {
    const long long db = 4LL * (open_part() - it.desc);
    it.descBytes = db <= ST_DESC ? (int)db : 0;
    if (it.descBytes == 0 || it.descBytes + it.desc2Bytes > ST_DESC) it.desc2Bytes = 0;
    // what a bulk copy needs: 16-byte boundaries, and room in a stage
    if ((it.bytes0 > 0 && off16(it.g0)) || (it.bytes1 > 0 && off16(it.g1)) || (it.bytes0 | it.bytes1) % 16 != 0 ||
        it.bytes0 + it.bytes1 > ST_DATA)
      throw std::runtime_error("solve plan: a piece of the factor does not fit its stage");
    produced[it.sig]++;
    items.push_back(it);
    phaseOf.push_back(phase);
  };
  auto push = [&](ApplyItem& it, const std::vector<int>& waits, std::initializer_list<int> header) {
    begin(it, waits);
    blob.insert(blob.end(), header.begin(), header.end());
    end(it);
  };

  // Row stride of partial sums: whole 32-byte sectors, so that an item stores
  // no part of one (words into a line long evicted cost its reader a fill from
  // DRAM: c2, 6 us in every reading item)
  auto part_ld = [](int n) { return (n + 7) & ~7; };
  // chunks of the larger interior supernodes: rows of G and of X per item
  struct Chunks {
    int nch, rc, per, staged, whole;
  };
  std::vector<Chunks> ch(nn);
  long long ipCur = 0;
  std::vector<long long> ipOff(nn, 0);
  fLen_ = 4;
  for (int s = 0; s < nn; ++s) {
    const SNode<T>& sn = nodes_[s];
    if (S.nodes[s].compressed || group_member(s)) continue;
    fLen_ = std::max(fLen_, sn.ldk);
    Chunks& c = ch[s];
    const int maxRows = ST_DATA / (sn.ldk * E);
    c.staged = maxRows >= 8;
    const int cap = c.staged ? maxRows : 32;   // too wide for a stage: 32 rows, read in place
    c.nch = std::max(1, (sn.n + sn.m + cap - 1) / cap);
    // (multiples of a sector, so that a chunk stores whole sectors of u and t,
    // where a stage holds two of them)
    const int al = cap >= 2 * (32 / E) ? 32 / E : 1;
    c.whole = al > 1;
    for (;; ++c.nch) {
      c.rc = ((sn.m + c.nch - 1) / c.nch + al - 1) / al * al;
      c.per = ((sn.n + c.nch - 1) / c.nch + al - 1) / al * al;
      if (c.rc + c.per <= cap && c.rc <= 64) break;
    }
    if (c.rc + c.per > GT) throw std::runtime_error("solve plan: a chunk has more rows than a group has threads");
    ipOff[s] = ipCur;
    ipCur += (long long)c.nch * part_ld(sn.n);
  }
  // groups of small supernodes, per level
  std::vector<std::vector<std::vector<int>>> groups(F_.interiorLevels.size());
  std::vector<int> childCount(nn, 0);
  int dev = 0;
  RSCHOL_CUDA(cudaGetDevice(&dev));
  RSCHOL_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
  for (size_t l = 0; l < F_.interiorLevels.size(); ++l) {
    long long bytes = 0, ints = 0;
    // one member a warp while the batched kernel's consumer groups (two CTAs an SM) are
    // enough to take a level so (up to eight always: 2D 40 x 37 FP64 100 against 94.5 us a
    // call, four columns 179 against 166; 2D 128^2, a step, 1802 against 1727)
    int members = 0;
    for (int s : F_.interiorLevels[l]) members += group_member(s);
    const int most = members <= GW * 2 * NGRP * sms_ ? GW : GRP;
    for (int s : F_.interiorLevels[l]) {
      if (!group_member(s)) continue;
      const SNode<T>& sn = nodes_[s];
      const long long b = (long long)(sn.n + sn.m) * sn.ldk * E;
      long long q = GH + 8 + sn.n + sn.m + 1;
      for (int c : S.children[s]) q += nodes_[c].m + 2;
      auto& g = groups[l];
      if (g.empty() || (int)g.back().size() == most || bytes + b > ST_DATA || 4 * (ints + q) > ST_DESC) {
        g.push_back({});
        bytes = ints = 0;
      }
      g.back().push_back(s);
      bytes += b;
      ints += q;
    }
  }
  // the pull lists of a supernode's columns and rows, in child order ...
  std::vector<int> pStart, pEnt, pFill;
  auto pull_prepare = [&](int s) {
    const int R = nodes_[s].n + nodes_[s].m;
    pStart.assign(R + 1, 0);
    for (int c : S.children[s]) {
      const int* rl = rel.data() + nodes_[c].relOff;
      for (int a = 0; a < nodes_[c].m; ++a) pStart[rl[a] + 1]++;
    }
    for (int t = 0; t < R; ++t) pStart[t + 1] += pStart[t];
    pEnt.resize(pStart[R]);
    pFill.assign(pStart.begin(), pStart.end() - 1);
    for (int c : S.children[s]) {
      const int* rl = rel.data() + nodes_[c].relOff;
      for (int a = 0; a < nodes_[c].m; ++a) pEnt[pFill[rl[a]]++] = nodes_[c].uOff + a;
    }
  };
  // ... and those of its rows [r0, r0 + count) of [columns; rows], appended to the
  // blob as offsets and entries
  auto pull_lists = [&](int r0, int count) {
    const int e0 = pStart[r0];
    for (int i = 0; i <= count; ++i) blob.push_back(pStart[r0 + i] - e0);
    blob.insert(blob.end(), pEnt.begin() + e0, pEnt.begin() + pStart[r0 + count]);
  };
  auto has_pull = [&](int s) {
    for (int c : S.children[s])
      if (nodes_[c].m > 0) return true;
    return false;
  };
  std::vector<int> waits;
  // ---- interior, forward
  for (size_t l = 0; l < F_.interiorLevels.size(); ++l) {
    ++phase;
    for (auto& g : groups[l]) {
      ApplyItem it{};
      it.kind = IT_FGRP;
      it.sig = counter();
      it.count = (int)g.size();
      const SNode<T>& first = nodes_[g[0]];
      it.g0 = first.G;
      it.g1 = first.X;
      waits.clear();
      long long gE = 0, xE = 0;
      for (int s : g) {
        gE += (long long)nodes_[s].m * nodes_[s].ldk;
        xE += (long long)nodes_[s].n * nodes_[s].ldk;
        for (int c : S.children[s]) pairs_of(waits, up[c]);
      }
      it.bytes0 = (int)(gE * E);
      it.bytes1 = (int)(xE * E);
      begin(it, waits);
      const size_t h0 = blob.size();
      blob.resize(h0 + GH * g.size(), 0);
      for (size_t q = 0; q < g.size(); ++q) {
        const int s = g[q];
        const SNode<T>& sn = nodes_[s];
        int* h = &blob[h0 + GH * q];
        h[0] = sn.n;
        h[1] = sn.m;
        h[2] = sn.c0;
        h[3] = sn.uOff;
        h[4] = (int)(sn.G - first.G);
        h[5] = (int)(gE + (sn.X - first.X));
        h[7] = sn.ldk;
        h[8] = sn.tOff;
        if (has_pull(s)) {
          h[6] = (int)blob.size() - it.desc;
          pull_prepare(s);
          pull_lists(0, sn.n + sn.m);
        }
        up[s] = fDone[s] = Done{it.sig, 1};
      }
      end(it);
    }
    for (int s : F_.interiorLevels[l]) {
      if (group_member(s)) continue;
      const SNode<T>& sn = nodes_[s];
      const Chunks& c = ch[s];
      waits.clear();
      for (int k : S.children[s]) pairs_of(waits, up[k]);
      up[s] = fDone[s] = Done{counter(), c.nch};
      const bool pull = has_pull(s);
      int shared = 0, sharedBytes = 0;
      if (pull) {   // the columns' lists, once for all chunks
        pull_prepare(s);
        shared = open_part();
        pull_lists(0, sn.n);
        sharedBytes = 4 * (open_part() - shared);
      }
      for (int b = 0; b < c.nch; ++b) {
        const int a0 = std::min(sn.m, b * c.rc), rows = std::min(c.rc, sn.m - a0);
        const int s0 = std::min(sn.n, b * c.per), sr = std::min(c.per, sn.n - s0);
        ApplyItem it{};
        it.kind = IT_FWD;
        it.sig = up[s].ctr;
        it.g0 = sn.G + (size_t)a0 * sn.ldk;
        it.g1 = sn.X + (size_t)s0 * sn.ldk;
        if (c.staged) {
          it.bytes0 = rows * sn.ldk * E;
          it.bytes1 = sr * sn.ldk * E;
        }
        it.desc2 = shared;
        it.desc2Bytes = sharedBytes;
        begin(it, waits);
        const int list = pull ? (int)blob.size() - it.desc + 10 : 0;
        blob.insert(blob.end(), {sn.n, rows, sn.c0, sn.uOff + a0, s0, sr, list, sn.ldk, sn.tOff, c.whole});
        if (pull) pull_lists(sn.n + a0, rows);
        end(it);
      }
    }
  }
  // ---- compressed levels
  const int L = (int)F_.compressedLevels.size();
  auto rows_per = [&](int r, int& staged) {   // rows of an r-wide matrix per item
    if (r == 0) {
      staged = 0;
      return ROWS8;
    }
    const int fit = ST_DATA / (r * E) & ~7;
    staged = fit >= 8;
    return staged ? std::min(ROWS8, fit) : 16;
  };
  long long zpCur = 0, spCur = 0, ypCur = 0, xpCur = 0;
  std::vector<long long> zpOff(nn), spOff(nn), ypOff(nn), xpOff(nn);
  // Many partials of z or s are added once, by items of CR_COLS columns, before
  // the items that read the sums: each of those would otherwise add all of them
  // (c2: 200 partials of s, 8 us in every item; with the extra step 1.5 + 1.5).
  // Up to CR_MIN partials the extra step costs more than it saves.
  constexpr int CR_COLS = 16, CR_MIN = 12;
  auto emit_cr = [&](Done& d, long long& off, int rp, int isS) {
    const int parts = d.target;
    if (parts <= CR_MIN) return parts;
    waits.clear();
    pairs_of(waits, d);
    const long long sums = off + (long long)parts * rp;   // the row after the partials
    const Done all{counter(), (rp + CR_COLS - 1) / CR_COLS};
    for (int k0 = 0; k0 < rp; k0 += CR_COLS) {
      ApplyItem it{};
      it.kind = IT_CR;
      it.sig = all.ctr;
      push(it, waits, {i32(off + k0), parts, rp, std::min(CR_COLS, rp - k0), i32(sums + k0), isS});
    }
    d = all;
    off = sums;
    return 1;
  };
  std::vector<int> zParts(nn, 0), sParts(nn, 0);
  std::vector<int> yBase(nn, -1);   // first of the supernode's per-row-block counters of y
  constexpr int YR = Y_ROWS, YC = Y_COLS<T>, TR = T_ROWS<T>;
  for (int j = 0; j < nn; ++j) {
    if (!S.nodes[j].compressed) continue;
    const SNode<T>& sn = nodes_[j];
    int sg = 0;
    const int cb = rows_per(sn.r, sg), rp = part_ld(sn.r);
    zpOff[j] = zpCur;
    zpCur += (long long)((sn.n + cb - 1) / cb + 1) * rp;
    spOff[j] = spCur;
    spCur += (long long)((sn.m + cb - 1) / cb + 1) * rp;
    ypOff[j] = ypCur;
    ypCur += (long long)part_ld(sn.n) * ((sn.n + YC - 1) / YC);
    xpOff[j] = xpCur;
    xpCur += (long long)part_ld(sn.n) * ((sn.n + TR - 1) / TR);
  }
  auto emit_cf = [&](int l) {
    ++phase;
    for (int j : F_.compressedLevels[l]) {
      const SNode<T>& sn = nodes_[j];
      int sg = 0;
      const int cb = rows_per(sn.r, sg), rp = part_ld(sn.r), nb = (sn.n + cb - 1) / cb;
      waits.clear();
      for (int c : S.children[j]) pairs_of(waits, up[c]);
      zDone[j] = Done{counter(), nb};
      up[j] = zDone[j];
      for (int b = 0; b < nb; ++b) {
        const int j0 = b * cb, cols = std::min(cb, sn.n - j0);
        ApplyItem it{};
        it.kind = IT_CF;
        it.sig = zDone[j].ctr;
        it.g0 = sn.W + (size_t)j0 * sn.r;
        it.bytes0 = sg ? bytes16((long long)cols * sn.r * E) : 0;
        begin(it, waits);
        const int list = (int)blob.size() - it.desc + 5;
        blob.insert(blob.end(), {sn.c0 + j0, cols, sn.r, i32(zpOff[j] + (long long)b * rp), list});
        const long long* cs = &cstart[sn.cOff + j0];
        for (int i = 0; i <= cols; ++i) blob.push_back(i32(cs[i] - cs[0]));
        blob.insert(blob.end(), ents.begin() + cs[0], ents.begin() + cs[cols]);
        end(it);
      }
    }
  };
  std::vector<Done> zSum(nn);   // z of a supernode ready to be read
  auto emit_cu = [&](int l) {
    ++phase;
    for (int j : F_.compressedLevels[l]) {
      zSum[j] = zDone[j];
      if (nodes_[j].m > 0 && nodes_[j].r > 0) zParts[j] = emit_cr(zSum[j], zpOff[j], part_ld(nodes_[j].r), 0);
    }
    for (int j : F_.compressedLevels[l]) {
      const SNode<T>& sn = nodes_[j];
      if (sn.m == 0 || sn.r == 0) continue;
      int sg = 0;
      const int rb = rows_per(sn.r, sg), nb = (sn.m + rb - 1) / rb;
      waits.clear();
      pairs_of(waits, zSum[j]);
      up[j] = Done{counter(), nb};
      for (int b = 0; b < nb; ++b) {
        const int a0 = b * rb, rows = std::min(rb, sn.m - a0);
        ApplyItem it{};
        it.kind = IT_CU;
        it.sig = up[j].ctr;
        it.g0 = sn.V + (size_t)a0 * sn.r;
        it.bytes0 = sg ? bytes16((long long)rows * sn.r * E) : 0;
        push(it, waits, {rows, sn.r, i32(zpOff[j]), zParts[j], sn.uOff + a0});
      }
    }
  };
  // a tile of X: its packed copy, one stage
  std::vector<PackTile> packs;
  std::vector<int> packItems;   // items whose g0 is the tile of the same place in packs
  auto tile_of = [&](ApplyItem& it, int j, int j0, int i0, int boxCols, int boxRows) {
    packItems.push_back((int)items.size());
    packs.push_back(PackTile{j, i0, j0, boxCols, boxRows});
    it.bytes0 = ST_DATA;
  };
  auto emit_y = [&](int l) {
    ++phase;
    for (int j : F_.compressedLevels[l]) {
      const SNode<T>& sn = nodes_[j];
      const int ncb = (sn.n + YC - 1) / YC, nt = (sn.n + TR - 1) / TR;
      waits.clear();
      pairs_of(waits, zDone[j]);
      yBase[j] = nCtr;
      for (int q = 0; q < nt; ++q) counter();
      for (int i0 = 0; i0 < sn.n; i0 += YR)
        for (int jb = 0; jb * YC <= i0 + YR - 1 && jb < ncb; ++jb) {
          const int j0 = jb * YC, rows = std::min(YR, sn.n - i0);
          const int cols = std::min({YC, sn.n - j0, i0 + rows - j0});   // up to the diagonal
          if (cols <= 0) throw std::runtime_error("solve plan: an empty tile");
          ApplyItem it{};
          it.kind = IT_Y;
          it.sig = yBase[j] + i0 / TR;
          tile_of(it, j, j0, i0, YC, YR);
          push(it, waits, {sn.c0 + j0, cols, rows, i32(ypOff[j] + (long long)jb * part_ld(sn.n) + i0)});
        }
    }
  };
  auto emit_t = [&](int l) {
    ++phase;
    for (int j : F_.compressedLevels[l]) {
      const SNode<T>& sn = nodes_[j];
      const int ncb = (sn.n + YC - 1) / YC, nt = (sn.n + TR - 1) / TR;
      tDone[j] = Done{counter(), 0};
      for (int ib = 0; ib < nt; ++ib) {
        const int i0 = ib * TR, rows = std::min(TR, sn.n - i0);
        std::vector<int> waits;
        pairs_of(waits, Done{yBase[j] + ib, produced[yBase[j] + ib]});
        for (int j0 = 0; j0 <= i0 + TR - 1 && j0 < sn.n; j0 += T_COLS) {
          const int cols = std::min(T_COLS, sn.n - j0);
          ApplyItem it{};
          it.kind = IT_XT;
          it.sig = tDone[j].ctr;
          tDone[j].target++;
          tile_of(it, j, j0, i0, T_COLS, TR);
          push(it, waits, {rows, cols, i32(ypOff[j] + i0), part_ld(sn.n), i0,
                                i32(xpOff[j] + (long long)ib * part_ld(sn.n) + j0), ncb});
        }
      }
    }
  };
  auto emit_cs = [&](int l) {
    ++phase;
    for (int j : F_.compressedLevels[l]) {
      const SNode<T>& sn = nodes_[j];
      if (sn.m == 0 || sn.r == 0) continue;
      int sg = 0;
      const int rb = rows_per(sn.r, sg), rp = part_ld(sn.r), nb = (sn.m + rb - 1) / rb;
      waits.clear();
      pairs_of(waits, solved[S.nodes[j].parent]);
      sDone[j] = Done{counter(), nb};
      for (int b = 0; b < nb; ++b) {
        const int a0 = b * rb, rows = std::min(rb, sn.m - a0);
        ApplyItem it{};
        it.kind = IT_CS;
        it.sig = sDone[j].ctr;
        it.g0 = sn.V + (size_t)a0 * sn.r;
        it.bytes0 = sg ? bytes16((long long)rows * sn.r * E) : 0;
        begin(it, waits);
        const int list = (int)blob.size() - it.desc + 4;
        blob.insert(blob.end(), {rows, sn.r, i32(spOff[j] + (long long)b * rp), list});
        blob.insert(blob.end(), S.nodes[j].rows.begin() + a0, S.nodes[j].rows.begin() + a0 + rows);
        end(it);
      }
    }
    for (int j : F_.compressedLevels[l])
      if (sDone[j].ctr >= 0) sParts[j] = emit_cr(sDone[j], spOff[j], part_ld(nodes_[j].r), 1);
  };
  auto emit_cx = [&](int l) {
    ++phase;
    for (int j : F_.compressedLevels[l]) {
      const SNode<T>& sn = nodes_[j];
      int sg = 0;
      const int cb = rows_per(sn.r, sg), nb = (sn.n + cb - 1) / cb, nt = (sn.n + TR - 1) / TR;
      waits.clear();
      pairs_of(waits, tDone[j]);
      if (sDone[j].ctr >= 0) pairs_of(waits, sDone[j]);
      solved[j] = Done{counter(), nb};
      for (int b = 0; b < nb; ++b) {
        const int j0 = b * cb, cols = std::min(cb, sn.n - j0);
        ApplyItem it{};
        it.kind = IT_CX;
        it.sig = solved[j].ctr;
        it.g0 = sn.W + (size_t)j0 * sn.r;
        it.bytes0 = sg && sDone[j].ctr >= 0 ? bytes16((long long)cols * sn.r * E) : 0;
        push(it, waits, {sn.c0 + j0, cols, sn.r, i32(spOff[j]), sParts[j],
                              i32(xpOff[j] + j0), part_ld(sn.n), j0, j0 / T_COLS * T_COLS / TR, nt});
      }
    }
  };
  // The products with X follow their level's up pieces one level behind, so
  // that the chain up the tree comes first and they fill its gaps.
  for (int l = 0; l < L; ++l) {
    emit_cf(l);
    emit_cu(l);
    if (l >= 1) emit_y(l - 1);
    if (l >= 2) emit_t(l - 2);
  }
  if (L >= 1) emit_y(L - 1);
  if (L >= 1) emit_t(L - 1);
  if (L >= 2) emit_t(L - 2);
  for (int l = L - 1; l >= 0; --l) {
    emit_cs(l);
    emit_cx(l);
  }
  // ---- interior, backward
  for (int l = (int)F_.interiorLevels.size() - 1; l >= 0; --l) {
    ++phase;
    auto wait_for = [&](int s, std::vector<int>& waits) {
      const int p = S.nodes[s].parent;
      pairs_of(waits, p >= 0 ? solved[p] : fDone[s]);
    };
    for (int s : F_.interiorLevels[l]) {
      if (group_member(s)) continue;
      const SNode<T>& sn = nodes_[s];
      const Chunks& c = ch[s];
      waits.clear();
      pairs_of(waits, fDone[s]);
      wait_for(s, waits);
      const int nch = std::max((sn.m + c.rc - 1) / std::max(1, c.rc), (sn.n + c.per - 1) / c.per);   // not empty
      const Done parts{counter(), nch};
      for (int b = 0; b < nch; ++b) {
        const int a0 = std::min(sn.m, b * c.rc), rows = std::min(c.rc, sn.m - a0);
        const int s0 = std::min(sn.n, b * c.per), sr = std::min(c.per, sn.n - s0);
        ApplyItem it{};
        it.kind = IT_BWD;
        it.early = 1;
        it.sig = parts.ctr;
        it.g0 = sn.G + (size_t)a0 * sn.ldk;
        it.g1 = sn.X + (size_t)s0 * sn.ldk;
        if (c.staged) {
          it.bytes0 = rows * sn.ldk * E;
          it.bytes1 = sr * sn.ldk * E;
        }
        begin(it, waits);
        const int list = (int)blob.size() - it.desc + 11;
        blob.insert(blob.end(),
                    {sn.n, rows, sn.c0, i32(ipOff[s]), b, nch, list, sn.ldk, part_ld(sn.n), sn.tOff + s0, sr});
        blob.insert(blob.end(), S.nodes[s].rows.begin() + a0, S.nodes[s].rows.begin() + a0 + rows);
        end(it);
      }
      solved[s] = parts;
    }
    for (auto& g : groups[l]) {
      ApplyItem it{};
      it.kind = IT_BGRP;
      it.sig = counter();
      it.count = (int)g.size();
      const SNode<T>& first = nodes_[g[0]];
      it.g0 = first.G;
      it.g1 = first.X;
      long long gE = 0, xE = 0;
      waits.clear();
      for (int s : g) pairs_of(waits, fDone[s]);   // (one item, forward)
      it.early = (int)waits.size() / 2;
      for (int s : g) {
        gE += (long long)nodes_[s].m * nodes_[s].ldk;
        xE += (long long)nodes_[s].n * nodes_[s].ldk;
        wait_for(s, waits);
      }
      it.bytes0 = (int)(gE * E);
      it.bytes1 = (int)(xE * E);
      begin(it, waits);
      const size_t h0 = blob.size();
      blob.resize(h0 + GH * g.size(), 0);
      for (size_t q = 0; q < g.size(); ++q) {
        const SNode<T>& sn = nodes_[g[q]];
        int* h = &blob[h0 + GH * q];
        h[0] = sn.n;
        h[1] = sn.m;
        h[2] = sn.c0;
        h[4] = (int)(sn.G - first.G);
        h[5] = (int)(gE + (sn.X - first.X));
        h[6] = (int)blob.size() - it.desc;
        h[7] = sn.ldk;
        h[8] = sn.tOff;
        blob.insert(blob.end(), S.nodes[g[q]].rows.begin(), S.nodes[g[q]].rows.end());
        solved[g[q]] = Done{it.sig, 1};
      }
      end(it);
    }
    ++phase;
    // the sums of a level's chunks after all of them: next to its chunks such
    // an item would hold up its group
    for (int s : F_.interiorLevels[l]) {
      if (group_member(s) || solved[s].target == 1) continue;
      ApplyItem it{};
      it.kind = IT_BR;
      it.sig = counter();
      waits.clear();
      pairs_of(waits, solved[s]);
      // many parts: by columns, 1024 entries an item, so that a block of right-hand
      // sides has no item that reads megabytes (3D 40^3, k = 32: an item of 100 parts
      // of 400 columns held the level up for 130 - 180 us)
      const int n = nodes_[s].n, parts = solved[s].target, w = std::max(16, 1024 / parts & ~15);
      for (int c = 0; c < n; c += w)
        push(it, waits, {std::min(w, n - c), nodes_[s].c0 + c, i32(ipOff[s] + c), parts, part_ld(n)});
      solved[s] = Done{it.sig, (n + w - 1) / w};
    }
  }
  nItems_ = (int)items.size();
  // shared memory: the stages, and per consumer group two areas of GT vectors
  // and the f buffer (or a group item's buffers in their place)
  work_ = (std::max(GW * (IW_N + IW_M), 2 * GT * Vec16<T>::V + std::min(fLen_, F_TILE<T>)) + 3) & ~3;
  smem_ = (size_t)NSTAGE * ST_BYTES + NGRP * sizeof(T) * (size_t)work_;
  // the limit belongs to the kernel, not to this factor: what the widest supernode needs
  constexpr int maxWork = std::max(GW * (IW_N + IW_M), 2 * GT * Vec16<T>::V + F_TILE<T>);
  constexpr int maxSmem = NSTAGE * ST_BYTES + NGRP * (int)sizeof(T) * maxWork;
  static_assert(3 * (maxSmem + 1536) <= 228 * 1024, "three CTAs an SM");   // (static and reserved shared memory beside)
  RSCHOL_CUDA(cudaFuncSetAttribute(apply_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxSmem));
  int per = 0;
  RSCHOL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, apply_kernel<T>, NGRP * GT + 32, smem_));
  grid_ = std::min(std::max(1, nItems_), sms_ * std::max(1, per));
  // phases that a few items per group work off
  std::vector<int> count(phase + 1, 0);
  for (int q : phaseOf) count[q]++;
  for (size_t q = 0; q < items.size(); ++q) items[q].shallow = count[phaseOf[q]] <= SHALLOW * NGRP * grid_;
  nSync_ = nCtr;
  auto upload = [&](DevBuf& b, const void* src, size_t bytes) {
    b.alloc(bytes);
    if (bytes) RSCHOL_CUDA(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, st));
  };
  nPacks_ = (int)packs.size();
  upload(dPackTiles_, packs.data(), packs.size() * sizeof(PackTile));
  dPacked_.alloc(packs.size() * (size_t)ST_DATA);
  for (size_t q = 0; q < packItems.size(); ++q)
    items[packItems[q]].g0 = dPacked_.as<unsigned char>() + q * (size_t)ST_DATA;
  upload(dItems_, items.data(), items.size() * sizeof(ApplyItem));
  upload(dBlob_, blob.data(), blob.size() * sizeof(int));
  dSync_.alloc(sizeof(int) * nCtr);
  RSCHOL_CUDA(cudaMemsetAsync(dSync_.p, 0, sizeof(int) * nCtr, st));
  dZp_.alloc(sizeof(T) * zpCur);
  dSp_.alloc(sizeof(T) * spCur);
  dYp_.alloc(sizeof(T) * ypCur);
  dXp_.alloc(sizeof(T) * xpCur);
  dIp_.alloc(sizeof(T) * ipCur);
  RSCHOL_CUDA(cudaStreamSynchronize(st));   // the host arrays go out of scope
}

template <class T>
void SolveEngine<T>::plan_inverse() {
  // X = L11^{-1} of every supernode of more than 64 columns by recursive doubling:
  // with the diagonal 64 x 64 inverses in place, for block sizes sz = 64, 128, ...
  // every pair (A, B) of consecutive sz-blocks gets X_BA = -X_BB (L_BA X_AA).
  // Both products run by 64-column (64-row) blocks whose K stops at the
  // triangle, so the work is n^3 / 3 per supernode.
  const Symbolic& S = F_.S;
  // X of a compressed supernode by split products on the tensor cores; what takes the
  // place of FP32 sums with the factor itself -- X and G of the interior supernodes, and
  // W -- by FP32 products.  (Those in split TF32 too, 22 bits an operand: the error of an
  // exact mixed application against 64 bits 1.3e-6 - 6.6e-6 on 3D 12^3 - 32x31x30,
  // sigma 0; with FP32 products 2.4e-7 - 3.9e-7, by substitution 4.3e-7 - 1.8e-6.)
  const bool tcX = std::is_same<T, float>::value && F_.tensor_cores();
  const int nn = (int)S.nodes.size();
  int maxN = 0;
  for (int s = 0; s < nn; ++s) maxN = std::max(maxN, S.nodes[s].n);
  long long t1Max = 1;
  for (int sz = SOLVE_RB; sz < maxN; sz *= 2) {
    long long t1 = 0;
    for (int s = 0; s < nn; ++s) {
      const int n = S.nodes[s].n;
      for (int A0 = 0; A0 + sz < n; A0 += 2 * sz) t1 += (long long)std::min(sz, n - A0 - sz) * sz;
    }
    t1Max = std::max(t1Max, t1);
  }
  dT1_.alloc(sizeof(T) * t1Max);
  std::vector<GemmTask<T>> tasks;
  xSteps_.clear();
  auto mk = [&](const T* A, int lda, const T* B, int ldb, T* C, int ldc, int M, int N, int K, T alpha) {
    GemmTask<T> t{};
    t.A = A;
    t.B = B;
    t.C = C;
    t.M = M;
    t.N = N;
    t.K = K;
    t.lda = lda;
    t.ldb = ldb;
    t.ldc = ldc;
    t.alpha = alpha;
    t.beta = T(0);
    t.split = 1;
    t.kSplit = 1;
    t.kLen = K;
    return t;
  };
  auto flush = [&](std::vector<GemmTask<T>>& batch, bool tc) {
    if (batch.empty()) return;
    int maxN = 0, maxK = 0;
    long long big = 0;
    for (auto& t : batch) {
      maxN = std::max(maxN, t.N);
      maxK = std::max(maxK, t.K);
      big += (long long)((t.M + 127) / 128) * ((t.N + 63) / 64);
    }
    // (the SIMT tiles of 128 rows where the factor's own launches take them)
    const bool rows128 = !tc && simt_rows128<T>(big, maxK);
    const int bn = tc ? tc_tile_n(maxN) : simt_tile<T>, rpt = tc || rows128 ? 128 : simt_tile<T>;
    int tiles = 0;
    for (auto& t : batch) {
      t.tilesN = (t.N + bn - 1) / bn;
      t.bn = bn;
      t.tileBase = tiles;
      tiles += ((t.M + rpt - 1) / rpt) * t.tilesN;
    }
    XStep xs{(long long)tasks.size(), (int)batch.size(), tiles, tc ? XS_TC : rows128 ? XS_ROWS128 : XS_SIMT};
    xs.bn = bn;
    xSteps_.push_back(xs);
    tasks.insert(tasks.end(), batch.begin(), batch.end());
    batch.clear();
  };
  for (int sz = SOLVE_RB; sz < maxN; sz *= 2) {
    std::vector<GemmTask<T>> b1[2], b2[2];   // interior, compressed
    long long t1cur = 0;
    for (int s = 0; s < nn; ++s) {
      const int n = S.nodes[s].n, ld = nodes_[s].ld, lx = nodes_[s].ldx;
      const T* L = nodes_[s].L;
      T* X = nodes_[s].X;
      const int c = S.nodes[s].compressed;
      for (int A0 = 0; A0 + sz < n; A0 += 2 * sz) {
        const int B0 = A0 + sz, bsz = std::min(sz, n - B0);
        T* T1 = dT1_.as<T>() + t1cur;
        t1cur += (long long)bsz * sz;
        for (int a = 0; a * SOLVE_RB < sz; ++a)   // T1[:, a] = L_BA[:, a:] X_AA[a:, a]
          b1[c].push_back(mk(L + (size_t)B0 * ld + A0 + a * SOLVE_RB, ld,
                          X + (size_t)(A0 + a * SOLVE_RB) * lx + A0 + a * SOLVE_RB, lx, T1 + a * SOLVE_RB, sz, bsz,
                          SOLVE_RB, sz - a * SOLVE_RB, T(1)));
        for (int b = 0; b * SOLVE_RB < bsz; ++b) {   // X_BA[b, :] = -X_BB[b, :b] T1[:b, :]
          const int hb = std::min(SOLVE_RB, bsz - b * SOLVE_RB), K = std::min(bsz, (b + 1) * SOLVE_RB);
          b2[c].push_back(mk(X + (size_t)(B0 + b * SOLVE_RB) * lx + B0, lx, T1, sz,
                          X + (size_t)(B0 + b * SOLVE_RB) * lx + A0, lx, hb, sz, K, T(-1)));
        }
      }
    }
    for (auto* b : {b1, b2}) {
      flush(b[0], false);
      flush(b[1], tcX);
    }
  }
  // then the products the apply reads: W = X^T U of the compressed supernodes and
  // G = L21 X of the interior ones of more than 64 columns, by blocks whose K starts
  // at the triangle
  std::vector<GemmTask<T>> bw, bi;
  for (int s = 0; s < nn; ++s) {
    const SNode<T>& sn = nodes_[s];
    const int n = sn.n, lx = sn.ldx;
    if (S.nodes[s].compressed) {
      constexpr int blk = simt_rows<T>;
      for (int j0 = 0; sn.r > 0 && j0 < n; j0 += blk) {
        GemmTask<T> t = mk(sn.X + (size_t)j0 * lx + j0, lx, sn.U + (size_t)j0 * sn.r, sn.r,
                           const_cast<T*>(sn.W) + (size_t)j0 * sn.r, sn.r, std::min(blk, n - j0), sn.r, n - j0, T(1));
        t.tA = 1;
        bw.push_back(t);
      }
    } else if (n > SOLVE_RB && sn.m > 0) {
      constexpr int blk = simt_tile<T>;
      for (int j0 = 0; j0 < n; j0 += blk)
        bi.push_back(mk(sn.L + (size_t)n * sn.ld + j0, sn.ld, sn.X + (size_t)j0 * lx + j0, lx, sn.G + j0, sn.ldk,
                        sn.m, std::min(blk, n - j0), n - j0, T(1)));
    }
  }
  flush(bw, false);
  flush(bi, false);
  dXGemm_.alloc(std::max<size_t>(16, tasks.size() * sizeof(GemmTask<T>)));
  if (!tasks.empty())
    RSCHOL_CUDA(cudaMemcpyAsync(dXGemm_.p, tasks.data(), tasks.size() * sizeof(GemmTask<T>), cudaMemcpyHostToDevice,
                                F_.stream));
}

template <class T>
int SolveEngine<T>::prepare(cudaStream_t st) {
  int launches = 0;
  if (nDinv_ > 0) {
    constexpr int smem = 2 * (int)sizeof(T) * SOLVE_RB * (SOLVE_RB + 1);
    static std::once_flag once;
    std::call_once(once, [] {
      RSCHOL_CUDA(cudaFuncSetAttribute(invert_diag_blocks<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    });
    invert_diag_blocks<T><<<nDinv_, SOLVE_RB, smem, st>>>(dDinvTasks_.as<DinvTask<T>>());
    RSCHOL_LAUNCH_CHECK();
    ++launches;
  }
  // G of the interior supernodes of up to 64 columns
  auto ops = [&](auto kernel, int cls, int nq) {
    if (opsClass_[cls].second == 0) return;
    const int smem = (int)sizeof(T) * (4 * nq + 64) * (4 * nq + 1);
    if (smem > 48 * 1024) RSCHOL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<opsClass_[cls].second, 256, smem, st>>>(dNodes_.as<SNode<T>>(),
                                                     dOpsWork_.as<RowBlock>() + opsClass_[cls].first);
    RSCHOL_LAUNCH_CHECK();
    ++launches;
  };
  ops(interior_ops_kernel<T, 4>, 0, 4);
  ops(interior_ops_kernel<T, 8>, 1, 8);
  ops(interior_ops_kernel<T, 16>, 2, 16);
  for (const XStep& x : xSteps_) {
    const GemmTask<T>* d = dXGemm_.as<GemmTask<T>>() + x.off;
    if constexpr (std::is_same<T, float>::value) {
      if (x.kind == XS_TC) launch_gemm_tc(d, x.count, x.tiles, F_.dFlag.template as<int>() + 1, st, x.bn);
      else if (x.kind == XS_ROWS128) launch_gemm_rows128(d, x.count, x.tiles, st);
      else launch_gemm<T>(d, x.count, x.tiles, st);
    } else {
      launch_gemm<T>(d, x.count, x.tiles, st);
    }
    ++launches;
  }
  if (nPacks_ > 0) {
    pack_tiles_kernel<T><<<nPacks_, 256, 0, st>>>(dNodes_.as<SNode<T>>(), dPackTiles_.as<PackTile>(), dPacked_.as<T>());
    RSCHOL_LAUNCH_CHECK();
    ++launches;
  }
  return launches;
}

template <class T>
int SolveEngine<T>::take_error(cudaStream_t st) {
  int e = 0;
  if (!dSync_.p) return 0;
  RSCHOL_CUDA(cudaMemcpyAsync(&e, dSync_.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  RSCHOL_CUDA(cudaStreamSynchronize(st));
  if (e) {
    // a wait gave up: counters and flags are in an unknown state; start over
    RSCHOL_CUDA(cudaMemsetAsync(dSync_.p, 0, sizeof(int) * nSync_, st));
    RSCHOL_CUDA(cudaStreamSynchronize(st));
  }
  return e;
}

template <class T>
void SolveEngine<T>::apply_inplace(double* w64, cudaStream_t st) {
  // FP32 factors are applied in FP32 (the PCG recurrences stay FP64)
  T* w = std::is_same<T, double>::value ? reinterpret_cast<T*>(w64) : dW_.as<T>();
  const int n = F_.S.n;
  if (!std::is_same<T, double>::value) {
    launch_k(convert_kernel<double, T>, dim3((n + 255) / 256), dim3(256), 0, st, w64, w, n);
    RSCHOL_LAUNCH_CHECK();
  }
  int* sync = dSync_.as<int>();
  const ApplyArgs<T> args{dItems_.as<ApplyItem>(), nItems_,         dBlob_.as<int>(), sync,          sync,         w,
                          dT_.as<T>(),             dWu_.as<T>(),    dZp_.as<T>(),     dSp_.as<T>(),  dYp_.as<T>(),
                          dXp_.as<T>(),            dIp_.as<T>(),    work_};
  launch_k(apply_kernel<T>, dim3(grid_), dim3(NGRP * GT + 32), smem_, st, args);
  RSCHOL_LAUNCH_CHECK();
  // ticket and counters are cleared by the apply's last kernel
  if (!std::is_same<T, double>::value) {
    launch_k(convert_out_kernel<T>, dim3((n + 255) / 256), dim3(256), 0, st, (const T*)w, w64, n, sync + 1, nSync_ - 1);
  } else {
    launch_k(clear_counters, dim3((nSync_ + 1023) / 1024), dim3(256), 0, st, sync + 1, nSync_ - 1);
  }
  RSCHOL_LAUNCH_CHECK();
}

template class SolveEngine<double>;
template class SolveEngine<float>;

}  // namespace rschol
