// Batched preconditioner apply: W (n x k, row-major, the k right-hand sides
// of a row contiguous) := M^{-1} W with one pass over the factor.
//
// The work items, their pieces of the factor and their order are those of the
// single-vector apply (solve.cu); only the products change: the pieces of the
// factor lie in shared memory, so a thread forms a tile of rows (or columns)
// of the piece times one 16-byte vector of right-hand sides.  A pass of an item
// covers up to KC columns (four vectors); wider blocks take several passes with
// the staged piece.  Factor bytes are read once per apply whatever k is; vector
// bytes scale with k.
//
// Width invariance: every (row, column) sum runs serially over the piece in one
// order, or in splits fixed by the piece alone; how threads cover (row, column)
// pairs depends on k, the arithmetic of a column does not.
//
// Bound: the latency of the items' gathers (a pass of an item is about 5 us of
// dependent loads whatever its bytes), FP64 its 1/64 rate.  Measured, one
// application against the earlier kernels (a triangular solve with a thread per
// (row, column) pair, six launches per compressed level): 2D 1024^2 FP32 k = 64
// 10.50 -> 6.5 ms, k = 8 3.62 -> 0.97 ms; 3D 40^3 FP32 k = 32 1.99 -> 0.69 ms,
// k = 8 1.81 -> 0.46 ms; 3D 64^3 FP32 k = 8 2.44 -> 0.97 ms; 3D 44x40x47 FP64
// k = 8 2.78 -> 1.52 ms.
#include <algorithm>
#include <mutex>
#include <stdexcept>
#include <type_traits>

#include "apply_dev.cuh"
#include "solve.cuh"
#include "solve_dev.cuh"

namespace rschol {

namespace {

using namespace solvedev;

constexpr int FB = 8192;   // bytes of a group's buffer of right-hand-side vectors
constexpr int FV = FB / 16;
// Persistent blocks per SM: two with 112 registers a thread; three with 72 spill
// in FP32 (2D 1024^2, k = 64: 5.99 against 7.06 ms an application)
constexpr int BATCH_BLOCKS = 2;
// rows (columns) of a piece a thread holds: FP64 pieces of a stage have half as
// many
template <class T> constexpr int NR = sizeof(T) == 8 ? 2 : 4;

template <class T>
struct Pass {   // one pass over up to four vectors of right-hand sides
  using Vt = typename Vec16<T>::type;
  const ApplyArgs<T>* A;
  int kp;        // row stride of the blocks (right-hand sides, padded to a vector)
  int cgN;       // vectors of the pass, rounded up to 1, 2 or 4
  int col;       // this thread's first column
  bool act;      // its vector holds columns of the block
  int cg, rg, nrg, tid;
  __device__ __forceinline__ Vt ld(const T* base, long long idx) const {
    return act ? __ldcg(reinterpret_cast<const Vt*>(base + idx * kp + col)) : vzero(T(0));
  }
  __device__ __forceinline__ void st(T* base, long long idx, Vt v) const {
    if (act) *reinterpret_cast<Vt*>(base + idx * kp + col) = v;
  }
};

__device__ __forceinline__ void vsub(float4& a, float4 b) {
  a.x -= b.x;
  a.y -= b.y;
  a.z -= b.z;
  a.w -= b.w;
}
__device__ __forceinline__ void vsub(double2& a, double2 b) {
  a.x -= b.x;
  a.y -= b.y;
}

// v[i] + the entries [b[i], e[i]) of a pull list, in order, for N targets at
// once: the loads of a round (two entries a target) are all in flight together.
template <class T, int N>
__device__ __forceinline__ void pulls(const Pass<T>& p, typename Vec16<T>::type (&v)[N], const int* ent, int (&b)[N],
                                      const int (&e)[N]) {
  bool more = true;
  while (more) {
    typename Vec16<T>::type x[N], y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = b[i] < e[i] ? p.ld(p.A->wu, ent[b[i]]) : vzero(T(0));
      y[i] = b[i] + 1 < e[i] ? p.ld(p.A->wu, ent[b[i] + 1]) : vzero(T(0));
    }
    more = false;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      vadd(v[i], x[i]);
      vadd(v[i], y[i]);
      b[i] += 2;
      more = more || b[i] < e[i];
    }
  }
}

// f of the columns [j0, j0 + jn) (offsets ps[j], entries ent; ps null: no
// children) into F, the caller's threads rg, rg + nrg, ... of every vector
template <class T>
__device__ __forceinline__ void gather_f(const Pass<T>& p, int c0, int j0, int jn, const int* ps, const int* ent,
                                         int rg, int nrg, typename Vec16<T>::type* F) {
  constexpr int N = 4;
  constexpr int V = Vec16<T>::V;
  const int jp = (jn + V - 1) / V * V;   // zeros up to a vector
  for (int jb = rg; jb < jp; jb += N * nrg) {
    typename Vec16<T>::type v[N];
    int b[N], e[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int j = jb + i * nrg;
      const bool in = j < jn;
      v[i] = in ? p.ld(p.A->w, c0 + j0 + j) : vzero(T(0));
      b[i] = ps && in ? ps[j0 + j] : 0;
      e[i] = ps && in ? ps[j0 + j + 1] : 0;
    }
    if (ps) pulls<T, N>(p, v, ent, b, e);
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (jb + i * nrg < jp) F[(jb + i * nrg) * p.cgN + p.cg] = v[i];
  }
}

__device__ __forceinline__ void vstep(float4& acc, const float4& m, const float4* F, int fs) {
  vaxpy(acc, F[0], m.x);
  vaxpy(acc, F[fs], m.y);
  vaxpy(acc, F[2 * fs], m.z);
  vaxpy(acc, F[3 * fs], m.w);
}
__device__ __forceinline__ void vstep(double2& acc, const double2& m, const double2* F, int fs) {
  vaxpy(acc, F[0], m.x);
  vaxpy(acc, F[fs], m.y);
}

// acc[i] += sum_k M_i[k] F[k], k < kn in order, for the thread's rows M_i = M +
// off[i] (off < 0: none); F: vectors, row stride fs.  ALIGNED: rows on 16-byte
// boundaries, zeros behind them (and in F) up to a vector: read in vectors -- the
// eight rows of a warp lie 16 floats apart in the commonest supernodes, four
// deep in the same banks when read by words.
template <class T, bool ALIGNED>
__device__ __forceinline__ void rows_dot(const T* M, const int (&off)[NR<T>], int k0, int kn,
                                         const typename Vec16<T>::type* F, int fs,
                                         typename Vec16<T>::type (&acc)[NR<T>]) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  if constexpr (ALIGNED) {
#pragma unroll 2
    for (int k = 0; k < kn; k += V) {
#pragma unroll
      for (int i = 0; i < NR<T>; ++i)
        if (off[i] >= 0) vstep(acc[i], *reinterpret_cast<const Vt*>(M + off[i] + k0 + k), F + k * fs, fs);
    }
  } else {
#pragma unroll 4
    for (int k = 0; k < kn; ++k) {
      const Vt f = F[k * fs];
#pragma unroll
      for (int i = 0; i < NR<T>; ++i)
        if (off[i] >= 0) vaxpy(acc[i], f, M[off[i] + k0 + k]);
    }
  }
}

// out(j, sum_{a < h} M[a * ld + j] X[a * xs]) for the thread's columns j < nc
template <class T, class Out>
__device__ __forceinline__ void cols_dot(const T* M, int ld, int h, int nc, const typename Vec16<T>::type* X, int xs,
                                         int j0, int step, Out out) {
  for (int jb = j0; jb < nc; jb += NR<T> * step) {
    typename Vec16<T>::type acc[NR<T>];
    const T* m[NR<T>];
#pragma unroll
    for (int i = 0; i < NR<T>; ++i) {
      acc[i] = vzero(T(0));
      m[i] = jb + i * step < nc ? M + jb + i * step : nullptr;
    }
#pragma unroll 4
    for (int a = 0; a < h; ++a) {
      const typename Vec16<T>::type x = X[a * xs];
#pragma unroll
      for (int i = 0; i < NR<T>; ++i)
        if (m[i]) vaxpy(acc[i], x, m[i][(size_t)a * ld]);
    }
#pragma unroll
    for (int i = 0; i < NR<T>; ++i)
      if (jb + i * step < nc) out(jb + i * step, acc[i]);
  }
}

// A group's members, a warp each; lanes over (row group, vector).
template <class T>
__device__ __forceinline__ void fgrp_k(const Pass<T>& p, const int* h0, const int* d, int cnt, const T* data,
                                       typename Vec16<T>::type* buf) {
  using Vt = typename Vec16<T>::type;
  const int lane = threadIdx.x & 31, warp = p.tid >> 5;
  const int rg = lane / p.cgN, nrg = 32 / p.cgN;
  Vt* F = buf + warp * 32 * p.cgN;
  for (int q = warp; q < cnt; q += GW) {
    const int* h = h0 + GH * q;
    const int n = h[0], m = h[1], c0 = h[2], ldk = h[7];
    const bool has = h[6] != 0;
    const int* ps = d + h[6];
    const int* ent = ps + n + m + 1;
    __syncwarp();
    gather_f<T>(p, c0, 0, n, has ? ps : nullptr, ent, rg, nrg, F);
    __syncwarp();
    for (int r0 = 0; r0 < m + n; r0 += NR<T> * nrg) {   // rows of G, then of X
      Vt acc[NR<T>];
      int off[NR<T>];
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        const int r = r0 + rg + i * nrg;
        off[i] = r < m ? h[4] + r * ldk : r < m + n ? h[5] + (r - m) * ldk : -1;
        acc[i] = vzero(T(0));
      }
      rows_dot<T, true>(data, off, 0, n, F + p.cg, p.cgN, acc);
      Vt u[NR<T>];
      if (has && r0 < m) {
        int b[NR<T>], e[NR<T>];
#pragma unroll
        for (int i = 0; i < NR<T>; ++i) {
          const int r = r0 + rg + i * nrg;
          u[i] = vzero(T(0));
          b[i] = r < m ? ps[n + r] : 0;
          e[i] = r < m ? ps[n + r + 1] : 0;
        }
        pulls<T, NR<T>>(p, u, ent, b, e);
      } else {
#pragma unroll
        for (int i = 0; i < NR<T>; ++i) u[i] = vzero(T(0));
      }
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        const int r = r0 + rg + i * nrg;
        if (r < m) {
          vsub(u[i], acc[i]);
          p.st(p.A->wu, h[3] + r, u[i]);
        } else if (r < m + n) {
          p.st(p.A->t, h[8] + r - m, acc[i]);
        }
      }
    }
  }
}

// Backward; early: X^T y, kept in the place of x, then x = that - G^T x_R.
template <class T>
__device__ __forceinline__ void bgrp_k(const Pass<T>& p, const int* h0, const int* d, int cnt, const T* data,
                                       typename Vec16<T>::type* buf, bool early) {
  using Vt = typename Vec16<T>::type;
  const int lane = threadIdx.x & 31, warp = p.tid >> 5;
  const int rg = lane / p.cgN, nrg = 32 / p.cgN;
  Vt* xs = buf + warp * 128;   // 128 vectors: NR<T> rows a lane
  for (int q = warp; q < cnt; q += GW) {
    const int* h = h0 + GH * q;
    const int n = h[0], c0 = h[2], ldk = h[7], rows = early ? n : h[1];
    const T* M = data + (early ? h[5] : h[4]);
    const int* rw = d + h[6];
    // the thread's columns j = rg + i nrg: 32 columns in 1, 2 or 4 sweeps of them
    const int tile = NR<T> * nrg;   // rows of y or x_R a tile
    auto load = [&](int a) {
      return a >= rows ? vzero(T(0)) : early ? p.ld(p.A->t, h[8] + a) : p.ld(p.A->w, rw[a]);
    };
    for (int jb = 0; jb < n; jb += NR<T> * nrg) {
      Vt acc[NR<T>], nx[NR<T>];
      const T* g[NR<T>];
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        acc[i] = vzero(T(0));
        g[i] = jb + rg + i * nrg < n ? M + jb + rg + i * nrg : nullptr;
        nx[i] = load(rg + i * nrg);
      }
      for (int a0 = 0; a0 < rows; a0 += tile) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NR<T>; ++i) xs[(rg + i * nrg) * p.cgN + p.cg] = nx[i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NR<T>; ++i) nx[i] = load(a0 + tile + rg + i * nrg);   // under this tile's products
        const int an = min(tile, rows - a0);
#pragma unroll 4
        for (int a = 0; a < an; ++a) {
          const Vt x = xs[a * p.cgN + p.cg];
#pragma unroll
          for (int i = 0; i < NR<T>; ++i)
            if (g[i]) vaxpy(acc[i], x, g[i][(size_t)(a0 + a) * ldk]);
        }
      }
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        const int j = jb + rg + i * nrg;
        if (j >= n) continue;
        if (early) {
          p.st(p.A->w, c0 + j, acc[i]);
        } else {
          Vt v = p.ld(p.A->w, c0 + j);
          vsub(v, acc[i]);
          p.st(p.A->w, c0 + j, v);
        }
      }
    }
  }
}

// One chunk: the rows of G, then of X (in a stage they follow each other; a
// supernode too wide for one is read where it is, G's rows and X's in turn).
template <class T>
__device__ __forceinline__ void fwd_k(const Pass<T>& p, const int* h, const int* d, const int* d2, const T* Gd,
                                      const T* Xd, bool staged, typename Vec16<T>::type* F) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V;
  const int n = h[0], rows = h[1], c0 = h[2], ldk = h[7];
  const bool has = h[6] != 0;
  const int* ps = d + h[6];
  const int* ent = ps + rows + 1;
  const int* ent2 = d2 + n + 1;
  const int ft = FV / p.cgN / V * V;   // rows of f a tile
  for (int part = 0; part < (staged ? 1 : 2); ++part) {
    const T* M = part ? Xd : Gd;
    const int first = part ? rows : 0, cnt = staged ? rows + h[5] : part ? h[5] : rows;
    // A wide supernode's chunk has few rows (300 columns in FP64: seven): K in GT /
    // slots slices, over the threads that would have no row -- a pass of fewer
    // vectors has more of them, so a thread takes one slice, or two or four -- and
    // the slices' sums added in order: the order of a sum does not depend on the
    // width of the block.  (With a thread for all of K one warp of four had the
    // work, FP64 at that: 3D 44x40x47, k = 8, 1.75 -> 1.50 ms an application.  The
    // gather of f, done over by every chunk, costs little beside: once for all
    // chunks, in items of its own, it gained nothing.)
    int slots = 1;
    while (slots < cnt) slots <<= 1;
    if (slots <= GT / 8) {
      const int row = p.rg & (slots - 1), sl = p.rg / slots, ns = p.nrg / slots, slices = GT / slots;
      const int per = ((n + V - 1) / V + slices - 1) / slices * V;
      Vt acc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = vzero(T(0));
      for (int j0 = 0; j0 < n; j0 += ft) {
        const int jn = min(ft, n - j0), jp = (jn + V - 1) / V * V;
        if (j0 > 0 || part > 0) cbar();
        gather_f<T>(p, c0, j0, jn, has ? d2 : nullptr, ent2, p.rg, p.nrg, F);
        cbar();
        if (row < cnt) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {   // slices sl, sl + ns, ... (vectors of the pass: as many)
            if (i >= p.cgN) break;
            const int ka = max((sl + i * ns) * per, j0), kb = min((sl + i * ns + 1) * per, j0 + jp);
#pragma unroll 2
            for (int k = ka; k < kb; k += V)
              vstep(acc[i], *reinterpret_cast<const Vt*>(M + row * ldk + k), F + (k - j0) * p.cgN + p.cg, p.cgN);
          }
        }
      }
      cbar();
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < p.cgN) F[((sl + i * ns) * slots + row) * p.cgN + p.cg] = acc[i];
      cbar();
      if (p.rg < cnt) {
        Vt v = F[row * p.cgN + p.cg], u[1] = {vzero(T(0))};
        for (int q = 1; q < slices; ++q) vadd(v, F[(q * slots + row) * p.cgN + p.cg]);
        const int r = first + row;
        int b[1] = {has && r < rows ? ps[r] : 0};
        const int e[1] = {has && r < rows ? ps[r + 1] : 0};
        pulls<T, 1>(p, u, ent, b, e);
        if (r < rows) {
          vsub(u[0], v);
          p.st(p.A->wu, h[3] + r, u[0]);
        } else {
          p.st(p.A->t, h[8] + h[4] + r - rows, v);
        }
      }
      continue;
    }
    for (int r0 = 0; r0 < cnt; r0 += NR<T> * p.nrg) {   // one sweep for the chunk heights in use
      Vt acc[NR<T>];
      int off[NR<T>];
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        const int r = r0 + p.rg + i * p.nrg;
        off[i] = r < cnt ? r * ldk : -1;
        acc[i] = vzero(T(0));
      }
      for (int j0 = 0; j0 < n; j0 += ft) {
        const int jn = min(ft, n - j0);
        if (j0 > 0 || r0 > 0 || part > 0) cbar();
        gather_f<T>(p, c0, j0, jn, has ? d2 : nullptr, ent2, p.rg, p.nrg, F);
        cbar();
        rows_dot<T, true>(M, off, j0, jn, F + p.cg, p.cgN, acc);
      }
      Vt u[NR<T>];
      int b[NR<T>], e[NR<T>];
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        const int r = first + r0 + p.rg + i * p.nrg;
        u[i] = vzero(T(0));
        b[i] = has && r < rows ? ps[r] : 0;
        e[i] = has && r < rows ? ps[r + 1] : 0;
      }
      if (has) pulls<T, NR<T>>(p, u, ent, b, e);
#pragma unroll
      for (int i = 0; i < NR<T>; ++i) {
        const int r = first + r0 + p.rg + i * p.nrg;
        if (off[i] < 0) continue;
        if (r < rows) {
          vsub(u[i], acc[i]);
          p.st(p.A->wu, h[3] + r, u[i]);
        } else {
          p.st(p.A->t, h[8] + h[4] + r - rows, acc[i]);
        }
      }
    }
  }
}

// F[kk] = sum of `parts` partial rows at idx0 + q * rp + kk, kk < kn
template <class T>
__device__ __forceinline__ void parts_k(const Pass<T>& p, const T* base, long long idx0, int rp, int kn, int parts,
                                        typename Vec16<T>::type* F) {
  using Vt = typename Vec16<T>::type;
  for (int kk = p.rg; kk < kn; kk += p.nrg) {
    Vt v = vzero(T(0));
    for (int q0 = 0; q0 < parts; q0 += 4) {
      Vt x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = q0 + q < parts ? p.ld(base, idx0 + (long long)(q0 + q) * rp + kk) : vzero(T(0));
#pragma unroll
      for (int q = 0; q < 4; ++q) vadd(v, x[q]);
    }
    F[kk * p.cgN + p.cg] = v;
  }
}

// out(i, sum_k M[i * r + k] y[k]) for the item's rows i < rows, y the sum of the
// partial rows
template <class T, class Out>
__device__ __forceinline__ void rows_parts_k(const Pass<T>& p, const T* Mx, int r, int rows, const T* base,
                                             long long idx0, int parts, typename Vec16<T>::type* F, Out out) {
  using Vt = typename Vec16<T>::type;
  const int rp = (r + 7) & ~7, ft = FV / p.cgN;
  int slots = 1;
  while (slots < rows) slots <<= 1;
  // Few rows (large ranks: 16 and fewer): K in GT / slots slices over the threads that
  // would have none, as in a chunk's forward products.  (A thread for all of K: FP64 3D
  // 44^3 at ranks up to 313 2.42 against 1.13 ms with two columns, 10.2 against 6.7 with
  // 40; FP32 at ranks up to 622 0.85 against 0.52 with two.)
  if (slots <= GT / 8) {
    const int row = p.rg & (slots - 1), sl = p.rg / slots, ns = p.nrg / slots, slices = GT / slots;
    const int per = (r + slices - 1) / slices;
    Vt acc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = vzero(T(0));
    for (int k0 = 0; k0 < r; k0 += ft) {
      const int kn = min(ft, r - k0);
      cbar();
      parts_k<T>(p, base, idx0 + k0, rp, kn, parts, F);
      cbar();
      if (row < rows) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // slices sl, sl + ns, ... (vectors of the pass: as many)
          if (i >= p.cgN) break;
          const int ka = max((sl + i * ns) * per, k0), kb = min((sl + i * ns + 1) * per, k0 + kn);
#pragma unroll 4
          for (int k = ka; k < kb; ++k) vaxpy(acc[i], F[(k - k0) * p.cgN + p.cg], Mx[(size_t)row * r + k]);
        }
      }
    }
    cbar();
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < p.cgN) F[((sl + i * ns) * slots + row) * p.cgN + p.cg] = acc[i];
    cbar();
    if (p.rg < rows) {
      Vt v = F[row * p.cgN + p.cg];
      for (int q = 1; q < slices; ++q) vadd(v, F[(q * slots + row) * p.cgN + p.cg]);
      out(row, v);
    }
    return;
  }
  for (int r0 = 0; r0 < rows; r0 += NR<T> * p.nrg) {
    Vt acc[NR<T>];
    int off[NR<T>];
#pragma unroll
    for (int i = 0; i < NR<T>; ++i) {
      const int q = r0 + p.rg + i * p.nrg;
      off[i] = q < rows ? q * r : -1;
      acc[i] = vzero(T(0));
    }
    for (int k0 = 0; k0 < r; k0 += ft) {
      const int kn = min(ft, r - k0);
      cbar();
      parts_k<T>(p, base, idx0 + k0, rp, kn, parts, F);
      cbar();
      rows_dot<T, false>(Mx, off, k0, kn, F + p.cg, p.cgN, acc);
    }
#pragma unroll
    for (int i = 0; i < NR<T>; ++i)
      if (r0 + p.rg + i * p.nrg < rows) out(r0 + p.rg + i * p.nrg, acc[i]);
  }
}

// red[s * cnt + o] (o < cnt outputs of a vector each, s < SP splits) added over s
// in order; every thread of the group must call it
template <class T, int SP, class Part, class Out>
__device__ __forceinline__ void split_sum(const Pass<T>& p, int outs, typename Vec16<T>::type* red, Part part, Out out) {
  using Vt = typename Vec16<T>::type;
  for (int e = p.rg; e < outs * SP; e += p.nrg) red[e * p.cgN + p.cg] = part(e / SP, e % SP);
  cbar();
  for (int o = p.rg; o < outs; o += p.nrg) {
    Vt v = vzero(T(0));
#pragma unroll
    for (int s = 0; s < SP; ++s) vadd(v, red[(o * SP + s) * p.cgN + p.cg]);
    out(o, v);
  }
}

template <class T>
__global__ void __launch_bounds__(NGRP * GT + 32, BATCH_BLOCKS) apply_batch_kernel(ApplyArgs<T> A, int kp, int slices, int width,
                                                                            int syncInts) {
  using Vt = typename Vec16<T>::type;
  constexpr int V = Vec16<T>::V, KC = 4 * V;
  extern __shared__ __align__(128) unsigned char absm[];
  // a slice of the columns: its own tickets and counters, every slices-th block
  const int slice = blockIdx.x % slices, colBeg = slice * width, colEnd = min(kp, colBeg + width);
  A.sync += slice * syncInts;
  __shared__ __align__(8) unsigned long long bars[2 * NSTAGE];
  __shared__ __align__(16) ApplyItem sItem[NSTAGE];
  int* const err = A.err;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(smem_u32(&bars[s]), 1);
      mbar_init(smem_u32(&bars[NSTAGE + s]), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x >= NGRP * GT) {
    apply_producer<T>(A, absm, sItem, smem_u32(&bars[0]), smem_u32(&bars[NSTAGE]));
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    return;
  }
  const int grp = threadIdx.x / GT, tid = threadIdx.x % GT, warp = tid >> 5;
  Vt* const F = reinterpret_cast<Vt*>(absm + NSTAGE * ST_BYTES + grp * FB);
  for (int k = grp;; k += NGRP) {
    const int s = k % NSTAGE;
    if (!wait_stage(k, smem_u32(&bars[0]))) {   // cannot happen while the producer runs
      if (tid == 0) atomicExch(err, 3);
      break;
    }
    const ApplyItem& it = sItem[s];
    const int kind = it.kind;
    if (kind == IT_END) break;
    const unsigned char* st = absm + (size_t)s * ST_BYTES;
    const T* data = reinterpret_cast<const T*>(st);
    const int* d = it.descBytes ? reinterpret_cast<const int*>(st + ST_DATA) : A.blob + it.desc;
    const int* h = d + 2 * it.waits;
    const int* d2 = it.desc2Bytes ? reinterpret_cast<const int*>(st + ST_DATA + it.descBytes) : A.blob + it.desc2;
    const int first = it.early ? it.early : it.waits;
    if (warp == 0) wait_list(d, first, A.sync, err);
    cbar();
    const T* g0 = it.bytes0 ? data : reinterpret_cast<const T*>(it.g0);
    const T* g1 = it.bytes1 ? data + it.bytes0 / sizeof(T) : reinterpret_cast<const T*>(it.g1);
    auto pass = [&](int col0) {
      Pass<T> p;
      p.A = &A;
      p.kp = kp;
      const int rem = (colEnd - col0) / V;
      p.cgN = rem >= 3 ? 4 : rem;
      p.tid = tid;
      p.cg = tid % p.cgN;
      p.rg = tid / p.cgN;
      p.nrg = GT / p.cgN;
      p.col = col0 + p.cg * V;
      p.act = p.col < colEnd;
      return p;
    };
    // a backward item's products with X, before the wait for its ancestors (2D 60 x 50
    // FP64, 5 columns: 232 against 250 us; never slower)
    if (it.early) {
      for (int col0 = colBeg; col0 < colEnd; col0 += KC) {
        const Pass<T> p = pass(col0);
        if (kind == IT_BGRP) {
          bgrp_k<T>(p, h, d, it.count, data, F, true);
          continue;
        }
        if (col0 > colBeg) cbar();
        for (int a = p.rg; a < h[10]; a += p.nrg) F[a * p.cgN + p.cg] = p.ld(A.t, h[9] + a);
        cbar();
        if (h[10] > 0)
          cols_dot<T>(g1, h[7], h[10], h[0], F + p.cg, p.cgN, p.rg, p.nrg, [&](int j, Vt v) {
            if (h[5] > 1) p.st(A.ip, h[3] + (long long)h[4] * h[8] + j, v);
            else p.st(A.w, h[2] + j, v);
          });
      }
      if (warp == 0) wait_list(d + 2 * first, it.waits - first, A.sync, err);
      cbar();
    }
    for (int col0 = colBeg; col0 < colEnd; col0 += KC) {
      const Pass<T> p = pass(col0);
      if (col0 > colBeg) cbar();   // the buffers of the last pass
      switch (kind) {
        case IT_FGRP: fgrp_k<T>(p, h, d, it.count, data, F); break;
        case IT_BGRP: bgrp_k<T>(p, h, d, it.count, data, F, false); break;
        case IT_FWD: fwd_k<T>(p, h, d, d2, it.bytes0 + it.bytes1 > 0 ? data : g0, g1, it.bytes0 + it.bytes1 > 0, F); break;
        case IT_BWD: {   // less G^T x_R
          const int rows = h[1];
          if (rows == 0) break;
#pragma unroll 2
          for (int a = p.rg; a < rows; a += p.nrg) F[a * p.cgN + p.cg] = p.ld(A.w, d[h[6] + a]);
          cbar();
          cols_dot<T>(g0, h[7], rows, h[0], F + p.cg, p.cgN, p.rg, p.nrg, [&](int j, Vt v) {
            T* const to = h[5] > 1 ? A.ip : A.w;
            const long long at = h[5] > 1 ? h[3] + (long long)h[4] * h[8] + j : h[2] + j;
            Vt x = h[10] > 0 ? p.ld(to, at) : vzero(T(0));
            vsub(x, v);
            p.st(to, at, x);
          });
          break;
        }
        case IT_BR: {
          for (int j = p.rg; j < h[0]; j += p.nrg) {
            Vt x = vzero(T(0));
            for (int q0 = 0; q0 < h[3]; q0 += 16) {
              Vt v[16];
#pragma unroll
              for (int q = 0; q < 16; ++q)
                v[q] = q0 + q < h[3] ? p.ld(A.ip, h[2] + (long long)(q0 + q) * h[4] + j) : vzero(T(0));
#pragma unroll
              for (int q = 0; q < 16; ++q) vadd(x, v[q]);
            }
            p.st(A.w, h[1] + j, x);
          }
          break;
        }
        case IT_CF: {
          const int cols = h[1], r = h[2];
          const int* ps = d + h[4];
          const int* ent = ps + cols + 1;
          for (int i = p.rg; i < cols; i += p.nrg) {   // (a column a thread: its list eight entries at a time)
            Vt v = p.ld(A.w, h[0] + i);
            const int e = ps[i + 1];
            for (int b = ps[i]; b < e; b += 8) {
              Vt x[8];
#pragma unroll
              for (int q = 0; q < 8; ++q) x[q] = b + q < e ? p.ld(A.wu, ent[b + q]) : vzero(T(0));
#pragma unroll
              for (int q = 0; q < 8; ++q) vadd(v, x[q]);
            }
            p.st(A.w, h[0] + i, v);
            F[i * p.cgN + p.cg] = v;
          }
          cbar();
          if (r > 0)
            cols_dot<T>(g0, r, cols, r, F + p.cg, p.cgN, p.rg, p.nrg, [&](int j, Vt v) { p.st(A.zp, h[3] + j, v); });
          break;
        }
        case IT_CU:
          rows_parts_k<T>(p, g0, h[1], h[0], A.zp, h[2], h[3], F, [&](int i, Vt v) {
            Vt u = vzero(T(0));
            vsub(u, v);
            p.st(A.wu, h[4] + i, u);
          });
          break;
        case IT_CR: {   // columns of partials, eight splits of the partials a column
          T* const base = h[5] ? A.sp : A.zp;
          split_sum<T, 8>(
              p, h[3], F,
              [&](int o, int sp) {
                Vt x = vzero(T(0));
                for (int q0 = sp; q0 < h[1]; q0 += 64) {
                  Vt v[8];
#pragma unroll
                  for (int q = 0; q < 8; ++q)
                    v[q] = q0 + 8 * q < h[1] ? p.ld(base, h[0] + (long long)(q0 + 8 * q) * h[2] + o) : vzero(T(0));
#pragma unroll
                  for (int q = 0; q < 8; ++q) vadd(x, v[q]);
                }
                return x;
              },
              [&](int o, Vt v) { p.st(base, h[4] + o, v); });
          break;
        }
        case IT_Y: {
          // the tile's rows in two halves of its columns (fixed), f in tiles
          const int cols = h[1], rows = h[2], ft = FV / p.cgN / 2;
          const int half = Y_COLS<T> / 2;
          Vt acc[2] = {vzero(T(0)), vzero(T(0))};   // (row, half) pairs rg, rg + nrg: 32 of them
          for (int j0 = 0; j0 < half; j0 += ft) {
            const int jn = min(ft, half - j0);
            cbar();
            for (int e = p.rg; e < 2 * jn; e += p.nrg) {   // both halves' rows of f
              const int hh = e >= jn, j = (hh ? e - jn : e) + j0 + hh * half;
              F[(hh * ft + (hh ? e - jn : e)) * p.cgN + p.cg] = j < cols ? p.ld(A.w, h[0] + j) : vzero(T(0));
            }
            cbar();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int e = p.rg + i * p.nrg, row = e >> 1, hh = e & 1;
              if (e < 2 * Y_ROWS && row < rows) {
                const T* m = data + row * Y_COLS<T> + hh * half + j0;
                const Vt* f = F + hh * ft * p.cgN + p.cg;
#pragma unroll 2
                for (int j = 0; j < jn; j += V)
                  vstep(acc[i], *reinterpret_cast<const Vt*>(m + j), f + j * p.cgN, p.cgN);
              }
            }
          }
          cbar();
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (p.rg + i * p.nrg < 2 * Y_ROWS) F[(p.rg + i * p.nrg) * p.cgN + p.cg] = acc[i];
          cbar();
          for (int i = p.rg; i < rows; i += p.nrg) {
            Vt v = F[2 * i * p.cgN + p.cg];
            vadd(v, F[(2 * i + 1) * p.cgN + p.cg]);
            p.st(A.yp, h[3] + i, v);
          }
          break;
        }
        case IT_XT: {
          for (int i = p.rg; i < h[0]; i += p.nrg) {
            const int nj = min(h[6], ((h[4] + i) / Y_ROWS * Y_ROWS + Y_ROWS - 1) / Y_COLS<T> + 1);
            Vt y = vzero(T(0));
            for (int j0 = 0; j0 < nj; j0 += 8) {
              Vt v[8];
#pragma unroll
              for (int q = 0; q < 8; ++q)
                v[q] = j0 + q < nj ? p.ld(A.yp, h[2] + (long long)(j0 + q) * h[3] + i) : vzero(T(0));
#pragma unroll
              for (int q = 0; q < 8; ++q) vadd(y, v[q]);
            }
            F[i * p.cgN + p.cg] = y;
          }
          cbar();
          cols_dot<T>(data, T_COLS, h[0], h[1], F + p.cg, p.cgN, p.rg, p.nrg,
                      [&](int j, Vt v) { p.st(A.xp, h[5] + j, v); });
          break;
        }
        case IT_CS: {
#pragma unroll 2
          for (int a = p.rg; a < h[0]; a += p.nrg) F[a * p.cgN + p.cg] = p.ld(A.w, d[h[3] + a]);
          cbar();
          cols_dot<T>(g0, h[1], h[0], h[1], F + p.cg, p.cgN, p.rg, p.nrg,
                      [&](int j, Vt v) { p.st(A.sp, h[2] + j, v); });
          break;
        }
        default: {   // IT_CX: t first (four splits of the row blocks), stored in place of x
          const int cols = h[1];
          split_sum<T, 4>(
              p, cols, F,
              [&](int j, int sp) {
                Vt x = vzero(T(0));
                const int first = max(h[8], (h[7] + j) / T_COLS * T_COLS / T_ROWS<T>);
                for (int i0 = h[8] + sp; i0 < h[9]; i0 += 32) {
                  Vt v[8];
#pragma unroll
                  for (int q = 0; q < 8; ++q) {
                    const int ib = i0 + 4 * q;
                    v[q] = ib < h[9] && ib >= first ? p.ld(A.xp, h[5] + (long long)ib * h[6] + j) : vzero(T(0));
                  }
#pragma unroll
                  for (int q = 0; q < 8; ++q) vadd(x, v[q]);
                }
                return x;
              },
              [&](int j, Vt v) { p.st(A.w, h[0] + j, v); });
          if (h[4] > 0) {
            cbar();
            rows_parts_k<T>(p, g0, h[2], cols, A.sp, h[3], h[4], F, [&](int j, Vt v) {
              Vt x = p.ld(A.w, h[0] + j);
              vsub(x, v);
              p.st(A.w, h[0] + j, x);
            });
          }
          break;
        }
      }
    }
    const int sig = it.sig;
    cbar();   // every consumer has stored and is done with the stage
    if (tid == GT - 32) {
      mbar_arrive(smem_u32(&bars[NSTAGE + s]));
      __threadfence();
      atomicAdd(A.sync + sig, 1);
    }
  }
}

// W64 (n x k) to the working block (n x kp, zeros in the padding)
template <class T>
__global__ void __launch_bounds__(256) widen_kernel(const double* __restrict__ src, T* __restrict__ dst, long long n,
                                                    int k, int kp) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n * kp; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / kp;
    const int c = (int)(i - r * kp);
    dst[i] = c < k ? (T)src[r * k + c] : T(0);
  }
}

// and back; the last kernel of a batched apply also zeroes the ticket and the
// counters (their last reader, the apply kernel, has finished)
template <class T>
__global__ void __launch_bounds__(256) narrow_kernel(const T* __restrict__ src, double* __restrict__ dst, long long n,
                                                     int k, int kp, int* __restrict__ clr, int nClr) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n * k; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / k;
    const int c = (int)(i - r * k);
    dst[i] = (double)src[r * kp + c];
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nClr; i += gridDim.x * blockDim.x) clr[i] = 0;
}

}  // namespace

template <class T>
int SolveEngine<T>::batch_capacity() const {
  return 64;
}

// Slices of columns that walk the items by themselves, beside each other: a pass over
// an item is a chain of loads (FP64: of multiply-adds, 64 clocks a warp), so passes
// one after the other leave most of the chip waiting.  Slices of a whole pass (four
// vectors); of two or one where the items are so few that the blocks outnumber
// them.  One application at one / two / four vectors a slice / all in turn: FP64 2D
// 75x70 (343 items) k = 16 270 / 303 / 419 / 749 us, 110x100 (750) k = 64 680 / 509 / 490 /
// 2863, 193x187 (2949) k = 16 884 / 713 / 749 / 1233; FP32 2D 193x187 (1371) k = 64 468 /
// 354 / 381 / 1093, 3D 40x38x40 (14058) k = 64 2976 / 1678 / 1091 / 1649.
template <class T>
int SolveEngine<T>::batch_slices(int kp) const {
  const long long nv = std::max(1, (kp + Vec16<T>::V - 1) / Vec16<T>::V), passes = nv * nItems_;
  const int w = passes <= 8000 ? 1 : passes <= 24000 ? 2 : 4;
  return (int)((nv + w - 1) / w);
}

// Buffers for blocks of kp columns; they only grow, so a changing width frees
// nothing and never synchronises the device.
template <class T>
void SolveEngine<T>::plan_batch(int kp) {
  if (kp <= kAllocB_) return;
  cudaStream_t st = F_.stream;
  auto widen = [&](DevBuf& b, const DevBuf& single) { b.alloc(single.bytes * (size_t)kp); };
  widen(dWuB_, dWu_);
  widen(dTB_, dT_);
  widen(dZpB_, dZp_);
  widen(dSpB_, dSp_);
  widen(dYpB_, dYp_);
  widen(dXpB_, dXp_);
  widen(dIpB_, dIp_);
  dWB_.alloc(sizeof(T) * (size_t)std::max(1, F_.S.n) * kp);   // the working copy of W
  if (!dSyncB_.p) {
    int slices = 1;
    for (int c = 1; c <= batch_capacity(); ++c) slices = std::max(slices, batch_slices(c));
    const size_t bytes = sizeof(int) * nSync_ * (size_t)slices;
    dSyncB_.alloc(bytes);
    RSCHOL_CUDA(cudaMemsetAsync(dSyncB_.p, 0, bytes, st));
  }
  kAllocB_ = kp;
  ++batchGen_;
}

template <class T>
int SolveEngine<T>::width_class(int k) const {
  int p = 1;
  while (p < k) p <<= 1;
  return p;
}

// The width class of k is k rounded up to a power of two.  Its one shape, the
// persistent blocks per SM, is timed at the full width on a zero block: fewer
// blocks leave fewer items waiting on one another at small widths.
template <class T>
const typename SolveEngine<T>::BatchCfg& SolveEngine<T>::config_for(int k, cudaStream_t st, bool tune) {
  const int kp = width_class(k);
  auto it = tuned_.find(kp);
  if (it != tuned_.end() && (it->second.ms > 0 || !tune)) return it->second;
  BatchCfg best;
  if (tune) {
    const size_t bytes = sizeof(double) * (size_t)std::max(1, F_.S.n) * kp;
    DevBuf zero;
    zero.alloc(bytes);
    RSCHOL_CUDA(cudaMemsetAsync(zero.p, 0, bytes, st));
    cudaEvent_t e0, e1;
    RSCHOL_CUDA(cudaEventCreate(&e0));
    RSCHOL_CUDA(cudaEventCreate(&e1));
    auto time_cfg = [&](const BatchCfg& c) {
      apply_batch_cfg(zero.as<double>(), kp, st, c);   // warm-up
      float bestMs = 1e30f;
      for (int rep = 0; rep < 2; ++rep) {
        RSCHOL_CUDA(cudaEventRecord(e0, st));
        apply_batch_cfg(zero.as<double>(), kp, st, c);
        RSCHOL_CUDA(cudaEventRecord(e1, st));
        RSCHOL_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        RSCHOL_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        bestMs = std::min(bestMs, ms);
      }
      return (double)bestMs;
    };
    best.ms = time_cfg(best);
    for (int b = 1; b < best.blocks; ++b) {
      BatchCfg c;
      c.blocks = b;
      c.ms = time_cfg(c);
      if (c.ms < best.ms) best = c;
    }
    RSCHOL_CUDA(cudaEventDestroy(e0));
    RSCHOL_CUDA(cudaEventDestroy(e1));
  }
  ++batchGen_;   // a new shape: a captured apply would use the old one
  return tuned_[kp] = best;
}

template <class T>
void SolveEngine<T>::autotune_batch(int kmax, cudaStream_t st) {
  kmax = std::min(kmax, batch_capacity());
  for (int k = 1; k <= kmax; k = width_class(k) + 1) config_for(k, st, true);
}

template <class T>
std::vector<std::array<double, 6>> SolveEngine<T>::batch_tuning() const {
  std::vector<std::array<double, 6>> out;
  for (const auto& kv : tuned_)
    out.push_back({(double)kv.first, (double)kv.second.blocks, 4.0 * Vec16<T>::V, 0.0, 0.0, kv.second.ms});
  return out;
}

template <class T>
void SolveEngine<T>::apply_batch(double* W64, int k, cudaStream_t st) {
  if (k <= 0) return;
  if (k > batch_capacity()) throw std::runtime_error("apply_batch: more right-hand sides than one pass handles");
  apply_batch_cfg(W64, k, st, config_for(k, st, autotune_));
}

template <class T>
void SolveEngine<T>::apply_batch_cfg(double* W64, int k, cudaStream_t st, const BatchCfg& cfg) {
  constexpr int V = Vec16<T>::V;
  const int kp = (k + V - 1) / V * V;
  plan_batch(kp);
  constexpr int smem = NSTAGE * ST_BYTES + NGRP * FB;
  static std::once_flag once;
  std::call_once(once, [] {
    RSCHOL_CUDA(cudaFuncSetAttribute(apply_batch_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  });
  const long long n = F_.S.n;
  T* w = dWB_.as<T>();
  const unsigned grid = (unsigned)std::min<long long>((n * kp + 255) / 256, 4096);
  launch_k(widen_kernel<T>, dim3(grid), dim3(256), 0, st, (const double*)W64, w, n, k, kp);
  RSCHOL_LAUNCH_CHECK();
  int* sync = dSyncB_.as<int>();
  const ApplyArgs<T> args{dItems_.as<ApplyItem>(), nItems_,         dBlob_.as<int>(), sync,           sync,          w,
                          dTB_.as<T>(),            dWuB_.as<T>(),   dZpB_.as<T>(),    dSpB_.as<T>(),  dYpB_.as<T>(),
                          dXpB_.as<T>(),           dIpB_.as<T>(),   0};
  const int slices = batch_slices(kp), width = ((kp / V + slices - 1) / slices) * V;
  const int blocks = (int)std::min<long long>(std::max(1LL, (long long)nItems_ * slices), (long long)sms_ * cfg.blocks);
  launch_k(apply_batch_kernel<T>, dim3(blocks), dim3(NGRP * GT + 32), smem, st, args, kp, slices, width, nSync_);
  RSCHOL_LAUNCH_CHECK();
  launch_k(narrow_kernel<T>, dim3(grid), dim3(256), 0, st, (const T*)w, W64, n, k, kp, sync + 1, nSync_ * slices - 1);
  RSCHOL_LAUNCH_CHECK();
}

template <class T>
int SolveEngine<T>::take_error_batch(cudaStream_t st) {
  int e = 0;
  if (!dSyncB_.p) return 0;
  RSCHOL_CUDA(cudaMemcpyAsync(&e, dSyncB_.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  RSCHOL_CUDA(cudaStreamSynchronize(st));
  if (e) {
    RSCHOL_CUDA(cudaMemsetAsync(dSyncB_.p, 0, dSyncB_.bytes, st));
    RSCHOL_CUDA(cudaStreamSynchronize(st));
  }
  return e;
}

#define RSCHOL_INST(T)                                                                               \
  template int SolveEngine<T>::batch_capacity() const;                                               \
  template int SolveEngine<T>::batch_slices(int) const;                                              \
  template void SolveEngine<T>::plan_batch(int);                                                     \
  template const SolveEngine<T>::BatchCfg& SolveEngine<T>::config_for(int, cudaStream_t, bool);      \
  template int SolveEngine<T>::width_class(int) const;                                               \
  template void SolveEngine<T>::autotune_batch(int, cudaStream_t);                                   \
  template void SolveEngine<T>::apply_batch_cfg(double*, int, cudaStream_t, const BatchCfg&);        \
  template std::vector<std::array<double, 6>> SolveEngine<T>::batch_tuning() const;                  \
  template void SolveEngine<T>::apply_batch(double*, int, cudaStream_t);                             \
  template int SolveEngine<T>::take_error_batch(cudaStream_t);
RSCHOL_INST(double)
RSCHOL_INST(float)
#undef RSCHOL_INST

}  // namespace rschol
