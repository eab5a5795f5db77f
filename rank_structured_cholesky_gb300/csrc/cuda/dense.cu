// Batched dense kernels (FP64 and FP32 instantiations).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "dense.cuh"
#include "solve_dev.cuh"

namespace rschol {

namespace {

using solvedev::ld_acquire;
using solvedev::st_release;
using solvedev::wait_geq;
using solvedev::wait_geq_lim;

constexpr int BM = 64, BN = 64, BK = 16, GEMM_THREADS = 256;

// One 64 x 64 tile of C = alpha op(A) op(B) + beta C at (row0, col0), by
// the 256 threads of the block.  Two shared stages: the next K slice is
// loaded into registers while the current one is multiplied (one barrier per
// slice); C is fetched before the K loop.  Each C entry's K order is the
// plain ascending one.
template <class T>
__device__ void gemm_tile(const GemmTask<T>& t, int row0, int col0, T (*As)[BK][BM + 1], T (*Bs)[BK][BN + 1]) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
  T cpre[4][4];
  if (t.beta != T(0)) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gi = row0 + ty + 16 * i, gj = col0 + tx + 16 * j;
        cpre[i][j] = (gi < t.M && gj < t.N) ? __ldcg(t.C + (size_t)gi * t.ldc + gj) : T(0);
      }
  }
  T ra[4], rb[4];
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int i, k;
      if (!t.tA) { i = (tid >> 4) + 16 * q; k = tid & 15; }
      else { i = tid & 63; k = (tid >> 6) + 4 * q; }
      const int gi = row0 + i, gk = k0 + k;
      ra[q] = (gi < t.M && gk < t.K) ? __ldcg(t.tA ? t.A + (size_t)gk * t.lda + gi : t.A + (size_t)gi * t.lda + gk)
                                       : T(0);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int j, k;
      if (!t.tB) { j = tid & 63; k = (tid >> 6) + 4 * q; }
      else { j = (tid >> 4) + 16 * q; k = tid & 15; }
      const int gj = col0 + j, gk = k0 + k;
      rb[q] = (gj < t.N && gk < t.K) ? __ldcg(t.tB ? t.B + (size_t)gj * t.ldb + gk : t.B + (size_t)gk * t.ldb + gj)
                                       : T(0);
    }
  };
  auto store = [&](int st) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int i, k;
      if (!t.tA) { i = (tid >> 4) + 16 * q; k = tid & 15; }
      else { i = tid & 63; k = (tid >> 6) + 4 * q; }
      As[st][k][i] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int j, k;
      if (!t.tB) { j = tid & 63; k = (tid >> 6) + 4 * q; }
      else { j = (tid >> 4) + 16 * q; k = tid & 15; }
      Bs[st][k][j] = rb[q];
    }
  };
  if (t.K > 0) {
    load(0);
    store(0);
  }
  __syncthreads();
  int st = 0;
  for (int k0 = 0; k0 < t.K; k0 += BK) {
    const bool more = k0 + BK < t.K;
    if (more) load(k0 + BK);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      T a[4], bb[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[st][k][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bb[j] = Bs[st][k][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], bb[j], acc[i][j]);
    }
    if (more) store(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gi = row0 + ty + 16 * i;
    if (gi >= t.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gj = col0 + tx + 16 * j;
      if (gj >= t.N) continue;
      T* c = t.C + (size_t)gi * t.ldc + gj;
      T v = t.alpha * acc[i][j];
      if (t.beta != T(0)) v = fma(t.beta, cpre[i][j], v);
      *c = v;
    }
  }
}

// FP64: one 32 x 32 tile.  The FP64 unit is the limit (two multiply-adds a
// clock and SM), so the tile is small enough to spread a launch over the SMs and
// the 16 x 16 blocks outside C are skipped; K in slices of 32, the next one
// loaded into registers under the current one's products.  Each C entry's K
// order is the plain ascending one.  (3D 37x41x35 FP64: the GEMM steps of a
// factorisation 18.0 ms in 64 x 64 tiles, 7.2 so, 5.1 with the launches of few
// tiles split along K.)
// part != null: the slice [kb, ke) of K, its plain product into part (32 x 32).
__device__ void gemm_tile_f64(const GemmTask<double>& t, int row0, int col0, int kb, int ke, double* part,
                              double (*As)[32][33], double (*Bs)[32][33]) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int nI = min(2, (t.M - row0 + 15) >> 4), nJ = min(2, (t.N - col0 + 15) >> 4);
  double acc[2][2] = {{0, 0}, {0, 0}}, cpre[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int gi = row0 + ty + 16 * i, gj = col0 + tx + 16 * j;
      cpre[i][j] = (t.beta != 0 && !part && gi < t.M && gj < t.N) ? __ldcg(t.C + (size_t)gi * t.ldc + gj) : 0.0;
    }
  double ra[4], rb[4];
  const int f = tid & 31, s0 = tid >> 5;   // fast and slow index of a thread's four elements (slow: s0 + 8 q)
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int s = s0 + 8 * q;
      const int gi = row0 + (t.tA ? f : s), ka = k0 + (t.tA ? s : f);
      ra[q] = (gi < t.M && ka < ke) ? __ldcg(t.A + (t.tA ? (size_t)ka * t.lda + gi : (size_t)gi * t.lda + ka)) : 0.0;
      const int gj = col0 + (t.tB ? s : f), kk = k0 + (t.tB ? f : s);
      rb[q] = (gj < t.N && kk < ke) ? __ldcg(t.B + (t.tB ? (size_t)gj * t.ldb + kk : (size_t)kk * t.ldb + gj)) : 0.0;
    }
  };
  auto store = [&](int st) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int s = s0 + 8 * q;
      if (t.tA) As[st][f][s] = ra[q];
      else As[st][s][f] = ra[q];
      if (t.tB) Bs[st][s][f] = rb[q];
      else Bs[st][f][s] = rb[q];
    }
  };
  if (ke > kb) {
    load(kb);
    store(0);
  }
  __syncthreads();
  int st = 0;
  for (int k0 = kb; k0 < ke; k0 += 32) {
    const bool more = k0 + 32 < ke;
    if (more) load(k0 + 32);
    const int kn = min(32, ke - k0);
    if (nI == 2 && nJ == 2) {
#pragma unroll 4
      for (int k = 0; k < kn; ++k) {
        const double a0 = As[st][ty][k], a1 = As[st][ty + 16][k], b0 = Bs[st][tx][k], b1 = Bs[st][tx + 16][k];
        acc[0][0] = fma(a0, b0, acc[0][0]);
        acc[0][1] = fma(a0, b1, acc[0][1]);
        acc[1][0] = fma(a1, b0, acc[1][0]);
        acc[1][1] = fma(a1, b1, acc[1][1]);
      }
    } else {
#pragma unroll 4
      for (int k = 0; k < kn; ++k) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            if (i < nI && j < nJ) acc[i][j] = fma(As[st][ty + 16 * i][k], Bs[st][tx + 16 * j][k], acc[i][j]);
      }
    }
    if (more) store(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int gi = row0 + ty + 16 * i, gj = col0 + tx + 16 * j;
      if (gi >= t.M || gj >= t.N) continue;
      if (part) {
        part[(ty + 16 * i) * 32 + tx + 16 * j] = acc[i][j];
        continue;
      }
      double v = t.alpha * acc[i][j];
      if (t.beta != 0) v = fma(t.beta, cpre[i][j], v);
      t.C[(size_t)gi * t.ldc + gj] = v;
    }
}

// FP32, launches of many tiles: 128 x 64 of C a block, 8 x 4 a thread.  What bounds
// the 64 x 64 tile is its instructions -- eight shared loads for 16 multiply-adds, and
// the addresses of a tile's loads and C -- (ncu: issue slots 70 % busy, FMA pipe
// 46 %); this one has three shared loads for 32.  Rows 4 ty + a and 64 + 4 ty + a,
// columns 2 tx + b and 32 + 2 tx + b; the sums as there, ascending in K.
// (Updates of rank 32 - 112: 3D 96^3 9.1 -> 7.6 ms a factorisation, 64^3 1.9 -> 1.6.)
constexpr int G2_ROWS = 128, G2_BK = 16;
__global__ void __launch_bounds__(GEMM_THREADS, 2) gemm_rows128_kernel(const GemmTask<float>* __restrict__ tasks,
                                                                       int nTasks) {
  __shared__ __align__(16) float As[2][G2_BK][132], Bs[2][G2_BK][68];
  int lo = 0, hi = nTasks - 1;
  const int bid = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tasks[mid].tileBase <= bid) lo = mid;
    else hi = mid - 1;
  }
  const GemmTask<float> t = tasks[lo];
  const int local = bid - t.tileBase, ti = local / t.tilesN, tj = local - ti * t.tilesN;
  const int row0 = ti * G2_ROWS, col0 = tj * 64;
  if (t.lower && row0 + G2_ROWS - 1 < col0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
  const bool aK = !t.tA, bK = t.tB != 0;
  // a thread's elements of a slice: along K a warp takes 4 rows x 8 k (whole sectors), else rows
  float ra[8], rb[4];
  auto arow = [&](int q) { return aK ? 4 * ((q * 8 + warp) & 31) + (lane & 3) : tid & 127; };
  auto ak = [&](int q) { return aK ? 8 * ((q * 8 + warp) >> 5) + (lane >> 2) : (tid >> 7) + 2 * q; };
  auto brow = [&](int q) { return bK ? 4 * ((q * 8 + warp) & 15) + (lane & 3) : tid & 63; };
  auto bk = [&](int q) { return bK ? 8 * ((q * 8 + warp) >> 4) + (lane >> 2) : (tid >> 6) + 4 * q; };
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int gi = row0 + arow(q), gk = k0 + ak(q);
      ra[q] = (gi < t.M && gk < t.K) ? __ldcg(aK ? t.A + (size_t)gi * t.lda + gk : t.A + (size_t)gk * t.lda + gi) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int gj = col0 + brow(q), gk = k0 + bk(q);
      rb[q] = (gj < t.N && gk < t.K) ? __ldcg(bK ? t.B + (size_t)gj * t.ldb + gk : t.B + (size_t)gk * t.ldb + gj) : 0.f;
    }
  };
  auto store = [&](int st) {
#pragma unroll
    for (int q = 0; q < 8; ++q) As[st][ak(q)][arow(q)] = ra[q];
#pragma unroll
    for (int q = 0; q < 4; ++q) Bs[st][bk(q)][brow(q)] = rb[q];
  };
  float acc[8][4];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
  if (t.K > 0) {
    load(0);
    store(0);
  }
  __syncthreads();
  int st = 0;
  for (int k0 = 0; k0 < t.K; k0 += G2_BK) {
    const bool more = k0 + G2_BK < t.K;
    if (more) load(k0 + G2_BK);
#pragma unroll 8
    for (int k = 0; k < G2_BK; ++k) {   // (zeros beyond K)
      const float4 a0 = *reinterpret_cast<const float4*>(&As[st][k][4 * ty]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[st][k][64 + 4 * ty]);
      const float2 b0 = *reinterpret_cast<const float2*>(&Bs[st][k][2 * tx]);
      const float2 b1 = *reinterpret_cast<const float2*>(&Bs[st][k][32 + 2 * tx]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(av[a], bv[b], acc[a][b]);
    }
    if (more) store(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
  const bool pairs = ((reinterpret_cast<uintptr_t>(t.C) & 7) | (t.ldc & 1)) == 0;   // two columns as one access
#pragma unroll
  for (int h = 0; h < 2; ++h) {   // (all C loads of a half before its first use)
    float c[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; b += 2) {
        const int gi = row0 + 64 * h + 4 * ty + a, gj = col0 + 16 * b + 2 * tx;
        const float* p = t.C + (size_t)gi * t.ldc + gj;
        c[a][b] = c[a][b + 1] = 0.f;
        if (t.beta == 0.f || gi >= t.M) continue;
        if (pairs && gj + 1 < t.N) {
          const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
          c[a][b] = v.x;
          c[a][b + 1] = v.y;
        } else {
          if (gj < t.N) c[a][b] = __ldcg(p);
          if (gj + 1 < t.N) c[a][b + 1] = __ldcg(p + 1);
        }
      }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; b += 2) {
        const int gi = row0 + 64 * h + 4 * ty + a, gj = col0 + 16 * b + 2 * tx;
        if (gi >= t.M) continue;
        float v0 = t.alpha * acc[4 * h + a][b], v1 = t.alpha * acc[4 * h + a][b + 1];
        if (t.beta != 0.f) {
          v0 = fmaf(t.beta, c[a][b], v0);
          v1 = fmaf(t.beta, c[a][b + 1], v1);
        }
        float* p = t.C + (size_t)gi * t.ldc + gj;
        if (pairs && gj + 1 < t.N) {
          *reinterpret_cast<float2*>(p) = make_float2(v0, v1);
        } else {
          if (gj < t.N) p[0] = v0;
          if (gj + 1 < t.N) p[1] = v1;
        }
      }
  }
}

template <class T>
__global__ void __launch_bounds__(GEMM_THREADS) gemm_kernel(const GemmTask<T>* __restrict__ tasks, int nTasks) {
  int lo = 0, hi = nTasks - 1;
  const int b = blockIdx.x;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (tasks[mid].tileBase <= b) lo = mid;
    else hi = mid - 1;
  }
  const GemmTask<T> t = tasks[lo];
  int local = b - t.tileBase, slice = 0;
  if (std::is_same<T, double>::value && t.kSplit > 1) {   // K slices: the tiles of each in turn
    const int tilesPer = ((t.M + 31) / 32) * t.tilesN;
    slice = local / tilesPer;
    local -= slice * tilesPer;
  }
  const int ti = local / t.tilesN, tj = local - ti * t.tilesN;
  constexpr int TL = simt_tile<T>;
  const int row0 = ti * TL, col0 = tj * TL;
  if (t.lower && row0 + TL - 1 < col0) return;
  if constexpr (std::is_same<T, double>::value) {
    __shared__ double As[2][32][33];
    __shared__ double Bs[2][32][33];
    double* part = nullptr;
    if (t.kSplit > 1)
      part = reinterpret_cast<double*>(t.ws) + ((size_t)slice * ((t.M + 31) / 32) * t.tilesN + local) * 1024;
    gemm_tile_f64(t, row0, col0, t.kSplit > 1 ? slice * t.kLen : 0,
                  t.kSplit > 1 ? min(t.K, (slice + 1) * t.kLen) : t.K, part, As, Bs);
  } else {
    __shared__ T As[2][BK][BM + 1];
    __shared__ T Bs[2][BK][BN + 1];
    gemm_tile<T>(t, row0, col0, As, Bs);
  }
}

// C = alpha * (sum of the K-slice products, in slice order) + beta * C for the
// split FP64 tasks of a launch; one thread per element of C.
__global__ void gemm_splitk_reduce_f64(const GemmTask<double>* __restrict__ tasks, const int* __restrict__ ids,
                                       int nIds, const long long* __restrict__ elemBase) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= elemBase[nIds]) return;
  int lo = 0, hi = nIds - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (elemBase[mid] <= e) lo = mid;
    else hi = mid - 1;
  }
  const GemmTask<double> t = tasks[ids[lo]];
  const long long le = e - elemBase[lo];
  const int i = (int)(le / t.N), j = (int)(le - (long long)i * t.N);
  const size_t tilesPer = (size_t)((t.M + 31) / 32) * t.tilesN;
  const double* p = reinterpret_cast<const double*>(t.ws) + ((size_t)(i >> 5) * t.tilesN + (j >> 5)) * 1024 +
                    (i & 31) * 32 + (j & 31);
  double s = 0.0;
  for (int sl = 0; sl < t.kSplit; ++sl) s += p[sl * tilesPer * 1024];
  double* c = t.C + (size_t)i * t.ldc + j;
  double v = t.alpha * s;
  if (t.beta != 0) v = fma(t.beta, *c, v);
  *c = v;
}

template <class T>
__global__ void __launch_bounds__(256) potrf_kernel(const PotrfTask<T>* __restrict__ tasks, int* flag) {
  // Right-looking Cholesky of one <= 64 x 64 tile in 16-column panels: one
  // warp factors the panel's diagonal block, every thread solves a row of
  // the panel below it, then all threads update the trailing triangle.
  const PotrfTask<T> t = tasks[blockIdx.x];
  __shared__ T a[64][65];
  __shared__ int bad;
  const int n = t.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int idx = tid; idx < n * n; idx += blockDim.x) {
    const int i = idx / n, j = idx - i * n;
    a[i][j] = (j <= i) ? t.A[(size_t)i * t.ld + j] : T(0);
  }
  if (tid == 0) bad = 0;
  __syncthreads();
  for (int p0 = 0; p0 < n; p0 += 16) {
    const int pw = min(16, n - p0);
    if (warp == 0) {
      for (int j = 0; j < pw; ++j) {
        const int jj = p0 + j;
        if (lane == 0) {
          T d = a[jj][jj];
          if (!(d > T(0))) {   // not positive definite (or NaN): keep going, report
            bad = 1;
            d = T(1);
          }
          a[jj][jj] = sqrt(d);
        }
        __syncwarp();
        if (lane > j && lane < pw) a[p0 + lane][jj] /= a[jj][jj];
        __syncwarp();
        if (lane > j && lane < pw) {
          const T lij = a[p0 + lane][jj];
          for (int k = j + 1; k <= lane; ++k) a[p0 + lane][p0 + k] -= lij * a[p0 + k][jj];
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for (int i = p0 + pw + tid; i < n; i += blockDim.x)
      for (int j = 0; j < pw; ++j) {
        T s = a[i][p0 + j];
        for (int k = 0; k < j; ++k) s -= a[i][p0 + k] * a[p0 + j][p0 + k];
        a[i][p0 + j] = s / a[p0 + j][p0 + j];
      }
    __syncthreads();
    const int q0 = p0 + pw, m = n - q0;
    for (int idx = tid; idx < m * m; idx += blockDim.x) {
      const int ii = idx / m, kk = idx - ii * m;
      if (kk <= ii) {
        T s = T(0);
        for (int c = 0; c < pw; ++c) s += a[q0 + ii][p0 + c] * a[q0 + kk][p0 + c];
        a[q0 + ii][q0 + kk] -= s;
      }
    }
    __syncthreads();
  }
  for (int idx = tid; idx < n * n; idx += blockDim.x) {
    const int i = idx / n, j = idx - i * n;
    if (j <= i) t.A[(size_t)i * t.ld + j] = a[i][j];
  }
  if (tid == 0 && bad) atomicMin(flag, t.code);
}

template <class T>
__global__ void __launch_bounds__(256) trsm_kernel(const TrsmTask<T>* __restrict__ tasks, int nTasks) {
  // B (64-row chunk x w) := B L^{-T} in 16-column panels: each row solves
  // with the panel's diagonal block (16 steps), then all threads update the
  // columns to the right.
  int lo = 0, hi = nTasks - 1;
  const int b = blockIdx.x;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (tasks[mid].chunkBase <= b) lo = mid;
    else hi = mid - 1;
  }
  const TrsmTask<T> t = tasks[lo];
  const int r0 = (b - t.chunkBase) * 64;
  const int nr = min(64, t.rows - r0);
  const int w = t.w, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char trsm_smem[];
  T (*L)[65] = reinterpret_cast<T (*)[65]>(trsm_smem);
  T (*X)[65] = reinterpret_cast<T (*)[65]>(trsm_smem + sizeof(T) * 64 * 65);
  for (int idx = tid; idx < w * w; idx += blockDim.x) {
    const int i = idx / w, j = idx - i * w;
    L[i][j] = (j <= i) ? t.L[(size_t)i * t.ldl + j] : T(0);
  }
  for (int idx = tid; idx < nr * w; idx += blockDim.x) {
    const int i = idx / w, j = idx - i * w;
    X[i][j] = t.B[(size_t)(r0 + i) * t.ldb + j];
  }
  __syncthreads();
  for (int p0 = 0; p0 < w; p0 += 16) {
    const int pw = min(16, w - p0);
    if (tid < nr)
      for (int j = 0; j < pw; ++j) {
        T s = X[tid][p0 + j];
        for (int k = 0; k < j; ++k) s -= X[tid][p0 + k] * L[p0 + j][p0 + k];
        X[tid][p0 + j] = s / L[p0 + j][p0 + j];
      }
    __syncthreads();
    const int q0 = p0 + pw, wq = w - q0;
    for (int idx = tid; idx < nr * wq; idx += blockDim.x) {
      const int i = idx / wq, q = q0 + (idx - i * wq);
      T s = T(0);
      for (int c = 0; c < pw; ++c) s += X[i][p0 + c] * L[q][p0 + c];
      X[i][q] -= s;
    }
    __syncthreads();
  }
  for (int idx = tid; idx < nr * w; idx += blockDim.x) {
    const int i = idx / w, j = idx - i * w;
    t.B[(size_t)(r0 + i) * t.ldb + j] = X[i][j];
  }
}

// FP32 variants: a register-resident POTRF (thread (i, g) keeps row i,
// columns g, g + 4, ... of the tile) and a TRSM that inverts the tile in
// every block and multiplies; they beat the panel-blocked kernels above in
// FP32, while FP64 prefers the blocked ones.  The tile bodies are device
// functions shared with the fused level kernel below.

// Right-looking Cholesky of one n x n (n <= 64) tile at A (row-major, ld) by
// the block's 256 threads as a 16 x 16 grid: thread (ti, tk) keeps the 4 x 4
// entries (ti + 16 a, tk + 16 b) in registers.  Column j is published
// unscaled (u_i = a_ij for i > j, zeros at rows <= j; the pivot p = a_jj
// apart) through a double-buffered shared vector laid out by (i % 16, i / 16),
// so one barrier per column suffices and a thread reads its four row values
// and its four column values as two 16-byte loads; every thread then runs
// the same 16 unpredicated FMAs a_ik -= (u_i / p) u_k (the zeros leave
// finished entries unchanged; entries right of the diagonal are never
// stored).  Finally L_jj = sqrt(p_j), L_ij = a_ij / sqrt(p_j).  A
// non-positive pivot is replaced by 1 and reported as atomicMin(flag, code).
// 1 / p on a POTRF's critical path: the fast reciprocal (MUFU-based,
// __fdividef, within 2 ulp) in FP32, whose factor carries larger rounding
// errors anyway; exact division in FP64.
__device__ __forceinline__ float pivot_recip(float p) { return __fdividef(1.0f, p); }
__device__ __forceinline__ double pivot_recip(double p) { return 1.0 / p; }

template <class T>
__device__ void potrf_tile_reg(T* A, int ld, int n, int code, int* flag) {
  __shared__ __align__(16) T col[2][64];
  __shared__ T piv[64];
  __shared__ int bad;
  const int tid = threadIdx.x, ti = tid >> 4, tk = tid & 15;
  T v[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = ti + 16 * a, k = tk + 16 * b;
      v[a][b] = (i < n && k <= i) ? __ldcg(A + (size_t)i * ld + k) : T(0);
    }
  if (tid == 0) bad = 0;
  __syncthreads();
#pragma unroll
  for (int b0 = 0; b0 < 4; ++b0) {
#pragma unroll 1
    for (int jj = 0; jj < 16; ++jj) {
      const int j = 16 * b0 + jj;
      if (j >= n) break;
      T* cj = col[j & 1];
      if (tk == jj) {   // the owners of column j: rows ti + 16 a
        T u[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const int i = ti + 16 * a;
          u[a] = v[a][b0];
          if (i == j) {
            T p = u[a];
            if (!(p > T(0))) {   // not positive definite (or NaN): keep going, report
              bad = 1;
              p = T(1);
            }
            piv[j] = p;
          }
          if (i <= j) u[a] = T(0);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) cj[4 * ti + a] = u[a];
      }
      __syncthreads();
      const T rp = pivot_recip(piv[j]);
      T ur[4], uc[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        ur[a] = cj[4 * ti + a] * rp;
        uc[a] = cj[4 * tk + a];
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) v[a][b] -= ur[a] * uc[b];
    }
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = ti + 16 * a, k = tk + 16 * b;
      if (i < n && k <= i) {
        const T d = sqrt(piv[k]);
        A[(size_t)i * ld + k] = (k == i) ? d : v[a][b] / d;
      }
    }
  if (tid == 0 && bad) atomicMin(flag, code);
  __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(256) potrf_reg_kernel(const PotrfTask<T>* __restrict__ tasks, int* flag) {
  const PotrfTask<T> t = tasks[blockIdx.x];
  potrf_tile_reg<T>(t.A, t.ld, t.n, t.code, flag);
}

// Li := L^{-1}, L the w x w lower tile at Lg (ld ldl) padded to 64 with a
// unit diagonal (so the leading w x w block of Li is the inverse; only the
// 16 x 16 blocks that cover it are formed).  Blocked: the 16 x 16 diagonal
// inverses by forward substitution (warp b inverts block b, lane c keeps
// column c in registers, the diagonal reciprocals formed up front), then the
// off-diagonal blocks by distance from the diagonal,
// Li[R][C] = -Li[R][R] sum_{K=C}^{R-1} L[R][K] Li[K][C], with unrolled
// fixed-length inner products.  L, Li: 64 x 65 shared; Tm: 3 x 16 x 17
// shared.  256 threads.
template <class T>
__device__ void tile_inverse(const T* Lg, int ldl, int w, T (*L)[65], T (*Li)[65], T (*Tm)[16][17]) {
  const int tid = threadIdx.x;
  // tile loads unrolled: all 16 loads of a thread in flight at once
#pragma unroll
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    const int i = idx >> 6, j = idx & 63;
    L[i][j] = (i < w && j <= i) ? __ldcg(Lg + (size_t)i * ldl + j) : (i == j ? T(1) : T(0));
    Li[i][j] = T(0);
  }
  __syncthreads();
  const int nb = (w + 15) >> 4;   // 16 x 16 blocks that cover the w x w inverse
  {
    const int wb = tid >> 5, c = tid & 15;
    if (wb < nb && (tid & 31) < 16) {
      const int o = 16 * wb;
      T d[16], x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) d[r] = T(1) / L[o + r][o + r];
      // x = column c of the block inverse: x_r = (delta_rc - sum_{k<r} L_rk x_k) / L_rr;
      // rows above c come out zero by themselves
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        T s = (r == c) ? T(1) : T(0);
#pragma unroll
        for (int k = 0; k < r; ++k) s -= L[o + r][o + k] * x[k];
        x[r] = s * d[r];
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) Li[o + r][o + c] = x[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (int d = 1; d < 4; ++d) {
    if (d >= nb) break;
    const int np = nb - d;   // block pairs (R, C = R - d)
    for (int e = tid; e < np * 256; e += 256) {
      const int pr = e >> 8, i = (e >> 4) & 15, j = e & 15;
      const int C = pr, R = pr + d;
      T s = T(0);
#pragma unroll
      for (int k = 0; k < 16 * d; ++k) s += L[16 * R + i][16 * C + k] * Li[16 * C + k][16 * C + j];
      Tm[pr][i][j] = s;
    }
    __syncthreads();
    for (int e = tid; e < np * 256; e += 256) {
      const int pr = e >> 8, i = (e >> 4) & 15, j = e & 15;
      const int C = pr, R = pr + d;
      T s = T(0);
#pragma unroll
      for (int k = 0; k < 16; ++k) s += Li[16 * R + i][16 * R + k] * Tm[pr][k][j];   // Li[R][R] is lower
      Li[16 * R + i][16 * C + j] = -s;
    }
    __syncthreads();
  }
}

// B (nr <= 64 rows x w) := B Li^T with Li = L^{-1} (64 x 65 shared, zero
// above the diagonal); X: 64 x 65 shared staging.  256 threads.
template <class T>
__device__ void trsm_chunk_mul(T* B, int ldb, int nr, int w, T (*X)[65], T (*Li)[65]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    const int i = idx >> 6, j = idx & 63;
    X[i][j] = (i < nr && j < w) ? __ldcg(B + (size_t)i * ldb + j) : T(0);
  }
  __syncthreads();
  // out[i][j] = sum_{k <= j} X[i][k] Li[j][k]; thread: rows ty + 16 a, columns tx + 16 c
  const int tx = tid & 15, ty = tid >> 4;
  T acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[a][c] = T(0);
#pragma unroll 4
  for (int k = 0; k < w; ++k) {
    T xa[4], lb[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) xa[a] = X[ty + 16 * a][k];
#pragma unroll
    for (int c = 0; c < 4; ++c) lb[c] = Li[tx + 16 * c][k];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = fma(xa[a], lb[c], acc[a][c]);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int i = ty + 16 * a;
    if (i >= nr) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = tx + 16 * c;
      if (j < w) B[(size_t)i * ldb + j] = acc[a][c];
    }
  }
  __syncthreads();
}

// Factor and invert one FP32 tile on the chain of the fused Cholesky: S (64 x 68
// shared) holds the n x n lower tile, padded with a unit diagonal; on return its L, but
// for the entries below the diagonal in the 16 x 16 diagonal blocks, which are still to
// be divided by their column's diagonal (tile_entry, when the tile is stored: divided
// here they cost the chain 2 of 18 ms a factorisation of 3D 64^3), and in Li (64 x 68)
// the inverse's lower blocks.  A column at a time (potrf_tile_reg
// and tile_inverse) every column costs a block barrier and a round through shared
// memory, 22 us a tile.  Here in blocks of 16: one warp eliminates the diagonal
// block and the identity beside it with shuffles, the rows below are multiplied by
// the inverse, and the same warp updates and eliminates the next diagonal block
// while the others update the rest and form the inverse's finished block row -- two
// barriers a block, 10 us a tile.  A pivot that is not positive (or NaN) is
// replaced by 1 and reported as atomicMin(flag, code).
__device__ __noinline__ void potrf_inverse_f32(float (*S)[68], float (*Li)[68], float (*Tm)[16][17], int n, bool invert,
                                               int code, int* flag) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = (n + 15) >> 4;
  const int lj = lane & 15, hi = lane >> 4;
  bool bad = false;
  // warp 0: the 16 x 16 block at o; lane r (and r + 16) holds row r in v, and row r
  // of the inverse of the unit lower factor in e
  auto diag = [&](int o, float (&v)[16]) {
    float e[16], pd = 1.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) e[k] = k == lj ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float p = __shfl_sync(0xffffffffu, v[j], j, 16);
      bad |= !(p > 0.f);
      p = p > 0.f ? p : 1.f;
      pd = lj == j ? p : pd;
      const float l = lj > j ? v[j] * pivot_recip(p) : 0.f;
#pragma unroll
      for (int k = j + 1; k < 16; ++k) v[k] -= l * __shfl_sync(0xffffffffu, v[j], k, 16);
#pragma unroll
      for (int k = 0; k < j; ++k) e[k] -= l * __shfl_sync(0xffffffffu, e[k], j, 16);
      e[j] -= l;
    }
    const float d = sqrtf(pd), rd = 1.f / d;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (hi == 0) {
        Li[o + lj][o + k] = e[k] * rd;
        if (k <= lj) S[o + lj][o + k] = k == lj ? d : v[k];
      }
  };
  // a warp: block (R, C) of the inverse, -Li[R][R] sum_{C <= K < R} L[R][K] Li[K][C];
  // lane: column lj, rows 2 q + hi
  auto inv_block = [&](int R, int C) {
    float t[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) t[q] = 0.f;
    for (int k = 16 * C; k < 16 * R; k += 4) {
      float y[4];
#pragma unroll
      for (int z = 0; z < 4; ++z) y[z] = Li[k + z][16 * C + lj];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 x = *reinterpret_cast<const float4*>(&S[16 * R + 2 * q + hi][k]);
        t[q] = fmaf(x.w, y[3], fmaf(x.z, y[2], fmaf(x.y, y[1], fmaf(x.x, y[0], t[q]))));
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) Tm[C][2 * q + hi][lj] = t[q];
    __syncwarp();
    float y[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) y[k] = Tm[C][k][lj];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float x = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k) x = fmaf(Li[16 * R + 2 * q + hi][16 * R + k], y[k], x);
      Li[16 * R + 2 * q + hi][16 * C + lj] = -x;
    }
  };
  if (warp == 0) {
    float v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = S[lj][k];
    diag(0, v);
  }
  __syncthreads();
  for (int kb = 0; kb + 1 < nb; ++kb) {
    const int o = 16 * kb, left = nb - kb - 1;   // blocks below
    {   // X := A Li(kb)^T: a half warp owns a row
      const int c = tid & 15, rr = tid >> 4;
      float lc[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) lc[k] = Li[o + c][o + k];
      for (int a = 1; a <= left; ++a) {
        const int i = o + 16 * a + rr;
        float x = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) x = fmaf(S[i][o + k], lc[k], x);
        __syncwarp();
        S[i][o + c] = x;
      }
    }
    __syncthreads();
    if (warp == 0) {   // the next diagonal block: each half warp forms eight columns of every row
      const int q = o + 16;
      float xr[16], w[8], v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) xr[k] = S[q + lj][o + k];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) s = fmaf(xr[k], S[q + 8 * hi + c][o + k], s);
        w[c] = S[q + lj][q + 8 * hi + c] - s;
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float other = __shfl_xor_sync(0xffffffffu, w[c], 16);
        v[c] = hi ? other : w[c];
        v[8 + c] = hi ? w[c] : other;
      }
      diag(q, v);
    } else {   // block row kb of the inverse; the other lower blocks (a, b) in units of 8 rows x 16 columns
      const int ni = invert ? kb : 0, units = left * (left + 1) - 2;
      for (int w = warp - 1; w < ni + units; w += 7) {
        if (w < ni) {
          inv_block(kb, w);
          continue;
        }
        const int u = w - ni;
        int a = 1, t = u >> 1;   // block t of (1, 0), (1, 1), (2, 0), ...
        while (t > a) t -= ++a;
        const int rb = o + 16 + 16 * a + 8 * (u & 1) + hi, cb = o + 16 + 16 * t + lj;
        float xj[16], s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 16; ++k) xj[k] = S[cb][o + k];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < 16; ++k) s[q] = fmaf(S[rb + 2 * q][o + k], xj[k], s[q]);
#pragma unroll
        for (int q = 0; q < 4; ++q) S[rb + 2 * q][cb] -= s[q];
      }
    }
    __syncthreads();
  }
  if (invert && warp < nb - 1) inv_block(nb - 1, warp);
  if (tid == 0 && bad) atomicMin(flag, code);
}

__device__ __forceinline__ float tile_entry(const float (*S)[68], int i, int k) {
  return (i >> 4) == (k >> 4) && k < i ? S[i][k] / S[k][k] : S[i][k];
}
__device__ __forceinline__ double tile_entry(const double (*S)[33], int i, int k) { return S[i][k]; }

// The same for one FP64 tile (n <= 32; S, Li 32 x 33, Tm 16 x 17 shared).  A warp's
// multiply-add holds its quarter of the FP64 unit for 64 clocks, so what counts is
// how many each warp issues: warp w keeps rows 4 w .. 4 w + 3 (a thread: one row, every eighth
// column), skips columns right of them and everything finished, and a row's
// multiplier is formed once; column j is published unscaled with the reciprocal of
// its pivot, one barrier a column.  Square roots and their reciprocals by one
// warp; the inverse's two 16 x 16 diagonal blocks by one warp, a column a lane.
// (Cholesky steps of 3D 37x41x35 FP64 12.3 -> 12.1 ms against every
// thread forming all its products on every column.)
__device__ __noinline__ void potrf_inverse_f64(double (*S)[33], double (*Li)[33], double (*Tm)[17], int n, bool invert,
                                               int code, int* flag) {
  __shared__ double col[2][32], rpv[2], piv[32], dia[32], rdia[32];
  __shared__ int bad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = 4 * warp + (lane >> 3), kc = lane & 7, rLast = 4 * warp + 3;
  double v[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) v[c] = S[i][kc + 8 * c];
  if (tid == 0) bad = 0;
  if (tid < 32) piv[tid] = 1.0;
  __syncthreads();
#pragma unroll
  for (int c0 = 0; c0 < 4; ++c0) {
    for (int jj = 0; jj < 8 && 8 * c0 + jj < n; ++jj) {
      const int j = 8 * c0 + jj, buf = j & 1;
      if (kc == jj) {
        double u = v[c0];
        if (i == j) {
          if (!(u > 0.0)) {   // not positive definite (or NaN): keep going, report
            bad = 1;
            u = 1.0;
          }
          piv[j] = u;
          rpv[buf] = pivot_recip(u);
        }
        col[buf][i] = i <= j ? 0.0 : u;
      }
      __syncthreads();
      if (rLast > j) {
        const double l = col[buf][i] * rpv[buf];
#pragma unroll
        for (int c = c0; c < 4; ++c)
          if (8 * c <= rLast) v[c] -= l * col[buf][kc + 8 * c];
      }
    }
  }
  __syncthreads();
  if (tid < 32) {
    const double d = sqrt(piv[tid]);
    dia[tid] = d;
    rdia[tid] = 1.0 / d;
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int k = kc + 8 * c;
    if (8 * c <= rLast && k <= i) S[i][k] = k == i ? dia[i] : v[c] / dia[k];
  }
  if (tid == 0 && bad) atomicMin(flag, code);
  if (!invert) return;   // (uniform; the caller's barrier follows)
  __syncthreads();
  if (warp == 0) {
    const int c = lane & 15, o = lane & 16;
    double x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = r == c ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      x[k] *= rdia[o + k];
#pragma unroll
      for (int r = k + 1; r < 16; ++r) x[r] -= S[o + r][o + k] * x[k];
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) Li[o + r][o + c] = x[r];
  }
  __syncthreads();
  if (n <= 16) return;
  {   // Li21 = -Li22 (L21 Li11): warp w columns 2 w, 2 w + 1 (zero above them), then rows 2 w, 2 w + 1
    const int f = lane & 15, p = 2 * warp + (lane >> 4);
    double t = 0.0;
    for (int k = 2 * warp; k < 16; ++k) t = fma(S[16 + f][k], Li[k][p], t);
    Tm[f][p] = t;
    __syncthreads();
    t = 0.0;
    for (int k = 0; k <= 2 * warp + 1; ++k) t = fma(Li[16 + p][16 + k], Tm[k][f], t);
    Li[16 + p][f] = -t;
  }
}

// out (32 x 32) := L^{-1}, L the w x w (w <= 32) lower tile at Lg padded with a
// unit diagonal: the 16 x 16 diagonal inverses by forward substitution (a warp
// each, lane c keeps column c), then the block below the diagonal.
__device__ void tile_inverse_f64(const double* Lg, int ldl, int w, double* out, double* smem) {
  double (*L)[33] = reinterpret_cast<double (*)[33]>(smem);
  double (*Li)[33] = reinterpret_cast<double (*)[33]>(smem + 32 * 33);
  __shared__ double Tm[16][17], rd[32];
  const int tid = threadIdx.x;
#pragma unroll
  for (int idx = tid; idx < 1024; idx += 256) {
    const int i = idx >> 5, j = idx & 31;
    L[i][j] = (i < w && j <= i) ? __ldcg(Lg + (size_t)i * ldl + j) : (i == j ? 1.0 : 0.0);
    Li[i][j] = 0.0;
  }
  __syncthreads();
  if (tid < 32) rd[tid] = 1.0 / L[tid][tid];
  __syncthreads();
  const int nb = (w + 15) >> 4;
  {
    const int wb = tid >> 5, c = tid & 15;
    if (wb < nb && (tid & 31) < 16) {
      const int o = 16 * wb;
      double x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        double s = (r == c) ? 1.0 : 0.0;
#pragma unroll
        for (int k = 0; k < r; ++k) s -= L[o + r][o + k] * x[k];
        x[r] = s * rd[o + r];
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) Li[o + r][o + c] = x[r];
    }
  }
  __syncthreads();
  if (nb == 2) {
    const int i = tid >> 4, j = tid & 15;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += L[16 + i][k] * Li[k][j];
    Tm[i][j] = s;
    __syncthreads();
    s = 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k <= (i | 1)) s += Li[16 + i][16 + k] * Tm[k][j];   // (lower; i | 1: the same for a warp)
    Li[16 + i][j] = -s;
    __syncthreads();
  }
#pragma unroll
  for (int idx = tid; idx < 1024; idx += 256) out[idx] = Li[idx >> 5][idx & 31];
}

template <class T>
__global__ void __launch_bounds__(256) trsm_inv_kernel(const TrsmTask<T>* __restrict__ tasks, int nTasks) {
  // B (64-row chunk x w) := B L^{-T}: the block inverts its w x w tile and
  // multiplies.
  int lo = 0, hi = nTasks - 1;
  const int b = blockIdx.x;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (tasks[mid].chunkBase <= b) lo = mid;
    else hi = mid - 1;
  }
  const TrsmTask<T> t = tasks[lo];
  const int rb0 = (b - t.chunkBase) * TRSM_ROWS_F32;
  extern __shared__ __align__(16) unsigned char trsm_smem[];
  T (*L)[65] = reinterpret_cast<T (*)[65]>(trsm_smem);
  T (*Li)[65] = reinterpret_cast<T (*)[65]>(trsm_smem + sizeof(T) * 64 * 65);
  T (*X)[65] = reinterpret_cast<T (*)[65]>(trsm_smem + 2 * sizeof(T) * 64 * 65);
  T (*Tm)[16][17] = reinterpret_cast<T (*)[16][17]>(trsm_smem + 3 * sizeof(T) * 64 * 65);   // 3 blocks
  tile_inverse<T>(t.L, t.ldl, t.w, L, Li, Tm);
  for (int sub = 0; sub < TRSM_ROWS_F32 / 64; ++sub) {
    const int r0 = rb0 + 64 * sub;
    if (r0 >= t.rows) break;
    trsm_chunk_mul<T>(t.B + (size_t)r0 * t.ldb, t.ldb, min(64, t.rows - r0), t.w, X, Li);
  }
}

// Blocked partial Cholesky of every front of a level in one launch.  A job
// factors the first nDiag columns of a front F (rows x rows, lower, row-major)
// in panels: the first w0 = nDiag - NB (P - 1) wide, the others NB (64, FP64 32),
// so that every later panel and every trailing block is aligned to the tile grid
// b(0) = 0, b(t) = w0 + NB (t - 1).  A work item is one lower tile (a, b) from its
// input to its result (left-looking): it subtracts X(a, q) X(b, q)^T of the panels
// q < min(b, P) in order, as they appear, from the tile in registers -- read once,
// before any wait, and written once -- and then
//   POTRF(p)      a = b = p: factors the tile and stores its inverse
//   TRSM(a, b)    b < P: multiplies by the inverse of tile b
//   GEMM(a, b)    b >= P: a tile of the trailing block, nothing more.
// A block takes the next item from a ticket counter; the items are listed in a
// topological order, so a block only waits, bounded, on items taken before its
// own: tdone[a] panels of row tile a stored, pdone[p] inverse p stored.
// What bounds it is the chain POTRF(p) -> TRSM(p + 1, p) -> POTRF(p + 1); as one
// item a tile and panel (right-looking) it was 36 us a panel, 22 of them the tile's
// factor and inverse, 5 the three hand-overs; now it is 22, and the updates read
// and write their tiles once (Cholesky steps of a factorisation: 3D 64^3 10.3 -> 7.5
// ms, 96^3 49.2 -> 35.2 ms, elasticity 30^3 6.3 -> 4.5 ms).
// sync[0] is the ticket, the counters follow (zeroed before every launch);
// a wait that gives up sets flag[1].  Data written by other blocks is read
// through L2 (ld.global.cg).
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned smid() {
  unsigned r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}

// A tile's registers and staging: 16 x 16 threads, R x R entries each -- FP32 rows
// 4 ty + a and columns 4 tx + b, so that a K step is two 16-byte shared loads for
// 16 FMAs; FP64 rows ty + 16 a and columns tx + 16 b, so that the 16 x 16 blocks
// outside the matrix or above the diagonal are skipped.  A panel's products are
// summed in ascending k and subtracted from the tile together.
template <class T>
struct CholTile;
// (c0, c1) += a (b0, b1): two FP32 multiply-adds in one instruction
__device__ __forceinline__ void fma2(float& c0, float& c1, float a, float b0, float b1) {
  asm("{\n.reg .b64 pa, pb, pc;\nmov.b64 pa, {%2, %2};\nmov.b64 pb, {%3, %4};\nmov.b64 pc, {%0, %1};\n"
      "fma.rn.f32x2 pc, pa, pb, pc;\nmov.b64 {%0, %1}, pc;\n}"
      : "+f"(c0), "+f"(c1)
      : "f"(a), "f"(b0), "f"(b1));
}
template <>
struct CholTile<float> {
  static constexpr int NB = 64, R = 4, Q = 8;
  typedef float Stage[32][68];   // k-major: conflict-free stores, 16-byte loads
  // element q of a thread in a 64 x 32 slice (a warp: 4 rows x 8 columns, full sectors)
  static __device__ int row(int q) { return 4 * ((q * 8 + ((int)threadIdx.x >> 5)) & 15) + (threadIdx.x & 3); }
  static __device__ int col(int q) { return 8 * ((q * 8 + ((int)threadIdx.x >> 5)) >> 4) + ((threadIdx.x & 31) >> 2); }
  static __device__ int ti(int a) { return 4 * (threadIdx.x >> 4) + a; }
  static __device__ int tj(int b) { return 4 * (threadIdx.x & 15) + b; }
  static __device__ float& at(Stage& s, int i, int k) { return s[k][i]; }
  static __device__ void mul(const Stage& A, const Stage& B, int kn, float (&acc)[4][4], bool, bool, bool) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
    for (int k = 0; k < kn; ++k) {
      const float4 av = *reinterpret_cast<const float4*>(&A[k][4 * ty]);
      const float4 bv = *reinterpret_cast<const float4*>(&B[k][4 * tx]);
      const float ar[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        fma2(acc[a][0], acc[a][1], ar[a], bv.x, bv.y);
        fma2(acc[a][2], acc[a][3], ar[a], bv.z, bv.w);
      }
    }
  }
};
template <>
struct CholTile<double> {
  static constexpr int NB = 32, R = 2, Q = 4;
  typedef double Stage[32][33];
  static __device__ int row(int q) { return (threadIdx.x >> 5) + 8 * q; }
  static __device__ int col(int) { return threadIdx.x & 31; }
  static __device__ int ti(int a) { return (threadIdx.x >> 4) + 16 * a; }
  static __device__ int tj(int b) { return (threadIdx.x & 15) + 16 * b; }
  static __device__ double& at(Stage& s, int i, int k) { return s[i][k]; }
  // w01, w10, w11: the blocks wanted besides (0, 0); kLeft: the K of the left ones
  static __device__ void mul(const Stage& A, const Stage& B, int kn, double (&acc)[2][2], bool w01, bool w10, bool w11,
                             int kLeft = 32) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
    for (int k = 0; k < kn; ++k) {
      const double a0 = A[ty][k], a1 = A[ty + 16][k], b0 = B[tx][k], b1 = B[tx + 16][k];
      if (k < kLeft) {
        acc[0][0] = fma(a0, b0, acc[0][0]);
        if (w10) acc[1][0] = fma(a1, b0, acc[1][0]);
      }
      if (w01) acc[0][1] = fma(a0, b1, acc[0][1]);
      if (w11) acc[1][1] = fma(a1, b1, acc[1][1]);
    }
  }
};
// dynamic shared memory: two stages of A and B, the TRSM's operands, or the POTRF's tiles
template <class T> constexpr int chol_smem = 4 * (int)sizeof(typename CholTile<T>::Stage) +
                                             (std::is_same<T, float>::value ? 3 * 16 * 17 * 4 : 0);

template <class T>
__global__ void __launch_bounds__(256, 3) chol_fused_kernel(const CholFusedJob<T>* __restrict__ jobs,
                                                            const CholItem* __restrict__ items, int nItems,
                                                            int* __restrict__ sync, T* __restrict__ ws, int* flag,
                                                            unsigned long long* __restrict__ trace) {
  typedef CholTile<T> C;
  typedef typename C::Stage Stage;
  constexpr int NB = C::NB, R = C::R;
  static_assert(NB == chol_nb<T>, "tile width");
  extern __shared__ __align__(16) unsigned char cf_smem[];
  Stage* As = reinterpret_cast<Stage*>(cf_smem);   // [2]
  Stage* Bs = As + 2;                              // [2]
  __shared__ int sTicket, sReady;
  __shared__ unsigned long long tStart, tReady;
  int* err = flag + 1;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    sTicket = atomicAdd(sync, 1);
    if (trace) tStart = tReady = globaltimer_ns();
  }
  __syncthreads();
  if (sTicket >= nItems) {   // counters not reset: report, touch nothing
    if (threadIdx.x == 0) atomicExch(err, 2);
    return;
  }
  const CholItem it = items[sTicket];
  const CholFusedJob<T> j = jobs[it.job];
  int* tdone = sync + 1 + j.cnt;   // TR: panels of row tile a stored
  int* pdone = tdone + j.TR;       // P: inverse of panel p stored
  const int a = it.a, b = it.b;
  const int* lim = flag + 2;   // polls before a wait gives up (set with the flags before the factorisation)
  auto bnd = [&](int t) { return t == 0 ? 0 : j.w0 + NB * (t - 1); };      // columns (and Cholesky rows)
  auto rbnd = [&](int t) { return t == 0 ? 0 : j.r1 + NB * (t - 1); };     // rows
  T* F = j.F;
  const int ld = j.ld, q0 = bnd(b);
  int* done = nullptr;
  int doneVal = 0;
  if (it.kind == CHOL_POTRF && j.L) {   // TRSM job: L is factored already, invert its diagonal tile
    const T* A = j.L + (size_t)q0 * j.ldl + q0;
    T* out = ws + j.inv + (size_t)b * NB * NB;
    const int w = bnd(b + 1) - q0;
    if constexpr (std::is_same<T, double>::value) {
      tile_inverse_f64(A, j.ldl, w, out, reinterpret_cast<double*>(cf_smem));
    } else {
      T (*L)[65] = reinterpret_cast<T (*)[65]>(cf_smem);
      T (*Li)[65] = L + 64;
      T (*Tm)[16][17] = reinterpret_cast<T (*)[16][17]>(Li + 64);
      tile_inverse<T>(A, j.ldl, w, L, Li, Tm);
#pragma unroll
      for (int idx = threadIdx.x; idx < 64 * 64; idx += 256) out[idx] = Li[idx >> 6][idx & 63];
    }
    done = pdone + b;
    doneVal = 1;
  } else {
    const int r0 = rbnd(a), m = min(rbnd(a + 1), j.nRows) - r0;
    const int n = (b < j.P ? bnd(b + 1) : min(bnd(b + 1), j.nUpd)) - q0;
    const bool same = !j.L && a == b;   // a diagonal tile: A = B, its upper blocks not wanted
    const int npan = min(b, j.P);
    T c[R][R];
#pragma unroll
    for (int x = 0; x < R; ++x)
#pragma unroll
      for (int y = 0; y < R; ++y) {
        const int i = C::ti(x), k = C::tj(y);
        c[x][y] = (i < m && k < n) ? __ldcg(F + (size_t)(r0 + i) * ld + q0 + k) : T(0);
      }
    const T* Ap = F + (size_t)r0 * ld;
    const T* Bp = j.L ? j.L + (size_t)q0 * j.ldl : F + (size_t)q0 * ld;   // TRSM job: X(a) L(b, q)^T
    const int ldb = j.L ? j.ldl : ld;
    const bool w01 = n > 16 && !same, w10 = m > 16, w11 = m > 16 && n > 16;   // (FP64)
    T ra[C::Q], rb[C::Q];
    auto load = [&](int k0, int k1) {
#pragma unroll
      for (int q = 0; q < C::Q; ++q) {
        const int i = C::row(q), k = k0 + C::col(q);
        ra[q] = (i < m && k < k1) ? __ldcg(Ap + (size_t)i * ld + k) : T(0);
        if (!same) rb[q] = (i < n && k < k1) ? __ldcg(Bp + (size_t)i * ldb + k) : T(0);
      }
    };
    auto store = [&](int st) {
#pragma unroll
      for (int q = 0; q < C::Q; ++q) {
        C::at(As[st], C::row(q), C::col(q)) = ra[q];
        if (!same) C::at(Bs[st], C::row(q), C::col(q)) = rb[q];
      }
    };
    // The panels that are there, in one pipelined pass; then wait for more.  (Tiles
    // far from their turn waiting for four panels at a time, out of step with each
    // other, to be less in the way of the next panel's: no gain.)
    for (int q = 0; q < npan;) {
      if (warp == 0) {
        const bool ok = wait_geq_lim(tdone + a, q + 1, err, lim) &&
                        (same || j.L || wait_geq_lim(tdone + b, q + 1, err, lim));
        if (threadIdx.x == 0) {
          int r = min(npan, ld_acquire(tdone + a));
          if (!same && !j.L) r = min(r, ld_acquire(tdone + b));
          sReady = ok ? r : -1;
          if (trace) tReady = globaltimer_ns();
        }
      }
      __syncthreads();
      const int r = sReady;
      if (r < 0) return;
      const int kEnd = bnd(r);
      int k0 = bnd(q), pe = bnd(q + 1), st = 0;   // pe: end of the current panel
      T acc[R][R];
#pragma unroll
      for (int x = 0; x < R; ++x)
#pragma unroll
        for (int y = 0; y < R; ++y) acc[x][y] = T(0);
      if (std::is_same<T, float>::value && same && r == q + 1 && pe - k0 == NB) {
        // one panel of a diagonal tile -- the chain's last: both slices in one round of loads
#pragma unroll
        for (int e = 0; e < C::Q; ++e) {
          const int i = C::row(e), k = k0 + C::col(e);
          ra[e] = i < m ? __ldcg(Ap + (size_t)i * ld + k) : T(0);
          rb[e] = i < m ? __ldcg(Ap + (size_t)i * ld + k + 32) : T(0);
        }
#pragma unroll
        for (int e = 0; e < C::Q; ++e) {
          C::at(As[0], C::row(e), C::col(e)) = ra[e];
          C::at(As[1], C::row(e), C::col(e)) = rb[e];
        }
        __syncthreads();
        C::mul(As[0], As[0], 32, acc, w01, w10, w11);
        C::mul(As[1], As[1], 32, acc, w01, w10, w11);
#pragma unroll
        for (int x = 0; x < R; ++x)
#pragma unroll
          for (int y = 0; y < R; ++y) c[x][y] -= acc[x][y];
        __syncthreads();
        q = r;
        continue;
      }
      load(k0, min(k0 + 32, pe));
      store(0);
      __syncthreads();
      while (true) {
        const int k1 = min(k0 + 32, pe);
        const bool last = k1 == pe, more = k1 < kEnd;
        const int peNext = last ? pe + NB : pe;
        if (more) load(k1, min(k1 + 32, peNext));
        C::mul(As[st], same ? As[st] : Bs[st], k1 - k0, acc, w01, w10, w11);
        if (last)
#pragma unroll
          for (int x = 0; x < R; ++x)
#pragma unroll
            for (int y = 0; y < R; ++y) {
              c[x][y] -= acc[x][y];
              acc[x][y] = T(0);
            }
        if (more) store(st ^ 1);
        __syncthreads();
        if (!more) break;
        k0 = k1;
        pe = peNext;
        st ^= 1;
      }
      q = r;
    }
    if (it.kind == CHOL_POTRF) {
      T* out = ws + j.inv + (size_t)b * NB * NB;
      const bool below = q0 + n < j.nRows;   // rows below: the TRSM items multiply by the inverse
      constexpr int PITCH = std::is_same<T, double>::value ? 33 : 68;
      T (*S)[PITCH] = reinterpret_cast<T (*)[PITCH]>(cf_smem);
      T (*Li)[PITCH] = S + NB;
#pragma unroll
      for (int x = 0; x < R; ++x)
#pragma unroll
        for (int y = 0; y < R; ++y) {
          const int i = C::ti(x), k = C::tj(y);
          S[i][k] = (k <= i && i < n) ? c[x][y] : (i == k ? T(1) : T(0));
        }
      __syncthreads();
      if constexpr (std::is_same<T, double>::value)
        potrf_inverse_f64(S, Li, reinterpret_cast<T (*)[17]>(Li + NB), n, below, j.code, flag);
      else potrf_inverse_f32(S, Li, reinterpret_cast<T (*)[16][17]>(Li + NB), n, below, j.code, flag);
      __syncthreads();
      if (below) {   // published before the tile itself, which no item of this launch reads
#pragma unroll
        for (int idx = threadIdx.x; idx < NB * NB; idx += 256) {
          const int i = idx / NB, k = idx % NB;
          out[idx] = k <= i && i < n ? Li[i][k] : T(0);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          __threadfence();
          st_release(pdone + b, 1);
        }
      }
#pragma unroll
      for (int idx = threadIdx.x; idx < NB * NB; idx += 256) {
        const int i = idx / NB, k = idx % NB;
        if (k <= i && i < n) F[(size_t)(r0 + i) * ld + q0 + k] = tile_entry(S, i, k);
      }
    } else if (it.kind == CHOL_TRSM) {   // X := C Li(b)^T, the inverse tile from the workspace
#pragma unroll
      for (int x = 0; x < R; ++x)
#pragma unroll
        for (int y = 0; y < R; ++y) {
          const int k = C::tj(y);   // C as the A operand: its columns are the k of the product
          C::at(As[k >> 5], C::ti(x), k & 31) = k < n ? c[x][y] : T(0);
        }
      if (warp == 0) {
        const bool ok = wait_geq_lim(pdone + b, 1, err, lim);
        if (threadIdx.x == 0) {
          sReady = ok;
          if (trace) tReady = globaltimer_ns();
        }
      }
      __syncthreads();
      if (!sReady) return;
      const T* Li = ws + j.inv + (size_t)b * NB * NB;
      T acc[R][R], rl[NB / 32][C::Q];
#pragma unroll
      for (int h = 0; h < NB / 32; ++h)
#pragma unroll
        for (int q = 0; q < C::Q; ++q) rl[h][q] = __ldcg(Li + C::row(q) * NB + 32 * h + C::col(q));
#pragma unroll
      for (int h = 0; h < NB / 32; ++h)
#pragma unroll
        for (int q = 0; q < C::Q; ++q) C::at(Bs[h], C::row(q), C::col(q)) = rl[h][q];
#pragma unroll
      for (int x = 0; x < R; ++x)
#pragma unroll
        for (int y = 0; y < R; ++y) acc[x][y] = T(0);
      __syncthreads();
      if constexpr (std::is_same<T, double>::value) {
        C::mul(As[0], Bs[0], n, acc, n > 16, m > 16, m > 16 && n > 16, 16);   // the inverse is lower triangular
      } else {
        C::mul(As[0], Bs[0], min(32, n), acc, true, true, true);
        if (n > 32) C::mul(As[1], Bs[1], n - 32, acc, true, true, true);
      }
#pragma unroll
      for (int x = 0; x < R; ++x)
#pragma unroll
        for (int y = 0; y < R; ++y) {
          const int i = C::ti(x), k = C::tj(y);
          if (i < m && k < n) F[(size_t)(r0 + i) * ld + q0 + k] = acc[x][y];
        }
      done = tdone + a;
      doneVal = b + 1;
    } else {   // a tile of the trailing block
#pragma unroll
      for (int x = 0; x < R; ++x)
#pragma unroll
        for (int y = 0; y < R; ++y) {
          const int i = C::ti(x), k = C::tj(y);
          if (i < m && k < n && (!same || k <= i)) F[(size_t)(r0 + i) * ld + q0 + k] = c[x][y];
        }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (done) {
      __threadfence();
      st_release(done, doneVal);
    }
    if (trace) {   // diagnostics: when the item started, was ready, ended (ns), and its SM
      unsigned long long* r = trace + 4 * (size_t)sTicket;
      r[0] = tStart;
      r[1] = tReady;
      r[2] = globaltimer_ns();
      r[3] = smid();
    }
  }
}

template <class T>
__global__ void __launch_bounds__(256) extadd_kernel(const ExtAddRow<T>* __restrict__ rows, int nRows,
                                                     const ExtAddSeg* __restrict__ segs,
                                                     const ExtAddSource<T>* __restrict__ src) {
  const int lane = threadIdx.x & 31;
  const int rw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (rw >= nRows) return;
  const ExtAddRow<T> R = rows[rw];
  for (int g = R.segBegin; g < R.segEnd; ++g) {
    const ExtAddSeg sg = segs[g];
    const ExtAddSource<T>& S = src[sg.src];
    const T* drow = S.D + (size_t)sg.a * S.ld;
    const int b1 = min(S.b1, sg.a + 1);
    for (int b = S.b0 + lane; b < b1; b += 32) {
      T* dst = R.Frow + S.rowRel[b];
      *dst = fma(S.sign, drow[b], *dst);
    }
    __syncwarp();   // the next source may hit the same target entries
  }
}

template <class T>
__global__ void scatter_kernel(const double* __restrict__ Avals, const long long* __restrict__ srcIdx,
                               const long long* __restrict__ dstIdx, long long count, T* __restrict__ dst) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < count;
       k += (long long)gridDim.x * blockDim.x)
    dst[dstIdx[k]] = (T)Avals[srcIdx[k]];
}

// ---------------------------------------------------------------------------
// Blocked Householder QR of the sketches (LAPACK dgeqrf + dorgqr: dlarfg
// reflectors with v_0 = 1, compact-WY panels of QR_PB columns, dlarft's
// forward column-wise T).  Per panel: one block per matrix factors the panel
// (in shared memory when it fits), then many blocks apply the panel's block
// reflector to the trailing columns.  Q = H_0 ... H_{r-1} [I; 0] is formed by
// applying the block reflectors to [I; 0] in reverse order.
constexpr int QR_PB = 16;          // panel width
constexpr int QRP_THREADS = 512;   // panel kernel
constexpr int QA_ROWS = 64;        // apply kernel: row chunk
constexpr int QA_CW = 16;          // apply kernel: columns per block
constexpr int QR_SMEM_MAX = 200 * 1024;

template <class R>
__device__ __forceinline__ R warp_sum_d(R v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of v[0..15] over the 32 lanes of a warp; lane l (l < 16) returns the
// total of v[l] (31 shuffles, fixed order).
template <class R>
__device__ __forceinline__ R warp_transpose_sum16(R (&v)[QR_PB]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 16);
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1) {
    const bool up = (lane & w) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const R send = up ? v[i] : v[i + w];
      const R keep = up ? v[i + w] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return v[0];
}

// Y (row-major n x r) -> W (column-major, ld n), 32 x 32 tiles.
template <class T>
__global__ void __launch_bounds__(256) qr_to_colmajor(const QrTask<T>* __restrict__ tasks) {
  __shared__ T tile[32][33];
  const QrTask<T> t = tasks[blockIdx.y];
  const int n = t.n, r = t.r;
  const int tr = (n + 31) / 32, tc = (r + 31) / 32;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  for (int tl = blockIdx.x; tl < tr * tc; tl += gridDim.x) {
    const int i0 = (tl / tc) * 32, j0 = (tl % tc) * 32;
    for (int y = ly; y < 32; y += 8)
      if (i0 + y < n && j0 + lx < r) tile[y][lx] = t.Y[(size_t)(i0 + y) * r + j0 + lx];
    __syncthreads();
    for (int y = ly; y < 32; y += 8)
      if (j0 + y < r && i0 + lx < n) t.W[(size_t)(j0 + y) * n + i0 + lx] = tile[lx][y];
    __syncthreads();
  }
}

// Y (row-major n x r) := [I; 0]
template <class T>
__global__ void qr_set_e(const QrTask<T>* __restrict__ tasks) {
  const QrTask<T> t = tasks[blockIdx.y];
  const long long tot = (long long)t.n * t.r;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < tot; k += (long long)gridDim.x * blockDim.x) {
    const long long i = k / t.r, j = k - i * t.r;
    t.Y[k] = (i == j) ? T(1) : T(0);
  }
}

// Factor columns j0 .. j0+pw-1 of W (rows j0 .. n-1).  On return the panel
// holds V below its diagonal and T (pw x pw, upper) in place of the upper
// triangle of its diagonal block (R is not needed: only Q is used).
template <class T>
__global__ void __launch_bounds__(QRP_THREADS) qr_panel_kernel(const QrTask<T>* __restrict__ tasks, int j0,
                                                               long long smemElems) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int NW = QRP_THREADS / 32;
  __shared__ T redA[NW];
  __shared__ T redC[NW][QR_PB];
  __shared__ T sred[QR_PB], sfin[QR_PB];
  __shared__ T Ts[QR_PB][QR_PB + 1];
  const QrTask<T> t = tasks[blockIdx.x];
  const int n = t.n, r = t.r;
  if (j0 >= r) return;
  const int pw = min(QR_PB, r - j0), nr = n - j0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T* Wg = t.W + (size_t)j0 * n + j0;   // panel element (i, c) at Wg[c * n + i]
  T* P = Wg;
  long long lp = n;
  const bool inSmem = (long long)nr * pw <= smemElems;
  if (inSmem) {   // a thread's loads of all panel columns in flight at once
    P = reinterpret_cast<T*>(smraw);
    lp = nr;
    for (int i = tid; i < nr; i += QRP_THREADS) {
      T tmp[QR_PB];
#pragma unroll
      for (int c = 0; c < QR_PB; ++c)
        if (c < pw) tmp[c] = Wg[(size_t)c * n + i];
#pragma unroll
      for (int c = 0; c < QR_PB; ++c)
        if (c < pw) P[c * lp + i] = tmp[c];
    }
  }
  for (int idx = tid; idx < QR_PB * (QR_PB + 1); idx += QRP_THREADS) (&Ts[0][0])[idx] = T(0);
  __syncthreads();
  for (int kk = 0; kk < pw; ++kk) {
    T* pk = P + kk * lp;
    // dlarfg on column kk
    T x2 = T(0);
    for (int i = kk + 1 + tid; i < nr; i += QRP_THREADS) x2 += pk[i] * pk[i];
    x2 = warp_sum_d(x2);
    if (lane == 0) redA[warp] = x2;
    __syncthreads();
    x2 = T(0);
#pragma unroll
    for (int q = 0; q < NW; ++q) x2 += redA[q];
    const T alpha = pk[kk];
    T tau = T(0), scal = T(1);
    if (x2 > T(0)) {
      const T beta = -copysign(sqrt(alpha * alpha + x2), alpha);
      tau = (beta - alpha) / beta;
      scal = T(1) / (alpha - beta);
      for (int i = kk + 1 + tid; i < nr; i += QRP_THREADS) pk[i] *= scal;
    }
    // s_c = P[kk][c] + sum_{i>kk} v_i P[i][c] for every panel column c
    T part[QR_PB];
#pragma unroll
    for (int c = 0; c < QR_PB; ++c) part[c] = T(0);
    for (int i = kk + 1 + tid; i < nr; i += QRP_THREADS) {
      const T vi = pk[i];
#pragma unroll
      for (int c = 0; c < QR_PB; ++c)
        if (c < pw) part[c] += P[c * lp + i] * vi;
    }
    const T ws = warp_transpose_sum16(part);
    if (lane < QR_PB) redC[warp][lane] = ws;
    __syncthreads();
    if (tid < pw) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < NW; ++q) s += redC[q][tid];
      sred[tid] = s + P[tid * lp + kk];
    }
    __syncthreads();
    // T column kk (dlarft): T[p][kk] = -tau sum_{q=p}^{kk-1} T[p][q] y_q, T[kk][kk] = tau
    if (tid < kk) {
      T s = T(0);
      for (int q = tid; q < kk; ++q) s += Ts[tid][q] * sred[q];
      Ts[tid][kk] = -tau * s;
    }
    if (tid == kk) Ts[kk][kk] = tau;
    if (tid < pw) sfin[tid] = tau * sred[tid];
    __syncthreads();
    // apply H_kk to the remaining panel columns
    if (tau != T(0)) {
      for (int c = kk + 1; c < pw; ++c) {
        const T w = sfin[c];
        T* pc = P + c * lp;
        for (int i = kk + 1 + tid; i < nr; i += QRP_THREADS) pc[i] -= w * pk[i];
        if (tid == 0) pc[kk] -= w;
      }
    }
    __syncthreads();
  }
  if (inSmem)
    for (int c = 0; c < pw; ++c)
      for (int i = tid; i < nr; i += QRP_THREADS) Wg[(size_t)c * n + i] = P[c * lp + i];
  __syncthreads();
  // T over the upper triangle of the diagonal block
  for (int idx = tid; idx < pw * pw; idx += QRP_THREADS) {
    const int a = idx / pw, b = idx - a * pw;
    if (a <= b) Wg[(size_t)b * n + a] = Ts[a][b];
  }
}

// The same panel factorisation with the panel in registers (FP32, at most
// 512 rows): thread t keeps row t of the 16 panel columns, so a column step touches shared memory only for its three block
// reductions (|x|^2 below the diagonal with row kk, the 16 dot products
// s_c = v^T P[:, c], the T column) -- three barriers per column.  Reflectors,
// T factor and layout as qr_panel_kernel (the sums run in another fixed order).
__global__ void __launch_bounds__(QRP_THREADS, 1) qr_panel_reg_kernel(const QrTask<float>* __restrict__ tasks,
                                                                      int j0) {
  constexpr int NW = QRP_THREADS / 32;
  __shared__ float redA[2][NW];
  __shared__ float redC[NW][QR_PB];
  __shared__ float rowk[QR_PB], sred[QR_PB];
  __shared__ float Ts[QR_PB][QR_PB + 1];
  const QrTask<float> t = tasks[blockIdx.x];
  const int n = t.n, r = t.r;
  if (j0 >= r) return;
  const int pw = min(QR_PB, r - j0), nr = n - j0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* Wg = t.W + (size_t)j0 * n + j0;   // panel element (i, c) at Wg[c * n + i]
  float a[QR_PB];
#pragma unroll
  for (int c = 0; c < QR_PB; ++c) a[c] = (tid < nr && c < pw) ? Wg[(size_t)c * n + tid] : 0.f;
  for (int idx = tid; idx < QR_PB * (QR_PB + 1); idx += QRP_THREADS) (&Ts[0][0])[idx] = 0.f;
  if (tid < QR_PB) sred[tid] = 0.f;   // columns beyond pw keep s = 0
#pragma unroll
  for (int kk = 0; kk < QR_PB; ++kk) {
    if (kk >= pw) break;
    // |x|^2 below the diagonal; row kk published (alpha and the unit row of the reflector)
    const bool below = tid > kk && tid < nr;
    float x2 = warp_sum_d(below ? a[kk] * a[kk] : 0.f);
    if (lane == 0) redA[kk & 1][warp] = x2;
    if (tid == kk)
#pragma unroll
      for (int c = 0; c < QR_PB; ++c) rowk[c] = a[c];
    __syncthreads();
    x2 = 0.f;
#pragma unroll
    for (int q = 0; q < NW; ++q) x2 += redA[kk & 1][q];
    const float alpha = rowk[kk];
    float tau = 0.f, scal = 1.f;
    if (x2 > 0.f) {
      const float beta = -copysignf(sqrtf(alpha * alpha + x2), alpha);
      tau = (beta - alpha) / beta;
      scal = 1.f / (alpha - beta);
    }
    const float v = below ? a[kk] * scal : 0.f;
    if (below) a[kk] = v;
    // s_c = P[kk][c] + sum_{i > kk} v_i P[i][c]
    float part[QR_PB];
#pragma unroll
    for (int c = 0; c < QR_PB; ++c) part[c] = v * a[c];
    const float ws = warp_transpose_sum16(part);
    if (lane < QR_PB) redC[warp][lane] = ws;
    __syncthreads();
    if (tid < pw) {
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < NW; ++q) sum += redC[q][tid];
      sred[tid] = sum + rowk[tid];
    }
    __syncthreads();
    // T column kk (dlarft): T[p][kk] = -tau sum_{q=p}^{kk-1} T[p][q] s_q, T[kk][kk] = tau
    if (tid < kk) {
      float sum = 0.f;
      for (int q = tid; q < kk; ++q) sum += Ts[tid][q] * sred[q];
      Ts[tid][kk] = -tau * sum;
    }
    if (tid == kk) Ts[kk][kk] = tau;
    // apply H_kk to the columns right of kk
    if (tau != 0.f) {
#pragma unroll
      for (int c = kk + 1; c < QR_PB; ++c) {
        const float w = tau * sred[c];
        a[c] -= w * v;
        if (tid == kk) a[c] -= w;
      }
    }
  }
  if (tid < nr)
#pragma unroll
    for (int c = 0; c < QR_PB; ++c)
      if (c < pw) Wg[(size_t)c * n + tid] = a[c];
  __syncthreads();
  // T over the upper triangle of the diagonal block
  for (int idx = tid; idx < pw * pw; idx += QRP_THREADS) {
    const int ra = idx / pw, cb = idx - ra * pw;
    if (ra <= cb) Wg[(size_t)cb * n + ra] = Ts[ra][cb];
  }
}

// The panel factorisation over a cluster of eight blocks, the panel's rows split
// between them in registers (thread t of block b: rows b rp + t + 256 q, q < R).
// One exchange a column: with x = column kk below the diagonal, the 16 products
// S_c = x^T P[:, c] give |x|^2 = S_kk and v^T P[:, c] = scal S_c + P[kk][c], so a
// column is one local reduction, one store of 16 partials into every block's
// shared memory, one cluster barrier, and the scalars (a square root, two
// divisions) by one warp.  Reflectors, T factor and layout as qr_panel_kernel.
// For FP64, whose adds and divisions run at 1/64 of the FP32 rate (every one of
// 512 threads forming the scalars and 16-term sums held the SM: QR steps of 3D
// 37x41x35 4.6 -> 1.7 ms), and for FP32 panels of more than 512 rows (those above
// 2048 went through shared memory or L2: 3D 96^3 24.7 -> 9.0 ms).
constexpr int QC = 8, QC_THREADS = 256;   // blocks of a cluster, threads of a block
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
template <class T>
__device__ __forceinline__ void st_cluster(T* local, unsigned rank, T v) {
  unsigned a = (unsigned)__cvta_generic_to_shared(local), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  if constexpr (sizeof(T) == 8) asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"((double)v) : "memory");
  else asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(r), "f"((float)v) : "memory");
}

template <class T, int R>
__global__ void __cluster_dims__(QC, 1, 1) __launch_bounds__(QC_THREADS)
    qr_panel_cluster_kernel(const QrTask<T>* __restrict__ tasks, int j0) {
  constexpr int NW = QC_THREADS / 32;
  __shared__ T wsum[NW][QR_PB];
  __shared__ T parts[2][QC][QR_PB], rowk[2][QR_PB];   // written by every block of the cluster / by block 0
  __shared__ T own[QR_PB], wv[QR_PB], sc[2];
  __shared__ T Ts[QR_PB][QR_PB + 1];
  const unsigned rank = blockIdx.x % QC;
  const QrTask<T> t = tasks[blockIdx.x / QC];
  const int n = t.n, r = t.r;
  if (j0 >= r) return;   // (every block of the cluster)
  const int pw = min(QR_PB, r - j0), nr = n - j0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rp = max(QR_PB, (nr + QC - 1) / QC), row0 = (int)rank * rp;   // <= QC_THREADS R rows a block
  const int rows = max(0, min(rp, nr - row0));
  const int nw = min(NW, (rows + 31) >> 5);   // warps that hold rows
  T* Wg = t.W + (size_t)j0 * n + j0;          // panel element (i, c) at Wg[c * n + i]
  T a[R][QR_PB];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int l = tid + QC_THREADS * q;
#pragma unroll
    for (int c = 0; c < QR_PB; ++c) a[q][c] = (l < rows && c < pw) ? Wg[(size_t)c * n + row0 + l] : T(0);
  }
  for (int idx = tid; idx < QR_PB * (QR_PB + 1); idx += QC_THREADS) (&Ts[0][0])[idx] = T(0);
  cluster_sync_all();   // every block runs before its shared memory is written
#pragma unroll
  for (int kk = 0; kk < QR_PB; ++kk) {
    if (kk >= pw) break;
    const int buf = kk & 1;
    if (warp < nw) {
      T part[QR_PB];
#pragma unroll
      for (int c = 0; c < QR_PB; ++c) part[c] = T(0);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int l = tid + QC_THREADS * q;
        const T x = (l < rows && row0 + l > kk) ? a[q][kk] : T(0);
#pragma unroll
        for (int c = 0; c < QR_PB; ++c) part[c] += x * a[q][c];
      }
      const T s = warp_transpose_sum16(part);
      if (lane < QR_PB) wsum[warp][lane] = s;
    }
    if (rank == 0 && tid == kk)
#pragma unroll
      for (int c = 0; c < QR_PB; ++c) own[c] = a[0][c];
    __syncthreads();
    if (tid < QC * QR_PB) {   // a thread per (block, column)
      const int c = tid % QR_PB;
      T s = T(0);
      for (int w = 0; w < nw; ++w) s += wsum[w][c];
      st_cluster(&parts[buf][rank][c], (unsigned)(tid / QR_PB), s);
      if (rank == 0) st_cluster(&rowk[buf][c], (unsigned)(tid / QR_PB), own[c]);
    }
    cluster_sync_all();
    if (warp == 0) {
      const int c = lane % QR_PB;
      T s = T(0);
#pragma unroll
      for (int b = 0; b < QC; ++b) s += parts[buf][b][c];
      const T x2 = __shfl_sync(0xffffffffu, s, kk), alpha = rowk[buf][kk];
      T tau = T(0), scal = T(1);
      if (x2 > T(0)) {
        const T beta = -copysign(sqrt(alpha * alpha + x2), alpha);
        tau = (beta - alpha) / beta;
        scal = T(1) / (alpha - beta);
      }
      const T y = scal * s + rowk[buf][c];   // v^T P[:, c]
      if (lane < QR_PB) wv[c] = tau * y;
      if (lane == 0) sc[buf] = scal;
      if (rank == 0) {   // T column kk (dlarft): T[p][kk] = -tau sum_{q=p}^{kk-1} T[p][q] y_q
        T sum = T(0);
        for (int q = 0; q < kk; ++q) {
          const T yq = __shfl_sync(0xffffffffu, y, q);
          if (lane < kk && q >= lane) sum += Ts[lane][q] * yq;
        }
        __syncwarp();
        if (lane < kk) Ts[lane][kk] = -tau * sum;
        if (lane == kk) Ts[kk][kk] = tau;
      }
    }
    __syncthreads();
    if (warp < nw) {   // v = scal x; the columns right of kk
      const T scal = sc[buf];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int l = tid + QC_THREADS * q;
        if (l < rows && row0 + l > kk) {
          const T v = a[q][kk] * scal;
          a[q][kk] = v;
#pragma unroll
          for (int c = kk + 1; c < QR_PB; ++c) a[q][c] -= wv[c] * v;
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int l = tid + QC_THREADS * q;
    if (l < rows)
#pragma unroll
      for (int c = 0; c < QR_PB; ++c)   // (T over the upper triangle of the diagonal block)
        if (c < pw) Wg[(size_t)c * n + row0 + l] = row0 + l <= c ? Ts[row0 + l][c] : a[q][c];
  }
}

// Apply the block reflector of panel j0 to the other columns, in parallel
// over (row block of QA_RB rows, group of QA_CW columns):
//   mode 0 (factor): W[j0:n, c] := (I - V T^T V^T) W[j0:n, c], c >= j0 + pw
//   mode 1 (form Q): Y[j0:n, c] := (I - V T V^T) Y[j0:n, c],   c >= j0
// in two launches: Zpart = V^T A per row block; then per row block Z = the
// row-block partials added in order, M = T^T Z (or T Z), A -= V M (every block
// of a column group forms the same small M instead of a launch of its own).
// ws holds Zpart (tasks x cgMax x rbMax x 16 x 16).
// Rows per block of the apply: one 64-row chunk, so a QR of few tall panels
// still spreads over many blocks (c2 factor 21.65 ms at 64 rows, 22.00 at
// 128, 22.85 at 256, 24.51 at 512).
constexpr int QA_RB = 64;

template <class T>
struct QrApplyView {
  const T* V;   // panel reflectors, column-major (ld n), V[p][i] at V[p * n + i], unit diagonal implied
  T* A;
  int n, r, nr, pw, c0, cw;
  int mode;
  __device__ size_t aidx(int j0, int i, int c) const {
    return mode == 0 ? (size_t)(c0 + c) * n + j0 + i : (size_t)(j0 + i) * r + c0 + c;
  }
  __device__ T v(int i, int p) const {   // reflector p at panel row i (i counted from j0)
    if (p >= pw) return T(0);
    return i == p ? T(1) : (i > p ? V[(size_t)p * n + i] : T(0));
  }
};

template <class T>
__device__ __forceinline__ bool qr_view(const QrTask<T>& t, int j0, int mode, int cg, QrApplyView<T>& w) {
  const int n = t.n, r = t.r;
  if (j0 >= r) return false;
  w.n = n;
  w.r = r;
  w.pw = min(QR_PB, r - j0);
  w.nr = n - j0;
  w.mode = mode;
  w.c0 = (mode == 0 ? j0 + w.pw : j0) + cg * QA_CW;
  if (w.c0 >= r) return false;
  w.cw = min(QA_CW, r - w.c0);
  w.V = t.W + (size_t)j0 * n + j0;
  w.A = mode == 0 ? t.W : t.Y;
  return true;
}

template <class T>
__global__ void __launch_bounds__(256) qr_zpart_kernel(const QrTask<T>* __restrict__ tasks, int j0, int mode,
                                                       T* __restrict__ ws, int cgMax, int rbMax) {
  __shared__ T Vs[QA_ROWS][QR_PB + 1];
  __shared__ T As[QA_ROWS][QA_CW + 1];
  const QrTask<T> t = tasks[blockIdx.y];
  const int cg = blockIdx.x % cgMax, rb = blockIdx.x / cgMax;
  QrApplyView<T> w;
  if (!qr_view(t, j0, mode, cg, w)) return;
  const int r0 = rb * QA_RB;
  if (r0 >= w.nr) return;
  const int r1 = min(w.nr, r0 + QA_RB);
  const int tid = threadIdx.x, zp = tid % QR_PB, zc = tid / QR_PB;
  T z = T(0);
  for (int i0 = r0; i0 < r1; i0 += QA_ROWS) {
    const int h = min(QA_ROWS, r1 - i0);
    for (int idx = tid; idx < QA_ROWS * QR_PB; idx += blockDim.x) {
      const int p = idx / QA_ROWS, i = idx - p * QA_ROWS;
      Vs[i][p] = i < h ? w.v(i0 + i, p) : T(0);
    }
    for (int idx = tid; idx < QA_ROWS * QA_CW; idx += blockDim.x) {
      int i, c;
      if (mode == 0) { c = idx / QA_ROWS; i = idx - c * QA_ROWS; }
      else { i = idx / QA_CW; c = idx - i * QA_CW; }
      As[i][c] = (i < h && c < w.cw) ? w.A[w.aidx(j0, i0 + i, c)] : T(0);
    }
    __syncthreads();
#pragma unroll 8
    for (int i = 0; i < QA_ROWS; ++i) z += Vs[i][zp] * As[i][zc];
    __syncthreads();
  }
  ws[(((size_t)blockIdx.y * cgMax + cg) * rbMax + rb) * (QR_PB * QA_CW) + zp * QA_CW + zc] = z;
}

template <class T>
__global__ void __launch_bounds__(256) qr_update_kernel(const QrTask<T>* __restrict__ tasks, int j0, int mode,
                                                        const T* __restrict__ ws, int cgMax, int rbMax) {
  __shared__ T Vs[QA_ROWS][QR_PB + 1];
  __shared__ T As[QA_ROWS][QA_CW + 1];
  __shared__ T M[QR_PB][QA_CW + 1];
  __shared__ T Z[QR_PB][QA_CW + 1];
  __shared__ T Ts[QR_PB][QR_PB + 1];
  const QrTask<T> t = tasks[blockIdx.y];
  const int cg = blockIdx.x % cgMax, rb = blockIdx.x / cgMax;
  QrApplyView<T> w;
  if (!qr_view(t, j0, mode, cg, w)) return;
  const int r0 = rb * QA_RB;
  if (r0 >= w.nr) return;
  const int r1 = min(w.nr, r0 + QA_RB);
  const int tid = threadIdx.x;
  {
    // M = T^T Z (mode 0) or T Z (mode 1), Z = V^T A summed over the row blocks'
    // partials in row-block order: every block of the column group forms the
    // same M (a 16 x 16 reduction, cheaper than a launch of its own)
    const int zp = tid % QR_PB, zc = tid / QR_PB;
    const int a = tid / QR_PB, b = tid - a * QR_PB;   // T over the upper triangle of the diagonal block
    Ts[a][b] = (a <= b && b < w.pw) ? w.V[(size_t)b * w.n + a] : T(0);
    const int nrb = (w.nr + QA_RB - 1) / QA_RB;
    const T* zpart = ws + ((size_t)blockIdx.y * cgMax + cg) * rbMax * (QR_PB * QA_CW) + zp * QA_CW + zc;
    T z = T(0);
    for (int q = 0; q < nrb; ++q) z += zpart[(size_t)q * (QR_PB * QA_CW)];
    Z[zp][zc] = z;
    __syncthreads();
    T m = T(0);
    if (mode == 0) {
      for (int q = 0; q <= zp; ++q) m += Ts[q][zp] * Z[q][zc];   // T^T Z
    } else {
      for (int q = zp; q < QR_PB; ++q) m += Ts[zp][q] * Z[q][zc];   // T Z
    }
    M[zp][zc] = m;
  }
  const int ai = tid % QA_ROWS, aq = (tid / QA_ROWS) * 4;
  for (int i0 = r0; i0 < r1; i0 += QA_ROWS) {
    const int h = min(QA_ROWS, r1 - i0);
    for (int idx = tid; idx < QA_ROWS * QR_PB; idx += blockDim.x) {
      const int p = idx / QA_ROWS, i = idx - p * QA_ROWS;
      Vs[i][p] = i < h ? w.v(i0 + i, p) : T(0);
    }
    for (int idx = tid; idx < QA_ROWS * QA_CW; idx += blockDim.x) {
      int i, c;
      if (mode == 0) { c = idx / QA_ROWS; i = idx - c * QA_ROWS; }
      else { i = idx / QA_CW; c = idx - i * QA_CW; }
      As[i][c] = (i < h && c < w.cw) ? w.A[w.aidx(j0, i0 + i, c)] : T(0);
    }
    __syncthreads();
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      T s = T(0);
#pragma unroll
      for (int p = 0; p < QR_PB; ++p) s += Vs[ai][p] * M[p][aq + cc];
      As[ai][aq + cc] -= s;
    }
    __syncthreads();
    for (int idx = tid; idx < QA_ROWS * QA_CW; idx += blockDim.x) {
      int i, c;
      if (mode == 0) { c = idx / QA_ROWS; i = idx - c * QA_ROWS; }
      else { i = idx / QA_CW; c = idx - i * QA_CW; }
      if (i < h && c < w.cw) w.A[w.aidx(j0, i0 + i, c)] = As[i][c];
    }
    __syncthreads();
  }
}

template <class T>
__global__ void set_identity_kernel(const IdentTask<T>* __restrict__ tasks) {
  const IdentTask<T> t = tasks[blockIdx.y];
  T* U = t.U;
  const int n = t.n, ld = t.ld;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < (long long)n * n;
       k += (long long)gridDim.x * blockDim.x) {
    int i = (int)(k / n), j = (int)(k - (long long)i * n);
    U[(size_t)i * ld + j] = (i == j) ? T(1) : T(0);
  }
}

template <class T>
__global__ void box_muller_kernel(const uint32_t* __restrict__ raw, long long count, T* __restrict__ out) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < count;
       k += (long long)gridDim.x * blockDim.x) {
    const double u1 = ((double)raw[2 * k] + 0.5) * (1.0 / 4294967296.0);
    const double u2 = (double)raw[2 * k + 1] * (1.0 / 4294967296.0);
    const double r = sqrt(-2.0 * log(1.0 - u1));
    const double phi = 2.0 * 3.14159265358979323846264338328 * u2;
    out[k] = (T)(r * cos(phi));
  }
}

int grid_for(long long n, int threads) {
  long long g = (n + threads - 1) / threads;
  if (g > 152LL * 32) g = 152LL * 32;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

template <class T> void launch_gemm(const GemmTask<T>* d, int n, int tiles, cudaStream_t s) {
  if (n <= 0 || tiles <= 0) return;
  gemm_kernel<T><<<tiles, GEMM_THREADS, 0, s>>>(d, n);
  RSCHOL_LAUNCH_CHECK();
}
void launch_gemm_rows128(const GemmTask<float>* d, int n, int tiles, cudaStream_t s) {
  if (n <= 0 || tiles <= 0) return;
  gemm_rows128_kernel<<<tiles, GEMM_THREADS, 0, s>>>(d, n);
  RSCHOL_LAUNCH_CHECK();
}
void launch_gemm_splitk_reduce(const GemmTask<double>* d, const int* ids, int nIds, const long long* elemBase,
                               long long elems, cudaStream_t s) {
  if (nIds <= 0 || elems <= 0) return;
  gemm_splitk_reduce_f64<<<(unsigned)((elems + 255) / 256), 256, 0, s>>>(d, ids, nIds, elemBase);
  RSCHOL_LAUNCH_CHECK();
}
template <class T> void launch_potrf(const PotrfTask<T>* d, int n, int* flag, cudaStream_t s) {
  if (n <= 0) return;
  if constexpr (std::is_same<T, float>::value) potrf_reg_kernel<T><<<n, 256, 0, s>>>(d, flag);
  else potrf_kernel<T><<<n, 256, 0, s>>>(d, flag);
  RSCHOL_LAUNCH_CHECK();
}
template <class T> void launch_trsm(const TrsmTask<T>* d, int n, int chunks, cudaStream_t s) {
  if (n <= 0 || chunks <= 0) return;
  static std::once_flag once;   // per instantiation; callers may be on several threads
  if constexpr (std::is_same<T, float>::value) {
    const int smem = (int)(3 * sizeof(T) * 64 * 65 + 3 * sizeof(T) * 16 * 17);
    std::call_once(once, [&] {
      RSCHOL_CUDA(cudaFuncSetAttribute(trsm_inv_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    });
    trsm_inv_kernel<T><<<chunks, 256, smem, s>>>(d, n);
  } else {
    const int smem = (int)(2 * sizeof(T) * 64 * 65);
    std::call_once(once, [&] {
      RSCHOL_CUDA(cudaFuncSetAttribute(trsm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    });
    trsm_kernel<T><<<chunks, 256, smem, s>>>(d, n);
  }
  RSCHOL_LAUNCH_CHECK();
}
template <class T>
void launch_chol_fused(const CholFusedJob<T>* jobs, const CholItem* items, int nItems, int* sync, long long syncInts,
                       T* ws, int* flag, unsigned long long* trace, cudaStream_t s) {
  if (nItems <= 0) return;
  RSCHOL_CUDA(cudaMemsetAsync(sync, 0, sizeof(int) * (size_t)syncInts, s));
  const int smem = chol_smem<T>;
  static std::once_flag once;
  std::call_once(once, [&] {
    RSCHOL_CUDA(cudaFuncSetAttribute(chol_fused_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  });
  chol_fused_kernel<T><<<nItems, 256, smem, s>>>(jobs, items, nItems, sync, ws, flag, trace);
  RSCHOL_LAUNCH_CHECK();
}
template <class T>
void launch_extadd(const ExtAddRow<T>* rows, int nRows, const ExtAddSeg* segs, const ExtAddSource<T>* src,
                   cudaStream_t s) {
  if (nRows <= 0) return;
  extadd_kernel<T><<<(nRows + 7) / 8, 256, 0, s>>>(rows, nRows, segs, src);
  RSCHOL_LAUNCH_CHECK();
}
// a block of 256 threads per (task, 64-row slab)
__global__ void block_convert_kernel(const CvtTask* __restrict__ tasks, int toDouble) {
  const CvtTask t = tasks[blockIdx.y];
  const int r0 = blockIdx.x * 64;
  if (r0 >= t.n) return;
  const int r1 = min(t.n, r0 + 64);
  for (int i = r0 + (threadIdx.x >> 5); i < r1; i += 8)
    for (int j = threadIdx.x & 31; j <= i; j += 32) {
      if (toDouble) t.D[(size_t)i * t.ldd + j] = (double)t.F[(size_t)i * t.ld + j];
      else t.F[(size_t)i * t.ld + j] = (float)t.D[(size_t)i * t.ldd + j];
    }
}

void launch_block_convert(const CvtTask* d, int nTasks, int maxN, int toDouble, cudaStream_t s) {
  if (nTasks <= 0 || maxN <= 0) return;
  block_convert_kernel<<<dim3((maxN + 63) / 64, nTasks), 256, 0, s>>>(d, toDouble);
  RSCHOL_LAUNCH_CHECK();
}

__global__ void init_flags_kernel(int* flag, int waitLimit) {
  flag[0] = INT_MAX;
  flag[1] = 0;
  flag[2] = waitLimit;
}

void launch_init_flags(int* flag, int waitLimit, cudaStream_t s) {
  init_flags_kernel<<<1, 1, 0, s>>>(flag, waitLimit);
  RSCHOL_LAUNCH_CHECK();
}

template <class T>
void launch_scatter(const double* A, const long long* si, const long long* di, long long count, T* dst,
                    cudaStream_t s) {
  if (count <= 0) return;
  scatter_kernel<T><<<grid_for(count, 256), 256, 0, s>>>(A, si, di, count, dst);
  RSCHOL_LAUNCH_CHECK();
}
long long householder_qr_workspace(int nTasks, int maxRows, int maxR) {
  const long long cgMax = (maxR + QA_CW - 1) / QA_CW, rbMax = (maxRows + QA_RB - 1) / QA_RB;
  return (long long)nTasks * cgMax * rbMax * (QR_PB * QA_CW);
}

template <class T>
int launch_householder_qr(const QrTask<T>* d, int n, int maxRows, int maxR, T* ws, cudaStream_t s) {
  if (n <= 0 || maxR <= 0) return 0;
  const int cgMax = (maxR + QA_CW - 1) / QA_CW, rbMax = (maxRows + QA_RB - 1) / QA_RB;
  int launches = 0;
  auto apply = [&](int j0, int mode) {
    qr_zpart_kernel<T><<<dim3(cgMax * rbMax, n), 256, 0, s>>>(d, j0, mode, ws, cgMax, rbMax);
    qr_update_kernel<T><<<dim3(cgMax * rbMax, n), 256, 0, s>>>(d, j0, mode, ws, cgMax, rbMax);
    RSCHOL_LAUNCH_CHECK();
    launches += 2;
  };
  static std::once_flag once;
  std::call_once(once, [] {
    RSCHOL_CUDA(cudaFuncSetAttribute(qr_panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, QR_SMEM_MAX));
  });
  const long long tiles = (long long)((maxRows + 31) / 32) * ((maxR + 31) / 32);
  qr_to_colmajor<T><<<dim3((unsigned)std::min<long long>(tiles, 64), n), 256, 0, s>>>(d);
  RSCHOL_LAUNCH_CHECK();
  launches += 1;
  const size_t smem = std::min<size_t>((size_t)QR_SMEM_MAX, sizeof(T) * (size_t)maxRows * QR_PB);
  const long long smemElems = (long long)(smem / sizeof(T));
  const int panels = (maxR + QR_PB - 1) / QR_PB;
  for (int p = 0; p < panels; ++p) {
    const int j0 = p * QR_PB;
    if constexpr (std::is_same<T, float>::value) {
      // up to 512 rows one block's registers hold the panel and a column costs three
      // block barriers; above, a cluster's one exchange a column is quicker (3D 64^3,
      // up to 2048 rows: 2.50 against 2.64 ms of QR steps)
      if (maxRows <= QRP_THREADS) qr_panel_reg_kernel<<<n, QRP_THREADS, 0, s>>>(d, j0);
      else if (maxRows <= QC * QC_THREADS) qr_panel_cluster_kernel<T, 1><<<QC * n, QC_THREADS, 0, s>>>(d, j0);
      else if (maxRows <= 2 * QC * QC_THREADS) qr_panel_cluster_kernel<T, 2><<<QC * n, QC_THREADS, 0, s>>>(d, j0);
      else if (maxRows <= 4 * QC * QC_THREADS) qr_panel_cluster_kernel<T, 4><<<QC * n, QC_THREADS, 0, s>>>(d, j0);
      else qr_panel_kernel<T><<<n, QRP_THREADS, smem, s>>>(d, j0, smemElems);
    } else {   // what a cluster's registers hold, else the panel in shared or global memory
      if (maxRows <= QC * QC_THREADS) qr_panel_cluster_kernel<T, 1><<<QC * n, QC_THREADS, 0, s>>>(d, j0);
      else if (maxRows <= 2 * QC * QC_THREADS) qr_panel_cluster_kernel<T, 2><<<QC * n, QC_THREADS, 0, s>>>(d, j0);
      else qr_panel_kernel<T><<<n, QRP_THREADS, smem, s>>>(d, j0, smemElems);
    }
    RSCHOL_LAUNCH_CHECK();
    ++launches;
    if (maxR - j0 - QR_PB > 0) apply(j0, 0);
  }
  const long long ecount = (long long)maxRows * maxR;
  qr_set_e<T><<<dim3((unsigned)std::max<long long>(1, std::min<long long>((ecount + 255) / 256, 256)), n), 256, 0, s>>>(d);
  RSCHOL_LAUNCH_CHECK();
  ++launches;
  for (int p = panels - 1; p >= 0; --p) apply(p * QR_PB, 1);
  return launches;
}
template <class T> void launch_set_identity(const IdentTask<T>* d, int n, cudaStream_t s) {
  if (n <= 0) return;
  set_identity_kernel<T><<<dim3(64, n), 256, 0, s>>>(d);
  RSCHOL_LAUNCH_CHECK();
}
template <class T> void launch_box_muller(const uint32_t* raw, long long count, T* out, cudaStream_t s) {
  if (count <= 0) return;
  box_muller_kernel<T><<<grid_for(count, 256), 256, 0, s>>>(raw, count, out);
  RSCHOL_LAUNCH_CHECK();
}

#define RSCHOL_INST(T)                                                                                   \
  template void launch_gemm<T>(const GemmTask<T>*, int, int, cudaStream_t);                              \
  template void launch_potrf<T>(const PotrfTask<T>*, int, int*, cudaStream_t);                           \
  template void launch_trsm<T>(const TrsmTask<T>*, int, int, cudaStream_t);                              \
  template void launch_chol_fused<T>(const CholFusedJob<T>*, const CholItem*, int, int*, long long, T*, int*,  \
                                     unsigned long long*, cudaStream_t);                                 \
  template void launch_extadd<T>(const ExtAddRow<T>*, int, const ExtAddSeg*, const ExtAddSource<T>*,      \
                                 cudaStream_t);                                                          \
  template void launch_scatter<T>(const double*, const long long*, const long long*, long long, T*,      \
                                  cudaStream_t);                                                         \
  template int launch_householder_qr<T>(const QrTask<T>*, int, int, int, T*, cudaStream_t);                  \
  template void launch_set_identity<T>(const IdentTask<T>*, int, cudaStream_t);                          \
  template void launch_box_muller<T>(const uint32_t*, long long, T*, cudaStream_t);
RSCHOL_INST(double)
RSCHOL_INST(float)

}  // namespace rschol
