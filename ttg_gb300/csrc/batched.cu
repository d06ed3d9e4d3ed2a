// Batched Cholesky solves of many independent SPD matrices of uneven sizes in ONE persistent
// launch (no host round trip, capturable in a CUDA graph).
//
// Each CTA takes matrices from a device-side queue in the order the caller gives (largest first is
// the longest-processing-time schedule) and for each matrix runs, on 128 or 256 threads:
//   plain (FP64):  left-looking Cholesky by 64 x 64 blocks, then the forward/backward solve for its
//                  right-hand sides, all in place;
//   fp32 + IR:     an FP32 factor of the same form, FP32 solve, then `refine` steps of FP64 iterative
//                  refinement x += (L L^T)^{-1} (b - A x) with the residual in FP64.
// Up to four right-hand sides are solved at once.
// Matrix i is column-major n_i x n_i (leading dimension n_i) at A + offA[i] (only the lower
// triangle is read); its right-hand sides are column-major n_i x nrhs at B + offB[i] and are
// overwritten by the solution.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <numeric>
#include <type_traits>
#include <vector>

#include "block_ops.cuh"
#include "gbx_common.cuh"
#include "gbx_potrf.h"

namespace gbx {
namespace batched {

constexpr int kMaxN = 1024;  // largest matrix order of the batched kernel (shared-memory vectors)
// One matrix keeps one CTA busy in spurts (a chain of pivots, a block product, a chain of panel solves), so
// a CTA is small and four matrices share an SM; two with twice the warps when there are few (gbx_dposv_batched_ex).
// 4096 matrices of 32 .. 512 rows: FP64 90.2 -> 52.7 ms with one CTA of 256 threads per SM before (the FP64 pipe alone
// needs 46), FP32 and two refinements 14.4 -> 8.9 (two CTAs of 256).
constexpr int kPan = 64;            // largest block edge of the factorisation
constexpr int kCk = 8;              // k-chunk of the block products
// shared memory of the FP64 factorisation: the panel's triangle, two chunks of both operands, the last columns, one int
constexpr size_t kFactor64Smem = (size_t)(kPan * kPan + 4 * kCk * kPan + 256) * sizeof(double) + 16;

// ---- FP64 ---------------------------------------------------------------------------------------------------
// Blocks of the factorisation live in registers: thread (warp, lane) has rows lane + 32 h of columns
// kWarps q + warp, h < 2, q < kCols. They hold what is to be subtracted from A (u), not the difference: the sums of
// products are small beside the diagonal, so that A's large entries are rounded once, when a column is due. A
// column's entries of A are read when the column before it in the same warp is done.

// u += L(r0.., 0:p0) L(p0.., 0:p0)^T; mb, pb: rows and columns present. k in chunks through shared memory, the next
// chunk in registers; a thread's columns stand in a row in the second operand.
// NG: groups of 16 columns; kLow: rows 32.. exist; kDiag: a diagonal block, whose first 32 rows have no columns past 32.
// (Parameters of the loop, since an FP64 instruction that a predicate turns off takes its time on the pipe all the same.)
template <int W, int NG, bool kLow, bool kDiag>
__device__ __forceinline__ void panel_update(double (&u)[2][kPan / W], const double* L, int ld, int r0, int p0, int mb, int pb,
                                             double* sm) {
  using T = double;
  constexpr int kWarps = W, kThr = 32 * W, kCols = kPan / W;
  constexpr int CK = kCk, NL = CK * kPan / kThr, KS = kThr / kPan;  // loads per thread, chunk and operand; their step in k
  T* As = sm;                 // [2][CK][64]
  T* Bs = sm + 2 * CK * kPan;  // [2][CK][64], column c at (c % kWarps) kCols + c / kWarps
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = tid & 63, kk = tid >> 6;
  const T* Ap = L + r0 + (row < mb ? row : 0);
  const T* Bp = L + p0 + (row < pb ? row : 0);
  const int at = (row % kWarps) * kCols + row / kWarps;
  T va[NL], vb[NL];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const long long k = (long long)(k0 + kk + KS * i) * ld;  // p0 is a multiple of 64: whole chunks
      va[i] = Ap[k];
      vb[i] = Bp[k];
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      As[(buf * CK + kk + KS * i) * kPan + row] = va[i];
      Bs[(buf * CK + kk + KS * i) * kPan + at] = vb[i];
    }
  };
  load(0);
  store(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < p0; k0 += CK, buf ^= 1) {
    if (k0 + CK < p0) load(k0 + CK);
#pragma unroll
    for (int k = 0; k < CK; ++k) {
      const T* ar = As + (buf * CK + k) * kPan + lane;
      const T* br = Bs + (buf * CK + k) * kPan + kCols * warp;
      const T a0 = ar[0], a1 = kLow ? ar[32] : T(0);
#pragma unroll
      for (int e = 0; e < NG * 16 / W; e += 2) {
        const double2 b = *(const double2*)(br + e);
        if (!kDiag || kWarps * e < 32) {
          u[0][e] = fma(a0, b.x, u[0][e]);
          u[0][e + 1] = fma(a0, b.y, u[0][e + 1]);
        }
        if (kLow) {
          u[1][e] = fma(a1, b.x, u[1][e]);
          u[1][e + 1] = fma(a1, b.y, u[1][e + 1]);
        }
      }
    }
    if (k0 + CK < p0) store(buf ^ 1);
    __syncthreads();
  }
}

// The block's columns in turn: for q, jj (column j = kWarps q + jj < n, owned by warp jj) f(q, jj) with q a constant
template <int W, typename F>
__device__ __forceinline__ void each_column(int n, F f) {
  constexpr int kWarps = W, kCols = kPan / W;
  auto round = [&](auto qc) {
    constexpr int q = decltype(qc)::value;
#pragma unroll 1
    for (int jj = 0; jj < kWarps; ++jj)
      if (kWarps * q + jj >= n || !f(qc, jj)) return false;
    return true;
  };
#define GBX_R(Q) if (!round(std::integral_constant<int, Q>{})) return;
  static_assert(kCols == 16 || kCols == 8, "rounds");
  GBX_R(0) GBX_R(1) GBX_R(2) GBX_R(3) GBX_R(4) GBX_R(5) GBX_R(6) GBX_R(7)
  if constexpr (kCols == 16) { GBX_R(8) GBX_R(9) GBX_R(10) GBX_R(11) GBX_R(12) GBX_R(13) GBX_R(14) GBX_R(15) }
#undef GBX_R
}

// Cholesky of the n x n diagonal block A - u, in place and, its columns divided by the diagonal, into tri. One barrier a column; the warp that owns the next pivot takes it before anything
// else and applies the current column to its others together with its own (as chol64_regs). cb: three columns, then
// the pivots' reciprocals. Returns 0 or the 1-based index of the first bad pivot.
template <int W>
__device__ __forceinline__ int chol_block(double (&u)[2][kPan / W], double* A, int ld, int n, double* tri, double* cb, int* flag) {
  using T = double;
  constexpr int kWarps = W, kCols = kPan / W;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool low = n > 32;  // rows 32.. exist
  T a[2];
  auto fetch = [&](int j) {  // column j of A
    a[0] = lane >= j && lane < n ? A[lane + (long long)j * ld] : T(0);
    a[1] = low && lane + 32 >= j && lane + 32 < n ? A[lane + 32 + (long long)j * ld] : T(0);
  };
  auto pivot = [&](auto qc, int j) {
    constexpr int q = decltype(qc)::value, h = kWarps * q / 32;
    const T v0 = a[0] - u[0][q], v1 = a[1] - u[1][q];
    const T d = __shfl_sync(0xffffffffu, h ? v1 : v0, j & 31);
    if (!(d > T(0))) {
      if (lane == 0) *flag = j + 1;
      return;
    }
    T l, inv;
    chol_pivot(d, l, inv);
    T* b = cb + 64 * (j % 3);
    const T x0 = lane == j ? l : v0 * inv, x1 = lane + 32 == j ? l : v1 * inv;
    if (h == 0) b[lane] = x0;
    if (low) b[lane + 32] = x1;
    if (lane == 0) cb[192 + j] = inv;
    if (h == 0 && lane >= j && lane < n) {
      A[lane + (long long)j * ld] = x0;
      tri[j * kPan + lane] = x0 * inv;
    }
    if (low && lane + 32 >= j && lane + 32 < n) {
      A[lane + 32 + (long long)j * ld] = x1;
      tri[j * kPan + lane + 32] = x1 * inv;
    }
    if (j + kWarps < n) fetch(j + kWarps);
  };
  if (warp < n) fetch(warp);
  if (warp == 0) pivot(std::integral_constant<int, 0>{}, 0);
  __syncthreads();
  each_column<W>(n, [&](auto qc, int jj) {
    constexpr int q = decltype(qc)::value;
    const int j = kWarps * q + jj;
    const int f = *(volatile int*)flag;  // (a later pivot's failure waits for its own turn)
    if (f != 0 && f <= j + 1) return false;
    auto apply = [&](int col, auto fromc, int first) {  // column `col` on the warp's columns >= first from round `from` on
      const T* b = cb + 64 * (col % 3);
      const T l0 = b[lane], l1 = low ? b[lane + 32] : T(0);
#pragma unroll
      for (int q2 = decltype(fromc)::value; q2 < kCols; ++q2) {
        const int c = kWarps * q2 + warp;
        if (c >= first && c < n) {
          const T lc = b[c];
          if (kWarps * q2 < 32) u[0][q2] = fma(l0, lc, u[0][q2]);
          if (low) u[1][q2] = fma(l1, lc, u[1][q2]);
        }
      }
    };
    const bool next = warp == (jj + 1) % kWarps && j + 1 < n;
    if (next) {
      const T* b = cb + 64 * (j % 3);
      const T lc = b[j + 1];
      auto take = [&](auto nc) {
        constexpr int qn = decltype(nc)::value;
        if (kWarps * qn < 32) u[0][qn] = fma(b[lane], lc, u[0][qn]);
        if (low) u[1][qn] = fma(b[lane + 32], lc, u[1][qn]);
        pivot(nc, j + 1);
      };
      if (jj < kWarps - 1) take(qc);
      else take(std::integral_constant<int, (q + 1 < kCols ? q + 1 : q)>{});
    } else {
      // the owner of column j: first what it put off while it took that pivot
      if (warp == jj && j > 0) apply(j - 1, std::integral_constant<int, (q + 1 < kCols ? q + 1 : q)>{}, j + 1);
      apply(j, qc, j + 1);
    }
    __syncthreads();
    return true;
  });
  return *(volatile int*)flag;
}

// A(mb rows, n columns) := (A - u) L11^{-T} against the triangle of chol_block; xb: 128 elements
template <int W>
__device__ __forceinline__ void solve_block(double (&u)[2][kPan / W], double* A, int ld, int mb, int n, const double* tri,
                                            const double* rinv, double* xb) {
  using T = double;
  constexpr int kWarps = W, kCols = kPan / W;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool low = mb > 32;
  T a[2];
  auto fetch = [&](int j) {
    a[0] = lane < mb ? A[lane + (long long)j * ld] : T(0);
    a[1] = low && lane + 32 < mb ? A[lane + 32 + (long long)j * ld] : T(0);
  };
  auto finish = [&](auto qc, int j) {  // column j is due
    constexpr int q = decltype(qc)::value;
    T* b = xb + 64 * (j & 1);
    const T v0 = a[0] - u[0][q], v1 = a[1] - u[1][q], ri = rinv[j];
    b[lane] = v0;
    if (low) b[lane + 32] = v1;
    if (lane < mb) A[lane + (long long)j * ld] = v0 * ri;
    if (low && lane + 32 < mb) A[lane + 32 + (long long)j * ld] = v1 * ri;
    if (j + kWarps < n) fetch(j + kWarps);
  };
  if (warp < n) fetch(warp);
  if (warp == 0) finish(std::integral_constant<int, 0>{}, 0);
  __syncthreads();
  each_column<W>(n, [&](auto qc, int jj) {
    constexpr int q = decltype(qc)::value;
    const int j = kWarps * q + jj;
    const T* b = xb + 64 * (j & 1);
    const T x0 = b[lane], x1 = low ? b[lane + 32] : T(0);
    const T* t = tri + j * kPan;
    if (j + 1 < n && warp == (jj + 1) % kWarps) {
      const T l = t[j + 1];
      auto take = [&](auto nc) {
        constexpr int qn = decltype(nc)::value;
        u[0][qn] = fma(x0, l, u[0][qn]);
        if (low) u[1][qn] = fma(x1, l, u[1][qn]);
        finish(nc, j + 1);
      };
      if (jj < kWarps - 1) take(qc);
      else take(std::integral_constant<int, (q + 1 < kCols ? q + 1 : q)>{});
    }
#pragma unroll
    for (int q2 = q; q2 < kCols; ++q2) {
      const int c = kWarps * q2 + warp;
      if (c > j + 1 && c < n) {
        const T l = t[c];
        u[0][q2] = fma(x0, l, u[0][q2]);
        if (low) u[1][q2] = fma(x1, l, u[1][q2]);
      }
    }
    __syncthreads();
    return true;
  });
}

// FP64 left-looking Cholesky of an n x n column-major matrix (ld), in place, by 64 x 64 blocks: bound by the FP64 pipe.
// Returns 0 or the 1-based index of the first bad pivot.
template <int W>
__device__ __forceinline__ int factor64(double* A, int n, int ld, unsigned char* smem) {
  constexpr int kCols = kPan / W;
  double* tri = (double*)smem;
  double* cb = tri + kPan * kPan;
  double* stage = cb + 256;
  int* flag = (int*)(stage + 4 * kCk * kPan);
  if (threadIdx.x == 0) *flag = 0;
  __syncthreads();
  for (int p0 = 0; p0 < n; p0 += kPan) {
    const int pb = min(kPan, n - p0);
    for (int r0 = p0; r0 < n; r0 += kPan) {
      const int mb = min(kPan, n - r0);
      double u[2][kCols];
#pragma unroll
      for (int q = 0; q < kCols; ++q) u[0][q] = u[1][q] = 0.0;
      if (p0 > 0) {
        if (r0 == p0) {  // the last one may be narrow
          if (pb <= 16) panel_update<W, 1, false, true>(u, A, ld, r0, p0, mb, pb, stage);
          else if (pb <= 32) panel_update<W, 2, false, true>(u, A, ld, r0, p0, mb, pb, stage);
          else if (pb <= 48) panel_update<W, 3, true, true>(u, A, ld, r0, p0, mb, pb, stage);
          else panel_update<W, 4, true, true>(u, A, ld, r0, p0, mb, pb, stage);
        } else if (mb <= 32) {
          panel_update<W, 4, false, false>(u, A, ld, r0, p0, mb, pb, stage);
        } else {
          panel_update<W, 4, true, false>(u, A, ld, r0, p0, mb, pb, stage);
        }
      }
      double* o = A + r0 + (long long)p0 * ld;
      if (r0 == p0) {
        const int info = chol_block<W>(u, o, ld, pb, tri, cb, flag);
        if (info) return p0 + info;
      } else {
        solve_block<W>(u, o, ld, mb, pb, tri, cb + 192, cb);
      }
      __syncthreads();
    }
  }
  return 0;
}

// ---- FP32 ---------------------------------------------------------------------------------------------------
// FP32 arithmetic is cheap beside a barrier or an instruction's issue, so here a thread has a row of 64 columns to
// itself: 64 products from one value of its own and 16 broadcast loads, and the solve against the triangle without
// any exchange. (The FP64 form above, in FP32, took three times as long.)
constexpr int kLdS = 68;  // leading dimension of the panel's triangle in shared memory (16-byte columns)
constexpr int kCk32 = 8;
constexpr size_t kFactor32Smem = (size_t)(kPan * kLdS + 2 * kCk32 * kPan + kPan) * sizeof(float) + 16;

// u[c] += sum over k < kd of L(row, k) L(brow + c, k), NC columns of the block at brow (pb of its rows present): the
// second operand through shared memory in chunks of kCk32, the next chunk and the thread's own values in registers.
// live: the warp has rows (else it only stages)
template <int W, int NC>
__device__ __forceinline__ void row_update(float (&u)[NC], const float* L, int ld, int row, int brow, int pb, int kd, int c0,
                                           bool live, float* Bs) {
  const int tid = threadIdx.x, bc = tid & 63, bk = tid >> 6;
  const float* Lr = L + row;
  const float* Lb = L + brow + (bc < pb ? bc : 0);
  constexpr int KS = 32 * W / kPan, NB = kCk32 / KS;  // step in k of a thread's loads, their number
  float a[kCk32], vb[NB];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < NB; ++i) vb[i] = Lb[(long long)(k0 + bk + KS * i) * ld];
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < NB; ++i) Bs[(buf * kCk32 + bk + KS * i) * kPan + bc] = vb[i];
  };
  load(0);
  store(0);
#pragma unroll
  for (int k = 0; k < kCk32; ++k) a[k] = Lr[(long long)k * ld];
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < kd; k0 += kCk32, buf ^= 1) {
    const bool more = k0 + kCk32 < kd;
    if (more) load(k0 + kCk32);
    if (live) {
#pragma unroll
      for (int k = 0; k < kCk32; ++k) {
        const float av = a[k];
        if (more) a[k] = Lr[(long long)(k0 + kCk32 + k) * ld];
        const float* b = Bs + (buf * kCk32 + k) * kPan + c0;
#pragma unroll
        for (int c = 0; c < NC; c += 4) {
          float bv[4];
          lds4(b + c, bv);
#pragma unroll
          for (int e = 0; e < 4; ++e) u[c + e] = fmaf(av, bv[e], u[c + e]);
        }
      }
    }
    if (more) store(buf ^ 1);
    __syncthreads();
  }
}

// FP32 left-looking Cholesky by 64-column panels: the lower triangle of A, converted as it is read, into L.
// As in FP64 the products are summed up by themselves and subtracted from A once.
template <int W>
__device__ __noinline__ int factor32(const double* A, float* L, int n, int ld, unsigned char* smem) {
  constexpr int kThr = 32 * W;
  float* S = (float*)smem;          // the panel's triangle, column c at c kLdS
  float* Bs = S + kPan * kLdS;      // [2][kCk32][64]
  float* rinv = Bs + 2 * kCk32 * kPan;
  int* flag = (int*)(rinv + kPan);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int p0 = 0; p0 < n; p0 += kPan) {
    const int pb = min(kPan, n - p0);
    {  // the diagonal block: thread = row (tid & 63), NC columns
      constexpr int NC = kPan * kPan / kThr;
      const int r = tid & 63, c0 = NC * (tid >> 6), row = p0 + min(r, pb - 1);
      float u[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) u[c] = 0.f;
      if (p0 > 0) row_update<W, NC>(u, L, ld, row, p0, pb, p0, c0, true, Bs);
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (r < pb && c0 + c <= r) S[(c0 + c) * kLdS + r] = (float)A[row + (long long)(p0 + c0 + c) * ld] - u[c];
    }
    __syncthreads();
    const int w1 = min(pb, 32), w2 = pb - w1;
    if (warp == 0) {
      const int bad = chol32_warp<kLdS>(S, w1, rinv);
      if (lane == 0) *flag = bad;
    }
    __syncthreads();
    if (*flag) return p0 + *flag;
    if (w2 > 0) {
      if (warp == 1) {  // rows 32.. against the first triangle
        float x[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) x[c] = lane < w2 ? S[c * kLdS + 32 + lane] : 0.f;
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          x[c] *= rinv[c];
#pragma unroll
          for (int c2 = c + 1; c2 < 32; ++c2) x[c2] = fmaf(-x[c], S[c * kLdS + c2], x[c2]);
        }
#pragma unroll
        for (int c = 0; c < 32; ++c) S[c * kLdS + 32 + lane] = x[c];  // (0 past the matrix)
      }
      __syncthreads();
      {
        constexpr int NE = 32 / W;  // columns per warp
        float acc[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) acc[e] = 0.f;
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
          const float a = S[k * kLdS + 32 + lane];
#pragma unroll
          for (int q = 0; q < NE; q += 4) {
            float b[4];
            lds4(S + k * kLdS + 32 + NE * warp + q, b);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[q + e] = fmaf(a, b[e], acc[q + e]);
          }
        }
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const int c = NE * warp + e;
          if (lane < w2 && c <= lane) S[(32 + c) * kLdS + 32 + lane] -= acc[e];
        }
      }
      __syncthreads();
      if (warp == 0) {
        const int bad = chol32_warp<kLdS>(S + 32 * kLdS + 32, w2, rinv + 32);
        if (lane == 0) *flag = bad;
      }
      __syncthreads();
      if (*flag) return p0 + 32 + *flag;
    }
    for (int e = tid; e < kPan * pb; e += kThr) {
      const int r = e & 63, c = e >> 6;
      if (r < pb && c <= r) L[p0 + r + (long long)(p0 + c) * ld] = S[c * kLdS + r];
    }
    // the rows below, a thread each (there are some only below a whole panel)
    for (int r0 = p0 + kPan; r0 < n; r0 += kThr) {
      const bool live = r0 + 32 * warp < n;
      const int row = min(r0 + tid, n - 1);
      float u[kPan];
#pragma unroll
      for (int c = 0; c < kPan; ++c) u[c] = 0.f;
      if (p0 > 0) row_update<W, kPan>(u, L, ld, row, p0, kPan, p0, 0, live, Bs);
      if (live) {
        const double* Ar = A + row + (long long)p0 * ld;
        float* Lr = L + row + (long long)p0 * ld;
        const bool mine = r0 + tid < n;
        double av[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) av[e] = Ar[(long long)e * ld];
#pragma unroll
        for (int c = 0; c < kPan; ++c) {
          const float x = ((float)av[c & 7] - u[c]) * rinv[c];
          if (c + 8 < kPan) av[c & 7] = Ar[(long long)(c + 8) * ld];
          if (mine) Lr[(long long)c * ld] = x;
#pragma unroll
          for (int q = (c + 1) / 4; q < kPan / 4; ++q) {
            float l[4];
            lds4(S + c * kLdS + 4 * q, l);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (4 * q + e > c) u[4 * q + e] = fmaf(x, l[e], u[4 * q + e]);
          }
        }
      }
    }
    __syncthreads();
  }
  return 0;
}

// (L L^T)^{-1} on R right-hand sides in shared memory (xs[r * ldx + i]) at once, by panels of 32: warp r solves
// the panel's triangle for right-hand side r; a thread applies it to its rows (forward), or a warp gathers the
// solved rows below for its columns (backward). tri: 2 * 32 * 33 elements.
template <int W, typename T, int R>
__device__ __forceinline__ void solve_multi(const T* L, int n, int ld, T* xs, int ldx, T* tri) {
  constexpr int kWarps = W, kThr = 32 * W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto load_tri = [&](int p0, T* t) {  // zeros outside the triangle and past n
#pragma unroll
    for (int u = 0; u < 32 / kWarps; ++u) {
      const int c = warp + kWarps * u;
      t[lane + 33 * c] = (p0 + lane < n && c <= lane) ? L[(p0 + lane) + (long long)(p0 + c) * ld] : T(0);
    }
  };
  load_tri(0, tri);
  __syncthreads();
  for (int p0 = 0, buf = 0; p0 < n; p0 += 32, buf ^= 1) {
    const int pw = min(32, n - p0);
    const T* t = tri + buf * 32 * 33;
    const int i0 = p0 + 32 + tid;
    T v[32];  // the first row's factor: in flight during the solve
    if (sizeof(T) == 4 && i0 < n)
#pragma unroll
      for (int c = 0; c < 32; ++c) v[c] = L[i0 + (long long)(p0 + c) * ld];
    if (p0 + 32 < n) load_tri(p0 + 32, tri + (buf ^ 1) * 32 * 33);
    if (warp < R) {
      T x = lane < pw ? xs[warp * ldx + p0 + lane] : T(0);
      const T ri = lane < pw ? T(1) / t[lane * 34] : T(0);
#pragma unroll 8
      for (int c = 0; c < pw; ++c) {
        const T xc = __shfl_sync(0xffffffffu, x * ri, c);
        if (lane == c) x = xc;
        else if (lane > c) x = fma(-t[lane + 33 * c], xc, x);
      }
      if (lane < pw) xs[warp * ldx + p0 + lane] = x;
    }
    __syncthreads();
    for (int i = i0; i < n; i += kThr) {  // (only full panels have rows below)
      T s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = T(0);
      if (sizeof(T) == 8 || i != i0)
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = L[i + (long long)(p0 + c) * ld];
#pragma unroll
      for (int c = 0; c < 32; c += 4)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          T y[4];
          lds4(xs + r * ldx + p0 + c, y);
#pragma unroll
          for (int e = 0; e < 4; ++e) s[r] = fma(v[c + e], y[e], s[r]);
        }
#pragma unroll
      for (int r = 0; r < R; ++r) xs[r * ldx + i] -= s[r];
    }
    __syncthreads();
  }
  const int last = ((n - 1) / 32) * 32;
  load_tri(last, tri);
  __syncthreads();
  for (int p0 = last, buf = 0; p0 >= 0; p0 -= 32, buf ^= 1) {
    const int pw = min(32, n - p0);
    const T* t = tri + buf * 32 * 33;
    if (p0 + 32 < n) {  // columns warp, warp + kWarps, ..: the solved rows below
      constexpr int C = 32 / kWarps;
      T s[C][R];
#pragma unroll
      for (int u = 0; u < C; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) s[u][r] = T(0);
#pragma unroll 2
      for (int i = p0 + 32 + lane; i < n; i += 32) {
        T l[C];
#pragma unroll
        for (int u = 0; u < C; ++u) l[u] = L[i + (long long)(p0 + warp + kWarps * u) * ld];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T y = xs[r * ldx + i];
#pragma unroll
          for (int u = 0; u < C; ++u) s[u][r] = fma(l[u], y, s[u][r]);
        }
      }
#pragma unroll
      for (int u = 0; u < C; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s[u][r] += __shfl_xor_sync(0xffffffffu, s[u][r], o);
          if (lane == 0) xs[r * ldx + p0 + warp + kWarps * u] -= s[u][r];
        }
    }
    if (p0 > 0) load_tri(p0 - 32, tri + (buf ^ 1) * 32 * 33);
    __syncthreads();
    if (warp < R) {
      T x = lane < pw ? xs[warp * ldx + p0 + lane] : T(0);
      const T ri = lane < pw ? T(1) / t[lane * 34] : T(0);
#pragma unroll 8
      for (int c = pw - 1; c >= 0; --c) {
        const T xc = __shfl_sync(0xffffffffu, x * ri, c);
        if (lane == c) x = xc;
        else if (lane < c) x = fma(-t[c + 33 * lane], xc, x);
      }
      if (lane < pw) xs[warp * ldx + p0 + lane] = x;
    }
    __syncthreads();
  }
}

// xf = (float)(b - A x) for R right-hand sides, A symmetric from its lower triangle, everything in FP64: one thread per
// row. (Past the diagonal a thread reads its own column of A, sixteen entries a cache line: bound by the FP64
// pipe all the same. Reading those coalesced and adding up across lanes took twice as long.)
template <int W, int R>
__device__ __forceinline__ void residual(const double* A, int n, const double* b, const double* xd, float* xf, int ldx) {
  for (int i = threadIdx.x; i < n; i += 32 * W) {
    double s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = b[i + (long long)r * n];
    const double* a = A + i;
#pragma unroll 8
    for (int c = 0; c <= i; ++c) {
      const double v = a[(long long)c * n];
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = fma(-v, xd[r * ldx + c], s[r]);
    }
    a = A + (long long)i * n;
#pragma unroll 8
    for (int c = i + 1; c < n; ++c) {
      const double v = a[c];
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = fma(-v, xd[r * ldx + c], s[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) xf[r * ldx + i] = (float)s[r];
  }
  __syncthreads();
}

struct Params {
  int batch;
  const int* n;
  const long long* offA;
  const long long* offB;
  const int* order;
  double* A;
  double* B;
  float* L32;    // fp32 factors (offA layout), fp32 + IR mode only
  int nrhs;
  int refine;    // IR steps
  int* info;     // per matrix: 0 or first bad pivot
  unsigned long long* head;  // matrices taken from the front of the order (low half) and its end (high half) after the first
  int front;                 // CTAs that take from the front
  int sms;
  bool own;                  // a CTA's first matrix is given by its number
};

// R right-hand sides b (column-major, n x R) of one factorised matrix, in place
template <int MODE, int W, int R>
__device__ __noinline__ void solve_rhs(const double* A, const float* L32, double* b, int n, int refine,
                                          unsigned char* smem) {
  const int ldx = (n + 3) & ~3;  // 16-byte rows
  const int tid = threadIdx.x;
  auto each = [&](auto f) {
    for (int e = tid; e < n; e += 32 * W)
#pragma unroll
      for (int r = 0; r < R; ++r) f(r * ldx + e, e + (long long)r * n);
    __syncthreads();
  };
  double* xd = (double*)smem;  // [R][ldx]
  if constexpr (MODE == 0) {
    double* tri = xd + R * ldx;
    each([&](int i, long long g) { xd[i] = b[g]; });
    solve_multi<W, double, R>(A, n, n, xd, ldx, tri);
    each([&](int i, long long g) { b[g] = xd[i]; });
  } else {
    float* xf = (float*)(xd + R * ldx);
    float* tri = xf + R * ldx;
    each([&](int i, long long g) { xf[i] = (float)b[g]; });
    solve_multi<W, float, R>(L32, n, n, xf, ldx, tri);
    each([&](int i, long long) { xd[i] = (double)xf[i]; });
    for (int it = 0; it < refine; ++it) {
      residual<W, R>(A, n, b, xd, xf, ldx);
      solve_multi<W, float, R>(L32, n, n, xf, ldx, tri);
      each([&](int i, long long) { xd[i] += (double)xf[i]; });
    }
    each([&](int i, long long g) { b[g] = xd[i]; });
  }
}
// shared memory of solve_rhs: up to four right-hand sides for n <= 512, two above
constexpr size_t solve_smem(int mode) {
  return mode == 0 ? 4 * 512 * 8 + 2 * 32 * 33 * 8 : 4 * 512 * (8 + 4) + 2 * 32 * 33 * 4;
}
constexpr size_t kSmem64 = std::max(kFactor64Smem, solve_smem(0));
constexpr size_t kSmem32 = std::max(kFactor32Smem, solve_smem(1));
// CTAs per SM, of four and of eight warps: 128 registers; FP64 50 KB of shared memory, FP32 33 KB
constexpr int ctas_per_sm(int W) { return 16 / W; }

// MODE 0: plain FP64; MODE 1: fp32 + IR; W: warps of a CTA
template <int MODE, int W>
__global__ void __launch_bounds__(32 * W, ctas_per_sm(W)) batched_kernel(Params P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_idx;
  // The first matrix is the CTA's own (P.own), so that it is known which ones share an SM (CTAs go to the SMs in turn, and they all
  // start at about the same time): every second round of SMs in reverse, and from the end of the order the other way round
  // than from its front. Then what is left, from the CTA's end.
  const int wave = (int)blockIdx.x / P.sms, in_wave = min(P.sms, P.front - wave * P.sms), at = (int)blockIdx.x % P.sms;
  int first = (int)blockIdx.x >= P.front ? P.batch - 1 - ((int)blockIdx.x - P.front)
                                         : wave * P.sms + (wave & 1 ? in_wave - 1 - at : at);
  if (!P.own) first = -1;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      long long t = first;
      if (first < 0) {
        const bool front = (int)blockIdx.x < P.front;
        const unsigned long long h = atomicAdd(P.head, front ? 1ULL : 1ULL << 32);
        const long long f = (P.own ? P.front : 0) + (long long)(h & 0xffffffffULL);
        const long long e = (P.own ? gridDim.x - P.front : 0) + (long long)(h >> 32);
        t = f + e >= P.batch ? -1 : front ? f : P.batch - 1 - e;  // (f and e of them are taken)
      }
      s_idx = t >= 0 ? P.order[t] : -1;
    }
    first = -1;
    __syncthreads();
    const int idx = s_idx;
    if (idx < 0) break;
    {
      const int n = P.n[idx];
      if (n <= 0 || n > kMaxN) {
        if (threadIdx.x == 0) P.info[idx] = -1;
        continue;
      }
      double* A = P.A + P.offA[idx];
      int inf;
      if constexpr (MODE == 0) inf = factor64<W>(A, n, n, smem_raw);
      else inf = factor32<W>(A, P.L32 + P.offA[idx], n, n, smem_raw);
      __syncthreads();
      if (threadIdx.x == 0) P.info[idx] = inf;
      if (inf) continue;
    }
    // (everything about the matrix is looked up again, so that the factorisation has the registers)
    const int id = *(volatile int*)&s_idx, n = P.n[id];
    const double* A = P.A + P.offA[id];
    const float* L = MODE == 1 ? P.L32 + P.offA[id] : nullptr;
    double* B = P.B + P.offB[id];
    const int most = n <= 512 ? 4 : 2;  // right-hand sides at once
    for (int j = 0; j < P.nrhs;) {
      double* b = B + (long long)j * n;
      const int left = P.nrhs - j;
      if (most == 4 && left >= 4) {
        solve_rhs<MODE, W, 4>(A, L, b, n, P.refine, smem_raw);
        j += 4;
      } else if (most == 4 && left == 3) {
        solve_rhs<MODE, W, 3>(A, L, b, n, P.refine, smem_raw);
        j += 3;
      } else if (left >= 2) {
        solve_rhs<MODE, W, 2>(A, L, b, n, P.refine, smem_raw);
        j += 2;
      } else {
        solve_rhs<MODE, W, 1>(A, L, b, n, P.refine, smem_raw);
        ++j;
      }
    }
  }
}

std::mutex g_mtx;
int g_sms = 0;
bool g_attr = false;
template <int MODE, int W>
int set_smem(size_t bytes) {
  return cudaFuncSetAttribute(batched_kernel<MODE, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess;
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double uniform_elem(uint64_t seed, long long i, long long j) {
  const uint64_t r = mix64(mix64(seed) ^ (((uint64_t)i << 32) | (uint64_t)(uint32_t)j));
  return __dsub_rn(__dmul_rn((double)(r >> 11), 1.0 / 9007199254740992.0), 0.5);
}

// matrix k of the batch: (M + M^T)/2 + n*I with M_ij uniform in [-0.5, 0.5) from the counter-based
// generator with seed (seed + k * 0x9e3779b97f4a7c15); one CTA-strided loop per matrix
__global__ void gen_batch_kernel(int batch, const int* n, const long long* offA, unsigned long long seed, double* A) {
  for (int k = blockIdx.x; k < batch; k += gridDim.x) {
    const int nk = n[k];
    const uint64_t sk = seed + (uint64_t)k * 0x9e3779b97f4a7c15ULL;
    double* out = A + offA[k];
    for (long long e = threadIdx.x; e < (long long)nk * nk; e += blockDim.x) {
      const int i = (int)(e % nk), j = (int)(e / nk);
      double v;
      if (i == j) v = __dadd_rn(uniform_elem(sk, i, i), (double)nk);
      else v = __dmul_rn(0.5, __dadd_rn(uniform_elem(sk, i, j), uniform_elem(sk, j, i)));
      out[e] = v;
    }
  }
}

}  // namespace batched
}  // namespace gbx

using namespace gbx;
using namespace gbx::batched;

extern "C" int gbx_dgen_uniform_sym_batched(int batch, const int* n, const long long* offA, unsigned long long seed,
                                            double* A, void* stream) {
  if (gbx::recording_stream(stream)) return GBX_ERR_ARG;  // not a CUDA stream
  if (batch < 0 || (batch > 0 && (!n || !offA || !A))) return GBX_ERR_ARG;
  if (batch == 0) return GBX_OK;
  gen_batch_kernel<<<std::min(batch, 4096), 256, 0, (cudaStream_t)stream>>>(batch, n, offA, seed, A);
  return cudaGetLastError() == cudaSuccess ? GBX_OK : GBX_ERR_CUDA;
}

extern "C" int gbx_batched_order(int batch, const int* n_host, int* order_host) {
  if (batch < 0 || (batch > 0 && (!n_host || !order_host))) return GBX_ERR_ARG;
  std::vector<int> o(batch);
  std::iota(o.begin(), o.end(), 0);
  std::stable_sort(o.begin(), o.end(), [&](int a, int b) { return n_host[a] > n_host[b]; });
  std::copy(o.begin(), o.end(), order_host);
  return GBX_OK;
}

extern "C" int gbx_dposv_batched(int batch, const int* n, const long long* offA, const long long* offB,
                                 const int* order, double* A, double* B, int nrhs, int mode, int refine, float* L32,
                                 int* info, void* work, size_t work_bytes, void* stream) {
  if (gbx::recording_stream(stream)) return GBX_ERR_ARG;  // not a CUDA stream
  return gbx_dposv_batched_ex(batch, n, offA, offB, order, A, B, nrhs, mode, refine, L32, info, 0, work, work_bytes,
                              stream);
}

extern "C" int gbx_dposv_batched_ex(int batch, const int* n, const long long* offA, const long long* offB,
                                    const int* order, double* A, double* B, int nrhs, int mode, int refine, float* L32,
                                    int* info, int ctas, void* work, size_t work_bytes, void* stream) {
  if (gbx::recording_stream(stream)) return GBX_ERR_ARG;  // not a CUDA stream
  if (batch < 0 || nrhs < 1 || (mode != 0 && mode != 1) || refine < 0 || ctas < 0) return GBX_ERR_ARG;
  if (batch == 0) return GBX_OK;
  if (!n || !offA || !offB || !order || !A || !B || !info || (mode == 1 && !L32)) return GBX_ERR_ARG;
  if (!work || work_bytes < 256) return GBX_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  {
    std::lock_guard<std::mutex> lk(g_mtx);
    if (!g_attr) {
      int dev = 0;
      cudaGetDevice(&dev);
      if (cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return GBX_ERR_CUDA;
      if (set_smem<0, 4>(kSmem64) || set_smem<0, 8>(kSmem64) || set_smem<1, 4>(kSmem32) || set_smem<1, 8>(kSmem32))
        return GBX_ERR_CUDA;
      g_attr = true;
    }
  }
  if (cudaMemsetAsync(work, 0, 256, s) != cudaSuccess) return GBX_ERR_CUDA;
  Params P;
  P.batch = batch;
  P.n = n;
  P.offA = offA;
  P.offB = offB;
  P.order = order;
  P.A = A;
  P.B = B;
  P.L32 = L32;
  P.nrhs = nrhs;
  P.refine = refine;
  P.info = info;
  P.head = (unsigned long long*)work;
  // All CTAs that are resident at once, `ctas` of them if given. As many as fit with eight warps have eight: then
  // the systems are few, and what counts is one system's time (64 systems of order 100: FP64 296 us with four warps, 236 with
  // eight, 128: 338 and 265, 1024: 60 ms and 51; 200 of 200 .. 900: 46 ms and 40, FP32 9.0 and 6.0); with more CTAs
  // two small ones in the place of a large one do more (600 of order 64: 158 against 200 us).
  int grid = std::min(ctas > 0 ? ctas : INT_MAX, ctas_per_sm(4) * g_sms);
  grid = std::max(1, std::min(grid, batch));
  P.sms = g_sms;
  // When every system has a CTA at once, one CTA per SM takes them from the front of the order and the others from its
  // end: largest first, an SM's other CTAs run small ones beside its large ones, and stop where the ends meet
  // (FP64, all from the front before: 600 systems of 100 .. 400 13.8 -> 7.4 ms, of 20 .. 100 511 -> 344 us). With more
  // systems the small ones are better kept for the end (4096 of 32 .. 512: FP64 62 against 55.7 ms, FP32 11.4 against 9.6).
  const bool one_round = batch <= ctas_per_sm(4) * g_sms;
  P.front = one_round ? std::min(grid, g_sms) : grid;
  // Many systems in FP32 are bound by latency, not by what an SM's systems add up to: the first comers take the largest
  // (4096 systems 8.85 ms, 9.0 by number, FP64 59.3 and 55.7; 1300 of up to 64 rows 139 us, 150 by number).
  P.own = one_round || mode == 0;
  if (grid <= ctas_per_sm(8) * g_sms) {
    if (mode == 0) batched_kernel<0, 8><<<grid, 256, kSmem64, s>>>(P);
    else batched_kernel<1, 8><<<grid, 256, kSmem32, s>>>(P);
  } else {
    if (mode == 0) batched_kernel<0, 4><<<grid, 128, kSmem64, s>>>(P);
    else batched_kernel<1, 4><<<grid, 128, kSmem32, s>>>(P);
  }
  return cudaGetLastError() == cudaSuccess ? GBX_OK : GBX_ERR_CUDA;
}
