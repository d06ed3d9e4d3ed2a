// Block operations of the tiled Cholesky, templated on the element type (double for the FP64
// path, float for the working precision of the mixed path). One CTA of 256 threads per call.
#pragma once
#include <type_traits>
#include <cuda_runtime.h>

namespace gbx {

constexpr int kThreads = 256;  // threads per CTA of every FP64 block kernel
constexpr int kBlk = 128;      // largest block edge handled by one CTA
constexpr int kKC = 16;        // k-chunk of the GEMM staging
constexpr int kPW = 32;        // panel width of the TRSM

// CTA barrier of the block operations: every thread of the CTA, or (kNamed) the first 256 threads
// only, with named barrier 1, so that a larger CTA can run an operation on 256 of its threads
template <bool kNamed>
__device__ __forceinline__ void ops_sync() {
  if (kNamed) asm volatile("bar.sync 1, 256;" ::: "memory");
  else __syncthreads();
}

// four consecutive elements from shared memory in 16-byte loads (p 16-byte aligned)
__device__ __forceinline__ void lds4(const float* p, float (&v)[4]) {
  const float4 f = *(const float4*)p;
  v[0] = f.x;
  v[1] = f.y;
  v[2] = f.z;
  v[3] = f.w;
}
__device__ __forceinline__ void lds4(const double* p, double (&v)[4]) {
  const double2 a = *(const double2*)p, b = *(const double2*)(p + 2);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}

// pivot of the Cholesky column: l = sqrt(d) and 1/l. FP32: hardware reciprocal square root with
// one Newton step (r <- r (3 - d r^2) / 2), a few ulp, short latency on the factor's serial chain;
// FP64: rsqrt (within an ulp or two) and one multiply.
__device__ __forceinline__ void chol_pivot(float d, float& l, float& inv) {
  float r = rsqrtf(d);
  r = r * fmaf(-0.5f * d * r, r, 1.5f);
  inv = r;
  l = d * r;
}
// 1/sqrt(d), d > 0, for the FP64 factor's serial chain: Newton's iteration (one third-order step from the
// 22-bit FP32 value) in 64-bit fixed point, so that nothing of it waits for the FP64 pipe, which the other warps keep
// busy (there each dependent operation takes 64 clocks and more; rsqrt() takes 371 of an idle pipe). With
// d = m 2^e, e even, m in [1, 4), and y ~ m^(-1/2) in Q31:  r = 1 - m y^2 (exact product, Q60),
// m^(-1/2) = y (1 + r/2 + 3/8 r^2 + O(r^3)), |r| < 2^-20: about 2^-60 off before the rounding to 53 bits.
__device__ __forceinline__ double rsqrt_fixed(double d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const int ex = (int)(b >> 52);
  if (ex == 0 || ex >= 0x7ff) return rsqrt(d);  // subnormal, infinite (or not positive)
  const int odd = (ex + 1) & 1;                 // e = ex - 1023 odd
  const unsigned long long frac = b & 0xFFFFFFFFFFFFFULL;
  const unsigned long long M = ((1ULL << 52) | frac) << (10 + odd);  // m, Q62
  const float y0 = rsqrtf(__uint_as_float(((unsigned)(127 + odd) << 23) | (unsigned)(frac >> 29)));
  const unsigned Y = min(__float2uint_rn(y0 * 2147483648.0f), 0x7FFFFFFFu);
  const unsigned long long P = __umul64hi(M, (unsigned long long)Y * Y);  // m y^2, Q60
  const long long R = (long long)((1ULL << 60) - P);
  const long long Rs = R >> 16;
  const long long C = 2 * R + ((3 * Rs * Rs) >> 29);  // r/2 + 3/8 r^2, Q62
  const long long Y63 = (long long)Y << 32;
  const unsigned long long V = (unsigned long long)(Y63 + __mul64hi(Y63, C << 2));  // m^(-1/2), Q63
  const unsigned long long V53 = (V + 512) >> 10;
  // 2^(-1 - e/2) (1 + (V53 - 2^52) / 2^52); V53 = 2^53 carries into the exponent
  const long long be = 1022 - (ex - 1023 - odd) / 2;
  return __longlong_as_double((be << 52) + (long long)(V53 - (1ULL << 52)));
}
__device__ __forceinline__ void chol_pivot(double d, double& l, double& inv) {
  inv = rsqrt_fixed(d);
  l = d * inv;
}

// ------------------------------------------------------------------------------------------------
// block GEMM:  C(m x n) := C - A(m x k) * B(n x k)^T   (lower: only i >= j of C is written)
// 256 threads, each owning an 8 x 8 micro-tile (rows 4tx..4tx+3 and 64+4tx..64+4tx+3, the same
// pattern of columns from ty), read from shared memory with 16-byte vector loads; k staged through
// double-buffered chunks of 16 with a register prefetch of the next chunk.
// kSmall (m, n <= 64): each thread owns only the first 4 x 4 quarter of that pattern, so a 64 x 64
// block keeps every thread's FMAs useful (the 8 x 8 form would spend three quarters on zeros).
// smem: 2 * 2 * 16 * 128 elements (64 KB in FP64)
// ------------------------------------------------------------------------------------------------
template <typename T, bool kSmall = false>
__device__ __forceinline__ void op_gemm_nt(const T* __restrict__ A, int lda, const T* __restrict__ B, int ldb, T* C,
                                           int ldc, int m, int n, int k, bool lower, T* sm) {
  constexpr int R = kSmall ? 4 : 8;  // micro-tile edge
  T* As = sm;                       // [2][kKC][kBlk]
  T* Bs = sm + 2 * kKC * kBlk;      // [2][kKC][kBlk]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int lrow = tid & 127, lk0 = tid >> 7;
  T acc[R][R];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[i][j] = T(0);

  const int nchunks = (k + kKC - 1) / kKC;
  T ra[8], rb[8];
  auto gload = [&](int k0) {
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int kk = k0 + lk0 + 2 * s;
      ra[s] = (lrow < m && kk < k) ? __ldcg(A + lrow + (long long)kk * lda) : T(0);
      rb[s] = (lrow < n && kk < k) ? __ldcg(B + lrow + (long long)kk * ldb) : T(0);
    }
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      As[(buf * kKC + lk0 + 2 * s) * kBlk + lrow] = ra[s];
      Bs[(buf * kKC + lk0 + 2 * s) * kBlk + lrow] = rb[s];
    }
  };
  if (nchunks > 0) {
    gload(0);
    sstore(0);
    __syncthreads();
    for (int c = 0; c < nchunks; ++c) {
      const int buf = c & 1;
      if (c + 1 < nchunks) gload((c + 1) * kKC);
      const T* as = As + buf * kKC * kBlk;
      const T* bs = Bs + buf * kKC * kBlk;
#pragma unroll
      for (int kk = 0; kk < kKC; ++kk) {
        T a0[4], a1[4], b0[4], b1[4];
        lds4(as + kk * kBlk + 4 * tx, a0);
        lds4(bs + kk * kBlk + 4 * ty, b0);
        if (!kSmall) {
          lds4(as + kk * kBlk + 64 + 4 * tx, a1);
          lds4(bs + kk * kBlk + 64 + 4 * ty, b1);
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int j = 0; j < R; ++j) {
            const T ai = i < 4 ? a0[i & 3] : a1[i & 3], bj = j < 4 ? b0[j & 3] : b1[j & 3];
            acc[i][j] = fma(ai, bj, acc[i][j]);
          }
      }
      if (c + 1 < nchunks) sstore(buf ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int col = (j < 4 ? 0 : 60) + 4 * ty + j;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = (i < 4 ? 0 : 60) + 4 * tx + i;
      if (row < m && col < n && (!lower || row >= col)) {
        T* p = C + row + (long long)col * ldc;
        __stcg(p, __ldcg(p) - acc[i][j]);
      }
    }
  }
  __syncthreads();
}

// FP32 reciprocal without a branch: the hardware approximation refined by one Newton-Raphson step,
// r <- r + r (1 - d r) (within an ulp or so of 1/d). The IEEE division carries a slow-path branch
// that splits an unrolled solve into many scheduling regions and keeps its loads from being hoisted.
__device__ __forceinline__ float rcp_nr(float d) {
  const float r = __fdividef(1.f, d);
  return fmaf(r, fmaf(-d, r, 1.f), r);
}

// ---- FP64 factor and solve of small blocks held in registers --------------------------------------
// On GB300 a warp-wide FP64 instruction occupies its sub-partition's share of the FP64 pipe for 64
// clocks (76 with all four busy: 1.68 FMA per clock and SM) however many lanes are active, and its
// latency is no longer than that. So these operations are bound by the warp instructions issued per
// sub-partition and by the serial chain over the pivots, not by latency: the block stays in registers
// (lane = row, columns dealt to the eight warps), one barrier per column, and the owner of the next
// column updates and publishes it before anything else. Measured as tasks of the executor (its timeline), before
// and now: 64 x 64 POTRF 87 -> 44.5 us; a 64 x 64 triangle against 16 rows 61 -> 21 us, 8 rows 16 us, 64 rows
// 85 -> 50 us; a 128 x 128 triangle against 32 rows 180 -> 106 us (16 rows 80, 8 rows 62).

// Cholesky of an n x n block (n <= 64), thread (warp, lane) holding rows lane + 32 h of columns
// 8 q + warp in x[h][q] (what lies above the diagonal is not read, and is garbage on return).
// cb: 3 * 64 + 64 doubles, the last three columns of L, then the 64 pivot reciprocals;
// *flag: 0 on entry (visible to all threads). Returns 0 or the 1-based index of the first bad pivot.
template <bool kNamed>
__device__ __forceinline__ int chol64_regs(double (&x)[2][8], int n, double* cb, int* flag) {
  const bool low = n > 32;  // rows 32.. exist
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto pivot = [&](auto qc, int j) {  // the warp that owns column j = 8 q + warp
    constexpr int q = decltype(qc)::value, h = q >> 2;
    const double d = __shfl_sync(0xffffffffu, x[h][q], j & 31);
    if (!(d > 0.0)) {
      if (lane == 0) *flag = j + 1;
      return;
    }
    double l, inv;
    chol_pivot(d, l, inv);
    if (lane == 0) cb[192 + j] = inv;
    double* b = cb + 64 * (j % 3);
    if (h == 0) {
      x[0][q] = lane == j ? l : x[0][q] * inv;
      b[lane] = x[0][q];
    }
    if (low) {
      x[1][q] = (h == 1 && lane == (j & 31)) ? l : x[1][q] * inv;
      b[lane + 32] = x[1][q];
    }
  };
  if (warp == 0) pivot(std::integral_constant<int, 0>{}, 0);
  ops_sync<kNamed>();
  bool stop = false;
  auto round = [&](auto qc) {  // columns 8 q .. 8 q + 7
    constexpr int q = decltype(qc)::value;
#pragma unroll 1
    for (int jj = 0; jj < 8; ++jj) {
      const int j = 8 * q + jj;
      if (j >= n) return;
      // pivot j failed (a later pivot's failure, which a faster warp may have set by now, waits for
      // its own turn, so that every warp leaves at the same column)
      const int f = *(volatile int*)flag;
      if (f != 0 && f <= j + 1) {
        stop = true;
        return;
      }
      const double* b = cb + 64 * (j % 3);
      const double l0 = b[lane], l1 = low ? b[lane + 32] : 0.0;
      auto update = [&](auto q2c) {
        constexpr int q2 = decltype(q2c)::value;
        const double lc = b[8 * q2 + warp];
        if (q2 < 4) x[0][q2] = fma(-l0, lc, x[0][q2]);
        if (low) x[1][q2] = fma(-l1, lc, x[1][q2]);
      };
      // the next pivot's column, and nothing else in its warp: the other columns of that warp get
      // column j together with column j + 1
      const bool next = warp == ((jj + 1) & 7) && j + 1 < n;
      if (next) {
        if (jj < 7) {
          update(qc);
          pivot(qc, j + 1);
        } else if (q < 7) {
          constexpr int qn = q < 7 ? q + 1 : 7;
          update(std::integral_constant<int, qn>{});
          pivot(std::integral_constant<int, qn>{}, j + 1);
        }
      } else {
        if (warp == jj && j > 0) {  // what this warp put off while it took pivot j
          const double* bp = cb + 64 * ((j - 1) % 3);
          const double m0 = bp[lane], m1 = low ? bp[lane + 32] : 0.0;
#pragma unroll
          for (int q2 = q + 1; q2 < 8; ++q2) {
            if (8 * q2 + warp < n) {
              const double lc = bp[8 * q2 + warp];
              if (q2 < 4) x[0][q2] = fma(-m0, lc, x[0][q2]);
              if (low) x[1][q2] = fma(-m1, lc, x[1][q2]);
            }
          }
        }
#pragma unroll
        for (int q2 = q; q2 < 8; ++q2) {
          const int c = 8 * q2 + warp;
          if (c > j && c < n) {
            const double lc = b[c];
            if (q2 < 4) x[0][q2] = fma(-l0, lc, x[0][q2]);
            if (low) x[1][q2] = fma(-l1, lc, x[1][q2]);
          }
        }
      }
      ops_sync<kNamed>();
    }
  };
  round(std::integral_constant<int, 0>{});
  if (!stop && n > 8) round(std::integral_constant<int, 1>{});
  if (!stop && n > 16) round(std::integral_constant<int, 2>{});
  if (!stop && n > 24) round(std::integral_constant<int, 3>{});
  if (!stop && n > 32) round(std::integral_constant<int, 4>{});
  if (!stop && n > 40) round(std::integral_constant<int, 5>{});
  if (!stop && n > 48) round(std::integral_constant<int, 6>{});
  if (!stop && n > 56) round(std::integral_constant<int, 7>{});
  return *(volatile int*)flag;
}

// X := X L^{-T} for up to R G rows (R = 8, 16 or 32) and n <= NC 256 / R columns. A warp holds R rows
// by 32 / R columns of each of G row groups: thread (warp, lane) the row lane % R (+ R g) and the columns
// col(q) = 256 / R q + 32 / R warp + lane / R in x[g][q]. The triangle comes with its columns divided by
// the diagonal, L(c, j) / L(j, j) at Ls[j ldl + c] (c > j), so that one FMA a column is on the serial chain; the
// divisions of the results are taken at the end. rinv: the reciprocals of L's diagonal; both in shared memory
// and visible; xb: 2 R G doubles.
template <int R, int G, int NC, bool kNamed>
__device__ __forceinline__ void trsm_regs(double (&x)[G][NC], int n, const double* Ls, int ldl, const double* rinv, double* xb) {
  constexpr int P = 256 / R;  // columns dealt in one round
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane % R, col = (32 / R) * warp + lane / R;
  if (col == 0)
#pragma unroll
    for (int g = 0; g < G; ++g) xb[g * R + r] = x[g][0];
  ops_sync<kNamed>();
  auto round = [&](auto qc) {
    constexpr int q = decltype(qc)::value;
#pragma unroll 1
    for (int jj = 0; jj < P; ++jj) {
      const int j = P * q + jj;
      if (j >= n) return;
      double xj[G];
#pragma unroll
      for (int g = 0; g < G; ++g) xj[g] = xb[(j & 1) * R * G + g * R + r];
      const double* Lj = Ls + (long long)j * ldl;
      auto publish = [&](auto q2c) {  // column j + 1: final after this update
        constexpr int q2 = decltype(q2c)::value;
        const double l = Lj[j + 1];
#pragma unroll
        for (int g = 0; g < G; ++g) {
          x[g][q2] = fma(-xj[g], l, x[g][q2]);
          xb[((j + 1) & 1) * R * G + g * R + r] = x[g][q2];
        }
      };
      if (j + 1 < n) {
        if (jj < P - 1) {
          if (col == jj + 1) publish(qc);
        } else if (q < NC - 1) {
          if (col == 0) publish(std::integral_constant<int, (q < NC - 1 ? q + 1 : q)>{});
        }
      }
#pragma unroll
      for (int q2 = q; q2 < NC; ++q2) {
        const int c = P * q2 + col;
        if (c > j + 1 && c < n) {
          const double l = Lj[c];
#pragma unroll
          for (int g = 0; g < G; ++g) x[g][q2] = fma(-xj[g], l, x[g][q2]);
        }
      }
      ops_sync<kNamed>();
    }
  };
  static_assert(NC <= 16, "rounds below");
  round(std::integral_constant<int, 0>{});
#define GBX_ROUND(Q) \
  if constexpr (NC > Q) { \
    if (n > P * Q) round(std::integral_constant<int, Q>{}); \
  }
  GBX_ROUND(1) GBX_ROUND(2) GBX_ROUND(3) GBX_ROUND(4) GBX_ROUND(5) GBX_ROUND(6) GBX_ROUND(7)
  GBX_ROUND(8) GBX_ROUND(9) GBX_ROUND(10) GBX_ROUND(11) GBX_ROUND(12) GBX_ROUND(13) GBX_ROUND(14) GBX_ROUND(15)
#undef GBX_ROUND
#pragma unroll
  for (int q = 0; q < NC; ++q)
    if (P * q + col < n) {
      const double ri = rinv[P * q + col];
#pragma unroll
      for (int g = 0; g < G; ++g) x[g][q] *= ri;
    }
}

// B(m x n) := B L^{-T} for few rows (m <= R G) and n <= NMAX, in registers: the triangle of L is staged in
// shared memory, then trsm_regs. smem: trsm_regs_smem(R G, NMAX) doubles.
constexpr int trsm_regs_smem(int rows, int nmax) { return nmax * nmax + nmax + 2 * rows; }
template <int R, int G, int NMAX, bool kNamed>
__device__ __forceinline__ void op_trsm_regs(const double* L, int ldl, double* B, int ldb, int m, int n, double* sm) {
  constexpr int P = 256 / R, NC = NMAX / P;
  static_assert(NC * P == NMAX, "whole rounds");
  double* Ls = sm;
  double* rinv = sm + NMAX * NMAX;
  double* xb = rinv + NMAX;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = lane % R, col = (32 / R) * warp + lane / R;
  double x[G][NC];
#pragma unroll
  for (int q = 0; q < NC; ++q)
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int r = r0 + R * g, c = P * q + col;
      x[g][q] = (r < m && c < n) ? __ldcg(B + r + (long long)c * ldb) : 0.0;
    }
  if (tid < n) rinv[tid] = 1.0 / __ldcg(L + tid + (long long)tid * ldl);
#pragma unroll 4
  for (int c = warp; c < n; c += 8)
#pragma unroll
    for (int t = 0; t < NMAX / 32; ++t) {
      const int r = lane + 32 * t;
      if (r >= c && r < n) Ls[c * NMAX + r] = __ldcg(L + r + (long long)c * ldl);
    }
  ops_sync<kNamed>();
#pragma unroll 4
  for (int c = warp; c < n; c += 8) {
    const double ri = rinv[c];
#pragma unroll
    for (int t = 0; t < NMAX / 32; ++t) {
      const int r = lane + 32 * t;
      if (r > c && r < n) Ls[c * NMAX + r] *= ri;
    }
  }
  ops_sync<kNamed>();
  trsm_regs<R, G, NC, kNamed>(x, n, Ls, NMAX, rinv, xb);
#pragma unroll
  for (int q = 0; q < NC; ++q)
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int r = r0 + R * g, c = P * q + col;
      if (r < m && c < n) __stcg(B + r + (long long)c * ldb, x[g][q]);
    }
  ops_sync<kNamed>();
}

// C(m x n) -= A(m x k) B(n x k)^T for a strip of m <= R rows (R = 8 or 16), n, k <= 64; with roff >= 0
// only the elements with roff + i >= j (a strip of a lower block that starts at its row roff). A thread owns row
// tid % R of every (256 / R)-th column, so that every FP64 instruction works on 32 elements.
// smem: 64 R + 64 * 64 doubles.
template <int R, bool kNamed = false>
__device__ __forceinline__ void op_strip_nt(const double* A, int lda, const double* B, int ldb, double* C, int ldc, int m,
                                            int n, int k, int roff, double* sm) {
  constexpr int P = 256 / R, NC = 64 / P;
  double* As = sm;           // [k][R]
  double* Bs = sm + 64 * R;  // [k][64]
  const int tid = threadIdx.x, r = tid % R, cb = tid / R;
  const int nn = roff < 0 ? n : min(n, roff + m);  // columns with any element
#pragma unroll
  for (int u = 0; u < R / 4; ++u) {
    const int e = tid + 256 * u, i = e % R, kk = e / R;
    As[e] = (i < m && kk < k) ? __ldcg(A + i + (long long)kk * lda) : 0.0;
  }
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int e = tid + 256 * u, j = e & 63, kk = e >> 6;
    Bs[e] = (j < nn && kk < k) ? __ldcg(B + j + (long long)kk * ldb) : 0.0;
  }
  double acc[NC], c0[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int c = cb + P * i;
    acc[i] = 0.0;
    c0[i] = (r < m && c < nn) ? __ldcg(C + r + (long long)c * ldc) : 0.0;
  }
  ops_sync<kNamed>();
#pragma unroll 4
  for (int kk = 0; kk < k; ++kk) {
    const double a = As[kk * R + r];
#pragma unroll
    for (int i = 0; i < NC; ++i)
      if (P * i < nn) acc[i] = fma(a, Bs[kk * 64 + cb + P * i], acc[i]);
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int c = cb + P * i;
    if (r < m && c < nn && (roff < 0 || roff + r >= c)) __stcg(C + r + (long long)c * ldc, c0[i] - acc[i]);
  }
  ops_sync<kNamed>();
}

// block POTRF in FP64, n <= 64, in registers. smem: 258 doubles
template <bool kNamed>
__device__ __forceinline__ int op_potrf64(double* A, int lda, int n, double* sm) {
  int* flag = (int*)(sm + 256);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) *flag = 0;
  double x[2][8];
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      x[h][q] = (r < n && c <= r) ? __ldcg(A + r + (long long)c * lda) : 0.0;
    }
  ops_sync<kNamed>();
  const int info = chol64_regs<kNamed>(x, n, sm, flag);
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      if (r < n && c <= r) __stcg(A + r + (long long)c * lda, x[h][q]);
    }
  ops_sync<kNamed>();
  return info;
}

// block POTRF in FP64 (n <= 128): 64 columns at a time in registers. n > 64: the rows below the first
// 64 columns are solved against their triangle, and the rank-64 update of the rest is taken while it is
// loaded. smem: kPotrf64Smem doubles.
constexpr int kPotrf64Smem = 2 * 64 * 64 + 256 + 2;
template <bool kNamed>
__device__ __forceinline__ int op_potrf_f64(double* A, int lda, int n, double* sm) {
  double* L11 = sm;              // [64 columns][64 rows], columns divided by the diagonal (trsm_regs)
  double* X21 = sm + 64 * 64;    // [64 columns][64 rows]: rows 64.. of the first 64 columns of L
  double* cb = sm + 2 * 64 * 64;
  int* flag = (int*)(cb + 256);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) *flag = 0;
  double x[2][8];
  const int n1 = min(n, 64), n2 = n - n1;
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      x[h][q] = (r < n1 && c <= r) ? __ldcg(A + r + (long long)c * lda) : 0.0;
    }
  ops_sync<kNamed>();
  int info = chol64_regs<kNamed>(x, n1, cb, flag);
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      if (r < n1 && c <= r) {
        __stcg(A + r + (long long)c * lda, x[h][q]);
        if (n2 > 0) L11[r + 64 * c] = x[h][q] * cb[192 + c];
      }
    }
  if (info != 0 || n2 <= 0) {
    ops_sync<kNamed>();
    return info;
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      x[h][q] = r < n2 ? __ldcg(A + 64 + r + (long long)c * lda) : 0.0;
    }
  ops_sync<kNamed>();
  trsm_regs<32, 2, 8, kNamed>(x, 64, L11, 64, cb + 192, cb);
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      if (r < n2) __stcg(A + 64 + r + (long long)c * lda, x[h][q]);
      X21[r + 64 * c] = x[h][q];
    }
  double* A22 = A + 64 + 64LL * lda;
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      x[h][q] = (r < n2 && c <= r) ? __ldcg(A22 + r + (long long)c * lda) : 0.0;
    }
  ops_sync<kNamed>();
#pragma unroll 2
  for (int k = 0; k < 64; ++k) {
    const double a0 = X21[lane + 64 * k], a1 = X21[lane + 32 + 64 * k];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (8 * q < n2) {
        const double b = X21[8 * q + warp + 64 * k];
        if (q < 4) x[0][q] = fma(-a0, b, x[0][q]);
        x[1][q] = fma(-a1, b, x[1][q]);
      }
  }
  info = chol64_regs<kNamed>(x, n2, cb, flag);
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h, c = 8 * q + warp;
      if (r < n2 && c <= r) __stcg(A22 + r + (long long)c * lda, x[h][q]);
    }
  ops_sync<kNamed>();
  return info != 0 ? 64 + info : 0;
}

// One row of a 32-column panel held in registers: x := x * L_blk^{-T} (row-wise forward
// substitution against the panel's lower triangle Lp, column-major with leading dimension ldp).
// rinv (optional): the 32 reciprocals of the panel's diagonal at rinv[rinv_at(c)], computed once
// for all rows (an FP64 division per row and column is ~500 clocks of a warp on GB300).
__device__ __forceinline__ int rinv_at(int c, int ldp) { return (c & 15) + ldp * (16 + (c >> 4)); }
template <typename T>
__device__ __forceinline__ void row_solve32(T (&x)[32], const T* Lp, int ldp, int pw, const T* rinv = nullptr) {
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    if (c < pw) {
      T s0 = x[c], s1 = T(0);
#pragma unroll
      for (int c2 = 0; c2 + 1 < c; c2 += 2) {
        s0 = fma(-x[c2], Lp[c + ldp * c2], s0);
        s1 = fma(-x[c2 + 1], Lp[c + ldp * (c2 + 1)], s1);
      }
      if (c & 1) s0 = fma(-x[c - 1], Lp[c + ldp * (c - 1)], s0);
      // the reciprocal does not depend on x: off the chain
      x[c] = (s0 + s1) * (rinv ? rinv[rinv_at(c, ldp)] : (T(1) / Lp[c + ldp * c]));
    }
  }
}
// the reciprocals of a 32 x 32 lower panel Lp (column-major, ldp) into its strict upper triangle at
// rinv_at(c): rows 0-15 of columns 16 and 17, never read as part of the lower triangle. One warp.
template <typename T>
__device__ __forceinline__ void panel_reciprocals(T* Lp, int ldp, int pw, int lane) {
  const T v = lane < pw ? T(1) / Lp[lane + ldp * lane] : T(0);
  __syncwarp();
  Lp[rinv_at(lane, ldp)] = v;
}

// The same solve column by column for a full FP32 panel: once x(c) is final it is subtracted from
// the later entries, so column c of Lp is read with 16-byte loads that do not depend on x, and the
// chain per column is one multiply and one FMA. Lp is 16-byte aligned and ldp a multiple of 4. The
// warp sync every 8 columns bounds how far ahead the compiler hoists the loads (register pressure
// inside the persistent mixed kernel). It is a full-warp sync: every caller runs this on all 32
// lanes of its warps (a partial warp would never meet the sync).
__device__ __forceinline__ void col_solve32(float (&x)[32], const float* Lp, int ldp) {
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    float l[32];
#pragma unroll
    for (int q = c / 4; q < 8; ++q) lds4(Lp + c * ldp + 4 * q, *reinterpret_cast<float(*)[4]>(&l[4 * q]));
    x[c] *= rcp_nr(l[c]);
#pragma unroll
    for (int r = c + 1; r < 32; ++r) x[r] = fmaf(-l[r], x[c], x[r]);
    if ((c + 1) % 8 == 0 && c < 31) __syncwarp();  // keeps the loads hoisted at most 8 columns ahead
  }
}

// ------------------------------------------------------------------------------------------------
// block TRSM (Right, Lower, Trans, NonUnit): B(m x n) := B * L^{-T}, m <= 128, any n.
// Column panels of 32: left-looking update of the panel from the already-solved columns (a
// 128 x 32 x p0 GEMM, 4 x 4 micro-tiles), then each thread solves its own row across the panel.
// smem: panel 32*128 + X chunk 16*128 + L chunk 16*32 + diagonal 32*32 doubles = 60 KB
// ------------------------------------------------------------------------------------------------
// k-chunk of the TRSM update: 64 for float (enough FMAs per chunk to cover the L2 latency of the
// next chunk's prefetch), 16 for double (the FP64 pipe already hides it)
template <typename T>
struct TrsmChunk {
  static constexpr int value = sizeof(T) == 4 ? 64 : kKC;
};
template <typename T>
constexpr size_t op_trsm_smem_elems() {
  return (size_t)kPW * kBlk + (size_t)TrsmChunk<T>::value * kBlk + (size_t)TrsmChunk<T>::value * kPW + kPW * kPW;
}

// kColSolve (FP32 only): the panel solve in the column-wise form with the branch-free reciprocal,
// for kernels with registers to spare; the default keeps the row-wise form and IEEE division.
template <typename T, bool kColSolve = false, bool kNamed = false>
__device__ void op_trsm(const T* __restrict__ L, int ldl, T* B, int ldb, int m, int n, T* sm) {
  constexpr int KC = TrsmChunk<T>::value;
  T* P = sm;                    // [kPW][128]  panel, P[c*128 + r]
  T* Xc = P + kPW * kBlk;       // [KC][128]
  T* Lc = Xc + KC * kBlk;       // [KC][kPW]
  T* Ld = Lc + KC * kPW;        // [kPW][kPW]  Ld[c2*32 + c] = L(p0+c, p0+c2)
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  for (int p0 = 0; p0 < n; p0 += kPW) {
    const int pw = min(kPW, n - p0);
    for (int idx = tid; idx < kPW * kBlk; idx += kThreads) {
      const int r = idx & (kBlk - 1), c = idx >> 7;
      P[idx] = (r < m && c < pw) ? __ldcg(B + r + (long long)(p0 + c) * ldb) : T(0);
    }
    for (int idx = tid; idx < kPW * kPW; idx += kThreads) {
      const int c = idx & 31, c2 = idx >> 5;
      Ld[idx] = (c < pw && c2 <= c) ? __ldcg(L + (p0 + c) + (long long)(p0 + c2) * ldl) : T(0);
    }
    ops_sync<kNamed>();
    if (p0 > 0) {
      // P -= X(:, 0:p0) L(p0:p0+pw, 0:p0)^T, k in chunks of KC; the next chunk is prefetched into
      // registers while the current one is multiplied (hides the L2 latency)
      T acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
      T rx[KC * kBlk / kThreads], rl[(KC * kPW + kThreads - 1) / kThreads];
      auto gload = [&](int k0) {
#pragma unroll
        for (int u = 0; u < KC * kBlk / kThreads; ++u) {
          const int idx = tid + u * kThreads;
          const int r = idx & (kBlk - 1), kk = idx >> 7;
          rx[u] = (r < m && k0 + kk < p0) ? __ldcg(B + r + (long long)(k0 + kk) * ldb) : T(0);
        }
#pragma unroll
        for (int u = 0; u < (KC * kPW + kThreads - 1) / kThreads; ++u) {
          const int idx = tid + u * kThreads;
          const int c = idx & 31, kk = idx >> 5;
          rl[u] = (idx < KC * kPW && c < pw && k0 + kk < p0) ? __ldcg(L + (p0 + c) + (long long)(k0 + kk) * ldl) : T(0);
        }
      };
      auto sstore = [&]() {
#pragma unroll
        for (int u = 0; u < KC * kBlk / kThreads; ++u) Xc[tid + u * kThreads] = rx[u];
#pragma unroll
        for (int u = 0; u < (KC * kPW + kThreads - 1) / kThreads; ++u)
          if (tid + u * kThreads < KC * kPW) Lc[tid + u * kThreads] = rl[u];
      };
      // m <= 32 (a row sub-task): lane = row, warp = four columns, so that no FP64 instruction
      // works on absent rows (a warp-wide FP64 instruction costs the same with any active lanes)
      const bool narrow = m <= 32;
      gload(0);
      for (int k0 = 0; k0 < p0; k0 += KC) {
        sstore();
        ops_sync<kNamed>();
        if (k0 + KC < p0) gload(k0 + KC);
        if (narrow) {
#pragma unroll
          for (int kk = 0; kk < KC; ++kk) {  // row tx x columns 4ty..4ty+3
            const T a = Xc[kk * kBlk + tx];
            T b[4];
            lds4(Lc + kk * kPW + 4 * ty, b);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0][j] = fma(a, b[j], acc[0][j]);
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < KC; ++kk) {  // rows 4tx..4tx+3 x columns 4ty..4ty+3, vector loads
            T a[4], b[4];
            lds4(Xc + kk * kBlk + 4 * tx, a);
            lds4(Lc + kk * kPW + 4 * ty, b);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
          }
        }
        ops_sync<kNamed>();
      }
      if (narrow) {
#pragma unroll
        for (int j = 0; j < 4; ++j) P[(4 * ty + j) * kBlk + tx] -= acc[0][j];
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) P[(4 * ty + j) * kBlk + 4 * tx + i] -= acc[i][j];
      }
      ops_sync<kNamed>();
    }
    if (!kColSolve) {  // the panel's reciprocals once, into Ld's unused upper triangle
      if (tid < 32) panel_reciprocals<T>(Ld, kPW, pw, tid);
      ops_sync<kNamed>();
    }
    // each thread solves its row of the panel in registers; the column-wise solve synchronises its
    // warp, so it runs on whole warps (rows past m are zero in P and are never stored back)
    const int solvers = kColSolve ? ((m + 31) & ~31) : m;
    if (tid < solvers && tid < kBlk) {
      const int r = tid;
      T x[kPW];
#pragma unroll
      for (int c = 0; c < kPW; ++c) x[c] = P[c * kBlk + r];
      if constexpr (kColSolve) {
        if (pw == kPW) col_solve32(x, Ld, kPW);
        else row_solve32<T>(x, Ld, kPW, pw);
      } else {
        row_solve32<T>(x, Ld, kPW, pw, Ld);  // Ld holds L(p0+c, p0+c2) at c + 32*c2
      }
#pragma unroll
      for (int c = 0; c < kPW; ++c) P[c * kBlk + r] = x[c];
    }
    ops_sync<kNamed>();
    for (int idx = tid; idx < kPW * kBlk; idx += kThreads) {
      const int r = idx & (kBlk - 1), c = idx >> 7;
      if (r < m && c < pw) __stcg(B + r + (long long)(p0 + c) * ldb, P[idx]);
    }
    ops_sync<kNamed>();
  }
}


// 32 x 32 Cholesky (pw <= 32 rows) at S (leading dimension LD) in FP32 by one warp: lane = row, columns exchanged by shuffles; rinv: the
// reciprocals of the pivots. Returns 0 or the 1-based index of the first bad pivot.
template <int LD>
__device__ __forceinline__ int chol32_warp(float* S, int pw, float* rinv) {
  const int lane = threadIdx.x & 31;
  float x[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) x[c] = (lane < pw && c <= lane) ? S[lane + LD * c] : 0.f;
  int bad = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (j < pw && bad == 0) {
      const float d = __shfl_sync(0xffffffffu, x[j], j);
      if (!(d > 0.f)) {
        bad = j + 1;
      } else {
        float l, inv;
        chol_pivot(d, l, inv);
        if (lane == 0) rinv[j] = inv;
        const float lij = lane == j ? l : (lane > j ? x[j] * inv : 0.f);
        x[j] = lij;
#pragma unroll
        for (int c = j + 1; c < 32; ++c) {
          const float lcj = __shfl_sync(0xffffffffu, lij, c);
          x[c] = fmaf(-lij, lcj, x[c]);  // (above the diagonal: not used)
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (c <= lane && lane < pw) S[lane + LD * c] = x[c];
  return bad;
}

// ---- FP32 block operations on 128 x 128 blocks for a serial chain of them (256 threads) -------------------------
// In a chain every operation finds its code evicted from the instruction cache by the tasks in between: a solve
// unrolled over 64 columns (7000 instructions) took 16 us warm and 47 in the chain. So these are loops over 16
// columns with short bodies, on operands that are brought into shared memory by 16-byte loads before the arithmetic
// starts. As mini-tasks of a diagonal tile (us, before and now): POTRF 88 -> 38, TRSM 52 -> 28, update 30 -> 22
// (a factor of N=5000: 6.3 -> 3.9 ms). Out of line, so that a kernel that calls them keeps its registers. Leading
// dimensions are multiples of 4 and 128 rows from a block's start on can be read; blocks that are not 16-byte aligned
// are read and written by single entries.
constexpr int kLdF = 132;  // leading dimension of a block in shared memory (16-byte columns)
constexpr size_t kChainF32Smem = (size_t)(2 * kBlk * kLdF + kBlk + 4) * sizeof(float);

__device__ __forceinline__ bool aligned16(const float* p) { return ((size_t)p & 15) == 0; }
__device__ __forceinline__ float4 ldcg4(const float* p, bool al) {
  return al ? __ldcg((const float4*)p) : make_float4(__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3));
}
// the block's first n columns (128 rows; rows past m as zero) into S, by 16-byte loads, sixteen in flight
__device__ __forceinline__ void chain_stage_f32(const float* A, int lda, int m, int n, float* S) {
  const int r = 4 * (threadIdx.x & 31), c0 = threadIdx.x >> 5;
  const bool al = aligned16(A);
  float4 v[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int c = c0 + 8 * u;
    v[u] = c < n ? ldcg4(A + r + (long long)c * lda, al) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    if (r + 0 >= m) v[u].x = 0.f;
    if (r + 1 >= m) v[u].y = 0.f;
    if (r + 2 >= m) v[u].z = 0.f;
    if (r + 3 >= m) v[u].w = 0.f;
    *(float4*)(S + (c0 + 8 * u) * kLdF + r) = v[u];
  }
}
// x[0..15] (a thread's row, columns p0..) against the 16 x 16 triangle at T (column c at c kLdF)
__device__ __forceinline__ void chain_row16_f32(float (&x)[16], const float* T, const float* rinv) {
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    x[c] *= rinv[c];
#pragma unroll
    for (int q = (c + 1) / 4; q < 4; ++q) {
      float l[4];
      lds4(T + c * kLdF + 4 * q, l);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (4 * q + e > c) x[4 * q + e] = fmaf(-x[c], l[e], x[4 * q + e]);
    }
  }
}

// n x n block (n <= 128), lower, in place; returns 0 or the 1-based index of the first bad pivot
static __device__ __noinline__ int chain_potrf_f32(float* A, int lda, int n, float* sm) {
  float* S = sm;  // column c at c kLdF
  float* rinv = sm + kBlk * kLdF;
  int* flag = (int*)(rinv + kBlk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  chain_stage_f32(A, lda, n, n, S);
  __syncthreads();
  int info = 0;
#pragma unroll 1
  for (int p0 = 0; p0 < n; p0 += 16) {
    const int pw = min(16, n - p0), rb = p0 + 16;
    float* Sp = S + p0 * kLdF + p0;
    if (warp == 0) {  // 16 x 16 by one warp: lane = row, columns exchanged by shuffles
      float x[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) x[c] = (lane < pw && c <= lane) ? Sp[c * kLdF + lane] : 0.f;
      int bad = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float d = __shfl_sync(0xffffffffu, x[j], j);
        if (j < pw && bad == 0 && !(d > 0.f)) bad = j + 1;
        float l, inv;
        chol_pivot(d, l, inv);
        if (lane == 0) rinv[p0 + j] = inv;
        x[j] = lane == j ? l : x[j] * inv;
#pragma unroll
        for (int c = j + 1; c < 16; ++c) x[c] = fmaf(-x[j], __shfl_sync(0xffffffffu, x[j], c), x[c]);
      }
#pragma unroll
      for (int c = 0; c < 16; ++c)
        if (c <= lane && lane < pw) Sp[c * kLdF + lane] = x[c];
      if (lane == 0) *flag = bad;
    }
    __syncthreads();
    if (*flag) {
      info = p0 + *flag;
      break;
    }
    if (rb >= n) break;
    if (rb + tid < n) {  // a row below: against the triangle
      float* Sr = S + p0 * kLdF + rb + tid;
      float x[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) x[c] = Sr[c * kLdF];
      chain_row16_f32(x, Sp, rinv + p0);
#pragma unroll
      for (int c = 0; c < 16; ++c) Sr[c * kLdF] = x[c];
    }
    __syncthreads();
    // rank-16 update of the rest: 32 rows x 8 columns per warp and turn
    const int rg = (n - rb + 31) >> 5;  // row groups; group g has 4 (g + 1) column groups
#pragma unroll 1
    for (int w = warp; w < 2 * rg * (rg + 1); w += 8) {
      int g = 0, cg = w;
      while (cg >= 4 * (g + 1)) cg -= 4 * ++g;
      const int r = rb + 32 * g + lane, c0 = rb + 8 * cg;
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float a = S[(p0 + k) * kLdF + r];
        float b0[4], b1[4];
        lds4(S + (p0 + k) * kLdF + c0, b0);
        lds4(S + (p0 + k) * kLdF + c0 + 4, b1);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[e] = fmaf(a, b0[e], acc[e]);
          acc[4 + e] = fmaf(a, b1[e], acc[4 + e]);
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (r < n && c0 + e <= r) S[(c0 + e) * kLdF + r] -= acc[e];
    }
    __syncthreads();
  }
  __syncthreads();
#pragma unroll 1
  for (int c = warp; c < n; c += 8)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int r = lane + 32 * t;
      if (r >= c && r < n) __stcg(A + r + (long long)c * lda, S[c * kLdF + r]);
    }
  __syncthreads();
  return info;
}

// B(m x n) := B L^{-T}, m, n <= 128: two threads a row, left-looking by 16 columns, of which each takes 8 in the
// update from the solved ones; the first of them then has all 16 for the triangle
static __device__ __noinline__ void chain_trsm_f32(const float* L, int ldl, float* B, int ldb, int m, int n, float* sm) {
  float* S = sm;                  // L, column c at c kLdF
  float* Xs = sm + kBlk * kLdF;   // B, then X
  float* rinv = sm + 2 * kBlk * kLdF;
  const int tid = threadIdx.x, r = tid & 127, h = tid >> 7;
  chain_stage_f32(L, ldl, n, n, S);
  chain_stage_f32(B, ldb, m, n, Xs);
  __syncthreads();
  if (tid < kBlk) rinv[tid] = tid < n ? 1.f / S[tid * (kLdF + 1)] : 0.f;
#pragma unroll 1
  for (int p0 = 0; p0 < n; p0 += 16) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    const float* Sk = S + p0 + 8 * h;
#pragma unroll 8
    for (int k = 0; k < p0; ++k) {
      const float x = Xs[k * kLdF + r];
      float l0[4], l1[4];
      lds4(Sk + k * kLdF, l0);
      lds4(Sk + k * kLdF + 4, l1);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[e] = fmaf(x, l0[e], acc[e]);
        acc[4 + e] = fmaf(x, l1[e], acc[4 + e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) Xs[(p0 + 8 * h + e) * kLdF + r] -= acc[e];
    __syncthreads();
    if (h == 0) {
      float x[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) x[c] = Xs[(p0 + c) * kLdF + r];
      chain_row16_f32(x, S + p0 * kLdF + p0, rinv + p0);
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        Xs[(p0 + c) * kLdF + r] = x[c];
        if (r < m && p0 + c < n) __stcg(B + r + (long long)(p0 + c) * ldb, x[c]);
      }
    }
    __syncthreads();
  }
}

// C(m x n) -= A(m x k) B(n x k)^T, m, n, k <= 128 (lower: only i >= j of C): both operands staged at once, 8 x 8
// micro-tiles as op_gemm_nt
static __device__ __noinline__ void chain_gemm_f32(const float* A, int lda, const float* B, int ldb, float* C, int ldc, int m,
                                                   int n, int k, bool lower, float* sm) {
  float* As = sm;
  float* Bs = sm + kBlk * kLdF;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  chain_stage_f32(A, lda, m, k, As);
  chain_stage_f32(B, ldb, n, k, Bs);
  // this thread's entries of C (four rows at a time) on their way meanwhile
  const bool al = aligned16(C);
  float4 cv[2][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int col = (j < 4 ? 0 : 60) + 4 * ty + j;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      cv[i][j] = col < n ? ldcg4(C + 64 * i + 4 * tx + (long long)col * ldc, al) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  __syncthreads();
#pragma unroll 2
  for (int kk = 0; kk < k; ++kk) {
    float a0[4], a1[4], b0[4], b1[4];
    lds4(As + kk * kLdF + 4 * tx, a0);
    lds4(As + kk * kLdF + 64 + 4 * tx, a1);
    lds4(Bs + kk * kLdF + 4 * ty, b0);
    lds4(Bs + kk * kLdF + 64 + 4 * ty, b1);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(i < 4 ? a0[i & 3] : a1[i & 3], j < 4 ? b0[j & 3] : b1[j & 3], acc[i][j]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int col = (j < 4 ? 0 : 60) + 4 * ty + j;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = 64 * i + 4 * tx;
      float* p = C + row + (long long)col * ldc;
      const float4 v = make_float4(cv[i][j].x - acc[4 * i][j], cv[i][j].y - acc[4 * i + 1][j], cv[i][j].z - acc[4 * i + 2][j],
                                   cv[i][j].w - acc[4 * i + 3][j]);
      if (al && col < n && row + 3 < m && (!lower || row >= col)) {
        __stcg((float4*)p, v);
      } else if (col < n) {
        if (row < m && (!lower || row >= col)) __stcg(p, v.x);
        if (row + 1 < m && (!lower || row + 1 >= col)) __stcg(p + 1, v.y);
        if (row + 2 < m && (!lower || row + 2 >= col)) __stcg(p + 2, v.z);
        if (row + 3 < m && (!lower || row + 3 >= col)) __stcg(p + 3, v.w);
      }
    }
  }
  __syncthreads();
}

}  // namespace gbx
