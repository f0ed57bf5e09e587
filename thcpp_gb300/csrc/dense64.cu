// FP64 dense linear algebra on CUDA cores: GEMM (products of little work, with known zeros or a
// flag; the others go to dgemm_tc.cu), blocked Cholesky and the triangular inverse.  These and the
// digit products carry the all-FP64 path, which replaces the reference's ScaLAPACK
// calls one for one:
//   pzgemm 'C','N'  (P = Phi_mu^H Phi, src/interpolating_vectors.cpp:117)  -> dgemm + square
//   pzgels 'N'      (least squares C X = Z, :416)             -> potrf_inv + chol_inverse + dgemm
//   pzherk 'L','C'  (M = zeta_hat^H zeta_hat, :278)                         -> dgemm lower
//   pzpotrf 'L'     (Luv, :289)                                             -> potrf_inv
// GB300 runs FP64 at a small fraction of its FP32 rate (about two FMA lanes per clock per
// SM), so these kernels are bound by the FP64 pipe, and a GEMM must spread over all SMs:
// dgemm picks 64, 32 or 16 tiles and a split of K from the problem shape.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "dense64.cuh"

namespace thc {

namespace {

constexpr int BK = 16;

// C[m, n] = epilogue(sum_k A(m, k) * dk[k] * B(k, n)); AK / BK select which operand
// index is unit-stride so that the shared-memory loads stay coalesced.  T x T tile per
// CTA of 256 threads (16 x 16), (T/16)^2 outputs per thread.
template <bool AK, bool BK_, int T>
__global__ void __launch_bounds__(256) dgemm_kernel(GemmArgs g)
{
  constexpr int R = T / 16;
  constexpr int LOADS = BK * T / 256;
  if (g.skip_flag && *g.skip_flag) return;
  long long m0 = (long long)blockIdx.y * T, n0 = (long long)blockIdx.x * T;
  if (g.lower_only && n0 > m0 + T - 1 + g.lower_offset) return;
  __shared__ double As[BK][T + 1];
  __shared__ double Bs[BK][T + 1];
  int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double acc[R][R] = {};
  int kbeg = 0, kend = g.K;
  if (g.ksplit > 1) {
    int kc = ((g.K + g.ksplit - 1) / g.ksplit + BK - 1) / BK * BK;
    kbeg = blockIdx.z * kc;
    kend = min(g.K, kbeg + kc);
  }
  // Tiles start at multiples of T >= BK, so the first nonzero k is a multiple of BK.
  if (g.a_zero_below) kbeg = max(kbeg, (int)m0);
  if (g.b_zero_below) kbeg = max(kbeg, (int)n0);
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
    for (int r = 0; r < LOADS; r++) {
      int e = threadIdx.x + 256 * r;
      int mm, kk;
      if (AK) { mm = e / BK; kk = e % BK; } else { kk = e / T; mm = e % T; }
      long long m = m0 + mm;
      int k = k0 + kk;
      double av = 0.0;
      if (m < g.M && k < kend) {
        av = g.A[m * g.sam + (long long)k * g.sak];
        if (g.dk) av *= g.dk[k >> g.dk_shift];
      }
      As[kk][mm] = av;
      int nn, kb;
      if (BK_) { nn = e / BK; kb = e % BK; } else { kb = e / T; nn = e % T; }
      long long n = n0 + nn;
      int kq = k0 + kb;
      Bs[kb][nn] = (n < g.N && kq < kend) ? g.B[n * g.sbn + (long long)kq * g.sbk] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      double a[R], b[R];
#pragma unroll
      for (int i = 0; i < R; i++) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < R; j++) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) acc[i][j] = __fma_rn(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < R; i++) {
    long long m = m0 + ty + 16 * i;
    if (m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < R; j++) {
      long long n = n0 + tx + 16 * j;
      if (n >= g.N) continue;
      if (g.lower_only && n > m + g.lower_offset) continue;
      double v = acc[i][j];
      if (g.ksplit > 1) {
        g.part[((long long)blockIdx.z * g.M + m) * g.N + n] = v;
        continue;
      }
      double* cp = g.C + m * g.ldc + n;
      if (g.mode == GEMM_SQUARE) v = v * v;
      else v = g.alpha * v;
      if (g.beta != 0.0) v += g.beta * *cp;
      *cp = v;
    }
  }
}

// Sum split-K partials in split order, then apply the epilogue.
__global__ void dgemm_reduce(GemmArgs g)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= g.M * g.N) return;
  long long m = e / g.N, n = e % g.N;
  if (g.lower_only && n > m + g.lower_offset) return;
  double v = 0.0;
  for (int z = 0; z < g.ksplit; z++) v += g.part[((long long)z * g.M + m) * g.N + n];
  double* cp = g.C + m * g.ldc + n;
  if (g.mode == GEMM_SQUARE) v = v * v;
  else v = g.alpha * v;
  if (g.beta != 0.0) v += g.beta * *cp;
  *cp = v;
}

// ---- Cholesky (lower, in place, row-major) --------------------------------------

// Edge of the diagonal blocks of the blocked Cholesky.
constexpr int NB = 64;

// 1/sqrt(d) for a positive normal d: an FP32 seed y0 (relative error e0 < 2^-22), then one
// third-order step of the binomial series for (1 - e)^(-1/2), e = 1 - d y0^2:
// y = y0 (1 + e/2 + 3e^2/8), which leaves O(e0^3) -- below FP64 rounding.  Four dependent
// FP64 operations: the pivot is on the critical path of every Cholesky step, and FP64 latency
// is long on this part.  The two conversions are integer arithmetic for the same reason.
__device__ __forceinline__ double rsqrt_fast(double d)
{
  const long long db = __double_as_longlong(d);
  const int ed = (int)((db >> 52) & 0x7ff);
  if (ed < 1023 - 100 || ed > 1023 + 100) return 1.0 / sqrt(d);   // outside FP32's range
  // (float)d, rounded to nearest even.
  const long long half = db + 0x0fffffffLL + ((db >> 29) & 1);
  const float f = __uint_as_float((unsigned)(half >> 29) - 0xc0000000u);   // exponent - 896
  const int yb = __float_as_int(rsqrtf(f));
  const double y = __hiloint2double((yb >> 3) + (896 << 20), yb << 29);
  const double e = __fma_rn(-d * y, y, 1.0);
  return __fma_rn(y * e, __fma_rn(0.375, e, 0.5), y);
}

// The diagonal block at (k0, k0), on one SM: a chain of 64 pivots.  A warp's FP64 instruction
// holds its quarter of the SM's pipe for 64 clocks whatever its active lanes, and a dependent
// one follows no sooner; a pivot is eight of them (reciprocal root, scaling, next pivot) and
// two shuffles behind the last.  So the chain runs on one warp with as little beside it as
// possible: panels of four columns, a lane per row, the pivot and the multipliers going
// between lanes by shuffles; a second warp on another quarter follows column by column with
// the rows the first has no lane for; then all warps bring the next panel's columns up to
// date, and while that panel runs the other warps update the columns behind it.  Every element
// takes its FMAs in the order of the columns, as the plain right-looking loop does, so the
// factor has that loop's bits.  Measured 40 us (the chain alone would be 25); that loop, with a
// barrier pair per column and the inverse's triangle in the same block, took 100 us, panels of
// 16 columns on one warp 94 us.  All of N_mu = 256: 0.50 -> 0.25 ms.
// Pivots at or below thr stop the factorisation (info = global 1-based index).  Writes L_kk into
// A (upper part zeroed) and the pivots' reciprocal roots, the diagonal of L_kk^{-1}, into dinv.
constexpr int CP = 4;                        // panel width
constexpr int CS = NB + 2;                   // shared row length: 16-byte rows, spread banks
__global__ void __launch_bounds__(256) chol_diag(double* A, long long ld, int n, int k0,
                                                 const double* thr_p, CholStatus* cs, double* dinv)
{
  if (cs->flag) return;
  const double thr = thr_p ? *thr_p : 0.0;
  __shared__ __align__(16) double a[NB][CS];
  __shared__ double rr[NB];
  __shared__ int bad;
  const int nb = min(NB, n - k0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  {
    double v[16];                            // all loads in flight at once
    const int c = threadIdx.x & 63, r0 = threadIdx.x >> 6;
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const int r = r0 + 4 * q;
      v[q] = (r < nb && c <= r) ? A[(long long)(k0 + r) * ld + k0 + c] : (r == c ? 1.0 : 0.0);
    }
#pragma unroll
    for (int q = 0; q < 16; q++) a[r0 + 4 * q][c] = v[q];
  }
  if (threadIdx.x == 0) bad = 0;
  double pmin = cs->min_piv, pmax = cs->max_piv;
  // d > thr (thr >= 0) as an integer comparison of the bit patterns, which order like the
  // values for non-negative doubles (a negative d compares below).
  const long long thr_bits = __double_as_longlong(thr > 0.0 ? thr : 0.0);
  __syncthreads();
  // a[i][c] -= sum_j a[i][j] a[c][j] over panel columns j = c0 .. c0 + 3, in order.
  auto update = [&](int i, int c, int c0) {
    double v = a[i][c];
    const double2 x0 = *(const double2*)&a[i][c0], x1 = *(const double2*)&a[i][c0 + 2];
    const double2 y0 = *(const double2*)&a[c][c0], y1 = *(const double2*)&a[c][c0 + 2];
    v = __fma_rn(-x0.x, y0.x, v);
    v = __fma_rn(-x0.y, y0.y, v);
    v = __fma_rn(-x1.x, y1.x, v);
    v = __fma_rn(-x1.y, y1.y, v);
    a[i][c] = v;
  };
  for (int c0 = 0; c0 < nb; c0 += CP) {
    if (warp == 0) {
      const int row = c0 + lane;
      double x[CP];
#pragma unroll
      for (int q = 0; q < CP; q++) x[q] = row < NB ? a[row][c0 + q] : 0.0;
      bool stop = false;
#pragma unroll
      for (int q = 0; q < CP; q++) {
        const int j = c0 + q;
        if (j >= nb) stop = true;
        if (!stop) {
          const double d = __shfl_sync(0xffffffffu, x[q], q);
          const long long db = __double_as_longlong(d);
          if (db > thr_bits && ((db >> 52) & 0x7ff) != 0x7ff) {
            const double r = rsqrt_fast(d);
            x[q] = __dmul_rn(x[q], r);
            if (lane == 0) rr[j] = r;
            if (row < NB && lane >= q) a[row][j] = x[q];
#pragma unroll
            for (int c = q + 1; c < CP; c++)
              x[c] = __fma_rn(-x[q], __shfl_sync(0xffffffffu, x[q], c), x[c]);
            // The smallest and largest pivot, compared as bit patterns (all are positive).
            if (db < __double_as_longlong(pmin)) pmin = d;
            if (db > __double_as_longlong(pmax)) pmax = d;
          } else {
            if (lane == 0) {
              cs->flag = 1;
              cs->info = k0 + j + 1;
              bad = 1;
            }
            stop = true;
          }
        }
        // Column j is in shared memory (or there is none): warp 1 may go on.
        __syncwarp();
        asm volatile("bar.arrive %0, 64;\n" ::"r"(1 + q) : "memory");
      }
    } else if (warp == 1) {
      const int row = c0 + 32 + lane;
      double x[CP];
#pragma unroll
      for (int q = 0; q < CP; q++) x[q] = row < NB ? a[row][c0 + q] : 0.0;
#pragma unroll
      for (int q = 0; q < CP; q++) {
        asm volatile("bar.sync %0, 64;\n" ::"r"(1 + q) : "memory");
        if (c0 + 32 >= NB || c0 + q >= nb || *(volatile int*)&bad) continue;
        x[q] = __dmul_rn(x[q], rr[c0 + q]);
#pragma unroll
        for (int c = q + 1; c < CP; c++) x[c] = __fma_rn(-x[q], a[c0 + c][c0 + q], x[c]);
      }
#pragma unroll
      for (int q = 0; q < CP; q++)
        if (row < NB) a[row][c0 + q] = x[q];
    } else if (c0 > 0 && warp != 4) {
      // The panel before this one, on the columns behind this one (not by warp 4, which shares
      // its quarter of the FP64 pipe with the chain).  Item e of the triangle's list, columns
      // from the last one back: column 63 - u holds items u (u + 1) / 2 .. + u.
      const int w = NB - c0 - CP;
      for (int e = (int)threadIdx.x - (warp < 4 ? 64 : 96); e < w * (w + 1) / 2; e += 160) {
        int u = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
        if (u * (u + 1) / 2 > e) u--;
        if ((u + 1) * (u + 2) / 2 <= e) u++;
        update(63 - (e - u * (u + 1) / 2), 63 - u, c0 - CP);
      }
    }
    __syncthreads();
    if (bad) break;
    // The next panel's columns, by this panel: an element a thread.
    {
      const int i = threadIdx.x & 63, c = c0 + CP + (threadIdx.x >> 6);
      if (c < NB && i >= c) update(i, c, c0);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    cs->min_piv = pmin;
    cs->max_piv = pmax;
  }
  if (bad) return;
  const int c = threadIdx.x & 63;
#pragma unroll
  for (int q = 0; q < 16; q++) {
    const int r = (threadIdx.x >> 6) + 4 * q;
    if (r >= nb || c >= nb) continue;
    A[(long long)(k0 + r) * ld + k0 + c] = c <= r ? a[r][c] : 0.0;
    if (r == c) dinv[(long long)r * nb + r] = rr[r];
  }
}

// L_kk^{-1} (nb x nb, row-major, zero above the diagonal) from the factored block and the
// reciprocal roots on dinv's diagonal: the columns are independent forward substitutions, a
// warp each on SMs of their own (inside the diagonal kernel they took two thirds of its FP64
// work).  Column c: v_j *= r_j, then v_i -= l_ij v_j for i > j, j ascending.
constexpr int IW = 4;                        // columns a block: one warp to each FP64 quarter
__global__ void __launch_bounds__(32 * IW) chol_diag_inv(const double* A, long long ld, int n,
                                                         int k0, const CholStatus* cs, double* dinv)
{
  if (cs->flag) return;
  __shared__ double a[NB][NB + 1];
  __shared__ double rr[NB];
  const int nb = min(NB, n - k0);
  const int lane = threadIdx.x & 31, c = blockIdx.x * IW + (threadIdx.x >> 5);
  {
    const int q = threadIdx.x & 63, r0 = threadIdx.x >> 6;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      double v[16];
#pragma unroll
      for (int t = 0; t < 16; t++) {
        const int r = r0 + 2 * t + 32 * h;
        v[t] = (r < nb && q < r) ? A[(long long)(k0 + r) * ld + k0 + q] : 0.0;
      }
#pragma unroll
      for (int t = 0; t < 16; t++) a[r0 + 2 * t + 32 * h][q] = v[t];
    }
    if (threadIdx.x < nb) rr[threadIdx.x] = dinv[(long long)threadIdx.x * nb + threadIdx.x];
  }
  __syncthreads();
  if (c >= nb) return;
  double v0 = lane == c ? 1.0 : 0.0, v1 = lane + 32 == c ? 1.0 : 0.0;
  // Rows 0-31, then (where they take part at all) rows 32-63 by every column.
  for (int j = c; j < min(nb, 32); j++) {
    const double vj = __dmul_rn(__shfl_sync(0xffffffffu, v0, j), rr[j]);
    const double t0 = __fma_rn(-a[lane][j], vj, v0);       // a is zero on and above the diagonal
    v1 = __fma_rn(-a[lane + 32][j], vj, v1);
    v0 = lane == j ? vj : (lane > j ? t0 : v0);
  }
  for (int j = max(c, 32); j < nb; j++) {
    const double vj = __dmul_rn(__shfl_sync(0xffffffffu, v1, j - 32), rr[j]);
    const double t1 = __fma_rn(-a[lane + 32][j], vj, v1);
    v1 = lane + 32 == j ? vj : (lane + 32 > j ? t1 : v1);
  }
  if (lane < nb && lane != c) dinv[(long long)lane * nb + c] = lane > c ? v0 : 0.0;
  if (lane + 32 < nb && lane + 32 != c) dinv[(long long)(lane + 32) * nb + c] = lane + 32 > c ? v1 : 0.0;
}

// L_panel = A_panel L_kk^{-T} in place, rows k0 + 64 .. n: a CTA owns R whole rows, so that
// nothing it overwrites is read elsewhere (the general GEMM went through partials and a second
// launch).  Two threads an entry sum k below and above 32, the order of that GEMM's split.
template <int R>
__global__ void __launch_bounds__(128 * R) chol_panel(double* P, long long ld, int rows,
                                                      const double* __restrict__ dinv,
                                                      const int* flag)
{
  if (*flag) return;
  __shared__ __align__(16) double v[NB][CS];
  __shared__ __align__(16) double x[R][NB];
  constexpr int T = 128 * R, LD = NB * NB / 2 / T;
  {
    double2 t[LD];
#pragma unroll
    for (int q = 0; q < LD; q++) t[q] = __ldg((const double2*)dinv + threadIdx.x + q * T);
    if (threadIdx.x < NB * R) {
      const long long row = blockIdx.x * (long long)R + threadIdx.x / NB;
      x[threadIdx.x / NB][threadIdx.x % NB] = row < rows ? P[row * ld + threadIdx.x % NB] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < LD; q++) {
      const int e = 2 * (threadIdx.x + q * T);
      *(double2*)&v[e / NB][e % NB] = t[q];
    }
  }
  __syncthreads();
  const int h = threadIdx.x & 1, c = (threadIdx.x >> 1) & (NB - 1), r = threadIdx.x / (2 * NB);
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < NB / 2; k += 2) {
    const double2 p = *(const double2*)&x[r][32 * h + k], q = *(const double2*)&v[c][32 * h + k];
    s = __fma_rn(p.x, q.x, s);
    s = __fma_rn(p.y, q.y, s);
  }
  const double s1 = __shfl_down_sync(0xffffffffu, s, 1);
  const long long row = blockIdx.x * (long long)R + r;
  if (h == 0 && row < rows) P[row * ld + c] = __dadd_rn(__dadd_rn(0.0, s), s1);
}

// C[m, n] -= sum_{k < 64} L[m, k] L[n, k] for n <= m (C and L row-major with ld): the small
// trailing updates.  A CTA of 256 threads owns 8 x 16 entries, two threads each for k below and
// above 32, added in that order as the general GEMM's split does; small tiles, because an SM
// takes two FMAs a clock and 192 rows are 1.2e6 of them.  (That GEMM and the sum of its
// partials were two launches of 12 and 4 us at 192 rows.)
constexpr int RM = 8, RN = 16;
__global__ void __launch_bounds__(256) chol_rank64(const double* __restrict__ L, double* C,
                                                   long long ld, int rows, const int* flag)
{
  // Tile t: row block i of 8 reaches column block i / 2 of 16; 2 q (q + 1) / 2 tiles lie
  // before row blocks 2q and 2q + 1, which have q + 1 each.
  const int t = blockIdx.x;
  int q = (int)((sqrtf(4.f * (float)t + 1.f) - 1.f) * 0.5f);
  while (q * (q + 1) > t) q--;
  while ((q + 1) * (q + 2) <= t) q++;
  const int rest = t - q * (q + 1);
  const int m0 = (2 * q + (rest > q ? 1 : 0)) * RM, n0 = (rest > q ? rest - q - 1 : rest) * RN;
  if (m0 >= rows || *flag) return;
  __shared__ __align__(16) double x[RM][CS], y[RN][CS];
  {
    double2 v[3];
#pragma unroll
    for (int s = 0; s < 3; s++) {             // 24 rows of 32 pairs
      const int e = threadIdx.x + 256 * s, r = e >> 5, k = 2 * (e & 31);
      const int row = r < RM ? m0 + r : n0 + r - RM;
      const double* p = L + (long long)row * ld + k;
      v[s] = row < rows ? make_double2(p[0], p[1]) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int s = 0; s < 3; s++) {
      const int e = threadIdx.x + 256 * s, r = e >> 5, k = 2 * (e & 31);
      *(double2*)(r < RM ? &x[r][k] : &y[r - RM][k]) = v[s];
    }
  }
  const int h = threadIdx.x & 1, j = (threadIdx.x >> 1) & (RN - 1), i = threadIdx.x / (2 * RN);
  const int m = m0 + i, n = n0 + j;
  const bool own = h == 0 && m < rows && n <= m;
  double* cp = C + (long long)m * ld + n;
  const double old = own ? *cp : 0.0;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < NB / 2; k += 2) {
    const double2 a = *(const double2*)&x[i][32 * h + k], b = *(const double2*)&y[j][32 * h + k];
    s = __fma_rn(a.x, b.x, s);
    s = __fma_rn(a.y, b.y, s);
  }
  const double s1 = __shfl_down_sync(0xffffffffu, s, 1);
  if (own) *cp = __dadd_rn(old, -__dadd_rn(__dadd_rn(0.0, s), s1));
}

__global__ void set_identity_k(double* A, long long ld, int n)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)n * n) return;
  long long r = e / n, c = e % n;
  A[r * ld + c] = r == c ? 1.0 : 0.0;
}

__global__ void add_diag(double* A, long long ld, int n, const double* trace_src, double rel,
                         double* shift_out)
{
  // shift = rel * trace / n, computed from the diagonal (trace_src = A itself).
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += trace_src[(long long)i * ld + i];
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    red[0] = rel * t / n;
    if (shift_out) *shift_out = red[0];
  }
  __syncthreads();
  double sh = red[0];
  for (int i = threadIdx.x; i < n; i += blockDim.x) A[(long long)i * ld + i] += sh;
}

__global__ void diag_mean_k(const double* A, long long ld, int n, double* out)
{
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += A[(long long)i * ld + i];
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    *out = t / n;
  }
}

// Complex Hermitian Cholesky (lower) for small matrices, single block, interleaved
// (re, im) row-major.  Pivots at or below thr set info and stop.
__global__ void zpotrf_small_k(double* A, int n, const double* thr_p, CholStatus* cs)
{
  double thr = thr_p ? *thr_p : 0.0;
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  for (int j = 0; j < n; j++) {
    if (threadIdx.x == 0) {
      double d = A[2 * ((long long)j * n + j)];
      if (!(d > thr)) {
        bad = 1;
        cs->flag = 1;
        cs->info = j + 1;
      } else {
        A[2 * ((long long)j * n + j)] = sqrt(d);
        A[2 * ((long long)j * n + j) + 1] = 0.0;
      }
    }
    __syncthreads();
    if (bad) return;
    double r = A[2 * ((long long)j * n + j)];
    for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) {
      A[2 * ((long long)i * n + j)] /= r;
      A[2 * ((long long)i * n + j) + 1] /= r;
    }
    __syncthreads();
    long long m = n - j - 1;
    for (long long e = threadIdx.x; e < m * m; e += blockDim.x) {
      int i = j + 1 + (int)(e / m), c = j + 1 + (int)(e % m);
      if (c > i) continue;
      // A[i][c] -= L[i][j] * conj(L[c][j])
      double ar = A[2 * ((long long)i * n + j)], ai = A[2 * ((long long)i * n + j) + 1];
      double br = A[2 * ((long long)c * n + j)], bi = -A[2 * ((long long)c * n + j) + 1];
      double* t = A + 2 * ((long long)i * n + c);
      t[0] -= ar * br - ai * bi;
      t[1] -= ar * bi + ai * br;
    }
    __syncthreads();
  }
}

}  // namespace

template <int T>
static void launch_dgemm(const GemmArgs& g, cudaStream_t s)
{
  dim3 grid((unsigned)cdiv(g.N, T), (unsigned)cdiv(g.M, T), (unsigned)std::max(1, g.ksplit));
  bool ak = g.sak == 1, bk = g.sbk == 1;
  if (ak && bk) dgemm_kernel<true, true, T><<<grid, 256, 0, s>>>(g);
  else if (ak && !bk) dgemm_kernel<true, false, T><<<grid, 256, 0, s>>>(g);
  else if (!ak && bk) dgemm_kernel<false, true, T><<<grid, 256, 0, s>>>(g);
  else dgemm_kernel<false, false, T><<<grid, 256, 0, s>>>(g);
}

// Tile and split of K so that the grid covers the SMs about twice.
static void choose_tile(GemmArgs& g)
{
  const long long want = 2LL * 152;
  auto tiles = [&](int t) {
    long long mt = cdiv(g.M, t), nt = cdiv(g.N, t);
    return g.lower_only ? (mt * nt + mt) / 2 : mt * nt;
  };
  g.tile = tiles(64) >= want / 2 ? 64 : (tiles(32) >= want / 2 ? 32 : 16);
  long long split = std::min<long long>(cdiv(want, tiles(g.tile)), std::max(1, g.K / 32));
  if (g.no_split) split = 1;
  g.ksplit = (int)std::max<long long>(1, std::min<long long>(split, cdiv(g.K, BK)));
}

int dgemm(Ctx* c, const GemmArgs& g_in)
{
  if (g_in.M <= 0 || g_in.N <= 0) return THC_OK;
  if (dgemm_tc_fits(c, g_in)) {
    bool done = false;
    const int st = dgemm_tc(c, g_in, &done);
    if (st || done) return st;
  }
  GemmArgs g = g_in;
  if (g.ksplit <= 1 && !g.part) {
    choose_tile(g);
    if (g.ksplit > 1) {
      g.part = (double*)ws_get(c, WS_DPART, sizeof(double) * g.ksplit * g.M * g.N);
      if (!g.part) {
        digits_release(c);
        g.part = (double*)ws_get(c, WS_DPART, sizeof(double) * g.ksplit * g.M * g.N);
      }
      if (!g.part) return set_error(c, THC_ERR_NOMEM, "dgemm: split-K partials");
    }
  }
  ProfScope prof(c, "dgemm");
  if (g.tile == 16) launch_dgemm<16>(g, c->stream);
  else if (g.tile == 32) launch_dgemm<32>(g, c->stream);
  else launch_dgemm<64>(g, c->stream);
  THC_LAUNCHED(c, "dgemm");
  return g.ksplit > 1 ? dgemm_reduce_partials(c, g) : THC_OK;
}

int dgemm_reduce_partials(Ctx* c, const GemmArgs& g)
{
  dgemm_reduce<<<(unsigned)cdiv(g.M * g.N, 256), 256, 0, c->stream>>>(g);
  THC_LAUNCHED(c, "dgemm_reduce");
  return THC_OK;
}

// C -= L L^T over a panel of 64 columns: the kernel for it where the general GEMM would split K
// in two (fewer tiles than twice the SMs), else that GEMM.
static int rank64_update(Ctx* c, const GemmArgs& g)
{
  GemmArgs t = g;
  choose_tile(t);
  if (t.ksplit != 2 || g.K != NB) return dgemm(c, g);
  const long long q = cdiv(g.M, 2 * RM);
  chol_rank64<<<(unsigned)(q * (q + 1)), 256, 0, c->stream>>>(g.A, g.C, g.ldc, (int)g.M,
                                                             g.skip_flag);
  THC_LAUNCHED(c, "chol_rank64");
  return THC_OK;
}

// Blocked Cholesky whose panel solve is a GEMM with the inverted diagonal block; the
// inverted diagonal blocks are kept in dinv (nblk x 64 x 64) for the triangular inverse.
int potrf_inv(Ctx* c, double* A, long long ld, int n, const double* thr, CholStatus* cs,
              double* dinv, bool last)
{
  ProfScope prof(c, "potrf_inv");
  cudaStream_t s = c->stream;
  // Look-ahead (n >= 512, with the context's second stream): after block k's panel, the
  // next diagonal block is updated first, on the main stream, and factored there while the
  // rest of block k's trailing update runs on the second stream; the next panel waits for
  // that update.  The diagonal blocks' one-SM chain then runs beside the FP64 GEMMs on the
  // other SMs instead of between them.
  const bool la = n >= 512 && c->aux_stream && c->aux_stream != s;
  cudaStream_t s2 = la && !c->one_stream ? c->aux_stream : s;
  bool trail_pending = false;
  for (int k0 = 0; k0 < n; k0 += NB) {
    int nb = std::min(NB, n - k0);
    double* di = dinv + (long long)(k0 / NB) * NB * NB;
    chol_diag<<<1, 256, 0, s>>>(A, ld, n, k0, thr, cs, di);
    THC_LAUNCHED(c, "chol_diag");
    int rest = n - k0 - nb;
    if (rest > 0 || last) {
      chol_diag_inv<<<NB / IW, 32 * IW, 0, s>>>(A, ld, n, k0, cs, di);
      THC_LAUNCHED(c, "chol_diag_inv");
    }
    if (rest <= 0) break;
    if (trail_pending) {     // the panel rows below were updated on the second stream
      THC_CUDA(c, cudaStreamWaitEvent(s, c->ev_trail, 0));
      trail_pending = false;
    }
    {
      double* panel = A + (long long)(k0 + nb) * ld + k0;
      // Rows a CTA: two while their blocks find an SM at once, else four, which share the copy
      // of the inverse block.
      if (rest <= 608) chol_panel<2><<<(unsigned)cdiv(rest, 2), 256, 0, s>>>(panel, ld, rest, di, &cs->flag);
      else chol_panel<4><<<(unsigned)cdiv(rest, 4), 512, 0, s>>>(panel, ld, rest, di, &cs->flag);
      THC_LAUNCHED(c, "chol_panel");
    }
    const double* l21 = A + (long long)(k0 + nb) * ld + k0;
    if (!la) {
      GemmArgs g{};
      g.M = rest; g.N = rest; g.K = nb;
      g.A = l21; g.sam = ld; g.sak = 1;
      g.B = l21; g.sbn = ld; g.sbk = 1;
      g.C = A + (long long)(k0 + nb) * ld + k0 + nb; g.ldc = ld;
      g.alpha = -1.0; g.beta = 1.0; g.lower_only = 1; g.mode = GEMM_STORE;
      g.skip_flag = &cs->flag;
      int st = rank64_update(c, g);
      if (st) return st;
      continue;
    }
    const int nb1 = std::min(NB, rest);
    {
      // The next diagonal block first (rows and columns k0 + nb .. k0 + nb + nb1).
      GemmArgs g{};
      g.M = nb1; g.N = nb1; g.K = nb;
      g.A = l21; g.sam = ld; g.sak = 1;
      g.B = l21; g.sbn = ld; g.sbk = 1;
      g.C = A + (long long)(k0 + nb) * ld + k0 + nb; g.ldc = ld;
      g.alpha = -1.0; g.beta = 1.0; g.lower_only = 1; g.mode = GEMM_STORE;
      g.skip_flag = &cs->flag;
      int st = rank64_update(c, g);
      if (st) return st;
    }
    if (rest > nb1) {
      // The rest of the trailing triangle (rows below the next diagonal block, columns from
      // it on) on the second stream, after the panel.
      if (s2 != s) {
        THC_CUDA(c, cudaEventRecord(c->ev_panel, s));
        THC_CUDA(c, cudaStreamWaitEvent(s2, c->ev_panel, 0));
      }
      GemmArgs g{};
      g.M = rest - nb1; g.N = rest; g.K = nb;
      g.A = l21 + (long long)nb1 * ld; g.sam = ld; g.sak = 1;
      g.B = l21; g.sbn = ld; g.sbk = 1;
      g.C = A + (long long)(k0 + nb + nb1) * ld + k0 + nb; g.ldc = ld;
      g.alpha = -1.0; g.beta = 1.0; g.lower_only = 1; g.lower_offset = nb1;
      g.mode = GEMM_STORE; g.no_split = 1;
      g.skip_flag = &cs->flag;
      int st;
      {
        StreamSwap on_s2(c, s2);
        st = dgemm(c, g);
      }
      if (st) return st;
      if (s2 != s) {
        THC_CUDA(c, cudaEventRecord(c->ev_trail, s2));
        trail_pending = true;
      }
    }
  }
  if (trail_pending) THC_CUDA(c, cudaStreamWaitEvent(s, c->ev_trail, 0));
  return THC_OK;
}

constexpr int kTensorInverse = 512;

// X = L^{-1} (lower, n x n, ld) from the factor L and its inverted diagonal blocks, block row
// by block row: X_ii = dinv_i, X[i, 0:i] = -dinv_i (L[i, 0:i] X[0:i, 0:i]), with the block
// edge NB that potrf_inv used.  T is an NB x n scratch.  Then Cinv = X^T X.
int chol_inverse(Ctx* c, const double* L, long long ld, int n, const double* dinv, double* X,
                 double* T, double* Cinv, const CholStatus* cs,
                 bool tensor)
{
  ProfScope prof(c, "chol_inverse");
  cudaStream_t s = c->stream;
  THC_CUDA(c, cudaMemsetAsync(X, 0, sizeof(double) * (size_t)n * ld, s));
  int nblk = (n + NB - 1) / NB;
  for (int bi = 0; bi < nblk; bi++) {
    int i0 = bi * NB, nb = std::min(NB, n - i0);
    const double* di = dinv + (long long)bi * NB * NB;
    THC_CUDA(c, cudaMemcpy2DAsync(X + (long long)i0 * ld + i0, sizeof(double) * ld, di,
                                  sizeof(double) * nb, sizeof(double) * nb, nb,
                                  cudaMemcpyDeviceToDevice, s));
    if (bi == 0) continue;
    GemmArgs g{};
    g.M = nb; g.N = i0; g.K = i0;                       // T = L[i, 0:i] X[0:i, 0:i]
    g.A = L + (long long)i0 * ld; g.sam = ld; g.sak = 1;
    g.B = X; g.sbn = 1; g.sbk = ld;
    g.b_zero_below = 1;                                 // X[0:i, 0:i] is lower triangular
    g.C = T; g.ldc = n;
    g.skip_flag = cs ? &cs->flag : nullptr;
    int st = dgemm(c, g);
    if (st) return st;
    GemmArgs h{};
    h.M = nb; h.N = i0; h.K = nb;                       // X[i, 0:i] = -dinv_i T
    h.A = di; h.sam = nb; h.sak = 1;
    h.B = T; h.sbn = 1; h.sbk = n;
    h.C = X + (long long)i0 * ld; h.ldc = ld;
    h.alpha = -1.0;
    h.skip_flag = cs ? &cs->flag : nullptr;
    st = dgemm(c, h);
    if (st) return st;
  }
  if (!Cinv) return THC_OK;
  GemmArgs g{};
  g.M = n; g.N = n; g.K = n;                            // Cinv = X^T X
  g.A = X; g.sam = 1; g.sak = ld;
  g.B = X; g.sbn = 1; g.sbk = ld;
  g.C = Cinv; g.ldc = n;
  // On the tensor cores from n 512 on, X's zeros and all, which the FP64 pipe skips: the inverse
  // takes 0.20 ms against 0.19 at n 320, 0.37 against 0.45 at 512, 1.20 against 2.19 at 1024.
  // Not for a caller whose results hang on the FMAs' rounding (tensor false).
  if (!(tensor && n >= kTensorInverse && c->gemm_tc)) {
    g.a_zero_below = g.b_zero_below = 1;                // X lower triangular
    g.skip_flag = cs ? &cs->flag : nullptr;
  }
  return dgemm(c, g);
}

int refine_polynomial(Ctx* c, const double* X, int n, double s, int k, double* G, double* T,
                      double* Xt)
{
  cudaStream_t st = c->stream;
  const size_t bytes = sizeof(double) * (size_t)n * n;
  int r;
  {
    GemmArgs g;                                   // G = s X X^T
    g.M = n; g.N = n; g.K = n;
    g.A = X; g.sam = n; g.sak = 1;
    g.B = X; g.sbn = n; g.sbk = 1;
    g.alpha = s;
    g.C = G; g.ldc = n;
    if ((r = dgemm(c, g))) return r;
  }
  // Horner: Xt = X + G (X + G (... X)); the last step lands in Xt.
  const double* cur = X;
  double* buf[2] = {Xt, T};
  if (k <= 0) THC_CUDA(c, cudaMemcpyAsync(Xt, X, bytes, cudaMemcpyDeviceToDevice, st));
  for (int j = 1; j <= k; j++) {
    double* dst = buf[(k - j) % 2];
    THC_CUDA(c, cudaMemcpyAsync(dst, X, bytes, cudaMemcpyDeviceToDevice, st));
    GemmArgs g;                                   // dst = X + G cur
    g.M = n; g.N = n; g.K = n;
    g.A = G; g.sam = n; g.sak = 1;
    g.B = cur; g.sbn = 1; g.sbk = n;
    g.beta = 1.0;
    g.C = dst; g.ldc = n;
    if ((r = dgemm(c, g))) return r;
    cur = dst;
  }
  return THC_OK;
}

namespace {

__global__ void __launch_bounds__(1024) balance_exponents_k(const double* a, long long stride,
                                                            int n, int* k, int* range,
                                                            double* scalars, bool twice)
{
  __shared__ int lo[32], hi[32];
  __shared__ double red[32];
  int mn = INT_MAX, mx = INT_MIN;
  double s = 0.0;                        // summed as diag_mean_k does
  for (int i = threadIdx.x; i < n; i += 1024) {
    const double v = a[i * stride];
    s += v;
    const int E = (__double2hiint(v) >> 20) & 0x7ff;
    const bool use = E != 0x7ff && v != 0.0;
    const int e = use ? (max(E, 1) - 1023) >> 1 : 0;
    k[i] = e;
    if (twice) k[n + i] = e;
    if (use) {
      mn = min(mn, e);
      mx = max(mx, e);
    }
  }
  mn = __reduce_min_sync(0xffffffffu, mn);
  mx = __reduce_max_sync(0xffffffffu, mx);
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) {
    lo[threadIdx.x >> 5] = mn;
    hi[threadIdx.x >> 5] = mx;
    red[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    mn = __reduce_min_sync(0xffffffffu, lo[threadIdx.x]);
    mx = __reduce_max_sync(0xffffffffu, hi[threadIdx.x]);
    if (threadIdx.x == 0) {
      range[0] = mn <= mx ? mn : 0;
      range[1] = mn <= mx ? mx : 0;
      if (scalars) {
        double t = 0.0;
        for (int w = 0; w < 32; w++) t += red[w];
        scalars[0] = t / n;
        scalars[1] = 1e-13 * scalars[0];
        scalars[2] = scalars[3] = 0.0;
      }
    }
  }
}

}  // namespace

int balance_exponents(Ctx* c, const double* a, long long stride, int n, int* k, int* range,
                      double* scalars, bool twice)
{
  balance_exponents_k<<<1, 1024, 0, c->stream>>>(a, stride, n, k, range, scalars, twice);
  THC_LAUNCHED(c, "balance_exponents");
  return THC_OK;
}

int set_identity(Ctx* c, double* A, long long ld, int n)
{
  set_identity_k<<<(int)cdiv((long long)n * n, 256), 256, 0, c->stream>>>(A, ld, n);
  THC_LAUNCHED(c, "set_identity");
  return THC_OK;
}

int add_diag_shift(Ctx* c, double* A, long long ld, int n, double rel, double* shift_out)
{
  add_diag<<<1, 1024, 0, c->stream>>>(A, ld, n, A, rel, shift_out);
  THC_LAUNCHED(c, "add_diag");
  return THC_OK;
}

int diag_mean(Ctx* c, const double* A, long long ld, int n, double* out)
{
  diag_mean_k<<<1, 1024, 0, c->stream>>>(A, ld, n, out);
  THC_LAUNCHED(c, "diag_mean");
  return THC_OK;
}

int zpotrf_small(Ctx* c, double* A, int n, const double* thr, CholStatus* cs)
{
  zpotrf_small_k<<<1, 1024, 0, c->stream>>>(A, n, thr, cs);
  THC_LAUNCHED(c, "zpotrf_small");
  return THC_OK;
}

}  // namespace thc
