// FP64 dense kernels shared by the ISDF driver.
#pragma once

#include "common.cuh"

namespace thc {

enum GemmMode : int { GEMM_STORE = 0, GEMM_SQUARE = 1 };

// C[m, n] = mode(alpha * sum_k A(m, k) dk[k >> dk_shift] B(k, n)) + beta C[m, n]
// with A(m, k) = A[m*sam + k*sak], B(k, n) = B[n*sbn + k*sbk] and row-major C.
// GEMM_SQUARE stores the squared product.  lower_only restricts C to n <= m.
struct GemmArgs {
  long long M = 0, N = 0;
  int K = 0;
  const double* A = nullptr;
  long long sam = 0, sak = 1;
  const double* B = nullptr;
  long long sbn = 0, sbk = 1;
  double* C = nullptr;
  long long ldc = 0;
  const double* dk = nullptr;
  int dk_shift = 0;
  const double* dkr = nullptr;       // sqrt(dk), where A == B and no dk is negative: lets the
                                     // tensor-core route cut one operand for both sides
  const int* kexp = nullptr;         // powers of two along k (K of them) that balance the operands'
                                     // rows before they are cut: A(m, k) 2^kexp, B(n, k) 2^-kexp
  double alpha = 1.0, beta = 0.0;
  int mode = GEMM_STORE;
  int lower_only = 0;
  const int* skip_flag = nullptr;   // if non-null and set, the kernel does nothing
  int ksplit = 1;                    // > 1: K is split over blockIdx.z into FP64 partials
  double* part = nullptr;            // ksplit x M x N partial buffer (row-major, ld = N)
  // Known zeros: A(m, k) = 0 for k < m (a_zero_below) / B(k, n) = 0 for k < n
  // (b_zero_below), as for a lower-triangular factor read transposed / as it is.  A tile
  // then starts its k loop at its first row / column: the skipped terms are exact zeros,
  // so the result is bit-identical.
  int a_zero_below = 0, b_zero_below = 0;
  int lower_offset = 0;              // lower_only keeps n <= m + lower_offset (C's own indices)
  int no_split = 0;                  // no split of K (no shared partial buffer: a GEMM that
                                     // runs beside others on a second stream)
  int fma_only = 0;                  // keep the FMA kernel (dgemm_tc_fits)
  int tile = 64;                     // CTA tile edge (64, 32 or 16; chosen by dgemm)
};

struct CholStatus {
  int flag;        // set on breakdown; later kernels of the same solve become no-ops
  int info;        // 1-based index of the failing pivot
  double min_piv;  // smallest / largest accepted pivot (before sqrt)
  double max_piv;
};

// With ksplit <= 1 and no part buffer, dgemm picks the tile edge and a split of K itself so
// that the grid covers the GPU (the FP64 pipe of one SM is narrow, so small GEMMs must spread
// over many SMs); split partials are summed in split order (deterministic).
int dgemm(Ctx* c, const GemmArgs& g);
// Products the tensor-core route takes (dgemm_tc.cu): at least this much work, no skip flag,
// no known-zero triangle and no caller's split.  Below it the FMA kernel's one
// launch is as fast as the cut of two operands and the product (97 x 1001 x 200, 3.9e7: 50 us
// against 36; 130 x 130 x 1000, 3.4e7: 52 against 46; 130 x 200 x 1000 row-contiguous, 5.2e7:
// 80 against 85; 256 x 4096 x 32, 6.7e7: 73 against 31).
constexpr double kDgemmTcFlops = 4e7;
bool dgemm_tc_fits(const Ctx* c, const GemmArgs& g);
// Runs g on the tensor cores; *done = false (and THC_OK) when it does not take it (no room
// for the digits), and the caller runs the FMA kernel.
int dgemm_tc(Ctx* c, const GemmArgs& g, bool* done);
// Split-K partials summed in split order, then the epilogue, into C.
int dgemm_reduce_partials(Ctx* c, const GemmArgs& g);
// Cholesky with GEMM panels; dinv receives the inverted NB x NB diagonal blocks
// (NB = 64: ceil(n/64) x 64 x 64 doubles), the last one's only with `last` (chol_inverse's).
int potrf_inv(Ctx* c, double* A, long long ld, int n, const double* thr, CholStatus* cs,
              double* dinv, bool last = true);
// Cinv = (L L^T)^{-1} via X = L^{-1}; X (n x ld) and T (64 x n) are scratch.
// With Cinv == nullptr only X = L^{-1} is formed.
// tensor: X^T X may take the tensor-core route (other roundings than the FMA kernel's).
int chol_inverse(Ctx* c, const double* L, long long ld, int n, const double* dinv, double* X,
                 double* T, double* Cinv, const CholStatus* cs, bool tensor = false);
// Iterative refinement of a shifted solve, in closed form.  With L L^T = C + sI and
// X = L^{-1} (n x n, ld n), k steps zeta_{j+1} = zeta_j + (C + sI)^{-1} (Z^T - C zeta_j)
// from zeta_0 = (C + sI)^{-1} Z^T give zeta_k = X^T P X Z^T, P = sum_{j<=k} (s X X^T)^j
// (eigenvalue lambda of C: filter 1 - (s / (lambda + s))^{k+1} on 1 / lambda).  Writes
// Xt = P X by Horner's rule in FP64 (k + 1 GEMMs of n^3); G and T are n x n scratch.
int refine_polynomial(Ctx* c, const double* X, int n, double s, int k, double* G, double* T,
                      double* Xt);
// The solve zeta = C^{-1} Z on the tensor cores.  C^{-1} scales as 1/d along k and Z as d,
// d = sqrt(diag C): a row cut relative to its largest entry holds the entries of the other points
// in few bits, and the error of zeta grows with d's range, from 10 on (two fragments of different
// amplitude, N_g 43200, N_mu 140: M 3.8 times the FMA kernel's error at a range of 1.5e4, 87
// times at 1.7e5).  So both operands are balanced by powers of two, 2^k_i = d_i to a factor of
// two (GemmArgs::kexp, exact); over 42 such systems the error then is the FMA kernel's within 5 %
// up to a range of 3e4, at 7e4 the smallest points' part of it is twice that.  Beyond
// 2^kBalancedBinades the FMA kernel takes the product, and C^{-1} = X^T X.
constexpr int kBalancedBinades = 13;
// k_i = floor(log2 sqrt|a_i|) of n values a_i, `stride` doubles apart (0 where a_i is 0 or not
// finite), and the smallest and the largest k_i of the others in range[0..1].
// scalars (optional): the mean of the a_i, the pivot threshold 1e-13 of it, and two zeros.
// twice: the k_i once more behind (real and imaginary parts).
int balance_exponents(Ctx* c, const double* a, long long stride, int n, int* k, int* range,
                      double* scalars = nullptr, bool twice = false);
int set_identity(Ctx* c, double* A, long long ld, int n);
int add_diag_shift(Ctx* c, double* A, long long ld, int n, double rel, double* shift_out);
int diag_mean(Ctx* c, const double* A, long long ld, int n, double* out);
int zpotrf_small(Ctx* c, double* A, int n, const double* thr, CholStatus* cs);

}  // namespace thc
