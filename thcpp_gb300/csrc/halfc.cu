// Half-rotated ISDF with complex orbitals (IVecs with rotate = true on complex aoR and
// aoR_half), FP64 throughout:
//   P      = Phi_mu^H Phi,  P_occ = Phi_occ,mu^H Phi_occ       setup_pseudo_dm, pzgemm 'C','N'
//                                                            (src/interpolating_vectors.cpp:117)
//   Z      = P_occ o conj(P)                                  setup_CZt_half (:143-161)
//   C      = Z[:, idx]   (complex, not Hermitian)             setup_CCt (:163-190)
//   X      = C^{-1} Z                                         least_squares, pzgels (:416)
//   zeta   = conj(X) (rows: zeta_mu(r))                       fft_vectors' Hermitian transpose
//   IVG    = forward, IVMG = backward unnormalised 3-D FFT    fft_vectors (:384-391)
//   M      = sum_G IVMG_mu(G) v(G) IVG_nu(G)                  construct_muv 'T','N' (:261-273)
// M is HalfTransformedMuv, written without a Cholesky factor (dump_thc_data, :317-328).
//
// C has full rank for a sensible point set but no symmetry, so the reference's QR solve is
// replaced by the inverse from Gauss-Jordan elimination with partial pivoting (one kernel per
// column, gj_step, on [C | I] from one buffer into another; N_mu^3 complex FMAs, small next to
// the N_mu^2 N_g of the products), then X = C^{-1} Z.  Complex values are (re, im) pairs; P
// and Z are kept as their real N_mu x N_g matrix and the imaginary one behind it, so that every
// complex product is one real GEMM (of twice the rows, or the terms) with each operand cut
// once.  IVMG(G) = IVG(-G), so one transform serves both.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "dense64.cuh"
#include "fft_tc.cuh"
#include "isdf.cuh"

namespace thc {
namespace {

// Rows of the pair-stored orbitals at the interpolating points: out[mu][*] = phi[idx[mu]][*]
// (kw doubles per row); rot (optional) = the rotated pairs (-im, re), for Im(a^H b) as a
// real dot product; orb (optional) = the (N_o, N_mu, 2) orbital output.
__global__ void gather_pairs(const double* __restrict__ phi, long long ng, int no,
                             const int* __restrict__ idx, int nmu, double* out, double* rot,
                             double* orb, int* bad)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)nmu * no) return;
  const int mu = (int)(e / no), i = (int)(e % no);
  const long long g = idx[mu];
  if (g < 0 || g >= ng) {
    atomicExch(bad, 1);
    return;
  }
  const double re = phi[(g * no + i) * 2], im = phi[(g * no + i) * 2 + 1];
  out[e * 2] = re;
  out[e * 2 + 1] = im;
  rot[e * 2] = -im;
  rot[e * 2 + 1] = re;
  if (orb) {
    orb[2 * ((long long)i * nmu + mu)] = re;
    orb[2 * ((long long)i * nmu + mu) + 1] = im;
  }
}

// Z = Q o conj(P) in place of (PR, PI):  ZR = QR PR + QI PI,  ZI = QI PR - QR PI.
__global__ void half_product(double* pr, double* pi, const double* __restrict__ qr,
                             const double* __restrict__ qi, long long n)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= n) return;
  const double a = pr[e], b = pi[e], c = qr[e], d = qi[e];
  pr[e] = __fma_rn(c, a, d * b);
  pi[e] = __fma_rn(d, a, -c * b);
}

// [C | I] (n x 2n complex, row-major) with C[mu][nu] = Z[mu][idx[nu]].
__global__ void build_augmented(const double* __restrict__ zr, const double* __restrict__ zi,
                                long long ng, const int* __restrict__ idx, int n, double* a)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)n * 2 * n) return;
  const int r = (int)(e / (2 * n)), c = (int)(e % (2 * n));
  double re = 0.0, im = 0.0;
  if (c < n) {
    const long long g = idx[c];
    if (g >= 0 && g < ng) {                            // gather_pairs has reported the others
      re = zr[(long long)r * ng + g];
      im = zi[(long long)r * ng + g];
    }
  } else {
    re = (c - n == r) ? 1.0 : 0.0;
  }
  a[2 * e] = re;
  a[2 * e + 1] = im;
}

struct GjStatus {
  int singular;        // 1-based column without a non-zero pivot
  int pad;
  double min_abs2;     // smallest / largest |pivot|^2
  double max_abs2;
};

// Step k of the elimination, in one kernel: the pivot p = argmax_{r >= k} |A[r][k]|^2 (lowest row
// on ties), rows k and p swapped, row k scaled by 1 / A[k][k], and A[r][c] -= A[r][k] A[k][c] for
// every other row and the columns c > k (those up to k are not read again).  From one buffer into
// the other, so that every block can find the pivot by itself and the swap is a choice of rows;
// with a pivot kernel of one block and an elimination in place the 144 steps at N_mu 144 took 2.4
// ms, now 0.9.  What bounds a step is the chain of column,
// pivot, reciprocal and row; R rows a thread are as few as keep the blocks resident at once.
constexpr int kGjCols = 64, kGjThreads = 256;   // 64 columns, 4 rows at a time
template <int R>
__global__ void __launch_bounds__(kGjThreads) gj_step(const double2* __restrict__ a, double2* o,
                                                      int n, int k, GjStatus* gs)
{
  __shared__ long long bv[kGjThreads / 32];
  __shared__ int bi[kGjThreads / 32];
  __shared__ double piv[2];
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long w = 2LL * n;                        // row length
  const int over = gs->singular;
  // Integer comparisons: an FP64 one holds its warp as long as an FP64 sum.  NaN never wins.
  long long best = -1;
  int arg = n;
  for (int r = k + tid; r < n; r += kGjThreads) {
    const double2 z = a[r * w + k];
    const double v = z.x * z.x + z.y * z.y;
    const long long b = v >= 0.0 ? __double_as_longlong(v) : -1;
    if (b > best) { best = b; arg = r; }
  }
  auto warp_best = [&]() {
    const int hi = __reduce_max_sync(full, (int)(best >> 32));
    bool in = (int)(best >> 32) == hi;
    const unsigned lo = __reduce_max_sync(full, in ? (unsigned)best : 0u);
    in = in && (unsigned)best == lo;
    arg = __reduce_min_sync(full, in ? arg : n);
    best = (long long)hi << 32 | lo;
  };
  warp_best();
  if (lane == 0) { bv[warp] = best; bi[warp] = arg; }
  __syncthreads();
  best = lane < kGjThreads / 32 ? bv[lane] : -1;
  arg = lane < kGjThreads / 32 ? bi[lane] : n;
  warp_best();
  if (over) return;
  const int p = arg;
  if (best <= 0 || p >= n) {
    if (blockIdx.x + blockIdx.y == 0 && tid == 0) gs->singular = k + 1;
    return;
  }
  const long long c = k + 1 + (long long)blockIdx.x * kGjCols + (tid & (kGjCols - 1));
  const int r0 = (int)blockIdx.y * 4 * R + tid / kGjCols;
  const bool in = c < w;
  double2 x = {0.0, 0.0}, y[R], f[R];
  if (in) x = a[p * w + c];
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int r = r0 + 4 * q, m = r == p ? k : r;
    y[q] = f[q] = {0.0, 0.0};
    if (in && r < n && r != k) {
      y[q] = a[m * w + c];
      f[q] = a[m * w + k];
    }
  }
  if (warp == 0) {
    // 1 / (x + i y) = (x - i y) / (x^2 + y^2), a lane each.
    const double2 z = a[p * w + k];
    const double d = z.x * z.x + z.y * z.y, v = (lane ? -z.y : z.x) / d;
    if (lane < 2) piv[lane] = v;
    if (blockIdx.x + blockIdx.y == 0 && lane == 0) {
      const double b = __longlong_as_double(best);
      gs->min_abs2 = k ? fmin(gs->min_abs2, b) : b;
      gs->max_abs2 = k ? fmax(gs->max_abs2, b) : b;
    }
  }
  __syncthreads();
  if (!in) return;
  const double2 xs = {x.x * piv[0] - x.y * piv[1], x.x * piv[1] + x.y * piv[0]};
#pragma unroll
  for (int q = 0; q < R; q++) {
    const int r = r0 + 4 * q;
    if (r >= n) continue;
    double2 z = xs;
    if (r != k) {
      z.x = __fma_rn(-f[q].x, xs.x, __fma_rn(f[q].y, xs.y, y[q].x));
      z.y = __fma_rn(-f[q].x, xs.y, __fma_rn(-f[q].y, xs.x, y[q].y));
    }
    o[r * w + c] = z;
  }
}

// zeta (interleaved complex, row mu = zeta_mu on the grid) = conj(XR + i XI).
__global__ void conj_interleave(const double* __restrict__ xr, const double* __restrict__ xi,
                                long long n, double* z)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= n) return;
  z[2 * e] = xr[e];
  z[2 * e + 1] = -xi[e];
}

// The left operand of M from the forward spectra: the backward transform of a field at G is its
// forward one at -G.  left1 = (re, -im) and left2 = (im, re) of IVMG(G) = IVG(-G), so that over
// (re, im) pairs left1 . IVG = Re(IVMG IVG) and left2 . IVG = Im; vs = v in the spectrum's order
// (zyx: kz, ky, kx with kx fastest, as fft_tc leaves it; else kz fastest).
__global__ void left_spectra(const double2* __restrict__ ivg, const double* __restrict__ v, int n0,
                             int n1, int n2, bool zyx, int nmu, double2* left1, double2* left2,
                             double* vs)
{
  const long long ng = (long long)n0 * n1 * n2;
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= ng) return;
  const int d0 = zyx ? n0 : n2;                       // fastest axis, then n1, then the other
  const int f = (int)(e % d0), k1 = (int)(e / d0 % n1), sl = (int)(e / d0 / n1);
  const int ds = zyx ? n2 : n0;
  const long long m = ((long long)((ds - sl) % ds) * n1 + (n1 - k1) % n1) * d0 + (d0 - f) % d0;
  if (blockIdx.y == 0) vs[e] = zyx ? v[((long long)f * n1 + k1) * n2 + sl] : v[e];
  for (int mu = blockIdx.y; mu < nmu; mu += gridDim.y) {
    const double2 p = ivg[mu * ng + m];
    left1[mu * ng + e] = make_double2(p.x, -p.y);
    left2[mu * ng + e] = make_double2(p.y, p.x);
  }
}

// [Re C^-1, -Im C^-1] over [Im C^-1, Re C^-1] (2n x 2n) from the right half of [C | I] after the
// elimination: with Z's real rows over its imaginary ones, one real product gives X's.
__global__ void inverse_pairs(const double* __restrict__ aug, int n, double* out)
{
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)n * n) return;
  const int r = (int)(e / n), c = (int)(e % n);
  const double re = aug[2 * ((long long)r * 2 * n + n + c)];
  const double im = aug[2 * ((long long)r * 2 * n + n + c) + 1];
  out[(long long)r * 2 * n + c] = re;
  out[(long long)r * 2 * n + n + c] = -im;
  out[(long long)(n + r) * 2 * n + c] = im;
  out[(long long)(n + r) * 2 * n + n + c] = re;
}

__global__ void interleave(const double* __restrict__ re, const double* __restrict__ im,
                           long long n, double* out)
{
  long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= n) return;
  out[2 * e] = re[e];
  out[2 * e + 1] = im[e];
}

}  // namespace

int isdf_half_complex_run(Ctx* c, const double* phi_in, long long ng, int no,
                          const double* occ_in, int nocc, const int* idx_in, int nmu,
                          const int* mesh_in, const double* coul_in, double* out_orb,
                          double* out_orb_occ, double* out_M, thc_isdf_stats* stats)
{
  c->zeta_elem = 0;
  if (!phi_in || !occ_in || !idx_in || !mesh_in || !coul_in || ng <= 0 || no <= 0 || nocc <= 0 ||
      nmu <= 0 || nmu > ng)
    return set_error(c, THC_ERR_ARG, "thc_isdf_half_complex: invalid arguments");
  int mesh[3];
  if (is_device_ptr(mesh_in)) {
    THC_CUDA(c, cudaMemcpy(mesh, mesh_in, sizeof(mesh), cudaMemcpyDeviceToHost));
  } else {
    std::copy(mesh_in, mesh_in + 3, mesh);
  }
  if (mesh[0] <= 0 || mesh[1] <= 0 || mesh[2] <= 0 ||
      (long long)mesh[0] * mesh[1] * mesh[2] != ng)
    return set_error(c, THC_ERR_SHAPE, "thc_isdf_half_complex: FFT mesh does not match N_g");
  cudaStream_t s = c->stream;
  int st = 0;
  const double* phi = (const double*)to_device(c, phi_in, sizeof(double) * 2 * ng * no, WS_PHI, &st);
  if (st) return st;
  const double* occ = (const double*)to_device(c, occ_in, sizeof(double) * 2 * ng * nocc,
                                               WS_PHIOCC, &st);
  if (st) return st;
  const int* idx = (const int*)to_device(c, idx_in, sizeof(int) * nmu, WS_IDX, &st);
  if (st) return st;
  const double* coul = (const double*)to_device(c, coul_in, sizeof(double) * ng, WS_COUL, &st);
  if (st) return st;
  const long long nmg = (long long)nmu * ng;
  const long long nn = (long long)nmu * nmu;
  // Gathered rows: Phi_mu, its rotation, Phi_occ,mu, its rotation.
  double* rows = (double*)ws_get(c, WS_PHIMU, sizeof(double) * 4 * nmu * (no + nocc));
  double* prpi = (double*)ws_get(c, WS_ZT, sizeof(double) * 2 * nmg);     // P, then Z, then zeta
  double* qrqi = (double*)ws_get(c, WS_ZETA, sizeof(double) * 2 * nmg);   // P_occ, then X
  double* spec = (double*)ws_get(c, WS_ZHAT, sizeof(double) * 4 * nmg);   // IVG, IVMG
  double* aug = (double*)ws_get(c, WS_C, sizeof(double) * 4 * nn);        // [C | I]
  double* aug2 = (double*)ws_get(c, WS_CINV, sizeof(double) * 4 * nn);
  double* Mw = (double*)ws_get(c, WS_M, sizeof(double) * 4 * nn);
  char* scr = (char*)ws_get(c, WS_SCRATCH, 4096);
  const bool orb_host = out_orb && !is_device_ptr(out_orb);
  const bool occ_host = out_orb_occ && !is_device_ptr(out_orb_occ);
  double* stage = nullptr;
  if (orb_host || occ_host)
    stage = (double*)ws_get(c, WS_ORB, sizeof(double) * 2 * nmu * (no + nocc));
  if (!rows || !prpi || !qrqi || !spec || !aug || !aug2 || !Mw || !scr ||
      ((orb_host || occ_host) && !stage))
    return set_error(c, THC_ERR_NOMEM, "thc_isdf_half_complex: workspace allocation failed");
  double* pmu = rows;
  double* pmu_rot = pmu + 2LL * nmu * no;
  double* omu = pmu_rot + 2LL * nmu * no;   // each followed by its rotation
  double* omu_rot = omu + 2LL * nmu * nocc;
  double *pr = prpi, *pi = prpi + nmg, *qr = qrqi, *qi = qrqi + nmg;   // Re and Im
  GjStatus* gs = (GjStatus*)scr;
  int* bad = (int*)(scr + 512);
  double* orb_dev = out_orb ? (orb_host ? stage : out_orb) : nullptr;
  double* occ_dev = out_orb_occ ? (occ_host ? stage + 2LL * nmu * no : out_orb_occ) : nullptr;
  THC_CUDA(c, cudaMemsetAsync(scr, 0, 1024, s));
  c->tc64_err = bad + 1;
  THC_CUDA(c, cudaEventRecord(c->ev0, s));
  gather_pairs<<<(int)cdiv((long long)nmu * no, 256), 256, 0, s>>>(phi, ng, no, idx, nmu, pmu,
                                                                  pmu_rot, orb_dev, bad);
  THC_LAUNCHED(c, "gather_pairs");
  gather_pairs<<<(int)cdiv((long long)nmu * nocc, 256), 256, 0, s>>>(occ, ng, nocc, idx, nmu, omu,
                                                                    omu_rot, occ_dev, bad);
  THC_LAUNCHED(c, "gather_pairs");
  if (orb_host)
    THC_CUDA(c, cudaMemcpyAsync(out_orb, orb_dev, sizeof(double) * 2 * nmu * no,
                                cudaMemcpyDeviceToHost, s));
  if (occ_host)
    THC_CUDA(c, cudaMemcpyAsync(out_orb_occ, occ_dev, sizeof(double) * 2 * nmu * nocc,
                                cudaMemcpyDeviceToHost, s));
  // Re(a^H b) and Im(a^H b) as real dot products over the (re, im) pairs: a . b and
  // rot(a) . b with rot(a) = (-im, re), whose rows follow a's; so do the results'.
  auto pseudo_dm = [&](const double* amu, const double* full, int k, double* out) -> int {
    GemmArgs g;
    g.M = 2LL * nmu; g.N = ng; g.K = 2 * k;
    g.A = amu; g.sam = 2 * k; g.sak = 1;
    g.B = full; g.sbn = 2 * k; g.sbk = 1;
    g.C = out; g.ldc = ng;
    return dgemm(c, g);
  };
  if ((st = pseudo_dm(pmu, phi, no, prpi))) return st;
  if ((st = pseudo_dm(omu, occ, nocc, qrqi))) return st;
  half_product<<<(int)cdiv(nmg, 256), 256, 0, s>>>(pr, pi, qr, qi, nmg);
  THC_LAUNCHED(c, "half_product");
  // C^{-1} by Gauss-Jordan elimination on [C | I].
  build_augmented<<<(int)cdiv(2 * nn, 256), 256, 0, s>>>(pr, pi, ng, idx, nmu, aug);
  THC_LAUNCHED(c, "build_augmented");
  int* bal = (int*)ws_get(c, WS_EQUIL, sizeof(int) * 2 * nmu);
  if (!bal) return set_error(c, THC_ERR_NOMEM, "thc_isdf_half_complex: workspace allocation failed");
  volatile int* h_range = (int*)c->pinned;     // written by the kernel, read after the event
  if ((st = balance_exponents(c, aug, 4LL * nmu + 2, nmu, bal, (int*)h_range, nullptr, true)))
    return st;
  THC_CUDA(c, cudaEventRecord(c->ev_fork, s));
  // The fewest rows a thread whose blocks the 152 SMs hold at once, eight each.
  int gr = 1;
  while (gr < 8 && cdiv(nmu, 4 * gr) * cdiv(2 * nmu, kGjCols) > 152 * 8) gr *= 2;
  auto step = gr == 1 ? gj_step<1> : gr == 2 ? gj_step<2> : gr == 4 ? gj_step<4> : gj_step<8>;
  for (int k = 0; k < nmu; k++) {
    const dim3 grid((unsigned)cdiv(2LL * nmu - k - 1, kGjCols), (unsigned)cdiv(nmu, 4 * gr));
    step<<<grid, kGjThreads, 0, s>>>((const double2*)aug, (double2*)aug2, nmu, k, gs);
    std::swap(aug, aug2);
  }
  c->launches += nmu;
  THC_LAUNCHED(c, "gj_step");
  // X = C^{-1} Z as one real product of 2 N_mu rows and 2 N_mu terms (into the P_occ buffers).
  {
    double* ci = (double*)ws_get(c, WS_DINV, sizeof(double) * 4 * nn);
    if (!ci) return set_error(c, THC_ERR_NOMEM, "thc_isdf_half_complex: inverse");
    inverse_pairs<<<(int)cdiv(nn, 256), 256, 0, s>>>(aug, nmu, ci);
    THC_LAUNCHED(c, "inverse_pairs");
    GemmArgs g;
    g.M = 2LL * nmu; g.N = ng; g.K = 2 * nmu;
    g.A = ci; g.sam = 2LL * nmu; g.sak = 1;
    g.B = prpi; g.sbn = 1; g.sbk = ng;
    g.kexp = bal;
    THC_CUDA(c, cudaEventSynchronize(c->ev_fork));   // long past, behind the elimination's launches
    g.fma_only = h_range[1] - h_range[0] > kBalancedBinades;
    g.C = qrqi; g.ldc = ng;
    if ((st = dgemm(c, g))) return st;
  }
  // zeta = conj(X), interleaved for cuFFT (in the P buffers), then both transforms.
  double* zc = prpi;
  conj_interleave<<<(int)cdiv(nmg, 256), 256, 0, s>>>(qr, qi, nmg, zc);
  THC_LAUNCHED(c, "conj_interleave");
  double* ivg = spec;
  double* left1 = spec + 2 * nmg;
  double* left2 = prpi;              // after the transform
  bool fft_products = false;
  if (fft_tc_fits(c, mesh[0], mesh[1], mesh[2], nmu) &&
      (st = fft_tc(c, mesh[0], mesh[1], mesh[2], nmu, false, zc, ivg, &fft_products)))
    return st;
  if (!fft_products) {
    ProfScope prof(c, "fft");
    for (int f0 = 0; f0 < nmu; f0 += kFftChunk) {
      const int nb = std::min(kFftChunk, nmu - f0);
      cufftHandle plan;
      if ((st = get_plan(c, mesh[0], mesh[1], mesh[2], nb, CUFFT_Z2Z, &plan))) return st;
      cufftDoubleComplex* src = (cufftDoubleComplex*)(zc + 2LL * ng * f0);
      if (cufftExecZ2Z(plan, src, (cufftDoubleComplex*)(ivg + 2LL * ng * f0), CUFFT_FORWARD) !=
          CUFFT_SUCCESS)
        return set_error(c, THC_ERR_CUFFT, "thc_isdf_half_complex: cufftExecZ2Z failed");
      c->launches++;
    }
  }
  double* vs = (double*)ws_get(c, WS_DSYM, sizeof(double) * ng);
  if (!vs) return set_error(c, THC_ERR_NOMEM, "thc_isdf_half_complex: Coulomb kernel");
  left_spectra<<<dim3((unsigned)cdiv(ng, 256), 16), 256, 0, s>>>(
      (const double2*)ivg, coul, mesh[0], mesh[1], mesh[2], fft_products, nmu, (double2*)left1,
      (double2*)left2, vs);
  THC_LAUNCHED(c, "left_spectra");
  c->zeta_last = nullptr;            // complex vectors: not served by the real accessor
  // M = sum_G v(G) IVMG_mu(G) IVG_nu(G) over (re, im) pairs: the real and the imaginary part.
  double* mr = Mw;
  double* mi = Mw + nn;
  {
    if (ng > 0x7fffffffLL) return set_error(c, THC_ERR_SHAPE, "thc_isdf_half_complex: mesh too large");
    constexpr long long kPart = 1LL << 30;           // the GEMM's K is an int
    for (long long k = 0; k < 2 * ng; k += kPart) {
      GemmArgs g;
      g.M = nmu; g.N = nmu; g.K = (int)std::min(kPart, 2 * ng - k);
      g.A = left1 + k; g.sam = 2 * ng; g.sak = 1;
      g.B = ivg + k; g.sbn = 2 * ng; g.sbk = 1;
      g.dk = vs + k / 2; g.dk_shift = 1;
      g.beta = k ? 1.0 : 0.0;
      g.C = mr; g.ldc = nmu;
      if ((st = dgemm(c, g))) return st;
      g.A = left2 + k;
      g.C = mi;
      if ((st = dgemm(c, g))) return st;
    }
  }
  double* mcx = Mw + 2 * nn;
  interleave<<<(int)cdiv(nn, 256), 256, 0, s>>>(mr, mi, nn, mcx);
  THC_LAUNCHED(c, "interleave");
  THC_CUDA(c, cudaEventRecord(c->ev1, s));
  if (out_M) THC_CUDA(c, cudaMemcpyAsync(out_M, mcx, sizeof(double) * 2 * nn, cudaMemcpyDefault, s));
  GjStatus hg{};
  int hbad = 0, herr = 0;
  THC_CUDA(c, cudaMemcpyAsync(&herr, c->tc64_err, sizeof(int), cudaMemcpyDeviceToHost, s));
  THC_CUDA(c, cudaMemcpyAsync(&hg, gs, sizeof(GjStatus), cudaMemcpyDeviceToHost, s));
  THC_CUDA(c, cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  THC_CUDA(c, cudaStreamSynchronize(s));
  if (hbad) return set_error(c, THC_ERR_ARG, "thc_isdf_half_complex: interpolating index out of range");
  if (herr)
    return set_error(c, THC_ERR_TIMEOUT, "thc_isdf_half_complex: tensor-core GEMM wait timed out");
  if (stats) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    stats->c_min_pivot = hg.max_abs2 > 0 ? hg.min_abs2 / hg.max_abs2 : 0.0;
    stats->chol_c_info = hg.singular;
    stats->device_ms = ms;
  }
  if (hg.singular)
    return set_error(c, THC_ERR_NOT_PD, "thc_isdf_half_complex: C is singular at column %d",
                     hg.singular);
  return THC_OK;
}

}  // namespace thc
