// FP64 3-D DFTs of many small fields as products with DFT matrices on the tensor cores.
//
// The reference transforms every interpolating vector with FFTW (fft_vectors,
// src/interpolating_vectors.cpp:331-404).  An FP64 FFT is bound by GB300's FP64 pipe (two
// operations a clock and SM): cuFFT took 2.39 of the 4.38 ms of a factorisation at N_g 48^3,
// N_mu 256.  A transform of length n along one axis is also a product with an n x n matrix, and
// dgemm_tc.cu's products cost about the same whatever n up to ~100, so the three axes run as
//     rows (field, x, y)   x (z)      -> (field, x, y, kz)
//     rows (field, x, kz)  x (y, re/im) -> (field, x, kz, ky)
//     rows (field, kz, ky) x (x, re/im) -> (field, kz, ky, kx)
// each complex product as a real one over (re, im) pairs.  Rows are what a product's A operand
// is cut by, so the result of one axis is cut across the next one and stored with that axis
// last; nothing is transposed on its own, and the spectrum comes out in (kz, ky, kx) order.
// Fields run in chunks that bound the buffers.  Every output is the rounded value
// of an exact sum over inputs of 55 bits and matrix entries of FP64, so its error is that of
// the entries' rounding, below the log n roundings of an FFT.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "dense64.cuh"
#include "digits64.cuh"
#include "fft_tc.cuh"
#include "ozgemm.cuh"

namespace thc {

namespace {

// Rows (s, q) over the middle axis of slabs [s][j][q] of complex values: k = (j, re/im).
struct SlabSrc {
  const double* x;
  long long rows;            // slabs x Q
  int Q, n;
};

// A block owns 64 rows: the maximum's pass reads along q, then 16 j x 64 rows at a time go
// through shared memory (as cut_cols does for a real matrix).
constexpr int kTR = 64;
__global__ void __launch_bounds__(256) cut_slab(SlabSrc a, Digits o, int* flag)
{
  __shared__ unsigned smx[4][kTR];
  __shared__ double t[32][kTR + 1];
  __shared__ int se[kTR];
  const long long r0 = blockIdx.x * (long long)kTR;
  const int rr = threadIdx.x & (kTR - 1), w = threadIdx.x / kTR;    // four j phases
  const long long r = r0 + rr;
  const bool live = r < a.rows;
  const long long s = live ? r / a.Q : 0;
  const double2* col = (const double2*)a.x + s * a.n * a.Q + (live ? r - s * a.Q : 0);
  unsigned mx = 0;
  if (live)
#pragma unroll 8
    for (int j = w; j < a.n; j += 4) {
      const double2 v = __ldg(col + (long long)j * a.Q);
      mx = max(mx, max(abs_hi(v.x), abs_hi(v.y)));
    }
  smx[w][rr] = mx;
  __syncthreads();
  if (threadIdx.x < kTR) {
    for (int q = 1; q < 4; q++) mx = max(mx, smx[q][rr]);
    const int e = row_exponent<CUT_PLAIN>(mx);
    se[rr] = e;
    o.e[r] = e;
    if (e == kNonFinite) atomicExch(flag, 1);
  }
  const int orow = threadIdx.x >> 2, oc = (threadIdx.x & 3) * 8;    // this thread's eight k
  for (int kt = 0; kt < (int)o.kpad; kt += 32) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int j = (kt >> 1) + w + 4 * q;
      double2 v = make_double2(0.0, 0.0);
      if (live && j < a.n) v = __ldg(col + (long long)j * a.Q);
      t[2 * (w + 4 * q)][rr] = v.x;
      t[2 * (w + 4 * q) + 1][rr] = v.y;
    }
    __syncthreads();
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = t[oc + j][orow];
    store8(o, r0 + orow, kt + oc, 1022 + se[orow], v);
  }
}

// Fields with a row that is not finite on any of the three axes (rows per field nz, ny, nx):
// the whole spectrum is NaN, as a transform's is.  One load when there is none.
__global__ void __launch_bounds__(256) fft_nonfinite(const int* ez, long long nz, const int* ey,
                                                     long long ny, const int* ex, long long nx,
                                                     double* out, long long len, const int* flag)
{
  if (!*flag) return;
  const long long f = blockIdx.x;
  bool bad = false;
  for (long long i = threadIdx.x; i < nz; i += blockDim.x) bad |= ez[f * nz + i] == kNonFinite;
  for (long long i = threadIdx.x; i < ny; i += blockDim.x) bad |= ey[f * ny + i] == kNonFinite;
  for (long long i = threadIdx.x; i < nx; i += blockDim.x) bad |= ex[f * nx + i] == kNonFinite;
  if (!__syncthreads_or(bad)) return;
  for (long long i = threadIdx.x; i < len; i += blockDim.x) out[f * len + i] = __longlong_as_double(0x7ff8000000000000LL);
}

// The digits of a DFT matrix, kept by the context: rows (k, re/im) of the forward transform
// over real inputs (half spectrum) or (re, im) pairs.
int dft_matrix(Ctx* c, int n, bool real, unsigned* rowmax, int* flag, Digits* out)
{
  const auto key = std::make_pair(n, real ? 1 : 0);
  auto it = c->dft.find(key);
  if (it == c->dft.end()) {
    const int nk = real ? n / 2 + 1 : n, K = real ? n : 2 * n, N = 2 * nk;
    std::vector<double> co(n), si(n), m((size_t)N * K);
    for (int i = 0; i < n; i++) {
      // Angles folded into [0, pi / 4], so that symmetric entries are equal to the last bit.
      const int q = 8 * i;                             // the angle in units of 2 pi / (8 n)
      auto ev = [&](int a, bool cosine) -> double {    // a in [0, 8n)
        bool neg = false;
        a %= 8 * n;
        if (a > 4 * n) { a = 8 * n - a; if (!cosine) neg = !neg; }
        if (a > 2 * n) { a = 4 * n - a; if (cosine) neg = !neg; }
        bool cs = cosine;
        if (a > n) { a = 2 * n - a; cs = !cs; }
        const long double x = 2.0L * 3.14159265358979323846264338327950288L * a / (8.0L * n);
        const double v = (double)(cs ? cosl(x) : sinl(x));
        return neg ? -v : v;
      };
      co[i] = ev(q, true);
      si[i] = ev(q, false);
    }
    for (int k = 0; k < nk; k++)
      for (int j = 0; j < n; j++) {
        const int a = (int)((long long)j * k % n);
        if (real) {
          m[(size_t)(2 * k) * K + j] = co[a];
          m[(size_t)(2 * k + 1) * K + j] = -si[a];
        } else {
          m[(size_t)(2 * k) * K + 2 * j] = co[a];
          m[(size_t)(2 * k) * K + 2 * j + 1] = si[a];
          m[(size_t)(2 * k + 1) * K + 2 * j] = -si[a];
          m[(size_t)(2 * k + 1) * K + 2 * j + 1] = co[a];
        }
      }
    const long long rp = oz_pad_mn(N), kp = oz_pad_k(K);
    const size_t dig = (size_t)rp * kp * kNS * 2;
    void* p = nullptr;
    double* md = (double*)ws_get(c, WS_FFTWORK, sizeof(double) * m.size());
    if (!md || cudaMallocAsync(&p, dig + sizeof(int) * rp, c->stream) != cudaSuccess) {
      cudaGetLastError();
      return THC_ERR_NOMEM;
    }
    THC_CUDA(c, cudaMemcpyAsync(md, m.data(), sizeof(double) * m.size(), cudaMemcpyHostToDevice,
                                c->stream));
    Digits d;
    d.s = (__nv_bfloat16*)p;
    d.e = (int*)((char*)p + dig);
    d.rows_pad = rp;
    d.kpad = kp;
    CutSrc a{md, N, K, 1, 0, K, nullptr, 0, K % 2 == 0};
    int st = digits_cut(c, a, d, rowmax, flag);
    if (st) {
      cudaFreeAsync(p, c->stream);
      return st;
    }
    THC_CUDA(c, cudaStreamSynchronize(c->stream));     // the host matrix goes out of scope
    it = c->dft.emplace(key, Ctx::Dft{p, rp, kp}).first;
  }
  const Ctx::Dft& f = it->second;
  out->s = (__nv_bfloat16*)f.p;
  out->e = (int*)((char*)f.p + (size_t)f.rows_pad * f.kpad * kNS * 2);
  out->rows_pad = f.rows_pad;
  out->kpad = f.kpad;
  return THC_OK;
}

}  // namespace

void dft_release(Ctx* c)
{
  for (auto& kv : c->dft) cudaFreeAsync(kv.second.p, c->stream);
  c->dft.clear();
}

bool fft_tc_fits(const Ctx* c, int n0, int n1, int n2, int count)
{
  return c->gemm_tc && std::max({n0, n1, n2}) <= kFftTcMaxN &&
         (double)n0 * n1 * n2 * count >= kFftTcMin;
}

int fft_tc(Ctx* c, int n0, int n1, int n2, int count, bool real, const double* in, double* out,
           bool* done)
{
  ProfScope prof(c, "fft");
  *done = false;
  const int nz = real ? n2 / 2 + 1 : n2, kin = real ? n2 : 2 * n2;
  const long long rz = (long long)n0 * n1, ry = (long long)n0 * nz, rx = (long long)nz * n1;
  const long long kz = oz_pad_k(kin), ky = oz_pad_k(2 * n1), kx = oz_pad_k(2 * n0);
  const size_t per = kNS * sizeof(__nv_bfloat16);
  const long long dig = std::max({rz * kz, ry * ky, rx * kx});         // per field
  const int F = (int)std::min<long long>(count, (long long)(std::min(c->digit_bytes / 4, kFftTcChunk) / (dig * per)));
  if (F < 1) return THC_OK;
  auto padded = [&](long long rows, long long kp) { return (size_t)oz_pad_mn(F * rows) * kp * per; };
  const long long e_rows = oz_pad_mn(F * rz) + oz_pad_mn(F * ry) + oz_pad_mn(F * rx);
  const size_t t1 = sizeof(double) * 2 * F * rz * nz, t2 = sizeof(double) * 2 * F * ry * n1;
  char* flags = (char*)ws_get(c, WS_T64_E, 256 + sizeof(int) * e_rows +
                                               sizeof(unsigned) * std::max<long long>(oz_pad_mn(F * rz), 1024));
  __nv_bfloat16* ds = (__nv_bfloat16*)ws_get(
      c, WS_T64_A, std::max({padded(rz, kz), padded(ry, ky), padded(rx, kx)}));
  if (!flags || !ds) return THC_OK;
  int* flag = (int*)flags;
  unsigned* rowmax = (unsigned*)(flags + 256);
  int* e0 = (int*)(rowmax + std::max<long long>(oz_pad_mn(F * rz), 1024));
  THC_CUDA(c, cudaMemsetAsync(flag, 0, sizeof(int), c->stream));
  int st;
  Digits mz, my, mx;
  if (c->dft.size() > 61) dft_release(c);              // at most 64 are kept
  if ((st = dft_matrix(c, n2, real, rowmax, flag, &mz)) ||
      (st = dft_matrix(c, n1, false, rowmax, flag, &my)) ||
      (st = dft_matrix(c, n0, false, rowmax, flag, &mx)))
    return st == THC_ERR_NOMEM ? THC_OK : st;
  // After the matrices: their staging shares the slot.
  char* tw = (char*)ws_get(c, WS_FFTWORK, t1 + t2 + 256);
  if (!tw) return THC_OK;
  double* a1 = (double*)tw;
  double* a2 = (double*)(tw + (t1 + 255) / 256 * 256);
  for (int f0 = 0; f0 < count; f0 += F) {
    const int nf = std::min(F, count - f0);
    Digits d;
    d.s = ds;
    auto axis = [&](const Digits& m, long long rows, int N, double* dst) -> int {
      GemmArgs g;
      g.M = rows; g.N = N;
      g.C = dst; g.ldc = N;
      return digits_product(c, d, m, g);
    };
    auto slab = [&](const double* x, long long rows, int Q, int n, long long kp, int* e) -> int {
      d.e = e;
      d.rows_pad = oz_pad_mn(rows);
      d.kpad = kp;
      SlabSrc a{x, rows, Q, n};
      ProfScope p2(c, "slice64");
      cut_slab<<<(unsigned)(d.rows_pad / kTR), 256, 0, c->stream>>>(a, d, flag);
      THC_LAUNCHED(c, "cut_slab");
      return THC_OK;
    };
    int* ez = e0;
    int* ey = ez + oz_pad_mn(F * rz);
    int* ex = ey + oz_pad_mn(F * ry);
    const double* src = in + (size_t)f0 * n0 * n1 * kin;
    d.e = ez;
    d.rows_pad = oz_pad_mn(nf * rz);
    d.kpad = kz;
    CutSrc a{src, nf * rz, kin, 1, 0, kin, nullptr, 0, kin % 2 == 0 && (uintptr_t)src % 16 == 0};
    if ((st = digits_cut(c, a, d, rowmax, flag))) return st;
    if ((st = axis(mz, nf * rz, 2 * nz, a1))) return st;
    if ((st = slab(a1, nf * ry, nz, n1, ky, ey))) return st;
    if ((st = axis(my, nf * ry, 2 * n1, a2))) return st;
    if ((st = slab(a2, nf * rx, nz * n1, n0, kx, ex))) return st;
    double* dst = out + (size_t)f0 * 2 * rx * n0;
    if ((st = axis(mx, nf * rx, 2 * n0, dst))) return st;
    fft_nonfinite<<<nf, 256, 0, c->stream>>>(ez, rz, ey, ry, ex, rx, dst, 2 * rx * n0, flag);
    THC_LAUNCHED(c, "fft_nonfinite");
  }
  *done = true;
  return THC_OK;
}

}  // namespace thc
