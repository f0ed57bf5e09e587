// FP64 GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA): dgemm()'s route for
// large products (dense64.cuh).
//
// GB300 issues two FP64 FMAs per clock and SM (1.25 TFLOP/s on the chip, tensor or not) but
// 2 PFLOP/s of BF16, so an FP64 product is cut into exact BF16 pieces.  Each row of A (each
// column of B) is taken relative to its largest entry, |x| < 2^e, to the 55-bit integer
// R = round(x 2^{55-e}) and split into seven balanced base-256 digits,
//     x = 2^{e-7} sum_{i<7} S_i 2^{-8i},   |S_i| <= 128,
// every digit an integer that BF16 holds exactly.  The product keeps the digit pairs with
// i + j <= 7 (34 of them):
//     C[m,n] = 2^{eA[m]+eB[n]-14} sum_{l<=7} 2^{-8l} V_l,   V_l = sum_{i+j=l} sum_k S_i T_j.
// The tensor cores sum V_l in FP32, exactly for l <= 4: over the 192 k between two drains
// |V_l| <= 5 192 2^14 < 2^24.  Levels 5 to 7 (weight <= 2^-40) could pass 2^24 only with
// digits of one sign throughout, and then round by less than 2^-55 of the sum.  A drain adds the
// sums to 96-bit integers in registers, which hold the sum over any K without rounding; it is
// rounded once, half away from zero, a negative one taken one unit (2^-70 2^{eA+eB}) smaller.  C is
// about 2^-57 sqrt(K) off relative to 2^{eA+eB}, where a chain of FP64 FMAs over terms of that
// size is 2^-54 sqrt(K) and more.  Where a row's entries meet small ones of the other operand
// only, the FMAs' error, relative to the terms, is the smaller one: operands that scale against
// each other along k are balanced first (GemmArgs::kexp; kBalancedBinades in dense64.cuh).
//
// Measured against the FMA kernel of dense64.cu, cut and product together (random operands of one
// size; errors relative to |a||b| of an entry's row and column, root mean square):
//     M x N x K                     FMA              tensor cores
//     256 x 110592 x 256            11.8 ms 3.4e-17  0.54 ms 3.7e-18   (27 TFLOP/s)
//     256 x 110592 x 32, squared    1.54 ms 3.5e-17  0.21 ms 9.9e-18
//     256 x 256 x 115200, lower     15.9 ms 2.6e-16  0.47 ms 9.5e-18
//     1024 x 1024 x 215040, lower    340 ms 7.2e-16  6.6 ms 4.8e-18   (69 TFLOP/s)
// What bounds the product is shared memory: the eleven MMAs of 16 k read 112 KB and the copies
// write 43 KB, 1211 clocks at 128 B, against 1088 of tensor work; without the drains 1350
// clocks are measured, with them 1580.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "dense64.cuh"
#include "digits64.cuh"
#include "ozgemm.cuh"
#include "tc_ptx.cuh"

namespace thc {

namespace {

constexpr int kLv = 8;                   // levels, one accumulator each
constexpr int kPeriod = 6;               // stages between drains: 192 k
constexpr int kBN = 64;                  // tile width (128 x 64: eight TMEM slots of 64 columns)
constexpr int kBK = 32;                  // k per pipeline stage
constexpr int kStages = 2;
constexpr int kABytes = TBM * kBK * 2;   // one digit tile of A
constexpr int kBBytes = kBN * kBK * 2;
constexpr int kStageBytes = kNS * (kABytes + kBBytes);
constexpr int kEpiWarps = 16;              // four per TMEM lane quadrant, 16 columns each
constexpr int kEC = 16;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr int kStgBytes = kEpiWarps * 32 * 8 * 8;   // results on their way to coalesced stores
constexpr size_t kSmem = 1024 + (size_t)kStages * kStageBytes + kStgBytes + 256 + 1024 + 8192;
static_assert(kSmem <= 227 * 1024, "shared memory");
static_assert(kStageBytes % 1024 == 0, "stage alignment");
// Level 4 is exact in FP32 between two drains, and level 0 (|S T| <= 2^14 a term) stays within the
// 2^22 that the epilogue's addition of 1.5 2^23 takes.
static_assert(5LL * kPeriod * kBK * (1 << 14) < (1 << 24), "exact levels");
static_assert((long long)kPeriod * kBK * (1 << 14) <= (1 << 22), "level 0");

constexpr long long kPair = 0x8b400000LL;  // 257 x the bits of 1.5 2^23, modulo 2^32

// ---- cutting an operand into digits (digits64.cuh) --------------------------------------

__device__ __forceinline__ void load8(const CutSrc& a, long long r, int k, double (&v)[8])
{
  const double* p = a.x + r * a.sr + (long long)(a.k0 + k) * a.sk;
  if (a.vec && k + 8 <= a.K) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const double2 t = __ldg((const double2*)p + q);
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = k + j < a.K ? __ldg(p + j * a.sk) : 0.0;
  }
}

__device__ __forceinline__ double scale_at(const CutSrc& a, int k)
{
  return k < a.K ? __ldg(a.scale + ((a.k0 + k) >> a.shift)) : 0.0;
}

__device__ __forceinline__ int shift_at(const CutSrc& a, int k)
{
  return k < a.K ? a.ksign * __ldg(a.kexp + a.k0 + k) : 0;
}

// The row maximum's contribution of x at column k.
template <CutScale SC>
__device__ __forceinline__ unsigned field_at(const CutSrc& a, int k, double x)
{
  if constexpr (SC == CUT_SCALED) return (unsigned)field_of(x, scale_at(a, k));
  if constexpr (SC == CUT_SHIFTED) return field_shifted(x, shift_at(a, k));
  return abs_hi(x);
}

// The maximum's contribution of eight columns.
template <CutScale SC>
__device__ __forceinline__ unsigned max8(const CutSrc& a, int k, const double (&v)[8], unsigned mx)
{
#pragma unroll
  for (int j = 0; j < 8; j++) mx = max(mx, field_at<SC>(a, k + j, v[j]));
  return mx;
}

template <CutScale SC>
__device__ __forceinline__ void scale8(const CutSrc& a, int k, double (&v)[8])
{
  if constexpr (SC == CUT_SCALED) {
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] *= scale_at(a, k + j);
  }
}

// Columns k .. k + 7 of row r, scaled already, as digits relative to 2^e.
template <CutScale SC>
__device__ __forceinline__ void cut8(const CutSrc& a, const Digits& o, long long r, int k, int e,
                                     const double (&v)[8])
{
  if constexpr (SC == CUT_SHIFTED)
    store8(o, r, k, 1022 + e, v, [&](int j) { return shift_at(a, k + j); });
  else
    store8(o, r, k, 1022 + e, v);
}

// Short rows (K <= kFusedK, k contiguous or nearly): lpr lanes per row, eight columns per
// lane and step, the row read twice (the second time from L1/L2).
constexpr int kFusedK = 4096;
template <CutScale SC>
__global__ void __launch_bounds__(256) cut_rows(CutSrc a, Digits o, int lpr, int* flag)
{
  const int lane = threadIdx.x & 31, sub = lane & (lpr - 1);
  const long long warp = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const long long r = warp * (32 / lpr) + lane / lpr;
  const bool live = r < a.rows;
  unsigned mx = 0;
  double v[8] = {};
  if (live)
    for (int k = 8 * sub; k < a.K; k += 8 * lpr) {
      load8(a, r, k, v);
      mx = max8<SC>(a, k, v, mx);
    }
  for (int off = lpr >> 1; off; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if (r >= o.rows_pad) return;
  const int e = row_exponent<SC>(mx);
  if (sub == 0) {
    o.e[r] = e;
    if (e == kNonFinite) atomicExch(flag, 1);
  }
  for (int k = 8 * sub; k < (int)o.kpad; k += 8 * lpr) {
    if (live && k < a.K) {
      // A row read in one step keeps its values from the maximum's pass.
      if (o.kpad > 8 * lpr) load8(a, r, k, v);
      scale8<SC>(a, k, v);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = 0.0;
    }
    cut8<SC>(a, o, r, k, e, v);
  }
}

// Long rows (the Coulomb product's K = 2 N_c): row maxima by column chunks, then the digits,
// each with the whole GPU on a few rows.
constexpr int kMaxChunk = 4096;
template <CutScale SC>
__global__ void __launch_bounds__(256) cut_rowmax(CutSrc a, int nch, unsigned* rowmax)
{
  const long long r = blockIdx.x / nch;
  const int c0 = (int)(blockIdx.x % nch) * kMaxChunk, c1 = min(a.K, c0 + kMaxChunk);
  unsigned mx = 0;
  double v[8];
  for (int k = c0 + 8 * threadIdx.x; k < c1; k += 2048) {
    load8(a, r, k, v);
    mx = max8<SC>(a, k, v, mx);
  }
  for (int off = 16; off; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(&rowmax[r], mx);
}

template <CutScale SC>
__global__ void __launch_bounds__(256) cut_long(CutSrc a, Digits o, int nch,
                                                const unsigned* __restrict__ rowmax, int* flag)
{
  const long long r = blockIdx.x / nch;
  const int ch = (int)(blockIdx.x % nch);
  const int k = (ch * 256 + threadIdx.x) * 8;
  const bool live = r < a.rows;
  const int e = live ? row_exponent<SC>(rowmax[r]) : 0;
  if (k == 0) {
    o.e[r] = e;
    if (e == kNonFinite) atomicExch(flag, 1);
  }
  if (k >= (int)o.kpad) return;
  double v[8] = {};
  if (live && k < a.K) {
    load8(a, r, k, v);
    scale8<SC>(a, k, v);
  }
  cut8<SC>(a, o, r, k, e, v);
}

// Row-contiguous operands (sr == 1: Z^T, N_mu x N_g, as the B of the zeta product): a block
// owns 64 rows; the maximum's pass reads coalesced along the rows, the second pass turns
// 32 k x 64 rows at a time through shared memory.
constexpr int kTR = 64;
template <CutScale SC>
__global__ void __launch_bounds__(256) cut_cols(CutSrc a, Digits o, int* flag)
{
  __shared__ unsigned smx[4][kTR];
  __shared__ double t[32][kTR + 1];
  __shared__ int se[kTR];
  const long long r0 = blockIdx.x * (long long)kTR;
  const int rr = threadIdx.x & (kTR - 1), w = threadIdx.x / kTR;    // four k phases
  const bool live = r0 + rr < a.rows;
  const double* col = a.x + r0 + rr + (long long)a.k0 * a.sk;
  unsigned mx = 0;
  if (live)
#pragma unroll 8
    for (int k = w; k < a.K; k += 4) {
      const double x = __ldg(col + k * a.sk);
      mx = max(mx, field_at<SC>(a, k, x));
    }
  smx[w][rr] = mx;
  __syncthreads();
  if (threadIdx.x < kTR) {
    for (int q = 1; q < 4; q++) mx = max(mx, smx[q][rr]);
    const int e = row_exponent<SC>(mx);
    se[rr] = e;
    o.e[r0 + rr] = e;
    if (e == kNonFinite) atomicExch(flag, 1);
  }
  const int orow = threadIdx.x >> 2, oc = (threadIdx.x & 3) * 8;    // this thread's eight k
  for (int kt = 0; kt < (int)o.kpad; kt += 32) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int k = kt + w + 4 * q;
      double x = 0.0;
      if (live && k < a.K) {
        x = __ldg(col + k * a.sk);
        if (SC == CUT_SCALED) x *= scale_at(a, k);
      }
      t[w + 4 * q][rr] = x;
    }
    __syncthreads();
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = t[oc + j][orow];
    cut8<SC>(a, o, r0 + orow, kt + oc, se[orow], v);
  }
}

// ---- the product ------------------------------------------------------------------------

struct Args {
  long long M, N;
  int stages;              // 32-k stages of the panel
  int ksplit, kt_per;      // k tiles per split
  const int* ea;
  const int* eb;
  double* C;
  long long ldc;
  double alpha, beta;
  int square, scaled, added;   // epilogue: the square, alpha != 1, beta != 0 (not with a split)
  int lower;
  unsigned two8, two16;    // 2^8 and 2^16: factors of integer multiply-adds, opaque (constants
                           // become shifts on the integer pipe)
  double* part;
  int* error;
  long long spin_limit;
  unsigned mtn, ntn, tiles;  // 32-bit: a 64-bit division is a hundred instructions, per warp
                             // and tile
};

constexpr int kGroupM = 16;    // m-tiles swept per n-tile: the CTAs of a wave share B tiles

__device__ __forceinline__ void tile_of(const Args& g, unsigned t, unsigned& mt, unsigned& nt)
{
  if (g.lower) {
    // Row i of 128 x 64 tiles reaches column 2i + 1: it starts at tile i (i + 1).
    unsigned i = (unsigned)((sqrtf(4.f * (float)t + 1.f) - 1.f) * 0.5f);
    while (i * (i + 1) > t) i--;
    while ((i + 1) * (i + 2) <= t) i++;
    mt = i;
    nt = t - i * (i + 1);
    return;
  }
  const unsigned per = kGroupM * g.ntn, grp = t / per, first = grp * kGroupM;
  const unsigned gm = min(g.mtn - first, (unsigned)kGroupM), r = t - grp * per;
  nt = r / gm;
  mt = first + r - nt * gm;
}

// 2^E v by ldexp: results that leave FP64's normal range.
__device__ __noinline__ double wide_double(unsigned hi, unsigned lo, int E, unsigned sign)
{
  const double v = ldexp((double)(((unsigned long long)hi << 32) | lo), E);
  return sign ? -v : v;
}

// The 96-bit integer (w2, w1, w0) times 2^E, rounded once to FP64 (half away from zero), in
// 32-bit integer arithmetic: the magnitude, its leading one brought to bit 63 of the top two
// words, and 53 bits of those with a rounding bit.  (Conversions and an FMA would be four
// operations of the FP64 pipe, 16,000 clocks a tile.)
template <bool WIDE>
__device__ __forceinline__ double to_double(unsigned w0, unsigned w1, unsigned w2, int E,
                                            bool& wide)
{
  // The magnitude as the one's complement of a negative sum: a unit of 2^-70 2^{eA+eB} less,
  // far below the expansion's truncation.
  const unsigned neg = (unsigned)((int)w2 >> 31);
  w0 ^= neg;
  w1 ^= neg;
  w2 ^= neg;
  const bool zero = (w0 | w1 | w2) == 0;
  int be = E + 95 + 1022;                             // biased exponent of bit 95, less one
  if (!w2) { w2 = w1; w1 = w0; w0 = 0; be -= 32; }
  if (WIDE) {
    if (zero) return 0.0;
    if (!w2) { w2 = w1; w1 = 0; be -= 32; }
  }
  const int n = __clz((int)w2);
  be -= n;
  const unsigned t1 = __funnelshift_l(w1, w2, n), t0 = __funnelshift_l(w0, w1, n);
  if (WIDE && (unsigned)be > 2044u) return wide_double(t1, t0, be - 1022 - 63, neg);
  wide |= !zero && ((unsigned)be > 2044u || !w2);
  unsigned m0 = __funnelshift_r(t0, t1, 11), m1 = (t1 >> 11) + ((unsigned)be << 20);
  asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, 0;\n"
      : "+r"(m0), "+r"(m1) : "r"((t0 >> 10) & 1u));
  m1 |= neg & 0x80000000u;
  return zero ? 0.0 : __hiloint2double((int)m1, (int)m0);
}

// One CTA per SM walks the items (tile, split of K).  Warp 0 is the TMA producer, warp 1
// allocates TMEM and issues the MMAs, warps 2-17 drain and store.  The eight level
// accumulators of a 128 x 64 tile fill TMEM (64 columns each, level l at column 64 l), so one
// MMA multiplies digit i of A with up to four digits of B at once: their tiles lie behind one
// another in shared memory, their products in the columns of consecutive levels.  A 16-k
// stage is 11 MMAs of up to 128 x 256 instead of 34 of 128 x 64, at the full rate of the
// tensor pipe (with one MMA per pair, each reads 6 KB of shared memory for 32 clocks of work
// and is issued alone: 0.996 ms for the zeta product at N_g 110592, N_mu 256, against 0.47 at
// once with these and 0.38 now).  Stages of 32 k with the 64-byte swizzle are 5 % faster than
// stages of 16 k with the 32-byte one.
// Every kPeriod stages (192 k) the levels are drained from the highest down; the next stage
// multiplies the lowest digits of A first and so follows the drain level by level instead of
// waiting for all of it.  Every wait is bounded (spin_limit); after one gives up, the kernel sets the
// error flag, waits for its own copies and MMAs, frees TMEM and returns.
// Digit i of A times digits j .. j + CNT - 1 of B, into levels i + j and up; a0 / b0 are the
// low descriptor words of the stage's operands.
template <int CNT>
__device__ __forceinline__ void mma_digits(uint32_t tmem, uint32_t a0, uint32_t b0, int i, int j,
                                           uint32_t acc)
{
  umma_lo<CNT * kBN, kBK>(tmem + (uint32_t)((i + j) * kBN), a0 + (uint32_t)(i * kABytes >> 4),
                          b0 + (uint32_t)(j * kBBytes >> 4), acc);
}

// Digit i of A times every digit j >= j0 of B with i + j <= 7, accumulated.
__device__ __forceinline__ void mma_run(uint32_t tmem, uint32_t a0, uint32_t b0, int i, int j0)
{
  const int end = (i == 0 ? kNS - 1 : kLv - 1 - i) + 1;
  int j = j0;
  if (end - j >= 4) { mma_digits<4>(tmem, a0, b0, i, j, 1u); j += 4; }
  if (end - j == 3) mma_digits<3>(tmem, a0, b0, i, j, 1u);
  else if (end - j == 2) mma_digits<2>(tmem, a0, b0, i, j, 1u);
  else if (end - j == 1) mma_digits<1>(tmem, a0, b0, i, j, 1u);
}

__global__ void __launch_bounds__(kThreads, 1)
    dgemm_tc_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                    Args g)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* stg_base = smem + kStages * kStageBytes;
  uint64_t* full = (uint64_t*)(stg_base + kStgBytes);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;      // the period's sums are final
  uint64_t* lev_free = acc_full + 1;         // [8] the level has been drained
  uint64_t* mma_done = lev_free + kLv;
  uint32_t* tmem_slot = (uint32_t*)(mma_done + 1);
  volatile int* abort = (volatile int*)(tmem_slot + 1);
  volatile int* issued = abort + 1;
  volatile int* consumed = issued + 1;
  int* sexp = (int*)((unsigned char*)full + 256);   // 16 warps x 16 column exponents

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned items = g.tiles * g.ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    for (int l = 0; l < kLv; l++) mbar_init(&lev_free[l], kEpiWarps);
    mbar_init(mma_done, 1);
    *abort = 0;
    *issued = 0;
    *consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(
                     su32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  const uint32_t tmem = *tmem_slot;

  // First stage and stage count of item t, and its tile.
  auto item_of = [&](unsigned t, unsigned& mt, unsigned& nt, int& st0, int& nst) {
    const unsigned z = g.ksplit > 1 ? t / g.tiles : 0u;
    tile_of(g, t - z * g.tiles, mt, nt);
    st0 = z * g.kt_per;
    nst = min(g.stages - st0, g.kt_per);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int git = 0;
      bool ok = true;
      for (unsigned t = blockIdx.x; t < items && ok; t += gridDim.x) {
        unsigned mt, nt;
        int st0, nst;
        item_of(t, mt, nt, st0, nst);
        for (int it = 0; it < nst; it++, git++) {
          const int s = git % kStages;
          if (!mbar_wait(&empty[s], (uint32_t)((git / kStages) & 1) ^ 1, abort, g.spin_limit)) {
            ok = false;
            break;
          }
          unsigned char* st = smem + s * kStageBytes;
          *issued = git + 1;
          mbar_expect_tx(&full[s], kStageBytes);
          const int y = (st0 + it) * kNS;
          tma_load_3d(st, &ta, 0, (int)(mt * TBM), y, &full[s]);
          tma_load_3d(st + kNS * kABytes, &tb, 0, (int)(nt * kBN), y, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int git = 0;
      uint32_t pc = 0;               // periods begun
      bool ok = true;
      for (unsigned t = blockIdx.x; t < items && ok; t += gridDim.x) {
        unsigned mt, nt;
        int st0, nst;
        item_of(t, mt, nt, st0, nst);
        int in_period = 0;
        for (int it = 0; it < nst; it++, git++) {
          const int s = git % kStages;
          if (!mbar_wait(&full[s], (uint32_t)((git / kStages) & 1), abort, g.spin_limit)) {
            ok = false;
            break;
          }
          *consumed = git + 1;
          asm volatile("tcgen05.fence::after_thread_sync;\n");
          const uint32_t sa = su32(smem + s * kStageBytes);
          const uint32_t a0 = sdesc_lo(sa), b0 = sdesc_lo(sa + kNS * kABytes);
          if (in_period == 0) {
            // The period's first stage: level i is free once drained, and its first pair
            // (i, 0) overwrites it; the levels above it are in use already.
            const uint32_t par = (pc & 1u) ^ 1u;
            pc++;
            ok = mbar_wait(&lev_free[7], par, abort, g.spin_limit);
#pragma unroll
            for (int i = kNS - 1; i >= 0; i--) {
              ok = ok && mbar_wait(&lev_free[i], par, abort, g.spin_limit);
              if (!ok) break;
              asm volatile("tcgen05.fence::after_thread_sync;\n");
              if (i == kNS - 1) {
                mma_digits<2>(tmem, a0, b0, i, 0, 0u);
              } else {
                mma_digits<1>(tmem, a0, b0, i, 0, 0u);
                mma_run(tmem, a0, b0, i, 1);
              }
            }
            if (!ok) break;
          } else {
#pragma unroll
            for (int i = 0; i < kNS; i++) mma_run(tmem, a0, b0, i, 0);
          }
          // The stage's second 16 k: 32 bytes further in every row.
#pragma unroll
          for (int i = 0; i < kNS; i++) mma_run(tmem, a0 + 2, b0 + 2, i, 0);
          umma_commit(&empty[s]);
          if (++in_period == kPeriod || it + 1 == nst) {
            umma_commit(acc_full);
            in_period = 0;
          }
        }
      }
      umma_commit(mma_done);
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int ew = warp - 2;
    const int quad = warp & 3;               // TMEM lane quadrant this warp may access
    const int col0 = (ew >> 2) * kEC;        // this warp's columns of the tile
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    int* seb = sexp + ew * kEC;
    double* stg = (double*)(stg_base + (size_t)ew * (32 * 8 * 8));
    uint32_t pc = 0;                         // periods drained
    bool ok = true;
    for (unsigned t = blockIdx.x; t < items && ok; t += gridDim.x) {
      unsigned mt, nt;
      int st0, nst;
      item_of(t, mt, nt, st0, nst);
      const long long m0 = (long long)mt * TBM, n0 = (long long)nt * kBN;
      if (lane < kEC) {
        const long long na = n0 + col0 + lane;
        seb[lane] = na < g.N ? g.eb[na] : 0;
      }
      const long long m = m0 + quad * 32 + lane;
      const int ea = (m < g.M ? g.ea[m] : 0) - 70;   // unit of the sums: 2^{-14 - 56}
      __syncwarp();
      // Sums of this thread's row, 16 columns, as 96-bit integers in units of 2^-56 (a set of
      // 64-bit pairs took 16 registers more and spilled), less what the drains add too much.
      unsigned w0[kEC], w1[kEC], w2[kEC];
      {
        const unsigned __int128 x = (unsigned __int128)((unsigned)((nst + kPeriod - 1) / kPeriod)) *
                                    kPair * 0x0001000100010001ULL;
#pragma unroll
        for (int q = 0; q < kEC; q++) {
          w0[q] = (unsigned)(0 - x);
          w1[q] = (unsigned)((0 - x) >> 32);
          w2[q] = (unsigned)((0 - x) >> 64);
        }
      }
      // P = 256 V_l + V_{l+1} of eight columns, plus kPair, in 32 bits: V plus a constant is
      // the bits of V + 1.5 2^23, exactly while |V| <= 2^22.  That always holds for level 0;
      // the squares of the others add up to `sq`, which stays below 2^43 unless their digits
      // have one sign nearly throughout.  (The sum runs on the FMA pipe; the integer pipe is
      // the one the epilogue fills.)
      auto pair8 = [&](uint32_t src, unsigned (&P)[8], float& sq, bool level0) {
        float a[8], c[8];
        tmem_ld8x2(src, src + kBN, a, c);
#pragma unroll
        for (int q = 0; q < 8; q++) {
          if (!level0) sq = __fmaf_rn(a[q], a[q], sq);
          sq = __fmaf_rn(c[q], c[q], sq);
          P[q] = __float_as_uint(__fadd_rn(a[q], 12582912.f)) * g.two8 +
                 __float_as_uint(__fadd_rn(c[q], 12582912.f));
        }
      };
      // Warps past the last column have nothing to collect or store.
      const bool act = n0 + col0 < g.N;
      for (int st = 0; st < nst; st += kPeriod, pc++) {
        if (!mbar_wait(acc_full, pc & 1u, abort, g.spin_limit)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n");
#pragma unroll
        for (int l = 4; l >= 0; l -= 4) {      // levels 4-7, then 0-3
#pragma unroll
          for (int b = 0; b < kEC && act; b += 8) {
            const uint32_t src = tmem + lane_base + (uint32_t)(l * kBN + col0 + b);
            unsigned P[8], Q[8];
            float sq = 0.f;
            pair8(src + 2 * kBN, P, sq, false);
            pair8(src, Q, sq, l == 0);
            if (!__any_sync(0xffffffffu, !(sq < 0x1p43f))) {
#pragma unroll
              for (int q = 0; q < 8; q++) {
                // 2^16 Q + P, 48 bits, at bit 0 (levels 4-7) or bit 32.
                unsigned long long x = P[q];
                asm("mad.wide.u32 %0, %1, %2, %0;\n" : "+l"(x) : "r"(Q[q]), "r"(g.two16));
                const unsigned lo = (unsigned)x, hi = (unsigned)(x >> 32);
                if (l)
                  asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, 0;\n"
                      : "+r"(w0[b + q]), "+r"(w1[b + q]), "+r"(w2[b + q]) : "r"(lo), "r"(hi));
                else
                  asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, %3;\n"
                      : "+r"(w1[b + q]), "+r"(w2[b + q]) : "r"(lo), "r"(hi));
              }
            } else {
              // By conversion (16 a clock and SM), level by level.
#pragma unroll 1
              for (int j = 0; j < 4; j++) {
                float v[8];
                tmem_ld8(src + (uint32_t)(j * kBN), v);
                const long long weight = 1LL << (24 - 8 * j);
                const long long more = j & 1 ? kPair << (j == 1 ? 16 : 0) : 0;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                  const long long x = __float2int_rn(v[q]) * weight + more;
                  const unsigned lo = (unsigned)x, hi = (unsigned)(x >> 32);
                  const unsigned top = (unsigned)(x >> 63);
                  if (l)
                    asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, %5;\n"
                        : "+r"(w0[b + q]), "+r"(w1[b + q]), "+r"(w2[b + q])
                        : "r"(lo), "r"(hi), "r"(top));
                  else
                    asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, %3;\n"
                        : "+r"(w1[b + q]), "+r"(w2[b + q]) : "r"(lo), "r"(hi));
                }
              }
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;\n");
          __syncwarp();
          if (lane < 4) mbar_arrive(&lev_free[l + lane]);
        }
      }
      if (!ok) break;
      if (!act) continue;
      const long long ld = g.ksplit > 1 ? g.N : g.ldc;
      double* base = g.ksplit > 1 ? g.part + (long long)(t / g.tiles) * g.M * g.N : g.C;
      // A tile inside the matrix with 16-byte aligned rows needs no checks per store.
      const bool whole = m0 + TBM <= g.M && n0 + kBN <= g.N && !g.lower && !g.added &&
                         !(ld & 1) && !((uintptr_t)base & 15);
#pragma unroll
      for (int b = 0; b < 2; b++) {          // 8 columns at a time through shared memory
        // Staging: row `lane`, pairs of columns swizzled so that 16-byte accesses spread over
        // the banks both ways.
        double2* row = (double2*)stg + lane * 4;
        const int sw = (lane >> 1) & 3;
        bool wide = false;
#pragma unroll
        for (int q = 0; q < 8; q += 2)
          row[(q >> 1) ^ sw] = make_double2(
              to_double<false>(w0[8 * b + q], w1[8 * b + q], w2[8 * b + q], ea + seb[8 * b + q],
                               wide),
              to_double<false>(w0[8 * b + q + 1], w1[8 * b + q + 1], w2[8 * b + q + 1],
                               ea + seb[8 * b + q + 1], wide));
        if (__any_sync(0xffffffffu, wide)) {
          // Rare: a result outside FP64's normal range, or below 2^-38 of 2^{eA+eB}.
#pragma unroll
          for (int q = 0; q < 8; q += 2)
            row[(q >> 1) ^ sw] = make_double2(
                to_double<true>(w0[8 * b + q], w1[8 * b + q], w2[8 * b + q], ea + seb[8 * b + q],
                                wide),
                to_double<true>(w0[8 * b + q + 1], w1[8 * b + q + 1], w2[8 * b + q + 1],
                                ea + seb[8 * b + q + 1], wide));
        }
        if (g.square) {                      // (the barriers keep these branches branches: a
          __syncwarp();                      // predicated-off FP64 operation costs its slot)
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const double2 v = row[q];
            row[q] = make_double2(__dmul_rn(v.x, v.x), __dmul_rn(v.y, v.y));
          }
        } else if (g.scaled) {
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const double2 v = row[q];
            row[q] = make_double2(v.x * g.alpha, v.y * g.alpha);
          }
        }
        __syncwarp();
        // Eight rows per pass: 4 lanes per row, two adjacent columns per lane.
        const long long n = n0 + col0 + 8 * b + 2 * (lane & 3);
        const long long r1 = m0 + quad * 32 + (lane >> 2);
        double* dst = base + r1 * ld + n;
        const double2* src = (const double2*)stg + (lane >> 2) * 4 + ((lane & 3) ^ ((lane >> 3) & 3));
        if (whole) {
#pragma unroll
          for (int r0 = 0; r0 < 32; r0 += 8) *(double2*)(dst + r0 * ld) = src[r0 * 4];
        } else {
          for (int r0 = 0; r0 < 32; r0 += 8) {
            const long long mr = r1 + r0;
            if (mr >= g.M) break;
            const bool v0 = n < g.N && !(g.lower && n > mr);
            const bool v1 = n + 1 < g.N && !(g.lower && n + 1 > mr);
            double2 v = src[r0 * 4];
            double* p = dst + r0 * ld;
            if (g.added) {
              if (v0) v.x += g.beta * p[0];
              if (v1) v.y += g.beta * p[1];
            }
            if (v0 && v1 && !((uintptr_t)p & 15)) {
              *(double2*)p = v;
            } else {
              if (v0) p[0] = v.x;
              if (v1) p[1] = v.y;
            }
          }
        }
        __syncwarp();   // the staging and the exponents are rewritten
      }
    }
  }
  // ---------------------------------------------------------------------- teardown
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  if (threadIdx.x == 0) {
    if (*abort) {
      atomicExch(g.error, 1);
      for (int it = *consumed; it < *issued; it++)
        mbar_drain(&full[it % kStages], (uint32_t)((it / kStages) & 1));
    }
    mbar_drain(mma_done, 0);
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
  }
}

// Entries whose row of A or column of B holds an Inf or NaN (their digits are zero): the FP64
// sum itself, added to what the product left there (beta C, or 0).  Does nothing, after one
// load, when there is no such row.
__global__ void __launch_bounds__(256) fix_nonfinite(GemmArgs g, int k0, int K,
                                                     const int* __restrict__ ea,
                                                     const int* __restrict__ eb,
                                                     const int* __restrict__ flag)
{
  if (!*flag) return;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < g.M * g.N; e += gridDim.x * 256LL) {
    const long long m = e / g.N, n = e % g.N;
    if ((g.lower_only && n > m) || (ea[m] != kNonFinite && eb[n] != kNonFinite)) continue;
    double s = 0.0;
    for (int k = k0; k < k0 + K; k++) {
      double av = g.A[m * g.sam + (long long)k * g.sak];
      if (g.dk) av *= g.dk[k >> g.dk_shift];
      s = __fma_rn(av, g.B[n * g.sbn + (long long)k * g.sbk], s);
    }
    g.C[m * g.ldc + n] += g.mode == GEMM_SQUARE ? s * s : g.alpha * s;
  }
}

// 3-D map of a digit buffer: x = k within its 32-wide tile, y = row, z = tile x digit.
int digit_map(Ctx* c, CUtensorMap* map, const Digits& d, int box_rows)
{
  auto enc = tensor_map_encoder();
  if (!enc) return set_error(c, THC_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {32, (cuuint64_t)d.rows_pad, (cuuint64_t)(d.kpad / 32 * kNS)};
  cuuint64_t strides[2] = {64, (cuuint64_t)d.rows_pad * 64};
  cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, (cuuint32_t)kNS};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d.s, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(c, THC_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return THC_OK;
}

template <CutScale SC>
int cut_operand_t(Ctx* c, const CutSrc& a, const Digits& d, unsigned* rowmax, int* flag)
{
  cudaStream_t s = c->stream;
  if (a.sr == 1 && a.sk != 1) {
    cut_cols<SC><<<(unsigned)(d.rows_pad / kTR), 256, 0, s>>>(a, d, flag);
    THC_LAUNCHED(c, "cut_cols");
    return THC_OK;
  }
  if (a.K <= kFusedK) {
    int lpr = 32;
    while (lpr > 4 && 8LL * (lpr >> 1) >= d.kpad) lpr >>= 1;
    const long long warps = cdiv(d.rows_pad, 32 / lpr);
    cut_rows<SC><<<(unsigned)cdiv(warps, 8), 256, 0, s>>>(a, d, lpr, flag);
    THC_LAUNCHED(c, "cut_rows");
    return THC_OK;
  }
  THC_CUDA(c, cudaMemsetAsync(rowmax, 0, sizeof(unsigned) * a.rows, s));
  const int n1 = (int)cdiv(a.K, kMaxChunk), n2 = (int)cdiv(d.kpad, 2048);
  cut_rowmax<SC><<<(unsigned)(a.rows * n1), 256, 0, s>>>(a, n1, rowmax);
  THC_LAUNCHED(c, "cut_rowmax");
  cut_long<SC><<<(unsigned)(d.rows_pad * n2), 256, 0, s>>>(a, d, n2, rowmax, flag);
  THC_LAUNCHED(c, "cut_long");
  return THC_OK;
}

}  // namespace

int digits_cut(Ctx* c, const CutSrc& a, const Digits& d, unsigned* rowmax, int* flag)
{
  ProfScope prof(c, "slice64");
  return a.scale  ? cut_operand_t<CUT_SCALED>(c, a, d, rowmax, flag)
         : a.kexp ? cut_operand_t<CUT_SHIFTED>(c, a, d, rowmax, flag)
                  : cut_operand_t<CUT_PLAIN>(c, a, d, rowmax, flag);
}

int digits_product(Ctx* c, const Digits& a, const Digits& b, const GemmArgs& g)
{
  int sms = 0, st;
  THC_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  THC_CUDA(c, cudaFuncSetAttribute(dgemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kSmem));
  Args t;
  t.M = g.M; t.N = g.N;
  t.stages = (int)(a.kpad / kBK);
  t.ea = a.e; t.eb = b.e;
  t.C = g.C; t.ldc = g.ldc; t.alpha = g.alpha; t.beta = g.beta;
  t.lower = g.lower_only;
  t.two8 = 1u << 8;
  t.two16 = 1u << 16;
  t.error = c->tc64_err;
  t.spin_limit = c->spin_limit;
  t.mtn = (unsigned)cdiv(g.M, TBM);
  t.ntn = (unsigned)cdiv(g.N, kBN);
  const long long tiles = g.lower_only
      ? ((long long)t.mtn - 1) * t.mtn + std::min(2 * t.mtn, t.ntn) : (long long)t.mtn * t.ntn;
  if (tiles > 1 << 22) return set_error(c, THC_ERR_SHAPE, "dgemm_tc: too many tiles");
  t.tiles = (unsigned)tiles;
  // Split of K: waves x (k tiles per item + ~3 k tiles' worth of fill and final drain).
  const int kt = t.stages;
  int best = 1;
  double cost = 0.0;
  for (int z = 1; z <= std::min(kt, 256); z++) {
    const int pk = (int)cdiv(kt, z);
    if ((size_t)z * g.M * g.N * 8 > ((size_t)1 << 30) && z > 1) break;
    const double w = (double)cdiv(tiles * cdiv(kt, pk), sms) * (pk + 3) + (z > 1 ? 2.0 : 0.0);
    if (z == 1 || w < 0.98 * cost) { cost = w; best = z; }
  }
  t.kt_per = (int)cdiv(kt, best);
  t.ksplit = (int)cdiv(kt, t.kt_per);
  t.part = nullptr;
  if (t.ksplit > 1) {
    t.part = (double*)ws_get(c, WS_DPART, sizeof(double) * t.ksplit * g.M * g.N);
    if (!t.part) { t.ksplit = 1; t.kt_per = kt; }
  }
  t.square = t.ksplit == 1 && g.mode == GEMM_SQUARE;
  t.scaled = t.ksplit == 1 && g.alpha != 1.0;
  t.added = t.ksplit == 1 && g.beta != 0.0;
  CUtensorMap ma, mb;
  if ((st = digit_map(c, &ma, a, TBM)) || (st = digit_map(c, &mb, b, kBN))) return st;
  const unsigned grid = (unsigned)std::min<long long>(tiles * t.ksplit, sms);
  {
    ProfScope prof(c, "dgemm_tc");
    dgemm_tc_kernel<<<grid, kThreads, kSmem, c->stream>>>(ma, mb, t);
    THC_LAUNCHED(c, "dgemm_tc");
  }
  if (t.ksplit > 1) {
    GemmArgs p = g;
    p.ksplit = t.ksplit;
    p.part = t.part;
    return dgemm_reduce_partials(c, p);
  }
  return THC_OK;
}

bool dgemm_tc_fits(const Ctx* c, const GemmArgs& g)
{
  if (!c->gemm_tc || g.fma_only || (g.kexp && g.dk) || g.skip_flag || g.a_zero_below ||
      g.b_zero_below ||
      g.lower_offset || g.no_split || g.ksplit > 1 || g.part || (g.lower_only && g.M != g.N))
    return false;
  return 2.0 * (double)g.M * (double)g.N * (double)g.K >= kDgemmTcFlops && g.K >= 8;
}

int dgemm_tc(Ctx* c, const GemmArgs& g, bool* done)
{
  *done = false;
  const long long mp = oz_pad_mn(g.M), np = oz_pad_mn(g.N), kp = oz_pad_k(g.K);
  const double* dkr = g.dkr;
  // One buffer of digits serves both operands of a symmetric product.
  const bool same = g.A == g.B && g.sam == g.sbn && g.sak == g.sbk && g.M == g.N &&
                    (!g.dk || dkr) && !g.kexp;
  // Panels: of N while A's digits and a panel of B's fit the budget, else of K (C accumulated
  // in FP64 over the panels).  A product whose smallest panels (128 columns of B, 512 k) pass the
  // budget is not taken.
  const size_t per = kNS * sizeof(__nv_bfloat16);
  const size_t budget = c->digit_bytes;
  long long npan = np;
  int kpan = (int)kp;
  if (!same && !g.lower_only && (size_t)(mp + np) * kp * per > budget &&
      (size_t)mp * kp * per <= budget / 2)
    npan = std::max<long long>(128, (long long)((budget / 2) / (kp * per)) / 128 * 128);
  else if ((size_t)(same ? mp : mp + np) * kp * per > budget)
    kpan = (int)std::max<long long>(512, (long long)(budget / ((same ? mp : mp + np) * per)) / 512 * 512);
  npan = std::min(npan, np);
  kpan = (int)std::min<long long>(std::min(kpan, 1 << 20), kp);   // < 2^21: 64-bit sums
  if (kpan < kp && g.mode == GEMM_SQUARE) return THC_OK;   // the square needs the whole sum
  const size_t abytes = (size_t)mp * kpan * per, bbytes = same ? 0 : (size_t)npan * kpan * per;
  // Coordinates and launch sizes are 32-bit.
  if (abytes + bbytes > budget || mp > 0x7fffff00LL || np > 0x7fffff00LL ||
      (mp / TBM) * (npan / kBN) > 1 << 22)
    return THC_OK;
  char* flags = (char*)ws_get(c, WS_T64_E, 256 + sizeof(int) * (mp + npan) +
                                               sizeof(unsigned) * std::max(mp, npan));
  Digits da, db;
  da.s = (__nv_bfloat16*)ws_get(c, WS_T64_A, abytes);
  db.s = same ? da.s : (__nv_bfloat16*)ws_get(c, WS_T64_B, bbytes);
  if (!flags || !da.s || !db.s) return THC_OK;             // no room: the FMA kernel
  unsigned* rowmax = (unsigned*)(flags + 256);
  da.e = (int*)(rowmax + std::max(mp, npan));
  da.rows_pad = mp;
  int* eb_own = da.e + mp;
  int* nonfin = (int*)flags;
  int sms = 0;
  THC_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  auto vec = [](const double* p, long long sr, long long sk) {
    return sk == 1 && sr % 2 == 0 && (uintptr_t)p % 16 == 0;
  };
  int st;
  for (int k0 = 0; k0 < g.K; k0 += kpan) {
    const int K = std::min(kpan, g.K - k0);
    da.kpad = db.kpad = oz_pad_k(K);
    THC_CUDA(c, cudaMemsetAsync(nonfin, 0, sizeof(int), c->stream));
    {
      CutSrc a{g.A, g.M, g.sam, g.sak, k0, K, same ? dkr : g.dk, g.dk_shift,
               vec(g.A, g.sam, g.sak), g.kexp, 1};
      if ((st = digits_cut(c, a, da, rowmax, nonfin))) return st;
    }
    for (long long n0 = 0; n0 < g.N; n0 += npan) {
      GemmArgs p = g;
      p.N = std::min(npan, g.N - n0);
      p.B = g.B + n0 * g.sbn;
      p.C = g.C + n0;
      if (k0 > 0) p.beta = 1.0;
      if (same) {
        db = da;
      } else {
        db.rows_pad = oz_pad_mn(p.N);
        db.e = eb_own;
        CutSrc b{p.B, p.N, g.sbn, g.sbk, k0, K, nullptr, 0, vec(p.B, g.sbn, g.sbk), g.kexp, -1};
        if ((st = digits_cut(c, b, db, rowmax, nonfin))) return st;
      }
      if ((st = digits_product(c, da, db, p))) return st;
      fix_nonfinite<<<(unsigned)(2 * sms), 256, 0, c->stream>>>(p, k0, K, da.e, db.e, nonfin);
      THC_LAUNCHED(c, "fix_nonfinite");
    }
  }
  *done = true;
  return THC_OK;
}

}  // namespace thc
