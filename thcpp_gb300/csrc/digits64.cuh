// Operands of the FP64 tensor-core products (dgemm_tc.cu) as base-256 digits: the device code
// that cuts rows, and the host calls that cut an operand and multiply two.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "dense64.cuh"

namespace thc {

constexpr int kNS = 7;                   // base-256 digits of an operand
constexpr int kNonFinite = 1 << 28;      // exponent mark of a row that holds an Inf or NaN

// A row's exponent e, |x| < 2^e for every entry, comes from the largest exponent field:
// entries are scanned by the high word of |x| (NaN and Inf above every finite value).  A
// scaled row takes the largest sum of the two fields, at most one above the exact exponent,
// which keeps the FP64 multiply (two a clock on this part) out of the first pass.
__device__ __forceinline__ unsigned abs_hi(double x)
{
  return (unsigned)__double2hiint(x) & 0x7fffffffu;
}

__device__ __forceinline__ int field_of(double x, double s)
{
  const int ex = (int)(abs_hi(x) >> 20), es = (int)(abs_hi(s) >> 20);
  return (ex == 0x7ff || es == 0x7ff) ? kNonFinite : ex + es;
}

// The exponent field of x 2^h, biased: 0 for x = 0 only.
constexpr int kShiftBias = 4096;         // |h| < 2^11
__device__ __forceinline__ unsigned field_shifted(double x, int h)
{
  const unsigned a = abs_hi(x), E = a >> 20;
  if (E == 0x7ff) return kNonFinite;
  if ((a | (unsigned)__double2loint(x)) == 0) return 0;
  return (unsigned)((int)max(E, 1u) + h + kShiftBias);
}

// What multiplies an operand along k: nothing, doubles (CutSrc::scale), or powers of two
// (CutSrc::kexp).
enum CutScale { CUT_PLAIN, CUT_SCALED, CUT_SHIFTED };

// e from the maximum of abs_hi (plain rows), of field_of (scaled rows) or of field_shifted.
template <CutScale SC>
__device__ __forceinline__ int row_exponent(unsigned mx)
{
  if (SC == CUT_SHIFTED)
    return mx == (unsigned)kNonFinite ? kNonFinite : mx ? (int)mx - kShiftBias - 1022 : -1021;
  if (SC == CUT_SCALED) return (int)mx - 2044 > 1024 ? kNonFinite : max((int)mx - 2044, -1021);
  const int E = (int)(mx >> 20);
  return E == 0x7ff ? kNonFinite : max(E, 1) - 1022;
}

// R = round(x 2^{55 - e}) (half away from zero) plus the bias 128 in each of its six low
// bytes, as two words: byte i of R then is digit 6 - i plus 128 (balanced digits in one
// addition), and the bits from 48 on are digit 0.  base = 1022 + e.  32-bit funnel shifts;
// a row marked kNonFinite shifts everything out (R = 0).
__device__ __forceinline__ void cut(double x, int base, unsigned& blo, unsigned& bhi)
{
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const int E = (int)((h & 0x7fffffffu) >> 20);
  const unsigned m = (h & 0xfffffu) | (E ? 0x100000u : 0u);
  unsigned qh = __funnelshift_l(l, m, 3), ql = l << 3;          // 8 x mantissa
  unsigned k = (unsigned)(base - max(E, 1));                    // >= 0: |x| < 2^e
  if (k >= 32) { ql = qh; qh = 0; k -= 32; }
  ql = __funnelshift_rc(ql, qh, k);
  qh = k >= 32 ? 0u : qh >> k;
  const unsigned long long q = (((unsigned long long)qh << 32 | ql) + 1) >> 1;
  const unsigned neg = (unsigned)((int)h >> 31);
  const unsigned long long r = (q ^ ((unsigned long long)neg << 32 | neg)) +
                               (0x0000808080808080ULL + (neg & 1u));
  blo = (unsigned)r;
  bhi = (unsigned)(r >> 32);
}

// Digits of two neighbouring columns as a BF16 pair, from byte n of their biased words:
// b - 128 = (128 + b mod 128) - (b < 128 ? 256 : 128), both terms BF16 bit patterns.
__device__ __forceinline__ unsigned digit_pair(unsigned w0, unsigned w1, int n)
{
  const unsigned x = __byte_perm(w0, w1, (unsigned)(n | n << 4 | (4 + n) << 8 | (4 + n) << 12));
  const unsigned a = (x & 0x007f007fu) | 0x43004300u, c = (~x & 0x00800080u) | 0x43004300u;
  const __nv_bfloat162 d = __hsub2(*(const __nv_bfloat162*)&a, *(const __nv_bfloat162*)&c);
  return *(const unsigned*)&d;
}

// Digit storage: [k / 32][digit][row][32] BF16, rows padded to 128 and k to 32 with zeros,
// so that the 32-k tile of 128 rows and all digits is one box of a 3-D tensor map.
struct Digits {
  __nv_bfloat16* s = nullptr;
  int* e = nullptr;
  long long rows_pad = 0, kpad = 0;
};

// Cuts columns k .. k + 7 of row r, column k + j times 2^h[j]: one 16-byte store per digit.
template <class H>
__device__ __forceinline__ void store8(const Digits& o, long long r, long long k, int base,
                                       const double (&v)[8], H h)
{
  unsigned lo[8], hi[8];
#pragma unroll
  for (int j = 0; j < 8; j++) cut(v[j], base - h(j), lo[j], hi[j]);
  __nv_bfloat16* p = o.s + (k >> 5) * (kNS * o.rows_pad * 32) + r * 32 + (k & 31);
  const long long step = o.rows_pad * 32;
  unsigned w[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    // (float)(hi >> 16) without the conversion pipe: |digit 0| <= 128.
    const float f0 = __int_as_float(0x4b400000 + ((int)hi[2 * q] >> 16)) - 12582912.f;
    const float f1 = __int_as_float(0x4b400000 + ((int)hi[2 * q + 1] >> 16)) - 12582912.f;
    const __nv_bfloat162 d = __floats2bfloat162_rn(f0, f1);
    w[q] = *(const unsigned*)&d;
  }
  *(uint4*)p = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
  for (int i = 1; i < kNS; i++) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      w[q] = i < 3 ? digit_pair(hi[2 * q], hi[2 * q + 1], 2 - i)
                   : digit_pair(lo[2 * q], lo[2 * q + 1], 6 - i);
    *(uint4*)(p + i * step) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ void store8(const Digits& o, long long r, long long k, int base,
                                       const double (&v)[8])
{
  store8(o, r, k, base, v, [](int) { return 0; });
}

// Where an operand's element (row r, index k) lies and what multiplies it.
struct CutSrc {
  const double* x;
  long long rows, sr, sk;    // x[r sr + k sk]
  int k0, K;                 // the panel's first k and its length
  const double* scale;       // CUT_SCALED: indexed (k0 + k) >> shift
  int shift;
  bool vec;                  // sk == 1, rows 16-byte aligned
  const int* kexp = nullptr; // CUT_SHIFTED: x 2^{ksign kexp[k0 + k]}
  int ksign = 1;
};

// Digits of one operand's panel (k0, K) into d; flag (device) is set if a row is not finite.
// rowmax: scratch, an unsigned per row.
int digits_cut(Ctx* c, const CutSrc& a, const Digits& d, unsigned* rowmax, int* flag);
// C = op(A B) of p (M, N, C, ldc, alpha, beta, mode, lower_only) from both operands' digits of
// the same k range; picks a split of K.  Rows marked kNonFinite count as zero.
int digits_product(Ctx* c, const Digits& a, const Digits& b, const GemmArgs& p);

}  // namespace thc
