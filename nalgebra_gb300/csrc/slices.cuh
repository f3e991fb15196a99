// FP64 products of short rows on the FP16 tensor cores, for the batched
// factorizations: rows of 16 doubles are cut into seven 8-bit digits each, the
// digit products summed exactly by mma.sync, the sums put together with integer
// instructions.
//
// Why: an FP64 multiply-add costs half a cycle of the SM's FP64 pipe; a
// 16-deep product of two rows 8 cycles.  The 28 digit products of an mma
// m16n8k16 tile cost 0.5 cycles per output, putting the sums together about 35
// integer instructions and one FP64 subtraction (about 1 cycle).
//
// Splitting (Ozaki, Ogita, Oishi & Rump 2012, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and its
// applications", with digits instead of floating-point slices): row r with
// largest exponent E_r becomes integers I = rint(v 2^(54 - E_r)), |I| <= 2^55,
// in balanced base-256 digits d_0 .. d_6 (d_0 in [-128, 128], the others in
// [-128, 127]), exact in FP16.  (FP16 and not BF16: with 11 significant bits a
// byte b placed under the exponent of 1024 is 1024 + b, so two digits take one
// byte permute and one packed subtraction.)  Level l collects the products d_p d_q with
// p + q = l; levels 0..6 are kept, 0..7 in the LU and the QR.  A sum of 16 * 7 such products stays below
// 2^21 (of 32: below 2^22), so with the accumulator starting at 1.5 2^23 every partial sum is an
// integer of FP32 and the low mantissa bits of the result are the sum itself.
//
// Error of one 16-deep product against 64 bits: rounding of I 2^-56 2^E of each
// factor and the levels left out 2^-54 2^(E_r + E_c), with an eighth level the sum's unit, 2^-56 (both
// relative to the largest entries of the two rows, so a caller whose depth runs over
// entries of different scale balances and checks, below); the FP64 loop's is 2^-53 of the partial
// sums, which contain the updated element itself.
#pragma once
#include "common.cuh"

namespace nacu {
namespace {

constexpr int kSlices = 7;
constexpr int kSliceRow = 32;            // bytes of one row's digits in one slice
constexpr int kBadRow = 1 << 20;         // exponent code of a row with inf or NaN
constexpr int kNoExponent = -(1 << 20);  // of zero, where rows are told from zero rows

__device__ __forceinline__ void mma_f16_16x8x16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// The digits of two values against the exponents e0 and e1, one word of two FP16
// digits per slice.  No digits where a value lies 2^60 below its exponent.
__device__ __forceinline__ void slice_digits(double v0, double v1, int e0, int e1, uint32_t (&w)[kSlices]) {
  uint32_t lo[2], hi[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const long long b = __double_as_longlong(k ? v1 : v0);
    const int ex = (int)((b >> 52) & 0x7ff);
    const long long m = (b & 0xfffffffffffffll) | (ex ? 0x10000000000000ll : 0ll);
    const int sh = (k ? e1 : e0) - max(ex, 1);  // >= 0, but for zeros: I = m 2^(2 - sh)
    long long i = (unsigned)sh > 60u ? 0 : ((((m << 3) >> sh) + 1) >> 1);
    // plus 128 in every digit: the bytes (the top one nine bits) are digit + 128
    i = (b < 0 ? -i : i) + 0x0080808080808080ll;
    lo[k] = (uint32_t)i;
    hi[k] = (uint32_t)(i >> 32);
  }
  auto minus = [](uint32_t x) {  // 1024 + 128 off both halves
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(0x64806480u));
    return r;
  };
  w[0] = minus(__byte_perm(hi[0], hi[1], 0x7632) | 0x64006400u);
  const uint32_t t54 = __byte_perm(hi[0], hi[1], 0x5140);  // bytes 4, 4, 5, 5 of the two values
  const uint32_t t32 = __byte_perm(lo[0], lo[1], 0x7362), t10 = __byte_perm(lo[0], lo[1], 0x5140);
  w[1] = minus(__byte_perm(t54, 0x64646464u, 0x4342));
  w[2] = minus(__byte_perm(t54, 0x64646464u, 0x4140));
  w[3] = minus(__byte_perm(t32, 0x64646464u, 0x4342));
  w[4] = minus(__byte_perm(t32, 0x64646464u, 0x4140));
  w[5] = minus(__byte_perm(t10, 0x64646464u, 0x4342));
  w[6] = minus(__byte_perm(t10, 0x64646464u, 0x4140));
}
// The same against a row's common exponent code em (slice_exponent).  em 2047 (inf or
// NaN in the row): zeros.
__device__ __forceinline__ int slice_exponent(double v) { return max((__double2hiint(v) >> 20) & 0x7ff, 1); }
__device__ __forceinline__ void slice_pair(double v0, double v1, int em, uint32_t (&w)[kSlices]) {
  const int e = em == 0x7ff ? kBadRow : em;
  slice_digits(v0, v1, e, e, w);
}
// A row's exponent code from its largest exponent: inf and NaN poison the row.
__device__ __forceinline__ int slice_code(int em) { return em == 0x7ff ? kBadRow : em; }

// A row's 16 doubles -> its seven slices at s0 + p * slice_bytes (32 bytes each,
// digits in the doubles' order) and its exponent code.
__device__ __forceinline__ int slice_row(const double (&v)[16], unsigned char* s0, int slice_bytes) {
  int em = 1;
#pragma unroll
  for (int k = 0; k < 16; ++k) em = max(em, slice_exponent(v[k]));
#pragma unroll
  for (int h = 0; h < 16; h += 8) {
    uint32_t w0[kSlices], w1[kSlices], w2[kSlices], w3[kSlices];
    slice_pair(v[h], v[h + 1], em, w0);
    slice_pair(v[h + 2], v[h + 3], em, w1);
    slice_pair(v[h + 4], v[h + 5], em, w2);
    slice_pair(v[h + 6], v[h + 7], em, w3);
#pragma unroll
    for (int p = 0; p < kSlices; ++p)
      *reinterpret_cast<uint4*>(s0 + p * slice_bytes + h * 2) = make_uint4(w0[p], w1[p], w2[p], w3[p]);
  }
  return slice_code(em);
}
__device__ __forceinline__ void slice_zero_row(unsigned char* s0, int slice_bytes) {
#pragma unroll
  for (int p = 0; p < kSlices; ++p) {
    uint4* out = reinterpret_cast<uint4*>(s0 + p * slice_bytes);
    out[0] = out[1] = make_uint4(0u, 0u, 0u, 0u);
  }
}

__device__ __forceinline__ void mma_f16_16x8x8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(b0));
}
template <int LEVELS>
__device__ __forceinline__ void slice_sums_start(float (&acc)[LEVELS][4]) {
#pragma unroll
  for (int l = 0; l < LEVELS; ++l)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[l][i] = 12582912.0f;
}

// Level sums of a 16 x 8 tile: rows sa .. sa + 15 against rows sb .. sb + 7
// (pointers to the first row's digits in slice 0).  A fragment's lane t holds
// the 16 products' terms 4 t .. 4 t + 3 (one 8-byte load), the same for both
// operands: the order of the terms is free.
template <int LEVELS>
__device__ __forceinline__ void slice_products_add(const unsigned char* sa, const unsigned char* sb, int slice_bytes,
                                                   int lane, float (&acc)[LEVELS][4]) {
  const int off = (lane >> 2) * kSliceRow + (lane & 3) * 8;
  uint32_t b[kSlices][2];
#pragma unroll
  for (int q = 0; q < kSlices; ++q) {
    const uint2 w = *reinterpret_cast<const uint2*>(sb + q * slice_bytes + off);
    b[q][0] = w.x;
    b[q][1] = w.y;
  }
#pragma unroll
  for (int p = 0; p < kSlices; ++p) {
    const uint2 w0 = *reinterpret_cast<const uint2*>(sa + p * slice_bytes + off);
    const uint2 w1 = *reinterpret_cast<const uint2*>(sa + p * slice_bytes + off + 8 * kSliceRow);
    const uint32_t a[4] = {w0.x, w1.x, w0.y, w1.y};
#pragma unroll
    for (int q = 0; q < kSlices && p + q < LEVELS; ++q) mma_f16_16x8x16(acc[p + q], a, b[q]);
  }
}

// ---- products whose factors' rows are graded ----------------------------------------------------------------
// The digits count from a row's largest entry.  Where the large entries of two rows
// do not meet, the product is far below that of the largest entries and the digits
// dropped weigh on it.  So a caller may (1) move powers of two from one factor to
// the other, term by term, by cutting against shifted exponents, and (2) let the
// magnitudes' leading digits be multiplied too: where their sum is under kMeet / 2^14
// = 1/8 of the largest entries' product, the products are to be formed in FP64.  The
// error, a few 2^-56 of the largest entries' product, is then below 2^-50 of the sum
// of the magnitudes, inside the bound 32 2^-53 of the FP64 loop's roundings.  Dense
// rows of one scale have sums of 1 to 4.
constexpr float kMeet = 2048.f;

// The exponent of v 2^shift; kNoExponent for zero, kBadRow for inf and NaN.
__device__ __forceinline__ int shifted_exponent(double v, int shift) {
  const int hi = __double2hiint(v) & 0x7fffffff, ex = hi >> 20;
  if (ex == 0x7ff) return kBadRow;
  return (hi | __double2loint(v)) == 0 ? kNoExponent : max(ex, 1) + shift;
}
// Likewise a row's code.
__device__ __forceinline__ int graded_code(int em) {
  return em >= kBadRow / 2 ? kBadRow : em <= kNoExponent / 2 ? kNoExponent : em;
}
// The digits of 16 elements, element k times 2^-shift[k] in the one factor and
// 2^shift[k] in the other (shift: 8-byte aligned).  Lowered, shift[k] is at least v[k]'s
// exponent, kBadRow for no entry and for inf or NaN (which the raised factor's code
// then tells).
__device__ __forceinline__ int slice_row_lowered(const double (&v)[16], const int* shift, unsigned char* s0, int slice_bytes) {
  int e[16], em = 2 * kNoExponent;
#pragma unroll
  for (int k = 0; k < 16; k += 2) {
    const int2 p = *reinterpret_cast<const int2*>(shift + k);
    e[k] = p.x, e[k + 1] = p.y;
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) em = max(em, slice_exponent(v[k]) - e[k]);
  uint32_t any = 0;
#pragma unroll
  for (int h = 0; h < 16; h += 8) {
    uint32_t w[4][kSlices];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = h + 2 * q;
      slice_digits(v[k], v[k + 1], em + e[k], em + e[k + 1], w[q]);
      any |= w[q][0];
    }
#pragma unroll
    for (int p = 0; p < kSlices; ++p)
      *reinterpret_cast<uint4*>(s0 + p * slice_bytes + h * 2) = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
  }
  if (any == 0) {  // no leading digit: a zero row, or its scale is that of its zeros (counted as 2^-1022)
    bool zero = true;
#pragma unroll
    for (int k = 0; k < 16; ++k) zero = zero && is_zero_bits(v[k]);
    if (zero) return kNoExponent;
  }
  return em;
}
__device__ __forceinline__ int slice_row_raised(const double (&v)[16], const int* shift, unsigned char* s0, int slice_bytes) {
  int em = kNoExponent;
#pragma unroll
  for (int k = 0; k < 16; ++k) em = max(em, shifted_exponent(v[k], shift[k]));
#pragma unroll
  for (int h = 0; h < 16; h += 8) {
    uint32_t w[4][kSlices];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = h + 2 * q;
      slice_digits(v[k], v[k + 1], em - shift[k], em - shift[k + 1], w[q]);
    }
#pragma unroll
    for (int p = 0; p < kSlices; ++p)
      *reinterpret_cast<uint4*>(s0 + p * slice_bytes + h * 2) = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
  }
  return graded_code(em);
}
// The sums of the leading digits' magnitudes.
__device__ __forceinline__ void slice_met(const unsigned char* sa, const unsigned char* sb, int lane, float (&met)[4]) {
  const int off = (lane >> 2) * kSliceRow + (lane & 3) * 8;
  constexpr uint32_t kAbs = 0x7fff7fffu;
  const uint2 w = *reinterpret_cast<const uint2*>(sb + off);
  const uint2 w0 = *reinterpret_cast<const uint2*>(sa + off), w1 = *reinterpret_cast<const uint2*>(sa + off + 8 * kSliceRow);
  const uint32_t a[4] = {w0.x & kAbs, w1.x & kAbs, w0.y & kAbs, w1.y & kAbs}, b[2] = {w.x & kAbs, w.y & kAbs};
  mma_f16_16x8x16(met, a, b);
}
// slice_products_add, and those.
template <int LEVELS>
__device__ __forceinline__ void slice_products_met(const unsigned char* sa, const unsigned char* sb, int slice_bytes,
                                                   int lane, float (&acc)[LEVELS][4], float (&met)[4]) {
  slice_products_add(sa, sb, slice_bytes, lane, acc);
  slice_met(sa, sb, lane, met);
}
__device__ __forceinline__ void slice_products(const unsigned char* sa, const unsigned char* sb, int slice_bytes, int lane,
                                               float (&acc)[kSlices][4]) {
  slice_sums_start(acc);
  slice_products_add(sa, sb, slice_bytes, lane, acc);
}

__device__ __noinline__ double slice_value_slow(long long w, int e) {
  if (e >= (kBadRow >> 1)) return __longlong_as_double(0x7ff8000000000000ll);  // a row with inf or NaN
  const int s = e - 2102;  // w 2^s
  const int s0 = max(min(s / 2, 1000), -1000), s1 = max(min(s - s0, 1000), -1000);
  return (double)w * __longlong_as_double((long long)(s0 + 1023) << 52) * __longlong_as_double((long long)(s1 + 1023) << 52);
}

// One product from its level sums (the accumulators' bit images); e the sum of
// the two rows' exponent codes.  W = sum_l S_l 2^(44 - 8 l), the value W 2^(e -
// 2046 - 56), rounded to 53 bits from the integer.  DEPTH 32: sums of up to 32
// products per level and slice pair (7 * 32 * 2^14 < 2^22 still fits the offset
// accumulators), W one bit shorter to stay below 2^63.  With an eighth level, S_7
// enters after S_6.
template <int DEPTH = 16, int LEVELS = kSlices>
__device__ __forceinline__ double slice_value(const float (&acc)[LEVELS][4], int i, int e) {
  constexpr int kDrop = DEPTH > 16 ? 1 : 0;
  const uint32_t s0 = __float_as_uint(acc[0][i]), s1 = __float_as_uint(acc[1][i]), s2 = __float_as_uint(acc[2][i]);
  const uint32_t s3 = __float_as_uint(acc[3][i]), s4 = __float_as_uint(acc[4][i]), s5 = __float_as_uint(acc[5][i]);
  const uint32_t s6 = __float_as_uint(acc[6][i]);
  constexpr uint32_t kM = 0x4b400000u, kM2 = kM * 256u + kM;  // the offset in one sum, and in 256 x + y
  const int a = (int)(s0 * 256u + s1 - kM2), b = (int)(s2 * 256u + s3 - kM2), c = (int)(s4 * 256u + s5 - kM2);
  int d = (int)(s6 - kM) >> (4 + kDrop);
  if constexpr (LEVELS > kSlices)
    d = (int)(s6 * 256u + __float_as_uint(acc[kSlices][i]) - kM2) >> (12 + kDrop);
  const long long w = (long long)b * (1ll << (20 - kDrop)) + ((long long)c * (16 >> kDrop) + d) +
                      ((long long)((unsigned long long)(uint32_t)a << (36 - kDrop)));
  const uint32_t sign = (uint32_t)((unsigned long long)w >> 63);
  unsigned long long m = (unsigned long long)(sign ? -w : w);
  if (m == 0) {
    return e < (kBadRow >> 1) ? 0.0 : slice_value_slow(w, e + kDrop);
  }
  const int z = __clzll((long long)m);  // >= 1: |w| < 2^63
  m <<= z - 1;                           // leading one at bit 62
  m += 0x200ull;                         // round to 53 bits (a carry to bit 63 moves into the exponent)
  const int ex = 63 - z + e - 1079 + kDrop;
  if ((unsigned)(ex - 1) >= 2044u) return slice_value_slow(w, e + kDrop);
  const uint32_t h = (uint32_t)(m >> 42) + ((uint32_t)(ex - 1) << 20) + (sign << 31);
  return __hiloint2double((int)h, (int)(uint32_t)(m >> 10));
}

}  // namespace
}  // namespace nacu
