// FP64 GEMM on the BF16 tensor cores by modular arithmetic: C = alpha * A * B
// + beta * C for column-major A (m x k), B (k x n), C (m x n), the GPU form of
// nalgebra's `Matrix::gemm` (src/base/blas.rs:729-746) for large products.
//
// Why: GB300 issues 2 FP64 multiply-adds per SM and cycle (1.25 TFLOP/s) and
// about 4096 BF16 ones through tcgen05.  An integer matrix product is exact on
// the tensor cores when it is taken modulo small numbers, and the Chinese
// remainder theorem puts the residues together again (Ozaki, Uchino & Imamura
// 2025, "Ozaki scheme II"; the classical reference is Knuth, TAOCP 4.3.2).
//
// Method:
//   1. Row i of A and column j of B are scaled by powers of two 2^s_i, 2^t_j
//      and rounded to integers a', b' of up to 62 bits, the scales chosen from
//      the rows' and columns' 2-norms so that |sum_l a'_il b'_lj| <= |a'_i||b'_j|
//      < P / 4, P the product of the 16 moduli below (125.4 bits).
//   2. For every modulus p the residues of a' (times the inverse of P/p) and b'
//      are small integers |r| <= 128, exact in BF16.
//   3. One BF16 GEMM per modulus.  1024 products of residues sum exactly in an
//      FP32 accumulator (1024 * 128^2 = 2^24); after each such chunk of K the
//      accumulator is reduced mod p into registers.  The result y_p goes to
//      memory as one byte.
//   4. X = sum_p y_p (P/p) - P * round(sum_p y_p / p) is the exact integer
//      product, formed in 21-bit limbs; C = alpha 2^-(s+t) X + beta C in FP64.
//
// Accuracy: the only errors are the rounding of a' and b' (half a unit of
// integers whose rows have norm about 2^61) and the conversion of X.  For data
// without large cancellation inside |A||B| the error is about 300 times below
// that of the FP64 FMA loop.  What can spoil it is a row of A and a column of
// B whose large entries never meet (|a|.|b| far below |a||b|).  So a
// seventeenth plane forms |a_i|.|b_j| / (|a_i||b_j|) in BF16, and where an
// output's ratio falls under 2^-7 -- also for NaN, infinities and exponents
// beyond +-800 -- its 128 x 128 tile is left to the FP64 kernel
// (gemm_fp64.cu), which skips all other tiles.
//
// Kernel: clusters of two CTAs share a 256 x 256 output tile
// (tcgen05.mma.cta_group::2, each CTA loads and holds 128 rows of A and 128
// columns of B, so the L2 -> shared-memory traffic per flop is half that of a
// 128 x 256 tile on one CTA), persistent over (plane, tile) units.  Warp 0:
// TMA producer, warp 1 (of the leading CTA): MMA issuer, warps 2-9: epilogue,
// 128 columns x 1 row per thread, reducing one TMEM accumulator (256 of the 512
// columns) while the next chunk's MMAs run in the other and storing its residues
// as 128-byte rows by TMA.  Every barrier wait is bounded.
//
// What bounds it: the tensor pipe, 17 BF16 products instead of one; for K in the
// hundreds the epilogue (156 us for the 17 planes of 4096 x 4096 x 128; 186 with
// byte stores from registers).  Measured (GB300, scratch warm): 8192^3 878 ->
// 16.1 ms (55x; 17 planes at 1.50 of the 1.90 PFLOP/s a BF16 GEMM reaches),
// 1000 x 777 x 1333 2.69 -> 0.13 ms, 256^3 266 -> 38 us.  Error against sums in
// short blocks, N(0,1) entries: 3.9e-16 relative at 4096^3 where the FP64 loop
// has 2.2e-15.
#include <cuda_bf16.h>

#include <algorithm>

#include "tc05.cuh"

namespace nacu {

namespace {

constexpr int kMod = 16;               // moduli
constexpr int kDigits = 15;            // base-256 digits of P / p (117.8 bits), balanced
constexpr int kKMax = 8;               // |sum_p y_p / p| <= 8: the multiples of P to subtract
constexpr int kPM = 256, kPN = 256;    // tile of a CTA pair
constexpr int kKB = 64;                // K of one stage: 128-byte rows, 128-byte swizzle
constexpr int kChunkBlocks = 16;       // k-blocks per exact FP32 sum: 1024 products
constexpr int kStagesC = 6;
constexpr uint32_t kStoreBytes = 32 * 128;  // one epilogue warp's residues: 32 rows x 128 columns
constexpr uint32_t kHalfTile = 128 * kKB * 2;       // 16 KB: one CTA's share of an operand tile
constexpr uint32_t kStageBytesC = 2 * kHalfTile;
constexpr int kCrtThreads = 320;       // producer, MMA issuer, eight epilogue warps
constexpr int kFlagTile = 128;
constexpr float kMinCos = 0.0078125f;  // 2^-7
constexpr int kMaxExp = 800;           // exponents of a row's / column's largest entry
constexpr int kBadScale = 0x40000000;  // a row / column for the FP64 kernel
constexpr int kZeroScale = 0x20000000; // an all-zero row / column: its products are exact zeros
// Columns of A per thread of the row statistics: a thread's loads are one
// dependent chain, so a short product (K = 128: 25 us with all of it on one
// thread) takes few; a long one fewer, larger partial sums to merge.
constexpr int stat_chunk(int k) { return k <= 512 ? 16 : 128; }

// ---- tables -------------------------------------------------------------------------------------------------
struct CrtTables {
  int p[kMod];          // the moduli, pairwise coprime, the largest such set below 257
  float pf[kMod], inv[kMod];
  int magic[kMod];      // round-up(2^38 / p)
  int wa[kMod][3];      // residues of q, q 2^21, q 2^42 with q = (P/p)^-1 mod p (for A), balanced
  int wb[kMod][3];      // residues of 1, 2^21, 2^42 (for B), balanced
  uint32_t digit[kMod / 4][kDigits];  // digit d of P / p for four moduli, a byte each
  uint32_t quot[kMod / 4];            // round(2^14 / p), a byte each
};

// k P + the digit sums' bias, k = -8 .. 8, as 128-bit numbers
struct CrtMultiples {
  uint4 v[2 * kKMax + 1];
};
constexpr int kDigitBias = 1 << 18;  // |16 digits x 128| < 2^18 keeps every digit sum positive

constexpr int balanced(long long v, int p) {
  long long r = v % p;
  if (r < 0) r += p;
  return (int)(2 * r > p ? r - p : r);
}

constexpr CrtTables make_tables() {
  CrtTables t{};
  const int ps[kMod] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
  for (int i = 0; i < kMod; ++i) {
    long long d[kDigits + 2] = {1};
    for (int j = 0; j < kMod; ++j) {
      if (j == i) continue;
      long long carry = 0;
      for (int l = 0; l < kDigits + 2; ++l) {
        const long long v = d[l] * ps[j] + carry;
        d[l] = v & 255;
        carry = v >> 8;
      }
    }
    for (int l = 0; l < kDigits; ++l) {
      if (d[l] >= 128) {
        d[l] -= 256;
        d[l + 1] += 1;
      }
      t.digit[i / 4][l] |= (uint32_t)(d[l] & 255) << (8 * (i % 4));
    }
    t.quot[i / 4] |= (uint32_t)(((1 << 15) / ps[i] + 1) / 2) << (8 * (i % 4));
  }
  for (int i = 0; i < kMod; ++i) {
    const int p = ps[i];
    long long r = 1;
    for (int j = 0; j < kMod; ++j)
      if (j != i) r = r * ps[j] % p;
    long long q = 1;
    while (r * q % p != 1) ++q;
    t.p[i] = p;
    t.pf[i] = (float)p;
    t.inv[i] = 1.0f / (float)p;
    t.magic[i] = (int)(((1ll << 38) + p - 1) / p);
    const long long b21 = (1ll << 21) % p, b42 = b21 * b21 % p;
    t.wb[i][0] = 1;
    t.wb[i][1] = balanced(b21, p);
    t.wb[i][2] = balanced(b42, p);
    t.wa[i][0] = balanced(q, p);
    t.wa[i][1] = balanced(q * b21, p);
    t.wa[i][2] = balanced(q * b42, p);
  }
  return t;
}
__constant__ CrtTables kT = make_tables();

constexpr CrtMultiples make_multiples() {
  CrtMultiples t{};
  const int ps[kMod] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
  long long d[16] = {1};  // P in base 256
  for (int j = 0; j < kMod; ++j) {
    long long carry = 0;
    for (int l = 0; l < 16; ++l) {
      const long long v = d[l] * ps[j] + carry;
      d[l] = v & 255;
      carry = v >> 8;
    }
  }
  for (int k = -kKMax; k <= kKMax; ++k) {
    uint32_t w[4] = {};
    long long carry = 0;
    for (int l = 0; l < 16; ++l) {
      const long long v = k * d[l] + (l < kDigits + 1 ? kDigitBias : 0) + carry;
      w[l / 4] |= (uint32_t)(v & 255) << (8 * (l % 4));
      carry = v >> 8;
    }
    t.v[k + kKMax].x = w[0];
    t.v[k + kKMax].y = w[1];
    t.v[k + kKMax].z = w[2];
    t.v[k + kKMax].w = w[3];
  }
  return t;
}
__constant__ CrtMultiples kP = make_multiples();

// ---- scaling ------------------------------------------------------------------------------------------------

// Running (max exponent, sum of squares relative to 2^(2 max)) of |x|; biased
// exponents, subnormals counted as the smallest normal number, inf / NaN as
// exponent 2047.
struct Norm {
  int e = 0;
  float s = 0.f;
  // x 2^shift; where it falls below the normal numbers, as the smallest of them
  __device__ __forceinline__ void add(double x, int shift) {
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu, lo = (unsigned)__double2loint(x);
    if ((hi | lo) == 0u) return;
    const int ex = hi >= 0x7ff00000u ? 2047 : min(max(max((int)(hi >> 20), 1) + shift, 1), 2047);
    // the mantissa rounded up to 21 bits: never below |x|
    const float f = __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | 7u);
    if (ex > e) {
      const int d = 2 * (e - ex);
      s = d < -120 ? 0.f : s * __int_as_float((127 + d) << 23);
      e = ex;
    }
    const int d = 2 * (ex - e);
    if (d >= -120) s = fmaf(f * f, __int_as_float((127 + d) << 23), s);
  }
  __device__ __forceinline__ void merge(int e2, float s2) {
    if (s2 == 0.f && e2 == 0) return;
    if (e2 > e) {
      const int d = 2 * (e - e2);
      s = (d < -120 ? 0.f : s * __int_as_float((127 + d) << 23)) + s2;
      e = e2;
    } else {
      const int d = 2 * (e2 - e);
      if (d >= -120) s = fmaf(s2, __int_as_float((127 + d) << 23), s);
    }
  }
  // The power of two that brings the 2-norm into (2^60.3, 2^61.6].
  __device__ __forceinline__ int scale() const {
    if (e == 0) return kZeroScale;
    const int ex = e - 1023;
    if (e == 2047 || ex > kMaxExp || ex < -kMaxExp) return kBadScale;
    return (int)floorf(61.59f - 0.5f * log2f(s)) - ex;
  }
};

// x * 2^s rounded to the nearest integer (|result| < 2^62), by integer shifts.
__device__ __forceinline__ long long scaled_int(double x, int s) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex == 0) return 0;  // zero or subnormal: below half a unit for every |s| a finite row can have
  const long long m = (b & 0xfffffffffffffll) | 0x10000000000000ll;
  const int sh = ex - 1075 + s;  // x 2^s = +-m 2^sh
  long long v;
  if (sh >= 0) v = m << sh;
  else if (sh < -54) v = 0;
  else v = ((m >> (-sh - 1)) + 1) >> 1;
  return b < 0 ? -v : v;
}

// Balanced residues of one integer, as floats' high halves (BF16 bit images).
struct Chunks {
  int c0, c1, c2;
  __device__ __forceinline__ explicit Chunks(long long v)
      : c0((int)(v & 0x1fffff)), c1((int)((v >> 21) & 0x1fffff)), c2((int)(v >> 42)) {}
};
__device__ __forceinline__ uint32_t residue_bits(const Chunks& c, const int* w, int i) {
  const int v = c.c0 * w[0] + c.c1 * w[1] + c.c2 * w[2];       // |v| < 2^30
  const int q = (__mulhi(v, kT.magic[i]) + 32) >> 6;           // round(v / p)
  const int r = v - q * kT.p[i];                               // |r| <= 128
  return __float_as_uint(__int_as_float(0x4b400000 + r) - 12582912.0f);
}
__device__ __forceinline__ uint32_t pack_hi(uint32_t lo, uint32_t hi) { return __byte_perm(lo, hi, 0x7632); }

// |x| relative to the norm's bound, for the plane that compares |a|.|b| with
// |a||b|; NaN sends the whole row or column to the FP64 kernel.
__device__ __forceinline__ uint32_t abs_bits(long long v, bool bad) {
  if (bad) return 0x7fff0000u;
  return __float_as_uint((float)llabs(v) * 2.168404344971009e-19f) + 0x8000u;  // 2^-62, rounded to BF16
}

// Partial row norms of A: thread per row and chunk of columns; part[chunk][row].
__global__ void __launch_bounds__(128) crt_row_stats_kernel(int m, int k, const double* A, int64_t lda,
                                                            int chunk, const int* bal,
                                                            int2* __restrict__ part, int* __restrict__ flags, int nflags) {
  wait_for_predecessor();
  const int i = blockIdx.x * 128 + threadIdx.x;
  for (int f = blockIdx.y * gridDim.x * 128 + i; f < nflags; f += gridDim.x * gridDim.y * 128) flags[f] = 0;
  if (i >= m) return;
  const int c0 = blockIdx.y * chunk, c1 = min(k, c0 + chunk);
  Norm nm;
  const double* a = A + (size_t)c0 * lda + i;
#pragma unroll 4
  for (int c = c0; c < c1; ++c, a += lda) nm.add(*a, bal ? bal[c] : 0);
  part[(size_t)blockIdx.y * m + i] = make_int2(nm.e, __float_as_int(nm.s));
}

// A -> residue planes [plane][mp][kp], K contiguous: 64 k x 32 rows per CTA,
// transposed through shared memory as scaled integers.  The CTAs of the first
// k tile also write the row scales.
__global__ void __launch_bounds__(256) crt_split_a_kernel(int m, int k, const double* A, int64_t lda,
                                                          const int2* part, int nparts, int mp, int kp,
                                                          const int* bal,
                                                          int* __restrict__ rscale, uint32_t* __restrict__ out) {
  __shared__ long long t[64][33];
  __shared__ int s_scale[32];
  const int i0 = blockIdx.y * 32, k0 = blockIdx.x * 64;
  const int tid = threadIdx.x;
  wait_for_predecessor();
  if (tid < 32) {
    Norm nm;
    if (i0 + tid < m)
      for (int c = 0; c < nparts; ++c) {
        const int2 v = part[(size_t)c * m + i0 + tid];
        nm.merge(v.x, __int_as_float(v.y));
      }
    const int sc = nm.scale();
    s_scale[tid] = sc;
    if (blockIdx.x == 0) rscale[i0 + tid] = sc;
  }
  __syncthreads();
  {
    const int r = tid & 31, sc = s_scale[r];
    const bool live = i0 + r < m && sc < kZeroScale;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int kk = (tid >> 5) + 8 * u;
      double x = (live && k0 + kk < k) ? A[(size_t)(k0 + kk) * lda + i0 + r] : 0.0;
      if (bal && k0 + kk < k) x = shift_exp(x, bal[k0 + kk]);
      t[kk][r] = scaled_int(x, live ? sc : 0);
    }
  }
  __syncthreads();
  const int lane = tid & 31;
  const size_t plane = (size_t)mp * kp / 2;
#pragma unroll 1
  for (int u = 0; u < 4; ++u) {
    const int r = (tid >> 5) * 4 + u;
    const long long v0 = t[2 * lane][r], v1 = t[2 * lane + 1][r];
    const Chunks a0(v0), a1(v1);
    uint32_t* o = out + ((size_t)(i0 + r) * kp + k0) / 2 + lane;
#pragma unroll
    for (int i = 0; i < kMod; ++i) o[i * plane] = pack_hi(residue_bits(a0, kT.wa[i], i), residue_bits(a1, kT.wa[i], i));
    const bool bad = s_scale[r] == kBadScale;
    o[kMod * plane] = pack_hi(abs_bits(v0, bad), abs_bits(v1, bad));
  }
}

// B (columns contiguous along K) -> residue planes [plane][np][kp] and the
// column scales; one CTA per (padded) column.
__global__ void __launch_bounds__(256) crt_split_b_kernel(int k, int n, const double* B, int64_t ldb, int np,
                                                          int kp, const int* bal,
                                                          int* __restrict__ cscale,
                                                          uint32_t* __restrict__ out) {
  __shared__ int s_e[8];
  __shared__ float s_s[8];
  __shared__ int s_scale;
  const int j = blockIdx.x, tid = threadIdx.x;
  wait_for_predecessor();
  const double* col = B + (size_t)j * ldb;
  auto at = [&](int c) { return bal ? shift_exp(col[c], -bal[c]) : col[c]; };
  Norm nm;
  if (j < n)
    for (int c = tid; c < k; c += 256) nm.add(col[c], bal ? -bal[c] : 0);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const int e2 = __shfl_xor_sync(0xffffffffu, nm.e, off);
    const float s2 = __shfl_xor_sync(0xffffffffu, nm.s, off);
    nm.merge(e2, s2);
  }
  if ((tid & 31) == 0) {
    s_e[tid >> 5] = nm.e;
    s_s[tid >> 5] = nm.s;
  }
  __syncthreads();
  if (tid == 0) {
    Norm all;
    for (int w = 0; w < 8; ++w) all.merge(s_e[w], s_s[w]);
    s_scale = all.scale();
    cscale[j] = s_scale;
  }
  __syncthreads();
  const int sc = s_scale;
  const bool live = j < n && sc < kZeroScale, bad = sc == kBadScale;
  const size_t plane = (size_t)np * kp / 2;
  for (int c = 2 * tid; c < kp; c += 512) {
    const long long v0 = (live && c < k) ? scaled_int(at(c), sc) : 0ll;
    const long long v1 = (live && c + 1 < k) ? scaled_int(at(c + 1), sc) : 0ll;
    const Chunks b0(v0), b1(v1);
    uint32_t* o = out + ((size_t)j * kp + c) / 2;
#pragma unroll
    for (int i = 0; i < kMod; ++i) o[i * plane] = pack_hi(residue_bits(b0, kT.wb[i], i), residue_bits(b1, kT.wb[i], i));
    o[kMod * plane] = pack_hi(abs_bits(v0, bad), abs_bits(v1, bad));
  }
}

// ---- the residue GEMMs --------------------------------------------------------------------------------------
// tcgen05 shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row
// groups 1024 bytes apart, descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffff) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Instruction descriptor, kind::f16: D = F32, A = B = BF16, both K-major, M = N = 256 over the CTA pair.
constexpr uint32_t kPairIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kPN >> 3) << 17) | ((uint32_t)(kPM >> 4) << 24);

__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// TMA load into this CTA's shared memory, its bytes counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y),
               "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(kPairIdesc), "r"(accum));
}
// Arrives on the barrier at this offset in both CTAs once the MMAs issued so far are done.
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void remote_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct CrtArgs {
  int m, n;            // valid rows / columns of this block
  int mp, np;          // padded to 256
  int kblocks;         // kp / 64
  int8_t* R;           // [kMod][mp][np] residues of the product, a row's columns contiguous
  const int* rscale;
  const int* cscale;
  int* flags;          // [np / 128][mp / 128]
};

// Unit -> (plane, tile): plane after plane, tiles in column stripes eight row
// tiles high, so the units in flight share A and B rows in L2.
__device__ __forceinline__ void unit_tile(int u, int tiles, int tm, int tn, int* plane, int* mi, int* ni) {
  *plane = u / tiles;
  const int t = u - *plane * tiles;
  const int stripe = t / (8 * tn), in = t - stripe * 8 * tn;
  const int h = min(8, tm - stripe * 8);
  *mi = stripe * 8 + in % h;
  *ni = in / h;
}

// Past this K a sum's remainder mod 255 needs a second reduction to fit a byte:
// 1 / 255 is 5.9e-8 too large in FP32, so from |x| = 8,454,907 on a quotient next to
// a tie rounds the wrong way and leaves +128.  Sums of 512 products stay below 2^23;
// the other odd moduli leave at most 127 up to 2^24.
constexpr int kOnceMaxK = 512;

// x - p round(x / p), exact for integers up to 2^24.
__device__ __forceinline__ float reduce_once(float x, float p, float inv) {
  return fmaf(-p, fmaf(x, inv, 12582912.f) - 12582912.f, x);
}

// Sixteen FP32 integers -> their balanced residues mod p as bytes (p = 256:
// 128 wraps to -128, the same residue).
__device__ __forceinline__ uint4 reduce_pack16(const uint32_t* v, float p, float inv) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float x = __uint_as_float(v[4 * j + i]);
      const float k = fmaf(x, inv, 12582912.f) - 12582912.f;
      b[i] = __float_as_uint(fmaf(-p, k, x) + 12582912.f);  // the integer in the low mantissa bits
    }
    w[j] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// kShort, kOneChunk: K <= 512 and K <= 1024, one exact sum per output and no register
// accumulators (the second reduction in the short products' code too costs the LU of
// order 8192, K = 128, 2.7%).
enum CrtForm { kShort, kOneChunk, kChunks };
template <CrtForm FORM>
__global__ void __launch_bounds__(kCrtThreads, 1) __cluster_dims__(2, 1, 1)
    crt_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                    const __grid_constant__ CUtensorMap mapR, const CrtArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[kStagesC], empty_bar[kStagesC], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int tm = g.mp / kPM, tn = g.np / kPN, tiles = tm * tn, units = tiles * (kMod + 1);
  const int nchunks = (g.kblocks + kChunkBlocks - 1) / kChunkBlocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesC; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 16);  // eight epilogue warps of each CTA
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;
  wait_for_predecessor();

  if (warp == 0 && lane == 0) {
    // producer: this CTA's 128 rows of A and 128 columns of B of every k-block
    int gk = 0;
    bool ok = true;
    for (int u = pair; u < units && ok; u += npairs) {
      int plane, mi, ni;
      unit_tile(u, tiles, tm, tn, &plane, &mi, &ni);
      const int ya = plane * g.mp + mi * kPM + (int)rank * 128, yb = plane * g.np + ni * kPN + (int)rank * 128;
      for (int kb = 0; kb < g.kblocks; ++kb, ++gk) {
        const int s = gk % kStagesC;
        if (!mbar_wait(&empty_bar[s], ((uint32_t)(gk / kStagesC) & 1u) ^ 1u)) {
          ok = false;
          break;
        }
        unsigned char* st = smem + (size_t)s * kStageBytesC;
        const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
        if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * kStageBytesC);
        tma_load_2d_pair(st, &mapA, kb * kKB, ya, bar);
        tma_load_2d_pair(st + kHalfTile, &mapB, kb * kKB, yb, bar);
      }
    }
    // before the CTAs leave: every stage consumed and its arrival received, or,
    // after a time-out, at least every load landed
    for (int i = max(0, gk - kStagesC); i < gk; ++i) {
      if (ok) mbar_wait(&empty_bar[i % kStagesC], (uint32_t)(i / kStagesC) & 1u);
      else if (rank == 0) mbar_wait(&full_bar[i % kStagesC], (uint32_t)(i / kStagesC) & 1u);
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // MMA issuer for the pair
    int gk = 0, gc = 0;
    bool ok = true;
    for (int u = pair; u < units && ok; u += npairs) {
      for (int kb = 0; kb < g.kblocks; ++kb, ++gk) {
        const int slot = gc & 1;
        if (kb % kChunkBlocks == 0) {
          if (!mbar_wait(&acc_empty[slot], ((uint32_t)(gc >> 1) & 1u) ^ 1u)) {
            ok = false;
            break;
          }
        }
        const int s = gk % kStagesC;
        if (!mbar_wait(&full_bar[s], (uint32_t)(gk / kStagesC) & 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = smem_u32(smem + (size_t)s * kStageBytesC);
        const uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + kHalfTile);
#pragma unroll
        for (int kk = 0; kk < kKB / 16; ++kk)  // K = 16 per instruction: +32 bytes in the swizzled row
          mma_pair(tmem + (uint32_t)slot * kPN, da + 2 * kk, db + 2 * kk, (kb % kChunkBlocks != 0 || kk > 0) ? 1u : 0u);
        commit_pair(&empty_bar[s]);
        if (kb % kChunkBlocks == kChunkBlocks - 1 || kb == g.kblocks - 1) {
          commit_pair(&acc_full[slot]);
          ++gc;
        }
      }
    }
  } else if (warp >= 2) {
    // epilogue: TMEM lanes 32 (warp mod 4) .. + 31 (this CTA's rows), 128 of the 256 columns
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int row_in = (int)rank * 128 + q * 32 + lane;
    unsigned char* stage_warp = smem + (size_t)kStagesC * kStageBytesC + (size_t)(warp - 2) * kStoreBytes;
    unsigned char* stage = stage_warp + lane * 128;
    int gc = 0;
    bool ok = true;
    for (int u = pair; u < units && ok; u += npairs) {
      int plane, mi, ni;
      unit_tile(u, tiles, tm, tn, &plane, &mi, &ni);
      const bool residue = plane < kMod;
      const float p = residue ? kT.pf[plane] : 0.f, inv = residue ? kT.inv[plane] : 0.f;
      const int row = mi * kPM + row_in, col0 = ni * kPN + half * 128;
      // this warp's staging: row `lane`, 16-byte column groups swizzled by the
      // row (the tensor map's 128-byte swizzle); its last store has been read
      if (residue) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
      }
      float acc[128];
      if constexpr (FORM == kChunks) {
#pragma unroll
        for (int i = 0; i < 128; ++i) acc[i] = 0.f;
      }
      for (int ch = 0; ch < nchunks; ++ch, ++gc) {
        const int slot = gc & 1;
        if (!mbar_wait(&acc_full[slot], (uint32_t)(gc >> 1) & 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(slot * kPN + half * 128);
#pragma unroll
        for (int c0 = 0; c0 < 128; c0 += 16) {
          uint32_t v[16];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(taddr + (uint32_t)c0));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          // p = 0 on the ratio plane: x itself
          if constexpr (FORM != kChunks) {
            if (residue) {
              if (FORM == kOneChunk && p == 255.f) {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(reduce_once(__uint_as_float(v[i]), p, inv));
              }
              *reinterpret_cast<uint4*>(stage + (((c0 / 16) ^ (lane & 7)) << 4)) = reduce_pack16(v, p, inv);
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) acc[c0 + i] = __uint_as_float(v[i]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[c0 + i] += reduce_once(__uint_as_float(v[i]), p, inv);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) remote_arrive(mapa_u32(smem_u32(&acc_empty[slot]), 0));
      }
      if (!ok) break;
      if (residue) {
        if constexpr (FORM == kChunks) {
#pragma unroll
          for (int c0 = 0; c0 < 128; c0 += 16)
            *reinterpret_cast<uint4*>(stage + (((c0 / 16) ^ (lane & 7)) << 4)) =
                reduce_pack16(reinterpret_cast<uint32_t*>(acc + c0), p, inv);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&mapR, col0, plane * g.mp + row, stage_warp);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      } else {
        bool bad = false;
        if (row < g.m) {
          // the exact zeros of an all-zero row or column pass (against a NaN they are NaN)
          const bool zero_row = g.rscale[row] == kZeroScale;
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (col0 + i < g.n && !(acc[i] >= kMinCos) &&
                !(acc[i] == 0.f && (zero_row || g.cscale[col0 + i] == kZeroScale)))
              bad = true;
        }
        if (bad) g.flags[(col0 / kFlagTile) * (g.mp / kFlagTile) + row / kFlagTile] = 1;
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  let_successor_in();
  cluster_barrier();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ---- residues -> C ------------------------------------------------------------------------------------------
__device__ __forceinline__ double pow2d(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// x 2^e for a signed 128-bit x (x.w the top word), rounded to nearest even by
// integer instructions: conversions and multiplies would each take the FP64
// pipe, which issues two lanes per cycle and SM.
__device__ __forceinline__ double scaled_double(uint4 x, int e) {
  const uint32_t sign = (uint32_t)((int)x.w >> 31);
  {  // |x|
    asm("{\n .reg .u32 c;\n and.b32 c, %4, 1;\n xor.b32 %0, %0, %4;\n xor.b32 %1, %1, %4;\n xor.b32 %2, %2, %4;\n"
        " xor.b32 %3, %3, %4;\n add.cc.u32 %0, %0, c;\n addc.cc.u32 %1, %1, 0;\n addc.cc.u32 %2, %2, 0;\n"
        " addc.u32 %3, %3, 0;\n}"
        : "+r"(x.x), "+r"(x.y), "+r"(x.z), "+r"(x.w)
        : "r"(sign));
  }
  // the leading one into the top word: whole words first (rare: |x| < 2^96)
  int lead = 127;
  while (x.w == 0u) {
    if ((x.x | x.y | x.z) == 0u) return 0.0;
    x.w = x.z;
    x.z = x.y;
    x.y = x.x;
    x.x = 0u;
    lead -= 32;
  }
  const int z = __clz((int)x.w);
  const uint32_t t1 = __funnelshift_l(x.z, x.w, z), t0 = __funnelshift_l(x.y, x.z, z);
  const uint32_t rest = (t0 & 0x7ffu) | (((x.y << z) | x.x) != 0u ? 1u : 0u);
  uint32_t hi = t1 >> 11, lo = __funnelshift_r(t0, t1, 11);
  const uint32_t up = (rest + (lo & 1u)) > 0x400u ? 1u : 0u;
  asm("add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, 0;" : "+r"(lo), "+r"(hi) : "r"(up));
  const int ex = 1023 + lead - z + e;  // biased exponent of the leading one
  if (ex > 0 && ex < 2046)  // hi's leading one adds the last 1; a carry moves on
    return __hiloint2double((int)((hi + ((uint32_t)(ex - 1) << 20)) | (sign & 0x80000000u)), (int)lo);
  // over- or underflow in the result: the scaling in two exact halves
  const double v = (double)(((unsigned long long)hi << 32) | lo);
  const int e0 = ex - 1023 - 52, e1 = e0 / 2;
  const double r = v * pow2d(max(min(e1, 1000), -1000)) * pow2d(max(min(e0 - e1, 1000), -1000));
  return sign ? -r : r;
}

// The digits of X for four elements at a time: byte dot products of the
// residues with the digits of P / p (dp4a, four moduli each), the sums carried
// into a 128-bit number, the nearest multiple of P subtracted (|X| < P / 4, so
// the quotient sum y_p / p needs no more than 14-bit weights).
//
// One thread: 4 rows x 4 columns, a warp 16 x 32 (32-byte pieces of R's rows
// and of C's columns).  Bound by instruction issue: 200 per element, 112 us for
// 4096 x 4096 (with 21-bit limbs in 64-bit words and FP64 conversions 280 and
// 200 us; the bytes would take 100).  C is read with the residues and alpha's and
// beta's cases are told apart on the host: an FP64 compare each per element and a
// load behind each store cost the LU of order 8192 62.1 ms against 57.6.
enum CombineMode { kPlain, kScaled, kAdded, kGeneral };  // beta = 0: alpha = 1 or not; beta = 1; neither
__global__ void __launch_bounds__(128) crt_combine_kernel(CrtArgs g, int mode, double alpha, double beta,
                                                          double* __restrict__ C, int64_t ldc) {
  __shared__ uint4 s_mult[2 * kKMax + 1];
  if (threadIdx.x < 2 * kKMax + 1) s_mult[threadIdx.x] = kP.v[threadIdx.x];
  __syncthreads();
  wait_for_predecessor();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * 64 + warp * 16 + (lane >> 3), j0 = blockIdx.y * 32 + (lane & 7) * 4;
  if (j0 >= g.n) return;
  if (g.flags[(j0 / kFlagTile) * (g.mp / kFlagTile) + i0 / kFlagTile]) return;  // the FP64 kernel's tile
  const size_t plane = (size_t)g.mp * g.np / 4;
  const int4 cs = *reinterpret_cast<const int4*>(g.cscale + j0);
#pragma unroll 1
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + 4 * r;
    if (i >= g.m) return;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(g.R) + ((size_t)i * g.np + j0) / 4;
    uint32_t y[kMod];
#pragma unroll
    for (int p = 0; p < kMod; ++p) y[p] = src[p * plane];
    const int rs = g.rscale[i];
    double* const cp = C + (size_t)j0 * ldc + i;
    double old[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) old[c] = mode >= kAdded && j0 + c < g.n ? cp[c * ldc] : 0.0;
    // 4 x 4 byte transposes: y[4 h + c] = the residues of column c for moduli 4 h .. 4 h + 3
#pragma unroll
    for (int h = 0; h < kMod; h += 4) {
      const uint32_t a = __byte_perm(y[h], y[h + 1], 0x5140), b = __byte_perm(y[h], y[h + 1], 0x7362);
      const uint32_t c = __byte_perm(y[h + 2], y[h + 3], 0x5140), d = __byte_perm(y[h + 2], y[h + 3], 0x7362);
      y[h] = __byte_perm(a, c, 0x5410);
      y[h + 1] = __byte_perm(a, c, 0x7632);
      y[h + 2] = __byte_perm(b, d, 0x5410);
      y[h + 3] = __byte_perm(b, d, 0x7632);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      int q = 1 << 13;
      uint32_t t[8];
#pragma unroll
      for (int h = 0; h < kMod / 4; ++h) q = __dp4a((int)y[4 * h + c], (int)kT.quot[h], q);
#pragma unroll
      for (int l = 0; l < 16; l += 2) {
        int s0 = kDigitBias, s1 = kDigitBias;
#pragma unroll
        for (int h = 0; h < kMod / 4; ++h) {
          s0 = __dp4a((int)y[4 * h + c], (int)kT.digit[h][l], s0);
          if (l + 1 < kDigits) s1 = __dp4a((int)y[4 * h + c], (int)kT.digit[h][l + 1], s1);
        }
        t[l / 2] = (uint32_t)s0 + ((uint32_t)s1 << 8);
      }
      const uint4 kp = s_mult[(q >> 14) + kKMax];
      unsigned long long u[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) u[l] = (unsigned long long)t[2 * l + 1] * 65536ull + t[2 * l];
      uint4 x;
      x.x = (uint32_t)u[0];
      asm("add.cc.u32 %0, %3, %4;\n addc.cc.u32 %1, %5, %6;\n addc.u32 %2, %7, %8;"
          : "=&r"(x.y), "=&r"(x.z), "=&r"(x.w)
          : "r"((uint32_t)(u[0] >> 32)), "r"((uint32_t)u[1]), "r"((uint32_t)(u[1] >> 32)), "r"((uint32_t)u[2]),
            "r"((uint32_t)(u[2] >> 32)), "r"((uint32_t)u[3]));
      asm("sub.cc.u32 %0, %0, %4;\n subc.cc.u32 %1, %1, %5;\n subc.cc.u32 %2, %2, %6;\n subc.u32 %3, %3, %7;"
          : "+r"(x.x), "+r"(x.y), "+r"(x.z), "+r"(x.w)
          : "r"(kp.x), "r"(kp.y), "r"(kp.z), "r"(kp.w));
      // an all-zero row or column has X = 0, whatever its scale's code
      const double v = scaled_double(x, -(rs + (c == 0 ? cs.x : c == 1 ? cs.y : c == 2 ? cs.z : cs.w)));
      if (j0 + c < g.n) {
        double w = v;
        if (mode == kScaled) w = alpha * v;
        else if (mode == kAdded) w = fma(alpha, v, old[c]);
        else if (mode == kGeneral) w = fma(alpha, v, beta * old[c]);
        cp[c * ldc] = w;
      }
    }
  }
}

int make_map(CUtensorMap* map, CUtensorMapDataType type, uint64_t elem, void* base, uint64_t rows, uint64_t cols,
             uint32_t box_rows, uint32_t box_cols) {
  EncodeTiledFn f = encode_fn();
  if (!f) return record_arg_error(-100, "dgemm: cuTensorMapEncodeTiled unavailable");
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * elem};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = f(map, type, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? NACU_SUCCESS : record_arg_error(-101, "dgemm: cuTensorMapEncodeTiled failed");
}

// A block of at most kBlockMN x kBlockMN outputs and kBlockK products per output.
constexpr int kBlockMN = 4096, kBlockK = 8192;

struct CrtLayout {
  int mb, nb, kb;  // block extents, padded
  size_t a_off, b_off, r_off, part_off, rs_off, cs_off, flag_off, total;
};
CrtLayout crt_layout(int m, int n, int k) {
  CrtLayout L;
  L.mb = (int)round_up((size_t)std::min(m, kBlockMN), kPM);
  L.nb = (int)round_up((size_t)std::min(n, kBlockMN), kPN);
  L.kb = (int)round_up((size_t)std::min(k, kBlockK), kKB);
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = round_up(o + bytes, 1024);
    return at;
  };
  L.a_off = take((size_t)(kMod + 1) * L.mb * L.kb * 2);
  L.b_off = take((size_t)(kMod + 1) * L.nb * L.kb * 2);
  L.r_off = take((size_t)kMod * L.mb * L.nb);
  L.part_off = take((size_t)((L.kb + stat_chunk(L.kb) - 1) / stat_chunk(L.kb)) * L.mb * sizeof(int2));
  L.rs_off = take((size_t)L.mb * 4);
  L.cs_off = take((size_t)L.nb * 4);
  L.flag_off = take((size_t)(L.mb / kFlagTile) * (L.nb / kFlagTile) * 4);
  L.total = o + 1024;  // room to align the caller's pointer
  return L;
}

}  // namespace

// The two forms' times in us, from measurements.  The FP64 kernel: 1.05 per unit
// of k until its tiles fill the chip, then 1.22 TFLOP/s.  The residues: six
// dependent launches a block, about 35 us (47 where each waits for the one before
// to end instead of being launched ahead), then 18 planes of each operand to write
// and read and 16 of the product.  Measured, FP64 against residues: 128^3 136 and
// 33, 256^3 266 and 38, 8192 x 1 x 8192 8523 and 1945, 1 x 1 x 8192 8266 and 156;
// with the launches one by one 64 x 64 x 32 38 and 46, 20000 x 4 x 64 197 and 256,
// 64 x 8192 x 64 72 and 132.
bool crt_gemm_pays(int m, int n, int k) {
  if (m <= 0 || n <= 0 || k <= 0) return false;
  const auto blocks = [](int x, int b) { return (double)((x + b - 1) / b); };
  const double mn = (double)m * n, fp64 = fmax(1.05 * k, 1.64e-6 * mn * k);
  const double crt = 42 * blocks(m, kBlockMN) * blocks(n, kBlockMN) * blocks(k, kBlockK) +
                     3e-5 * ((double)m * k + (double)k * n) + 2e-5 * mn;
  return crt < fp64;
}

size_t crt_gemm_workspace_bytes(int m, int n, int k) {
  return (m <= 0 || n <= 0 || k <= 0) ? 0 : crt_layout(m, n, k).total;
}

// CTA pairs the device keeps resident (a die whose SM count is odd leaves one SM without a partner).
static int crt_max_pairs(size_t smem) {
  static int pairs = 0;
  if (pairs == 0 && ensure_dynamic_smem(crt_gemm_kernel<kChunks>, smem) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)sm_count() & ~1u);
    cfg.blockDim = dim3(kCrtThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int c = 0;
    if (cudaOccupancyMaxActiveClusters(&c, crt_gemm_kernel<kChunks>, &cfg) != cudaSuccess || c < 1) {
      (void)cudaGetLastError();
      c = std::max(1, sm_count() / 2);
    }
    pairs = c;
  }
  return std::max(pairs, 1);
}

int crt_gemm_run(int m, int n, int k, double alpha, const double* A, int64_t lda, const double* B, int64_t ldb,
                 double beta, double* C, int64_t ldc, void* workspace, size_t workspace_bytes, cudaStream_t s,
                 const char* name, const int* balance) {
  const CrtLayout L = crt_layout(m, n, k);
  if (!workspace || workspace_bytes < L.total) return record_arg_error(-13, "dgemm: workspace too small");
  unsigned char* ws = reinterpret_cast<unsigned char*>(round_up(reinterpret_cast<uintptr_t>(workspace), 1024));
  uint32_t* ap = reinterpret_cast<uint32_t*>(ws + L.a_off);
  uint32_t* bp = reinterpret_cast<uint32_t*>(ws + L.b_off);
  int2* part = reinterpret_cast<int2*>(ws + L.part_off);
  int* rs = reinterpret_cast<int*>(ws + L.rs_off);
  int* cs = reinterpret_cast<int*>(ws + L.cs_off);
  int* flags = reinterpret_cast<int*>(ws + L.flag_off);
  constexpr int planes = kMod + 1;  // and the ratio plane
  constexpr size_t smem = (size_t)kStagesC * kStageBytesC + 8 * kStoreBytes + 1024;
  const auto kern = k <= kOnceMaxK            ? crt_gemm_kernel<kShort>
                    : k <= kChunkBlocks * kKB ? crt_gemm_kernel<kOneChunk>
                                              : crt_gemm_kernel<kChunks>;
  cudaError_t e = ensure_dynamic_smem(kern, smem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  const int pairs = crt_max_pairs(smem);
  if (balance && k > kBlockK) balance = nullptr;  // one block's depth
  for (int k0 = 0; k0 < k; k0 += kBlockK) {
    const int kc = std::min(kBlockK, k - k0), kp = (int)round_up((size_t)kc, kKB);
    const double bt = k0 == 0 ? beta : 1.0;
    for (int n0 = 0; n0 < n; n0 += kBlockMN) {
      const int nc = std::min(kBlockMN, n - n0), np = (int)round_up((size_t)nc, kPN);
      e = launch_chained(crt_split_b_kernel, dim3(np), 256, 0, s, kc, nc, B + (size_t)n0 * ldb + k0, ldb, np, kp,
                         balance, cs, bp);
      if (e != cudaSuccess) return record_cuda_error(e, name);
      for (int m0 = 0; m0 < m; m0 += kBlockMN) {
        const int mc = std::min(kBlockMN, m - m0), mp = (int)round_up((size_t)mc, kPM);
        const double* a = A + (size_t)k0 * lda + m0;
        double* c = C + (size_t)n0 * ldc + m0;
        const int chunk = stat_chunk(L.kb), nparts = (kc + chunk - 1) / chunk;
        const int nflags = (mp / kFlagTile) * (np / kFlagTile);
        e = launch_chained(crt_row_stats_kernel, dim3((mc + 127) / 128, nparts), 128, 0, s, mc, kc, a, lda, chunk,
                           balance, part, flags, nflags);
        if (e == cudaSuccess)
          e = launch_chained(crt_split_a_kernel, dim3(kp / 64, mp / 32), 256, 0, s, mc, kc, a, lda, part, nparts, mp, kp,
                             balance, rs, ap);
        if (e != cudaSuccess) return record_cuda_error(e, name);
        CUtensorMap mapA, mapB, mapR;
        int rc = make_map(&mapA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ap, (uint64_t)planes * mp, kp, 128, kKB);
        if (rc == NACU_SUCCESS)
          rc = make_map(&mapB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, bp, (uint64_t)planes * np, kp, 128, kKB);
        if (rc == NACU_SUCCESS)
          rc = make_map(&mapR, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ws + L.r_off, (uint64_t)kMod * mp, np, 32, 128);
        if (rc != NACU_SUCCESS) return rc;
        CrtArgs g{mc, nc, mp, np, kp / kKB, reinterpret_cast<int8_t*>(ws + L.r_off), rs, cs, flags};
        const int units = (mp / kPM) * (np / kPN) * planes;
        // The large LU's updates (balance) run beside its panels, whose clusters wait
        // for a whole kernel where every SM holds a CTA to its end: two rounds of
        // shorter ones take n = 8192 from 64.5 to 62.2 ms (four rounds 62.1, eight 63.5).
        e = launch_chained(kern, dim3(2 * std::min(units, balance ? 2 * pairs : pairs)), kCrtThreads, smem, s, mapA, mapB, mapR, g);
        const int mode = bt == 0.0 ? (alpha == 1.0 ? kPlain : kScaled) : bt == 1.0 ? kAdded : kGeneral;
        if (e == cudaSuccess)
          e = launch_chained(crt_combine_kernel, dim3((mc + 63) / 64, (nc + 31) / 32), 128, 0, s, g, mode, alpha, bt, c, ldc);
        if (e != cudaSuccess) return record_cuda_error(e, name);
        rc = dgemm_fp64_run(mc, nc, kc, alpha, a, lda, B + (size_t)n0 * ldb + k0, ldb, bt, c, ldc, flags,
                              mp / kFlagTile, s);
        if (rc != NACU_SUCCESS) return rc;
      }
    }
  }
  return NACU_SUCCESS;
}

int crt_gemm_error(int* flag) {
  const cudaError_t e = cudaMemcpyFromSymbol(flag, g_tc_error, sizeof(int));
  return e == cudaSuccess ? NACU_SUCCESS : record_cuda_error(e, "nacu_split_gemm_error");
}

}  // namespace nacu
