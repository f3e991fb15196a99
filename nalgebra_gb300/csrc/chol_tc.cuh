// Cholesky factor and solve of one matrix by one CTA with the trailing updates
// on the tensor cores (slices.cuh), the FMA form of chol_ragged.cu's larger
// orders.  Follows src/linalg/cholesky.rs:221-272 (lower triangle only) in
// right-looking blocks of 16 columns, the right-hand sides riding along as
// extra rows (their forward solve, cholesky.rs:122-129).
//
// Per block of 16 columns:
//   head   warp 0 factors the 16 x 16 diagonal block while the other warps
//          finish the previous block's trailing update;
//   rows   one thread per row below solves its 16 entries against the head in
//          registers (no barrier inside) and leaves their digit slices in
//          shared memory;
//   update warps take 16-row tiles x 32 columns of the trailing lower triangle:
//          28 mma per 16 x 8 tile, the result subtracted in global memory (L2).
//          The next block's columns come first, so its head can start.
// Three barriers per 16 columns.  The back solve goes the same way, with rows of
// the factor in place of rows below the head.
#pragma once
#include "chol_device.cuh"
#include "slices.cuh"

namespace nacu {
namespace {

constexpr int kTcBlock = 16;
constexpr int kTcMaxRhs = 16;  // right-hand sides that ride along

// Slots of the slices: rows below the first head (of 16) and 16 for the right-hand sides.
__host__ __device__ constexpr int tc_slots(int n_max) { return (n_max + 15) / 16 * 16; }
__host__ __device__ constexpr int tc_slice_bytes(int n_max) { return tc_slots(n_max) * kSliceRow; }
// Shared memory: slices, X (nrhs columns), 1 / L_ii, the head and its scratch,
// the slices' exponents and patterns, the factor's row exponents.
__host__ __device__ constexpr size_t tc_smem_bytes(int n_max, int nrhs) {
  return (size_t)kSlices * tc_slice_bytes(n_max) + ((size_t)(n_max | 1) * (nrhs + 1) + 1 + 16 * 17) * 8 +
         (size_t)3 * tc_slots(n_max) * 4;
}

// Element e of a 16 x 16 lower triangle packed by columns: 16 r + c.
__device__ __forceinline__ int tc_packed(int e) {
  int c = 0;
  while (e >= 16 - c) {
    e -= 16 - c;
    ++c;
  }
  return 16 * (c + e) + c;
}

// The 16 x 16 head at column J0 (w <= 16 columns of the matrix; the rest an
// identity): factored by one warp, written to the matrix, to Hd[j * 16 + r]
// (column j) and 1 / L_jj to rdiag.  The 136 elements lie packed over the
// lanes, five each, so an elimination step's FMAs fill the warp (a warp-wide
// FP64 instruction costs its full time however few lanes are active: 40 FMA
// instructions against 72 with a row per lane pair); column j goes through
// shared memory.  The elimination is the square-root-free one,
// a_rc -= a_rj (a_cj / d_j), so a step's chain has a reciprocal (three dependent
// FP64 instructions) and not a reciprocal root (five); the roots of all 16
// pivots are taken together at the end.  S: 16 doubles of scratch.
__device__ __noinline__ void tc_head(int n, double* __restrict__ a, int J0, double* Hd, double* rdiag,
                                     const uint8_t* packed, int* s_info, int has_subst, double subst, int lane) {
  const int w = min(kTcBlock, n - J0);
  double* S = Hd + 256;
  double v[5];
  int rc[5];
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int e = lane + 32 * s;
    rc[s] = e < 136 ? packed[e] : 0;  // past the end: (0, 0), never updated
    const int r = rc[s] >> 4, c = rc[s] & 15;
    v[s] = r < w ? a[(size_t)(J0 + c) * n + J0 + r] : (r == c ? 1.0 : 0.0);
    if (e < 16) Hd[e] = v[s];
  }
  __syncwarp();
  int fail = 0;
  constexpr int base[17] = {0, 16, 31, 45, 58, 70, 81, 91, 100, 108, 115, 121, 126, 130, 133, 135, 136};
#pragma unroll
  for (int j = 0; j < kTcBlock; ++j) {
    double* col = Hd + j * 16;
    double d = col[j];
    const double x = col[lane & 15];
    if (!pos_or_inf(d)) {  // cholesky.rs:237-268, as chol_pivot
      if (has_subst && !(subst <= 0.0) && subst >= 0.0) d = subst;
      else if (fail == 0) fail = J0 + j + 1;
    }
    if (j == kTcBlock - 1) {
      __syncwarp();
      if (lane == 0) col[j] = d;
      break;
    }
    S[lane & 15] = x * rcp_cubic(d);  // both half warps: the same values
    __syncwarp();
    if (lane == 0) col[j] = d;
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      if (32 * s + 31 >= base[j + 1]) {
        const int r = rc[s] >> 4, c = rc[s] & 15;
        if (c > j) v[s] = fma(-S[r], col[c], v[s]);
        if (c == j + 1) Hd[c * 16 + r] = v[s];
      }
    }
    __syncwarp();
  }
  if (fail) {
    if (lane == 0) *s_info = fail;
    return;
  }
  __syncwarp();
  {
    const double d = Hd[(lane & 15) * 17], r = rsqrt_halley(d);
    __syncwarp();
    S[lane & 15] = r;
    if (lane < w) rdiag[J0 + lane] = r;
    if (lane < 16) Hd[lane * 17] = d * r;
  }
  __syncwarp();
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int e = lane + 32 * s, r = rc[s] >> 4, c = rc[s] & 15;
    const double x = r > c ? Hd[c * 16 + r] * S[c] : Hd[c * 17];
    if (e < 136) {
      if (r > c) Hd[c * 16 + r] = x;
      if (r < w) a[(size_t)(J0 + c) * n + J0 + r] = x;
    }
  }
}

// A row's pattern: bit k for a nonzero entry k, and kTcThin where fewer than ten of its 16
// entries are within 1/16 of the largest.  Rows that are not thin meet in four entries at
// least: their products hold 1/64 of the largest entries' product, and the digits' error
// is within the FP64 loop's bound (slices.cuh).  Dense rows are thin once in some hundreds.
constexpr uint32_t kTcThin = 1u << 16;
__device__ __forceinline__ uint32_t tc_pattern(const double (&x)[16]) {
  int h[16], hm = 0, near = 0;
  uint32_t bits = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    h[k] = __double2hiint(x[k]) & 0x7fffffff;
    hm = max(hm, h[k]);
    bits |= (h[k] | __double2loint(x[k])) != 0 ? 1u << k : 0u;
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) near += h[k] >= hm - (4 << 20) ? 1 : 0;
  return bits | (near < 10 ? kTcThin : 0u);
}

// The elements of one 16 x 8 tile with a thin row whose large terms do not meet (slices.cuh),
// by FP64 sums over the entries that both rows hold; a bit for each of a lane's four that
// are done so.  l: row 0 of the tile's rows at the block's columns.
__device__ __noinline__ int tc_update_thin(int n, const double* l, int64_t row_stride, int64_t stride, const double* lc,
                                           double* p, int64_t p_row, int64_t p_col, int on, const unsigned char* sa,
                                           const unsigned char* sc, const int* ea, const int* ec, const uint32_t* pa,
                                           const uint32_t* pc, int lane) {
  const int g = lane >> 2, t = lane & 3;
  float met[4] = {0.f, 0.f, 0.f, 0.f};
  slice_met(sa, sc, lane, met);
  int done = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = g + (i >> 1) * 8, c = 2 * t + (i & 1);
    if (!(on >> i & 1) || met[i] >= kMeet || ea[r] + ec[c] >= kBadRow) continue;
    double s = 0.0;
    for (uint32_t b = pa[r] & pc[c] & 0xffffu; b != 0; b &= b - 1) {
      const int k = __ffs((int)b) - 1;
      s = fma(l[r * row_stride + k * stride], lc[c + (size_t)k * n], s);
    }
    p[r * p_row + c * p_col] -= s;
    done |= 1 << i;
  }
  return done;
}

// A tile of the trailing update: rows of tile `rt` (16 rows from j1 + 16 rt, or
// the right-hand sides) against columns c0 .. c1 (relative to j1, multiples of
// 8), a warp.  Tiles with thin rows are checked: parts of a system that are coupled
// weakly, or whose right-hand sides have other scales, keep what the loop in FP64 keeps
// (a coupling or a right-hand side of 2^-60 beside one of 1 was lost).  The checks take
// 20,000 systems of 8..256 from 17.7 to 18.8 ms, 600 sparse ones (5% of B in B B^T) of
// order 256 from 1.5 to 3.9 (all in FP64 4.0); those of right-hand sides alone 18.9.
__device__ __noinline__ void tc_update(int n, double* __restrict__ a, double* X, int ldx, int nrhs, int j1, int rt,
                                          bool rhs, int rhs_slot, int c0, int c1, const unsigned char* SL, int sb,
                                          const int* ex, const uint32_t* pat, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const int slot = rhs ? rhs_slot : 16 * rt;
  const bool thin = __any_sync(0xffffffffu, pat[slot + (lane & 15)] & kTcThin);
  const unsigned char* sa = SL + slot * kSliceRow;
  const int e0 = ex[slot + g], e1 = ex[slot + g + 8];
  const int r0 = rhs ? g : j1 + slot + g;  // rows r0 and r0 + 8
  const int rmax = rhs ? nrhs : n;
  for (int c = c0; c < c1; c += 8) {
    const int col = j1 + c + 2 * t;  // columns col and col + 1
    double* p[4];
    double v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = r0 + (i >> 1) * 8, cc = col + (i & 1);
      const bool on = rr < rmax && cc < n && (rhs || cc <= rr);
      p[i] = !on ? nullptr : rhs ? X + (size_t)rr * ldx + cc : a + (size_t)cc * n + rr;
      v[i] = on ? *p[i] : 0.0;
    }
    if (thin || __any_sync(0xffffffffu, pat[c + (lane & 7)] & kTcThin)) {
      const int k0 = j1 - kTcBlock, on = (p[0] ? 1 : 0) | (p[1] ? 2 : 0) | (p[2] ? 4 : 0) | (p[3] ? 8 : 0);
      const int first = j1 + c;
      const int done = rhs ? tc_update_thin(n, X + k0, ldx, 1, a + (size_t)k0 * n + first, X + first, ldx, 1, on, sa,
                                            SL + c * kSliceRow, ex + slot, ex + c, pat + slot, pat + c, lane)
                           : tc_update_thin(n, a + (size_t)k0 * n + j1 + slot, 1, n, a + (size_t)k0 * n + first,
                                            a + (size_t)first * n + j1 + slot, 1, n, on, sa, SL + c * kSliceRow,
                                            ex + slot, ex + c, pat + slot, pat + c, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (done >> i & 1) p[i] = nullptr;
    }
    float acc[kSlices][4];
    slice_products(sa, SL + c * kSliceRow, sb, lane, acc);
    const int f0 = ex[c + 2 * t], f1 = ex[c + 2 * t + 1];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double x = slice_value(acc, i, (i >> 1 ? e1 : e0) + (i & 1 ? f1 : f0));
      if (p[i]) *p[i] = v[i] - x;
    }
  }
}

// Factor the matrix a (n x n, column-major, in place) and, for nrhs <= 16
// columns in X, the forward solve.  *s_info 0 or the first failing pivot; rexp the
// largest exponents of L's rows left of their diagonal blocks, kBadRow past the last.
__device__ __forceinline__ void chol_tc_cta(int n, double* __restrict__ a, int n_max, int nrhs, double* X, int ldx,
                                            unsigned char* SL, double* rdiag, double* Hd, int* ex, int* rexp, uint32_t* pat,
                                            const uint8_t* packed, int* s_info, int* s_next, int has_subst, double subst) {
  const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;
  const int sb = tc_slice_bytes(n_max);
  if (warp == 0) tc_head(n, a, 0, Hd, rdiag, packed, s_info, has_subst, subst, lane);
  __syncthreads();
  for (int J0 = 0; J0 < n; J0 += kTcBlock) {
    if (*s_info != 0) return;
    const int j1 = J0 + kTcBlock, m = max(0, n - j1);
    const int w = min(kTcBlock, n - J0);
    const int mt = (m + 15) >> 4, rhs_slot = 16 * mt, slots = rhs_slot + (nrhs > 0 ? 16 : 0);
    // rows below the head
    for (int s = tid; s < slots; s += nthr) {
      const bool rhs = s >= rhs_slot;
      const int r = rhs ? s - rhs_slot : j1 + s;
      unsigned char* s0 = SL + s * kSliceRow;
      if (rhs ? r >= nrhs : r >= n) {
        slice_zero_row(s0, sb);
        ex[s] = 1;
        pat[s] = 0;
        if (!rhs) rexp[r] = kBadRow;
        continue;
      }
      double* p = rhs ? X + (size_t)r * ldx + J0 : a + (size_t)J0 * n + r;
      const size_t st = rhs ? 1 : (size_t)n;
      double x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = j < w ? p[j * st] : 0.0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        x[j] *= j < w ? rdiag[J0 + j] : 0.0;
#pragma unroll
        for (int c = j + 1; c < 16; ++c) x[c] = fma(-x[j], Hd[j * 16 + c], x[c]);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < w) p[j * st] = x[j];
      const int em = slice_row(x, s0, sb);
      ex[s] = em;
      pat[s] = tc_pattern(x);
      if (!rhs) rexp[r] = J0 == 0 ? em : max(rexp[r], em);
    }
    if (tid == 0) *s_next = nw - 1;
    __syncthreads();
    if (m == 0) break;
    // the next block's columns
    for (int rt = warp; rt < mt + (nrhs > 0 ? 1 : 0); rt += nw)
      tc_update(n, a, X, ldx, nrhs, j1, rt, rt == mt, rhs_slot, 0, 16, SL, sb, ex, pat, lane);
    __syncthreads();
    // the rest, in units of 16 rows x 32 columns: row tile i > 0 has ceil(i / 2), tiles 2 k - 1 and 2 k
    // together 2 k, so the first 2 k tiles k (k + 1)
    const int k1 = mt >> 1;  // tiles 1 .. mt - 1
    const int tri = (mt & 1) ? k1 * (k1 + 1) : k1 * k1;
    const int units = tri + (nrhs > 0 ? (max(0, m - 16) + 31) / 32 : 0);
    int u = warp - 1;
    if (warp == 0) {
      tc_head(n, a, j1, Hd, rdiag, packed, s_info, has_subst, subst, lane);
      u = units;
      if (nw == 1) u = 0;
      else {
        if (lane == 0) u = atomicAdd(s_next, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
      }
    }
    while (u < units) {
      if (u < tri) {
        int k = (int)((1.0f + sqrtf(1.0f + 4.0f * (float)u)) * 0.5f);
        if (k * (k - 1) > u) --k;
        if (k * (k + 1) <= u) ++k;
        const int rem = u - k * (k - 1);
        const int i = rem < k ? 2 * k - 1 : 2 * k, grp = rem < k ? rem : rem - k;
        tc_update(n, a, X, ldx, nrhs, j1, i, false, 0, 16 + 32 * grp, min(48 + 32 * grp, 16 * i + 16), SL, sb, ex, pat, lane);
      } else {
        const int c0 = 16 + 32 * (u - tri);
        tc_update(n, a, X, ldx, nrhs, j1, 0, true, rhs_slot, c0, min(c0 + 32, (m + 7) & ~7), SL, sb, ex, pat, lane);
      }
      if (nw == 1) {
        ++u;
      } else {
        if (lane == 0) u = atomicAdd(s_next, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
      }
    }
    __syncthreads();
  }
  __syncthreads();
}

// One block of the back solve by one warp: the 16 x 16 transposed triangle at J0, four
// right-hand sides at a time, eight lanes of two rows each; the rows pre-scaled by
// 1 / L_jj, so the chain is one FMA per step.
__device__ __forceinline__ void tc_backward_block(int n, const double* __restrict__ a, int J0, int nrhs, double* X, int ldx,
                                                  const double* rdiag, double* Hd, int lane) {
  const int w = min(16, n - J0);
  // Hd[j * 16 + i] = L_ji / L_jj (row j of the block)
  for (int e = lane; e < 256; e += 32) {
    const int i = e >> 4, j = e & 15;
    Hd[j * 16 + i] = (j < w && i < j) ? a[(size_t)(J0 + i) * n + J0 + j] * rdiag[J0 + j] : 0.0;
  }
  __syncwarp();
  for (int c0 = 0; c0 < nrhs; c0 += 4) {
    const int c = c0 + (lane >> 3), q = lane & 7;
    double* xc = X + (size_t)min(c, nrhs - 1) * ldx + J0;
    double y0 = q < w ? xc[q] : 0.0, y1 = q + 8 < w ? xc[q + 8] : 0.0;
#pragma unroll
    for (int j = 15; j > 0; --j) {
      const double yj = __shfl_sync(0xffffffffu, j >= 8 ? y1 : y0, (lane & 24) + (j & 7));
      y0 = fma(-yj, Hd[j * 16 + q], y0);  // zero for rows >= j
      if (j > 8) y1 = fma(-yj, Hd[j * 16 + q + 8], y1);
    }
    if (c < nrhs) {
      if (q < w) xc[q] = y0 * rdiag[J0 + q];
      if (q + 8 < w) xc[q + 8] = y1 * rdiag[J0 + q + 8];
    }
  }
}

// x = L^-T y for the nrhs columns of X, in blocks of 16 rows from the bottom, in FP64:
// a block solved by warp 0 while the other warps' threads load a row of L above it each
// (column i's 16 entries are contiguous), then y_i -= sum_r L_ri x_r, a thread per row.
__device__ __noinline__ void chol_tc_backward_fp64_cta(int n, const double* __restrict__ a, int nrhs, double* X, int ldx,
                                                       const double* rdiag, double* Hd) {
  const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int first = warp == 0 ? nthr - 32 + tid : tid - 32;  // this thread's first row
  for (int J0 = (n - 1) / 16 * 16; J0 >= 0; J0 -= 16) {
    const int w = min(16, n - J0);
    double l[16];
    const auto load = [&](int i) {
      const double* p = a + (size_t)i * n + J0;
#pragma unroll
      for (int r = 0; r < 16; ++r) l[r] = i < J0 && r < w ? p[r] : 0.0;
    };
    if (warp == 0) tc_backward_block(n, a, J0, nrhs, X, ldx, rdiag, Hd, lane);
    else load(first);
    __syncthreads();
    for (int i = first; i < J0; i += nthr) {
      if (warp == 0 || i != first) load(i);
      for (int c = 0; c < nrhs; ++c) {
        double* const x = X + (size_t)c * ldx;
        double s = 0.0;  // summed apart: one rounding of y a block
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (r < w) s = fma(l[r], x[J0 + r], s);
        x[i] -= s;
      }
    }
    __syncthreads();
  }
}

// One sum of the back solve in FP64; out of line, most blocks have none.
__device__ __noinline__ void tc_backward_fp64(const double* l, const double* x, int w, double* y) {
  double s = 0.0;
  for (int r = 0; r < w; ++r) s = fma(l[r], x[r], s);
  *y -= s;
}

// The same for the nrhs <= 16 columns with the products on the tensor cores: the other
// warps cut the block's row of L into slices while warp 0 solves its triangle, then
// y_i -= sum_r L_ri x_r for all rows i above, 16 x 8 tiles on the tensor cores.
// For A = D A0 D the entries L_ri go as d_r and x_r as 1 / d_r, where the factor's and
// the forward solve's slices, along rows, hold one scale each.  So L_ri is cut against
// row r's largest exponent and x_r the other way; where that leaves sums whose large
// terms do not meet (slices.cuh; in proportion to the terms where the last block has
// fewer than 16), an FP64 loop forms them.  (Without it, D of 2^+-20 left 1e-4 of an
// error of 3e-14.)
__device__ __forceinline__ void chol_tc_backward_cta(int n, const double* __restrict__ a, int n_max, int nrhs, double* X,
                                                     int ldx, unsigned char* SL, const double* rdiag, double* Hd, int* ex,
                                                     const int* rexp) {
  const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;
  const int sb = tc_slice_bytes(n_max);
  const int rhs_slots = nrhs > 8 ? 16 : 8;
  for (int J0 = (n - 1) / 16 * 16; J0 >= 0; J0 -= 16) {
    const int w = min(16, n - J0);
    if (warp == 0) {
      tc_backward_block(n, a, J0, nrhs, X, ldx, rdiag, Hd, lane);
      __syncwarp();
      if (lane < rhs_slots && J0 > 0) {  // the solved block as slices
        unsigned char* s0 = SL + (J0 + lane) * kSliceRow;
        if (lane < nrhs) {
          double x[16];
#pragma unroll
          for (int r = 0; r < 16; ++r) x[r] = r < w ? X[(size_t)lane * ldx + J0 + r] : 0.0;
          ex[J0 + lane] = slice_row_raised(x, rexp + J0, s0, sb);
        } else {
          slice_zero_row(s0, sb);
          ex[J0 + lane] = kNoExponent;
        }
      }
    }
    if (J0 == 0) break;
    if (warp > 0 || nw == 1)
      for (int i = nw == 1 ? tid : tid - 32; i < J0; i += nw == 1 ? nthr : nthr - 32) {
        const double* p = a + (size_t)i * n + J0;
        double x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) x[r] = r < w ? p[r] : 0.0;
        ex[i] = slice_row_lowered(x, rexp + J0, SL + i * kSliceRow, sb);
      }
    __syncthreads();
    const int tiles = (J0 >> 4) * (rhs_slots >> 3);
    const float meet = kMeet / 16.f * (float)w;
    for (int u = warp; u < tiles; u += nw) {
      const int it = rhs_slots > 8 ? u >> 1 : u, c8 = rhs_slots > 8 ? (u & 1) * 8 : 0;
      const int g = lane >> 2, t = lane & 3;
      const int i0 = 16 * it + g, c = c8 + 2 * t;
      float acc[kSlices + 1][4], met[4] = {0.f, 0.f, 0.f, 0.f};
      slice_sums_start(acc);
      slice_products_met(SL + 16 * it * kSliceRow, SL + (J0 + c8) * kSliceRow, sb, lane, acc, met);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int i = i0 + (v >> 1) * 8, cc = c + (v & 1);
        const int el = ex[i], er = ex[J0 + cc];
        const double x = slice_value(acc, v, el + er);
        double* const y = X + (size_t)cc * ldx;
        if (cc >= nrhs) continue;
        if (er == kBadRow || (met[v] < meet && el != kNoExponent && er != kNoExponent))
          tc_backward_fp64(a + (size_t)i * n + J0, y + J0, w, y + i);
        else
          y[i] -= x;
      }
    }
    __syncthreads();
  }
  __syncthreads();
}

}  // namespace
}  // namespace nacu
