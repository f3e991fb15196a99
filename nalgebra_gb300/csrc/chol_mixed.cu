// Ragged batched SPD solve in mixed precision: FP32 Cholesky factor, FP64
// iterative refinement.  The chosen precision form of nalgebra's
// `m.cholesky().solve(&b)` (src/linalg/cholesky.rs:221-272, 122-143): same
// inputs and outputs as the FP64 form, solutions refined until the normwise
// backward error ||b - A x||_inf / (||A||_inf ||x||_inf + ||b||_inf) is at the
// FP64 target (n * eps64 by default).
//
// Why: on GB300 FP32 runs at ~74x the FP64 rate.  The O(n^3) factorization
// and the triangular solves move to FP32; only the O(n^2) residual
// r = b - A x, the correction accumulation x += d and the fallback stay FP64.
//
// Per matrix (one CTA, persistent grid, largest matrices first):
//   1. A's lower triangle is converted to FP32 into the caller's workspace
//      (A itself is read-only); ||A||_inf comes from the first FP64 residual;
//   2. FP32 Cholesky (the same left-looking panel code as the FP64 kernel);
//   3. x0 = solve32(b), then repeat: r = b - A x in FP64 (A read from its lower
//      triangle, symmetric), stop if the backward error meets the target, else
//      d = solve32(r) (right-hand sides scaled by powers of two so FP32 never
//      under- or overflows) and x += d in FP64.  After two corrections the
//      contraction rate rho = ||d_k|| / ||d_{k-1}|| predicts the error of the
//      next iterate; when rho * ||d_k|| is far below the target the last
//      residual is skipped (NACU_FLAG_VERIFY forces it).
//   4. A matrix that is not SPD in FP32, or whose refinement stagnates
//      (rho > 1/2) or runs out of iterations, is refactored in FP64 in the
//      workspace and solved there: the per-matrix `iters` output records it.
#include "chol_device.cuh"

namespace nacu {
namespace {

constexpr double kEps64 = 2.220446049250313e-16;

struct MixedArgs {
  int count;
  int n_max;
  const int32_t* ns;
  const int64_t* aoff;
  const double* A;
  int nrhs;
  const int64_t* boff;
  const double* B;
  double* X;
  int32_t* info;
  int32_t* iters;
  const int32_t* order;
  int32_t* counter;
  double* W;  // per matrix n*n doubles at W + aoff[s]
  double tol_units;
  int max_iter;
  int verify;
  int has_subst;
  double subst;
};

__device__ __forceinline__ unsigned long long abs_bits(double x) { return abs_bits_f64(x); }

// max over the CTA of per-thread values (non-negative doubles compared as
// integers: no FP64 instructions); red: kRhsChunk x 4 warps scratch.
__device__ __forceinline__ void block_max4(unsigned long long (&v)[kRhsChunk], unsigned long long* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < kRhsChunk; ++c) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[c], off);
      v[c] = o > v[c] ? o : v[c];
    }
  }
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c) red[warp * kRhsChunk + c] = v[c];
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kRhsChunk; ++c) {
    unsigned long long m = 0;
    for (int w = 0; w < kCholThreads / 32; ++w) m = red[w * kRhsChunk + c] > m ? red[w * kRhsChunk + c] : m;
    v[c] = m;
  }
}

// R = B - A X for the symmetric A stored in its lower triangle (column-major,
// lda = n), nr <= 4 right-hand sides; X and R in shared memory (ld = ldx).
// Lane = row: elements left of the diagonal block come from column j (row
// i of L, coalesced), elements right of it from column i (A_ij = A_ji).
// The FP64 pipe bounds it, so the four warps take equal runs of the (32 rows x 8
// columns) pieces: whole row blocks, one warp each, left half the warps idle at
// n = 160 or 192.  A row block that a warp takes over in the middle goes to `part`
// (3 x 128 doubles, and 3 x 32 floats after the n row sums in rsum) and is added
// in the warps' order.
__device__ __noinline__ void residual_fp64(int n, const double* __restrict__ a, const double* __restrict__ b, int nr,
                              const double* Xd, double* Rd, int ldx, double* part, float* rsum, bool with_norm,
                              float* rowmax) {
  constexpr int U = 8;  // independent loads in flight per thread
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunks = (n + U - 1) / U, blocks = (n + 31) / 32;
  const int pieces = chunks * blocks;
  const int p1 = pieces * (warp + 1) / 4;
  for (int p = pieces * warp / 4; p < p1;) {
    const int blk = p / chunks, c0 = p - blk * chunks;
    const int c1 = min(chunks, c0 + p1 - p);
    p += c1 - c0;
    const int rb = blk * 32, i = rb + lane;
    const bool valid = i < n;
    const int ii = valid ? i : n - 1;
    double acc[kRhsChunk];
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c) acc[c] = (c0 == 0 && c < nr) ? b[(size_t)c * n + ii] : 0.0;
    float rs = 0.0f;  // sum |A_ij| over the row in FP32 (first residual only; off the FP64 pipe)
    const int dend = min(rb + 32, n);
    const double* colii = a + (size_t)ii * n;
    // element (ii, j): column j (left of / in the diagonal block, j <= ii) or
    // column ii (right of it), both from the lower triangle
    for (int j0 = c0 * U; j0 < c1 * U; j0 += U) {
      double av[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = j0 + u;
        av[u] = (j < n) ? ((j <= ii && j < dend) ? a[(size_t)j * n + ii] : colii[j]) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = j0 + u;
        if (j < n) {
          if (with_norm) rs += abs_f32_lower(av[u]);
#pragma unroll
          for (int c = 0; c < kRhsChunk; ++c) acc[c] = fma(-av[u], Xd[(size_t)c * ldx + j], acc[c]);
        }
      }
    }
    if (c0 > 0) {
#pragma unroll
      for (int c = 0; c < kRhsChunk; ++c) part[(warp - 1) * 128 + c * 32 + lane] = acc[c];
      rsum[n + (warp - 1) * 32 + lane] = rs;
    } else if (valid) {
#pragma unroll
      for (int c = 0; c < kRhsChunk; ++c)
        if (c < nr) Rd[(size_t)c * ldx + i] = acc[c];
      rsum[i] = rs;
    }
  }
  __syncthreads();
  // warp 0 adds what the others took over (at most one row block each)
  if (warp == 0)
    for (int w = 1; w < 4; ++w) {
      const int p = pieces * w / 4, blk = p / chunks, i = blk * 32 + lane;
      if (p - blk * chunks > 0 && p < pieces * (w + 1) / 4 && i < n) {
#pragma unroll
        for (int c = 0; c < kRhsChunk; ++c)
          if (c < nr) Rd[(size_t)c * ldx + i] += part[(w - 1) * 128 + c * 32 + lane];
        rsum[i] += rsum[n + (w - 1) * 32 + lane];
      }
    }
  __syncthreads();
  if (with_norm) {
    float m = 0.0f;
    for (int i = tid; i < n; i += kCholThreads) m = fmaxf(m, rsum[i]);
    *rowmax = m;
  }
}

// block_max4 whose result goes to shared memory (out[0..kRhsChunk)), so the
// norms do not occupy registers across the solves.
__device__ __forceinline__ void block_max4_to(unsigned long long (&v)[kRhsChunk], unsigned long long* red,
                                              unsigned long long* out) {
  block_max4(v, red);
  if (threadIdx.x < kRhsChunk) out[threadIdx.x] = v[threadIdx.x & (kRhsChunk - 1)];
  __syncthreads();
}

// Asynchronous copy of one float to shared memory (zero where !valid).
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// X <- L^-T L^-1 X for the FP32 factor L (lower triangle in global memory,
// lda = n), X in shared memory as one float4 of right-hand sides per row, padded
// with zero rows to a multiple of 32.  tiles: 4 x kTile floats.
//
// The chain through a 32 x 32 diagonal block, one warp's shuffles, and the
// latency of the loads bound a solve of this size, not its arithmetic.  So warp
// 0 runs one block ahead: it applies the block solved last to its own block only
// and goes on, while warps 1-3 apply it to everything else and fetch warp 0's
// next two 32 x 32 tiles.  One barrier a block, and no load on the chain.
// 20,000 matrices of 8..256, four right-hand sides: the solves are 18% of the
// refinement's 14.6 ms; with loads on the chain and all warps waiting for it they
// were 31% of 16.2 ms.
constexpr int kTile = 32 * 33;
__device__ __noinline__ void solve32_cta(int n, const float* __restrict__ a, float4* X, const float* rdiag, float* tiles) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = (n + 31) / 32;
  // tile (rb, cb) of L into T[c * 33 + r]: column c's rows in 32 different banks, and row r's columns too
  const auto fetch = [&](int rb, int cb, float* T, int w, int nw) {
    const int r = rb * 32 + lane;
    for (int c = w; c < 32; c += nw) {
      const int col = cb * 32 + c;
      const bool valid = r < n && col <= r;
      copy_async(T + c * 33 + lane, valid ? a + (size_t)col * n + r : a, valid);
    }
  };
  fetch(0, 0, tiles, warp, 4);
  copies_wait();
  __syncthreads();
  for (int k = 0; k < nb; ++k) {
    float* const cur = tiles + (k & 1) * 2 * kTile;
    float* const nxt = tiles + ((k + 1) & 1) * 2 * kTile;
    if (warp == 0) {
      const int r = k * 32 + lane;
      float4 b = X[r];
      if (k > 0) {
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
          const float l = cur[kTile + i * 33 + lane];
          const float4 y = X[(k - 1) * 32 + i];
          b.x = fmaf(-y.x, l, b.x);
          b.y = fmaf(-y.y, l, b.y);
          b.z = fmaf(-y.z, l, b.z);
          b.w = fmaf(-y.w, l, b.w);
        }
      }
      const float rd = r < n ? rdiag[r] : 0.f;
#pragma unroll 8
      for (int i = 0; i < 32; ++i) {
        const float l = cur[i * 33 + lane];
        const float4 y = make_float4(b.x * rd, b.y * rd, b.z * rd, b.w * rd);
        const float yx = __shfl_sync(0xffffffffu, y.x, i), yy = __shfl_sync(0xffffffffu, y.y, i);
        const float yz = __shfl_sync(0xffffffffu, y.z, i), yw = __shfl_sync(0xffffffffu, y.w, i);
        if (lane > i) {
          b.x = fmaf(-yx, l, b.x);
          b.y = fmaf(-yy, l, b.y);
          b.z = fmaf(-yz, l, b.z);
          b.w = fmaf(-yw, l, b.w);
        }
      }
      if (r < n) X[r] = make_float4(b.x * rd, b.y * rd, b.z * rd, b.w * rd);
    } else {
      if (k + 1 < nb) {
        fetch(k + 1, k + 1, nxt, warp - 1, 3);
        fetch(k + 1, k, nxt + kTile, warp - 1, 3);
      }
      if (k > 0)
        for (int r = (k + 1) * 32 + tid - 32; r < n; r += kCholThreads - 32) {
          const float* lp = a + (size_t)(k - 1) * 32 * n + r;
          float4 b = X[r];
#pragma unroll
          for (int i0 = 0; i0 < 32; i0 += 16) {
            float l[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) l[u] = lp[(size_t)(i0 + u) * n];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
              const float4 y = X[(k - 1) * 32 + i0 + u];
              b.x = fmaf(-y.x, l[u], b.x);
              b.y = fmaf(-y.y, l[u], b.y);
              b.z = fmaf(-y.z, l[u], b.z);
              b.w = fmaf(-y.w, l[u], b.w);
            }
          }
          X[r] = b;
        }
      copies_wait();
    }
    __syncthreads();
  }
  // Backward: the last diagonal tile is still in place; a tile lies transposed
  // here, lane = column.
  for (int k = nb - 1; k >= 0; --k) {
    float* const cur = tiles + (k & 1) * 2 * kTile;
    float* const nxt = tiles + ((k + 1) & 1) * 2 * kTile;
    if (warp == 0) {
      const int r = k * 32 + lane;
      float4 y = X[r];
      if (k + 1 < nb) {
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
          const float l = cur[kTile + lane * 33 + i];
          const float4 x = X[(k + 1) * 32 + i];
          y.x = fmaf(-x.x, l, y.x);
          y.y = fmaf(-x.y, l, y.y);
          y.z = fmaf(-x.z, l, y.z);
          y.w = fmaf(-x.w, l, y.w);
        }
      }
      const float rd = r < n ? rdiag[r] : 0.f;
#pragma unroll 8
      for (int i = 31; i >= 0; --i) {
        const float l = cur[lane * 33 + i];
        const float4 x = make_float4(y.x * rd, y.y * rd, y.z * rd, y.w * rd);
        const float xx = __shfl_sync(0xffffffffu, x.x, i), xy = __shfl_sync(0xffffffffu, x.y, i);
        const float xz = __shfl_sync(0xffffffffu, x.z, i), xw = __shfl_sync(0xffffffffu, x.w, i);
        if (lane < i) {
          y.x = fmaf(-xx, l, y.x);
          y.y = fmaf(-xy, l, y.y);
          y.z = fmaf(-xz, l, y.z);
          y.w = fmaf(-xw, l, y.w);
        }
      }
      if (r < n) X[r] = make_float4(y.x * rd, y.y * rd, y.z * rd, y.w * rd);
    } else if (k > 0) {
      fetch(k - 1, k - 1, nxt, warp - 1, 3);
      fetch(k, k - 1, nxt + kTile, warp - 1, 3);
      // y of block k - 1 less what the blocks below k give: four columns a
      // warp, lanes along the rows, and a reduce-scatter of the 16 sums
      const int r0 = (k + 1) * 32;
      if (r0 < n)
        for (int cb = (k - 1) * 32 + (warp - 1) * 4; cb < k * 32; cb += 12) {
          float v[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = 0.f;
          const float* lp = a + (size_t)cb * n;
          for (int rl = r0 + lane; rl < n; rl += 96) {
            float l[3][4];
#pragma unroll
            for (int h = 0; h < 3; ++h)
#pragma unroll
              for (int j = 0; j < 4; ++j) l[h][j] = rl + 32 * h < n ? lp[(size_t)j * n + rl + 32 * h] : 0.f;
#pragma unroll
            for (int h = 0; h < 3; ++h) {
              if (rl + 32 * h >= n) break;
              const float4 x = X[rl + 32 * h];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                v[j * 4 + 0] = fmaf(l[h][j], x.x, v[j * 4 + 0]);
                v[j * 4 + 1] = fmaf(l[h][j], x.y, v[j * 4 + 1]);
                v[j * 4 + 2] = fmaf(l[h][j], x.z, v[j * 4 + 2]);
                v[j * 4 + 3] = fmaf(l[h][j], x.w, v[j * 4 + 3]);
              }
            }
          }
#pragma unroll
          for (int half = 8; half >= 1; half >>= 1) {
            const bool up = (lane & half) != 0;
#pragma unroll
            for (int t = 0; t < half; ++t) {
              const float keep = up ? v[t + half] : v[t];
              const float give = up ? v[t] : v[t + half];
              v[t] = keep + __shfl_xor_sync(0xffffffffu, give, half);
            }
          }
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
          if (lane < 16) reinterpret_cast<float*>(X + cb + (lane >> 2))[lane & 3] -= v[0];
        }
      copies_wait();
    }
    __syncthreads();
  }
}

// FP32 solve with the FP32 factor: X32 <- L^-T L^-1 (src * 2^-e_c), returned
// in FP64 times 2^e_c (power-of-two scaling: exact, keeps FP32 in range).
__device__ __noinline__ void solve32_scaled(int n, const float* L32, const double* src, int ldsrc, int nr,
                               const unsigned long long* srcnorm, float4* X32, float* tiles, const float* rdiag32,
                               int ldx, double* dst, bool accumulate, unsigned long long* dnorm_out,
                               unsigned long long* red) {
  const int tid = threadIdx.x;
  // scale factors 2^-e and 2^e with e = the exponent of ||src_c||_inf, built
  // from the exponent bits (no FP64 instructions)
  __shared__ double s_down[kRhsChunk], s_up[kRhsChunk];
  if (tid < kRhsChunk) {
    long long ex = (long long)((srcnorm[tid] >> 52) & 0x7ff);
    if (ex == 0 || ex == 0x7ff) ex = 1023;  // zero/denormal/inf/NaN: no scaling
    const long long e = ex - 1023;
    const long long e_dn = (e < -1000) ? -1000 : (e > 1000 ? 1000 : e);
    s_down[tid] = __longlong_as_double((1023 - e_dn) << 52);
    s_up[tid] = __longlong_as_double((1023 + e_dn) << 52);
  }
  __syncthreads();
  for (int r = tid; r < (n + 31) / 32 * 32; r += kCholThreads) {
    float v[kRhsChunk];
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c)
      v[c] = (c < nr && r < n) ? (float)(src[(size_t)c * ldsrc + r] * s_down[c]) : 0.f;
    X32[r] = make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();  // src may lie where the tiles go
  solve32_cta(n, L32, X32, rdiag32, tiles);
  unsigned long long dn[kRhsChunk] = {0, 0, 0, 0};
  for (int r = tid; r < n; r += kCholThreads) {
    const float4 x = X32[r];
    const float v[kRhsChunk] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c)
      if (c < nr) {
        const double d = (double)v[c] * s_up[c];
        const unsigned long long ab = abs_bits(d);
        dn[c] = ab > dn[c] ? ab : dn[c];
        if (accumulate) dst[(size_t)c * ldx + r] += d;
        else dst[(size_t)c * ldx + r] = d;
      }
  }
  if (dnorm_out) block_max4_to(dn, red, dnorm_out);
}

// FP32 left-looking Cholesky for the refinement form.  Same panel structure as
// chol_factor_cta, but the panel itself is factored by warp 0 alone
// (warp-synchronous, no CTA barriers per column): in FP32 the arithmetic is
// cheap and the per-column barriers, not the math, set the time.
// b0, b1: two buffers of kb_cols staged columns of L with leading dimension ldl
// (a multiple of 4 that covers n_max: float4 reads past `rows` stay inside the
// buffer and only feed discarded accumulators); b1 may share P's space.
// One matrix of 256, all phases: 916 us with blocks loaded between two barriers
// (and the solves waiting for theirs), 660 us so.
__device__ __noinline__ void chol_factor32_cta(int n, float* __restrict__ a, int ldp, float* __restrict__ P, float* b0,
                                  float* b1, int kb_cols, int ldl, float* Hs, float* rdiag, int* s_info, int has_subst,
                                  double subst) {
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31;
  for (int J0 = 0; J0 < n; J0 += kNB) {
    const int jb = min(kNB, n - J0);
    const int rows = n - J0;
    // P = A[J0.., J0..J0+jb] - L[J0.., 0..J0] L[J0..J0+jb, 0..J0]^T: the
    // earlier columns are copied to shared memory kb_cols at a time, the next
    // block under this one's products: one barrier a block.
    const int cg = warp * 4;  // 4 warps x 4 columns = kNB
    for (int rb = 0; rb < rows; rb += kRowsPerPass) {
      // lane owns rows rb + 4*lane + 128*h + {0..3}, h = 0, 1
      float acc[2][4][4];  // [h][row][col]
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = rb + 4 * lane + 128 * h + i, c = cg + j;
            acc[h][i][j] = (r < rows && c < jb && r >= c) ? a[(size_t)(J0 + c) * n + J0 + r] : 0.f;
          }
      const auto stage = [&](int kb, float* Lb) {
        for (int c = warp; c < kb_cols; c += nthr >> 5) {
          const float* src = a + (size_t)(kb + c) * n + J0;
          float* dst = Lb + (size_t)c * ldl;
#pragma unroll 4
          for (int r = lane; r < rows; r += 32) copy_async(dst + r, src + r, true);
        }
      };
      if (J0 > 0) stage(0, b0);
      for (int kb = 0; kb < J0; kb += kb_cols) {  // kb_cols divides kNB, kNB divides J0
        float* const Lb = ((kb / kb_cols) & 1) ? b1 : b0;
        copies_wait();
        __syncthreads();
        if (kb + kb_cols < J0) stage(kb + kb_cols, ((kb / kb_cols) & 1) ? b0 : b1);
        if (cg < jb) {
#pragma unroll 2
          for (int k = 0; k < kb_cols; ++k) {
            const float* lk = Lb + (size_t)k * ldl;
            const float4 lc = *reinterpret_cast<const float4*>(lk + cg);  // L[cg..cg+3][k]
            float4 lr[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
              lr[h] = (rb + 4 * lane + 128 * h < rows) ? *reinterpret_cast<const float4*>(lk + rb + 4 * lane + 128 * h)
                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (h == 1 && rb + 128 >= rows) break;  // no row of the upper half
              const float rv[4] = {lr[h].x, lr[h].y, lr[h].z, lr[h].w};
              const float cv[4] = {lc.x, lc.y, lc.z, lc.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[h][i][j] = fmaf(-cv[j], rv[i], acc[h][i][j]);
            }
          }
        }
      }
      if (J0 > 0) __syncthreads();  // the buffers are free: P, and the next pass
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = rb + 4 * lane + 128 * h + i, c = cg + j;
            if (r < rows && c < jb && r >= c) P[(size_t)c * ldp + r] = acc[h][i][j];
          }
    }
    __syncthreads();
    // Panel, without CTA barriers per column: every warp factors the jb x jb
    // head of the panel redundantly (lanes 0..jb-1 hold its rows in
    // registers), keeps L_head and 1/L_jj in its own shared scratch, then
    // updates its share of the rows below the head, each row entirely in
    // registers.
    {
      float* hl = Hs + warp * (kNB * kNB + kNB);  // L_head[c][j] at hl[j*kNB + c], 1/L_jj at hl[kNB*kNB + j]
      float v[kNB];
#pragma unroll
      for (int c = 0; c < kNB; ++c) v[c] = (lane < jb && c <= lane && c < jb) ? P[(size_t)c * ldp + lane] : 0.f;
      bool fail = false;
#pragma unroll
      for (int j = 0; j < kNB; ++j) {
        if (j < jb && !fail) {
          const float d = __shfl_sync(0xffffffffu, v[j], j);
          float denom, rcp;
          if (!chol_pivot<false, float>(d, has_subst, subst, &denom, &rcp)) {
            fail = true;
            if (warp == 0 && lane == 0) *s_info = J0 + j + 1;
          } else {
            if (lane == j) v[j] = denom;
            else if (lane > j) v[j] *= rcp;
            if (lane == 0) hl[kNB * kNB + j] = rcp;
#pragma unroll
            for (int c = j + 1; c < kNB; ++c) {
              const float lcj = __shfl_sync(0xffffffffu, v[j], c);  // L[c][j]
              if (c < jb && lane >= c) v[c] = fmaf(-v[j], lcj, v[c]);
            }
          }
        }
      }
      if (lane < jb)
#pragma unroll
        for (int j = 0; j < kNB; ++j) hl[j * kNB + lane] = v[j];  // row `lane` of L_head
      __syncwarp();
      if (!fail) {
        float* const out = a + (size_t)J0 * n + J0;
        if (warp == 0 && lane < jb) {
#pragma unroll
          for (int c = 0; c < kNB; ++c)
            if (c <= lane && c < jb) out[(size_t)c * n + lane] = v[c];
          rdiag[J0 + lane] = hl[kNB * kNB + lane];
        }
        for (int r = jb + warp * 32 + lane; r < rows; r += nthr) {
          float w[kNB];
#pragma unroll
          for (int c = 0; c < kNB; ++c) w[c] = (c < jb) ? P[(size_t)c * ldp + r] : 0.f;
#pragma unroll
          for (int j = 0; j < kNB; ++j) {
            w[j] *= hl[kNB * kNB + j];  // L[r][j]; zero columns stay zero
#pragma unroll
            for (int c = (j + 1) / 4 * 4; c < kNB; c += 4) {
              const float4 h = *reinterpret_cast<const float4*>(hl + j * kNB + c);
              const float hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (c + q > j) w[c + q] = fmaf(-w[j], hv[q], w[c + q]);
            }
            // keep the compiler from hoisting all the head's loads into registers
            asm volatile("" ::: "memory");
          }
#pragma unroll
          for (int c = 0; c < kNB; ++c)
            if (c < jb) out[(size_t)c * n + r] = w[c];
        }
      }
    }
    __syncthreads();
    if (*s_info != 0) return;
  }
}

// Dynamic shared memory of the refinement kernel (byte offsets):
//   X32  (n_max to a multiple of 32, x 4 floats)  FP32 right-hand sides / solutions; the residual's row sums
//   rd32 (ldp floats)      1 / L_ii of the FP32 factor
//   u    union { P32 panel (ldp x kNB floats) ; Rd residual (ldp x 4 doubles) and
//                its parts (3 x 128 doubles) ; the solves' tiles ; staged L columns, where a panel is one pass }
//   xd   union { staged L columns during the factor ;
//                Xd, the FP64 iterate (ldp x 4 doubles) }
// A panel of more than kRowsPerPass rows is updated in passes that leave their
// result in P32: there both buffers of staged columns lie in xd, at half the size.
struct MixedSmem {
  size_t x32, rd32, u, xd, total;
  int ldl, kb_cols;
  bool shared_panel;  // staged columns in u
};
constexpr int kHeadFloats = (kCholThreads / 32) * (kNB * kNB + kNB);
__host__ __device__ inline MixedSmem mixed_smem_layout(int n_max) {
  MixedSmem L;
  const size_t ldp = (size_t)(n_max | 1);
  L.ldl = ((n_max + 3 + 3) / 4) * 4;  // float4 reads may run 3 past the last row
  L.shared_panel = n_max <= kRowsPerPass;
  L.kb_cols = L.shared_panel ? 8 : 4;
  const auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
  const auto larger = [](size_t x, size_t y) { return x > y ? x : y; };
  L.x32 = 0;
  // X32 is idle during the factor: the per-warp 16 x 16 heads of the FP32
  // panel share its space (no static shared memory for them)
  const size_t x32 = (size_t)((n_max + 31) / 32) * 32 * kRhsChunk * sizeof(float);
  L.rd32 = up16(L.x32 + larger(x32, (size_t)kHeadFloats * sizeof(float)));
  L.u = up16(L.rd32 + ldp * sizeof(float));
  const size_t lb = (size_t)L.ldl * 8 * sizeof(float);
  size_t u = larger(ldp * kNB * sizeof(float), (ldp * kRhsChunk + 3 * 128) * sizeof(double));
  u = larger(u, 4 * kTile * sizeof(float));
  if (L.shared_panel) u = larger(u, lb);
  L.xd = up16(L.u + u);
  L.total = up16(L.xd + larger(ldp * kRhsChunk * sizeof(double), lb));
  return L;
}

// Norms kept in shared memory (indices into nrm[]).
constexpr int kBn = 0, kRn = 4, kXn = 8, kDn = 12, kDprev = 16, kNrmSize = 20;

__device__ void mixed_one(const MixedArgs& g, int s, unsigned char* smem, int* s_info, double* s_scal,
                          unsigned long long* red, float* hs, unsigned long long* nrm) {
  const int tid = threadIdx.x;
  const int n = g.ns[s];
  if (n < 0 || n > g.n_max) {
    if (tid == 0) {
      if (g.info) g.info[s] = -1;
      if (g.iters) g.iters[s] = 0;
    }
    return;
  }
  const int ldp = g.n_max | 1;
  const double* a = g.A + g.aoff[s];
  const double* b = g.B + g.boff[s];
  double* x = g.X + g.boff[s];
  MixedSmem L = mixed_smem_layout(g.n_max);
  float4* X32 = reinterpret_cast<float4*>(smem + L.x32);
  float* rd32 = reinterpret_cast<float*>(smem + L.rd32);
  float* P32 = reinterpret_cast<float*>(smem + L.u);
  double* Rd = reinterpret_cast<double*>(smem + L.u);
  double* Xd = reinterpret_cast<double*>(smem + L.xd);
  float* tiles = reinterpret_cast<float*>(smem + L.u);
  float* W32 = reinterpret_cast<float*>(g.W + g.aoff[s]);

  // 1. convert A's lower triangle to FP32 (one conversion per element: on
  //    this part a hardware FP64<->FP32 conversion costs an FP64 issue slot,
  //    so the normal-range conversion is done with integer instructions).
  //    Only the lower triangle is read: warp w takes the column pairs
  //    (c, n-1-c), c = w, w + 4, ..., whose n + 1 rows are one run of
  //    coalesced 32-row chunks, up to 9 loads in flight per lane.
  //    ||A||_inf is accumulated by the first FP64 residual pass.
  if (tid == 0) *s_info = 0;
  {
    constexpr int U = 9;
    const int warp = tid >> 5, lane = tid & 31;
    for (int c = warp; c < (n + 1) / 2; c += kCholThreads / 32) {
      const int c2 = n - 1 - c;
      const int len1 = n - c;                             // rows c..n-1 of column c
      const int len = (c2 == c) ? len1 : len1 + (c + 1);  // and rows c2..n-1 of column c2
      for (int k0 = 0; k0 < len; k0 += U * 32) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int k = k0 + u * 32 + lane;
          const int idx = (k < len1) ? c * n + c + k : c2 * n + c2 + (k - len1);  // n*n < 2^31
          v[u] = (k < len) ? a[idx] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int k = k0 + u * 32 + lane;
          const int idx = (k < len1) ? c * n + c + k : c2 * n + c2 + (k - len1);
          if (k < len) W32[idx] = f64_to_f32_rn(v[u]);
        }
      }
    }
  }
  {
    unsigned long long bv[kRhsChunk] = {0, 0, 0, 0};
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c)
      if (c < g.nrhs)
        for (int r = tid; r < n; r += kCholThreads) {
          const unsigned long long ab = abs_bits(b[(size_t)c * n + r]);
          bv[c] = ab > bv[c] ? ab : bv[c];
        }
    block_max4_to(bv, red, nrm + kBn);
  }
  double anorm = 0.0;
  // 2. FP32 factor.
  {
    float* b0 = reinterpret_cast<float*>(smem + L.xd);
    float* b1 = L.shared_panel ? reinterpret_cast<float*>(smem + L.u) : b0 + L.kb_cols * L.ldl;
    chol_factor32_cta(n, W32, ldp, P32, b0, b1, L.kb_cols, L.ldl, hs, rd32, s_info, g.has_subst, g.subst);
  }
  int status = *s_info;  // non-zero: not SPD in FP32 -> FP64 fallback
  __syncthreads();
  int used = 0;
  bool converged = false;
  const int nr = g.nrhs;
  const double tol = g.tol_units * (double)(n > 0 ? n : 1) * kEps64;
  if (status == 0 && n > 0) {
    // 3. x0 = solve32(b), then refinement with FP64 residuals.
    solve32_scaled(n, W32, b, n, nr, nrm + kBn, X32, tiles, rd32, ldp, Xd, false, nullptr, red);
    if (tid < kRhsChunk) nrm[kDprev + tid] = 0;
    for (int it = 0; it < g.max_iter; ++it) {
      __syncthreads();
      float rowmax = 0.0f;
      residual_fp64(n, a, b, nr, Xd, Rd, ldp, Rd + 4 * ldp, reinterpret_cast<float*>(X32), it == 0, &rowmax);
      ++used;
      if (it == 0) {  // ||A||_inf: max over the CTA (integer compare on the bits)
        unsigned long long av[kRhsChunk] = {(unsigned long long)__float_as_uint(rowmax), 0, 0, 0};
        block_max4(av, red);
        anorm = (double)__uint_as_float((unsigned)av[0]);  // FP32 row sums; inf only past FLT_MAX
      }
      {
        unsigned long long rn[kRhsChunk] = {0, 0, 0, 0}, xn[kRhsChunk] = {0, 0, 0, 0};
#pragma unroll
        for (int c = 0; c < kRhsChunk; ++c)
          if (c < nr)
            for (int r = tid; r < n; r += kCholThreads) {
              const unsigned long long ra = abs_bits(Rd[(size_t)c * ldp + r]);
              const unsigned long long xa = abs_bits(Xd[(size_t)c * ldp + r]);
              rn[c] = ra > rn[c] ? ra : rn[c];
              xn[c] = xa > xn[c] ? xa : xn[c];
            }
        block_max4_to(rn, red, nrm + kRn);
        block_max4_to(xn, red, nrm + kXn);
      }
      bool ok = true, finite = !isinf(anorm);  // ||A||_inf beyond FP32: the FP64 form takes over
      for (int c = 0; c < nr; ++c) {
        if (nrm[kRn + c] >= 0x7ff0000000000000ull || nrm[kXn + c] >= 0x7ff0000000000000ull) finite = false;
        const double rr = __longlong_as_double((long long)nrm[kRn + c]);
        const double den = anorm * __longlong_as_double((long long)nrm[kXn + c]) +
                           __longlong_as_double((long long)nrm[kBn + c]);
        if (!(rr <= 0.5 * tol * den)) ok = false;
      }
      if (!finite) break;  // FP32 overflow or a non-finite input: FP64 fallback
      if (ok) {
        converged = true;
        break;
      }
      solve32_scaled(n, W32, Rd, ldp, nr, nrm + kRn, X32, tiles, rd32, ldp, Xd, true, nrm + kDn, red);
      // contraction rate and predicted backward error of the new iterate
      bool stagnant = false, predicted = (it >= 1) && !g.verify;
      for (int c = 0; c < nr; ++c) {
        const double d = __longlong_as_double((long long)nrm[kDn + c]);
        const double dp = __longlong_as_double((long long)nrm[kDprev + c]);
        const double rho = (it >= 1 && dp > 0.0) ? d / dp : 1.0;
        if (it >= 1 && rho > 0.5) stagnant = true;
        const double den = anorm * __longlong_as_double((long long)nrm[kXn + c]) +
                           __longlong_as_double((long long)nrm[kBn + c]);
        if (!(anorm * rho * d <= 0.125 * tol * den)) predicted = false;
      }
      __syncthreads();
      if (tid < kRhsChunk) nrm[kDprev + tid] = nrm[kDn + tid];
      if (stagnant) break;
      if (predicted) {
        converged = true;
        break;
      }
    }
  }
  __syncthreads();
  if (!converged && n > 0) {
    // 4. queue the matrix for the FP64 fallback kernel (runs after this one)
    if (tid == 0) {
      const int slot = atomicAdd(g.counter + 1, 1);
      g.counter[4 + slot] = s;
      if (g.info) g.info[s] = 0;
      if (g.iters) g.iters[s] = -(used + 1);
    }
    __syncthreads();
    return;
  }
  if (status == 0)
    for (int c = 0; c < nr; ++c)
      for (int r = tid; r < n; r += kCholThreads) x[(size_t)c * n + r] = Xd[(size_t)c * ldp + r];
  if (tid == 0) {
    if (g.info) g.info[s] = status;
    if (g.iters) g.iters[s] = used;
  }
  __syncthreads();
}

// FP64 fallback for the matrices the refinement kernel queued: factor a copy
// of A in the workspace and solve, exactly the FP64 form's arithmetic.
__global__ void __launch_bounds__(kCholThreads, 4) chol_mixed_fallback_kernel(MixedArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_item;
  __shared__ int s_info;
  __shared__ double s_scal[2 + kCholThreads / 32];
  const int tid = threadIdx.x;
  const int ldp = g.n_max | 1;
  double* P64 = reinterpret_cast<double*>(smem_raw);
  double* Xd = P64 + (size_t)ldp * kNB;
  double* rd64 = Xd + (size_t)ldp * kRhsChunk;
  for (;;) {
    if (tid == 0) s_item = atomicAdd(g.counter + 2, 1);
    __syncthreads();
    const int idx = s_item;
    __syncthreads();
    if (idx >= g.counter[1]) break;
    const int s = g.counter[4 + idx];
    const int n = g.ns[s];
    const int nr = g.nrhs;
    const double* a = g.A + g.aoff[s];
    const double* b = g.B + g.boff[s];
    double* x = g.X + g.boff[s];
    double* W64 = g.W + g.aoff[s];
    for (int e = tid; e < n * n; e += kCholThreads) W64[e] = a[e];
    if (tid == 0) s_info = 0;
    __syncthreads();
    chol_factor_cta<false, double>(n, W64, ldp, P64, rd64, &s_info, s_scal, g.has_subst, g.subst);
    const int status = s_info;
    if (status == 0) {
      for (int e = tid; e < n * nr; e += kCholThreads) {
        const int c = e / n, r = e - c * n;
        Xd[(size_t)c * ldp + r] = b[e];
      }
      __syncthreads();
      chol_forward_cta<false, double>(n, W64, Xd, ldp, nr, rd64);
      chol_backward_fast_cta<double>(n, W64, Xd, ldp, nr, rd64);
      for (int e = tid; e < n * nr; e += kCholThreads) {
        const int c = e / n, r = e - c * n;
        x[e] = Xd[(size_t)c * ldp + r];
      }
    }
    if (tid == 0 && g.info) g.info[s] = status;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kCholThreads, 7) chol_mixed_kernel(MixedArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_item;
  __shared__ int s_info;
  __shared__ double s_scal[2 + kCholThreads / 32];
  __shared__ unsigned long long red[4 * kRhsChunk];
  __shared__ unsigned long long nrm[kNrmSize];
  float* hs = reinterpret_cast<float*>(smem_raw + mixed_smem_layout(g.n_max).x32);
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(g.counter, 1);
    __syncthreads();
    const int idx = s_item;
    __syncthreads();
    if (idx >= g.count) break;
    const int s = g.order ? g.order[idx] : idx;
    mixed_one(g, s, smem_raw, &s_info, s_scal, red, hs, nrm);
  }
}

size_t mixed_smem_bytes(int n_max) { return mixed_smem_layout(n_max).total; }

size_t fallback_smem_bytes(int n_max) {
  const size_t ldp = (size_t)(n_max | 1);
  return ldp * (kNB + kRhsChunk + 1) * sizeof(double);
}

}  // namespace
}  // namespace nacu

extern "C" {

// Workspace: [0,16): queue heads; [16, 16 + 4*count): fallback list, rounded
// up to 256; then 8 bytes per matrix element (FP32 factor or FP64 fallback).
static size_t mixed_head_bytes(int count) { return ((size_t)16 + 4 * (size_t)count + 255) & ~(size_t)255; }

size_t nacu_mixed_workspace_bytes(int count, int64_t total_matrix_elements) {
  return mixed_head_bytes(count) + (size_t)total_matrix_elements * sizeof(double);
}

int nacu_dposv_ragged_mixed(int count, int n_max, const int32_t* ns, const int64_t* a_offsets, const double* A,
                            int nrhs, const int64_t* b_offsets, const double* B, double* X, int32_t* info,
                            int32_t* iters, const int32_t* order, int64_t total_matrix_elements, void* workspace,
                            size_t workspace_bytes, double tol_units, int max_iter, double substitute, int flags,
                            nacu_stream_t stream) {
  using namespace nacu;
  if (count < 0) return record_arg_error(-1, "dposv_ragged_mixed: negative count");
  if (n_max < 0 || n_max > NACU_CHOL_RAGGED_MAX_N)
    return record_arg_error(-2, "dposv_ragged_mixed: n_max out of range [0, 512]");
  if (count == 0) return NACU_SUCCESS;
  if (!ns || !a_offsets || !A) return record_arg_error(-3, "dposv_ragged_mixed: null ns, a_offsets or A");
  if (nrhs < 1 || nrhs > kRhsChunk) return record_arg_error(-6, "dposv_ragged_mixed: nrhs out of range [1, 4]");
  if (!b_offsets || !B || !X) return record_arg_error(-7, "dposv_ragged_mixed: null b_offsets, B or X");
  if (!info) return record_arg_error(-10, "dposv_ragged_mixed: null info");
  if (total_matrix_elements < 0) return record_arg_error(-13, "dposv_ragged_mixed: negative total_matrix_elements");
  if (!workspace || workspace_bytes < nacu_mixed_workspace_bytes(count, total_matrix_elements))
    return record_arg_error(-14, "dposv_ragged_mixed: workspace too small");
  if (flags & NACU_FLAG_EXACT) return record_arg_error(-19, "dposv_ragged_mixed: NACU_FLAG_EXACT does not apply");
  MixedArgs g{count, n_max, ns, a_offsets, A, nrhs, b_offsets, B, X, info, iters, order,
              reinterpret_cast<int32_t*>(workspace),
              reinterpret_cast<double*>(static_cast<unsigned char*>(workspace) + mixed_head_bytes(count)),
              tol_units > 0.0 ? tol_units : 1.0, max_iter > 0 ? max_iter : 10,
              (flags & NACU_FLAG_VERIFY) ? 1 : 0, (flags & NACU_FLAG_SUBSTITUTE) ? 1 : 0, substitute};
  const size_t smem = mixed_smem_bytes(n_max);
  const size_t smem_fb = fallback_smem_bytes(n_max);
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = ensure_dynamic_smem(chol_mixed_kernel, smem);
  if (e == cudaSuccess)
    e = ensure_dynamic_smem(chol_mixed_fallback_kernel, smem_fb);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dposv_ragged_mixed");
  int per_sm = 0, per_sm_fb = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chol_mixed_kernel, kCholThreads, smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_fb, chol_mixed_fallback_kernel, kCholThreads, smem_fb);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dposv_ragged_mixed");
  int grid = sm_count() * (per_sm < 1 ? 1 : per_sm);
  if (grid > count) grid = count;
  int grid_fb = sm_count() * (per_sm_fb < 1 ? 1 : per_sm_fb);
  if (grid_fb > count) grid_fb = count;
  e = cudaMemsetAsync(workspace, 0, 16, s);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dposv_ragged_mixed");
  chol_mixed_kernel<<<grid, kCholThreads, smem, s>>>(g);
  int rc = check_launch("nacu_dposv_ragged_mixed");
  if (rc != NACU_SUCCESS) return rc;
  // Runs after the refinement kernel on the same stream; exits at once when
  // no matrix was queued.
  chol_mixed_fallback_kernel<<<grid_fb, kCholThreads, smem_fb, s>>>(g);
  return check_launch("nacu_dposv_ragged_mixed: fallback");
}

}  // extern "C"
