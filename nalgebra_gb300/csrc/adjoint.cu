// Reverse-mode adjoint of the batched Cholesky solve and log-determinant, for
// batches of equal-order SPD matrices (n <= 128), in FP64 and FP32.
//
// Forward (nalgebra's `m.cholesky()`, `.solve(&b)`, `.ln_determinant()`,
// src/linalg/cholesky.rs:221-272, 122-143, 172-185): x = A^-1 b and
// logdet A = sum ln(L_ii^2); the factor L is written out (the "store" form)
// or discarded (the "recompute" form keeps only A).
//
// Backward, for the cotangents w = dl/dx and g = dl/dlogdet of a loss l
// (default g = 1: the loss l = sum_s w_s^T x_s + logdet A_s; nalgebra has no
// autodiff, this is the chosen differentiation form):
//   v  = A^-1 w                       (dl/db)
//   Abar = -v x^T + g A^-1            (dl/dA for an unstructured A)
// nalgebra reads only the lower triangle, so the parameters are the lower
// entries theta_ij (i >= j) with A_ij = A_ji = theta_ij; the gradient
// returned in dA's lower triangle is
//   dA_ii = Abar_ii = -v_i x_i + g (A^-1)_ii,
//   dA_ij = Abar_ij + Abar_ji = -(v_i x_j + v_j x_i) + 2 g (A^-1)_ij  (i > j),
// which is what central differences on theta_ij measure.  (Giles 2008,
// "Collected matrix derivative results for forward and reverse mode AD";
// Murray 2016, "Differentiation of the Cholesky decomposition".)
//
// Design: one CTA (256 threads) per matrix with the matrix's packed lower
// triangle in shared memory (66 KB at n = 128 in FP64, so three CTAs share an
// SM where the full square allowed one), so the factorization, the in-place
// triangular inverse L -> L^-1 and the product A^-1 = L^-T L^-1 run out of
// shared memory.  Trailing updates use a
// pair-folded index over the lower triangle (column c paired with column
// m-1-c fills an (m+1) x ceil(m/2) rectangle), so no lane idles on the
// triangle's empty half.
#include "chol_tc.cuh"

namespace nacu {
namespace {

constexpr int kAdjThreads = 256;
constexpr int kAdjMaxN = 128;

template <typename T>
__device__ __forceinline__ T fma_t(T a, T b, T c) {
  if constexpr (sizeof(T) == 8) return fma(a, b, c);
  else return fmaf(a, b, c);
}

// Pair-folded enumeration of the lower triangle (rows >= column) of an m x m
// block: rectangle index (k, q), k in [0, m+1), q in [0, ceil(m/2)).
__device__ __forceinline__ bool fold(int m, int k, int q, int* r, int* c) {
  const int len = m - q;  // column q holds rows q..m-1
  if (k < len) {
    *c = q;
    *r = q + k;
    return true;
  }
  const int c2 = m - 1 - q;
  if (c2 <= q) return false;  // odd m: the middle column appears once
  *c = c2;
  *r = c2 + (k - len);
  return *r < m;
}

// Element (r, c), r >= c, of the lower triangle in shared memory sits at
// S[cb[c] + r]: cb[c] = c * ld for a full column-major square, or
// c * n - c (c + 1) / 2 for the packed triangle (column c's rows c..n-1 follow
// column c-1's), which halves the backward kernel's shared memory.

// Right-looking Cholesky of the n x n matrix in S (lower triangle).
// Returns info (0 ok, j+1 first failing pivot) in *s_info.
template <typename T>
__device__ void chol_smem(int n, T* S, const int* cb, int* s_info, T* s_sc) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (int j = 0; j < n; ++j) {
    T* cj = S + cb[j];
    if (tid == 0) {
      const T d = cj[j];
      if (!(d <= T(0)) && d >= T(0)) {
        const T r = rsqrt(d);  // L_jj = d * rsqrt(d), 1/L_jj = rsqrt(d): one dependent FP64 chain
        cj[j] = d * r;
        s_sc[0] = r;
      } else if (*s_info == 0) {
        *s_info = j + 1;
      }
    }
    __syncthreads();
    if (*s_info != 0) return;
    const T rcp = s_sc[0];
    for (int r = j + 1 + tid; r < n; r += nthr) cj[r] *= rcp;
    __syncthreads();
    const int m = n - j - 1;
    if (m > 0) {
      const int qn = (m + 1) >> 1, total = (m + 1) * qn;
      for (int e = tid; e < total; e += nthr) {
        const int q = e / (m + 1), k = e - q * (m + 1);
        int r, c;
        if (fold(m, k, q, &r, &c)) {
          r += j + 1;
          c += j + 1;
          S[cb[c] + r] = fma_t(-cj[r], cj[c], S[cb[c] + r]);
        }
      }
    }
    __syncthreads();
  }
}

// In place L -> L^-1 (lower), columns from right to left (LAPACK trti2 order):
// L^-1[i][j] = -(1/L_jj) * sum_{k=j+1..i} L^-1[i][k] L[k][j]  (i > j).
// Two threads per row i (k split by parity, combined by a shuffle), so all
// warps share each column's dot products; fused multiply-adds; the
// reciprocals of the diagonal (rdiag) are formed once beforehand.  Columns go
// two at a time (j and j-1 share each L^-1[i][k] load and one pair of
// barriers): with s0, s1 the sums over k > j,
//   L^-1[i][j] = -s0 / L_jj,  L^-1[i][j-1] = -(s1 + L^-1[i][j] L[j][j-1]) / L_{j-1,j-1}.
// tmp holds 2n values.
template <typename T>
__device__ void trinv_smem(int n, T* S, const int* cb, T* tmp, const T* rdiag) {
  const int tid = threadIdx.x;
  const int ri = tid >> 1, h = tid & 1;
  int j = n - 1;
  for (; j >= 1; j -= 2) {
    const T* cj = S + cb[j];
    const T* cj1 = S + cb[j - 1];
    const T ajj = rdiag[j], aj1 = rdiag[j - 1];
    const int i = j + 1 + ri;
    T s0 = T(0), s1 = T(0);
    if (i < n)
      for (int k = j + 1 + h; k <= i; k += 2) {
        const T li = S[cb[k] + i];  // L^-1[i][k]
        s0 = fma_t(li, cj[k], s0);
        s1 = fma_t(li, cj1[k], s1);
      }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    if (i < n && h == 0) {
      const T x0 = -ajj * s0;
      tmp[i] = x0;
      tmp[n + i] = -aj1 * fma_t(x0, cj1[j], s1);
    }
    __syncthreads();
    T* cw = S + cb[j];
    T* cw1 = S + cb[j - 1];
    for (int r = j + 1 + tid; r < n; r += blockDim.x) {
      cw[r] = tmp[r];
      cw1[r] = tmp[n + r];
    }
    if (tid == 0) {
      cw1[j] = -aj1 * (ajj * cw1[j]);  // L^-1[j][j-1] = -L[j][j-1] / (L_jj L_{j-1,j-1})
      cw[j] = ajj;
      cw1[j - 1] = aj1;
    }
    __syncthreads();
  }
  if (j == 0) {  // odd n: the first column on its own
    const T* c0 = S + cb[0];
    const T a00 = rdiag[0];
    const int i = 1 + ri;
    T acc = T(0);
    if (i < n)
      for (int k = 1 + h; k <= i; k += 2) acc = fma_t(S[cb[k] + i], c0[k], acc);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    if (i < n && h == 0) tmp[i] = -a00 * acc;
    __syncthreads();
    T* cw = S + cb[0];
    for (int r = 1 + tid; r < n; r += blockDim.x) cw[r] = tmp[r];
    if (tid == 0) cw[0] = a00;
    __syncthreads();
  }
}

// In place L^-1 -> A^-1 = L^-T L^-1 (lower triangle):
// (A^-1)_ij = sum_{k >= i} Linv_ki Linv_kj  (i >= j).  Given L^-1 the columns
// are independent, and column j needs only columns >= j, so four columns are
// formed per pair of barriers (each Linv_ki load feeds four FMAs) into tmp and
// written back over their L^-1 columns.  Two threads per row, k split by
// parity.  tmp holds 4n values.
template <typename T>
__device__ void inv_from_trinv_smem(int n, T* S, const int* cb, T* tmp) {
  const int tid = threadIdx.x;
  const int ri = tid >> 1, h = tid & 1;
  for (int j = 0; j < n; j += 4) {
    const int jw = min(4, n - j);
    const int i = j + ri;
    T acc[4] = {T(0), T(0), T(0), T(0)};
    if (i < n) {
      const T* ci = S + cb[i];
      const T* cju[4] = {S + cb[j], S + cb[min(j + 1, n - 1)], S + cb[min(j + 2, n - 1)], S + cb[min(j + 3, n - 1)]};
      for (int k = i + h; k < n; k += 2) {
        const T lki = ci[k];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < jw && i >= j + u) acc[u] = fma_t(lki, cju[u][k], acc[u]);  // Linv[k][j+u], k >= i >= j+u
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], 1);
      if (i < n && h == 0 && u < jw && i >= j + u) tmp[u * n + i] = acc[u];
    }
    __syncthreads();
    for (int u = 0; u < jw; ++u) {
      T* cw = S + cb[j + u];
      for (int r = j + u + tid; r < n; r += blockDim.x) cw[r] = tmp[u * n + r];
    }
    __syncthreads();
  }
}

// Forward: S <- A (lower), factor, x = A^-1 b (forward + back substitution in
// shared memory), logdet; write L (store form) or nothing.
template <typename T>
__global__ void __launch_bounds__(kAdjThreads) adj_forward_kernel(int n, const T* __restrict__ A, int64_t strideA,
                                                                  const T* __restrict__ B, T* __restrict__ X,
                                                                  T* __restrict__ Lout, T* __restrict__ logdet,
                                                                  int32_t* __restrict__ info, int batch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_info;
  __shared__ T s_sc[2];
  __shared__ int cb[kAdjMaxN];
  T* S = reinterpret_cast<T*>(smem_raw);  // the packed lower triangle
  T* y = S + (size_t)n * (n + 1) / 2;
  const int tid = threadIdx.x;
  for (int c = tid; c < n; c += blockDim.x) cb[c] = c * n - c * (c + 1) / 2;
  __syncthreads();  // every column base is set before any thread stores through it
  for (int s = blockIdx.x; s < batch; s += gridDim.x) {
    const T* a = A + (size_t)s * strideA;
    for (int e = tid; e < n * n; e += blockDim.x) {
      const int c = e / n, r = e - c * n;
      if (r >= c) S[cb[c] + r] = a[e];
    }
    for (int i = tid; i < n; i += blockDim.x) y[i] = B[(size_t)s * n + i];
    if (tid == 0) s_info = 0;
    __syncthreads();
    chol_smem<T>(n, S, cb, &s_info, s_sc);
    const int inf = s_info;
    if (inf == 0) {
      // L y = b then L^T x = y; one warp (n <= 128: four rows per lane)
      if (tid < 32) {
        for (int i = 0; i < n; ++i) {
          if (tid == 0) y[i] = y[i] / S[cb[i] + i];
          __syncwarp();
          const T yi = y[i];
          for (int r = i + 1 + tid; r < n; r += 32) y[r] = fma_t(-yi, S[cb[i] + r], y[r]);
          __syncwarp();
        }
        for (int i = n - 1; i >= 0; --i) {
          T sacc = T(0);
          for (int r = i + 1 + tid; r < n; r += 32) sacc = fma_t(S[cb[i] + r], y[r], sacc);
          sacc = warp_sum(sacc);
          if (tid == 0) y[i] = (y[i] - sacc) / S[cb[i] + i];
          __syncwarp();
        }
      }
      __syncthreads();
      for (int i = tid; i < n; i += blockDim.x) X[(size_t)s * n + i] = y[i];
      if (tid == 0) {
        T sum = T(0);
        for (int i = 0; i < n; ++i) {
          const T d = S[cb[i] + i];
          sum += log(d * d);
        }
        logdet[s] = sum;
      }
      if (Lout)
        for (int e = tid; e < n * n; e += blockDim.x) {
          const int c = e / n, r = e - c * n;
          Lout[(size_t)s * strideA + e] = (r >= c) ? S[cb[c] + r] : T(0);
        }
    }
    if (tid == 0 && info) info[s] = inf;
    __syncthreads();
  }
}

// Backward: from L (store form) or A (recompute form) build A^-1 in shared
// memory, then db = v = A^-1 w and the lower-triangle gradient dA.
template <typename T>
__global__ void __launch_bounds__(kAdjThreads) adj_backward_kernel(int n, const T* AL, int64_t strideA,
                                                                   int recompute, const T* __restrict__ X,
                                                                   const T* __restrict__ Wt,
                                                                   const T* __restrict__ Glog, T* dA,
                                                                   T* __restrict__ db, int32_t* __restrict__ info,
                                                                   int batch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_info;
  __shared__ T s_sc[2];
  __shared__ int cb[kAdjMaxN];
  T* S = reinterpret_cast<T*>(smem_raw);  // the packed lower triangle, n (n + 1) / 2 entries
  T* tmp = S + (size_t)n * (n + 1) / 2;
  T* v = tmp + n;
  T* xs = v + n;
  T* ws = xs + n;
  T* rdiag = ws + n;
  const int tid = threadIdx.x;
  for (int c = tid; c < n; c += blockDim.x) cb[c] = c * n - c * (c + 1) / 2;
  __syncthreads();
  for (int s = blockIdx.x; s < batch; s += gridDim.x) {
    const T* a = AL + (size_t)s * strideA;
    for (int e = tid; e < n * n; e += blockDim.x) {
      const int c = e / n, r = e - c * n;
      if (r >= c) S[cb[c] + r] = a[e];
    }
    if (tid == 0) s_info = 0;
    __syncthreads();
    if (recompute) chol_smem<T>(n, S, cb, &s_info, s_sc);  // refactor instead of storing L
    const int inf = s_info;
    if (inf == 0) {
      for (int i = tid; i < n; i += blockDim.x) rdiag[i] = T(1) / S[cb[i] + i];
      __syncthreads();
      trinv_smem<T>(n, S, cb, tmp, rdiag);     // tmp, v: 2n of scratch
      inv_from_trinv_smem<T>(n, S, cb, tmp);   // tmp, v, xs, ws: 4n of scratch
      for (int i = tid; i < n; i += blockDim.x) {
        xs[i] = X[(size_t)s * n + i];
        ws[i] = Wt[(size_t)s * n + i];
      }
      __syncthreads();
      // v = A^-1 w from the lower triangle of the symmetric A^-1
      for (int i = tid; i < n; i += blockDim.x) {
        T acc = T(0);
        for (int k = 0; k <= i; ++k) acc = fma_t(S[cb[k] + i], ws[k], acc);
        for (int k = i + 1; k < n; ++k) acc = fma_t(S[cb[i] + k], ws[k], acc);
        v[i] = acc;
      }
      __syncthreads();
      for (int i = tid; i < n; i += blockDim.x) db[(size_t)s * n + i] = v[i];
      T* g = dA + (size_t)s * strideA;
      const T gl = Glog ? Glog[s] : T(1);
      const T gl2 = T(2) * gl;
      for (int e = tid; e < n * n; e += blockDim.x) {
        const int c = e / n, r = e - c * n;
        T val = T(0);
        if (r == c) val = fma_t(-v[r], xs[r], gl * S[cb[c] + r]);
        else if (r > c) val = fma_t(-v[r], xs[c], fma_t(-v[c], xs[r], gl2 * S[cb[c] + r]));
        g[e] = val;
      }
    }
    if (tid == 0 && info) info[s] = inf;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// FP64 backward on the tensor cores (slices.cuh), orders above kAdjTcMinOrder.
//
// With X = L^-T stored by rows (row i = column i of L^-1) the inverse is the
// product of X's rows, (A^-1)_ij = sum_k X_ik X_jk, and X is the forward solve
// of the identity: its rows ride along below the factor's rows, as right-hand
// sides do in chol_tc.cuh.  So one sweep over blocks of 16 columns does
// everything: the rows' 16 entries are solved against the block's head (one
// thread per row, FP64), cut into slices, and 16-deep products of the slices
//   - update the factor's remaining columns (recompute form only),
//   - update X's remaining columns,
//   - accumulate A^-1,
//   - take w along: z = L^-1 w, then v = A^-1 w = X z.
// Everything lives in the output dA (L2): A^-1 and, ahead of it, the trailing
// matrix in the lower triangle (an entry's factor value is dead once its
// block is sliced, A^-1_ij starts at block i), X in the strict upper one.  So the
// output may be the stored factor's own buffer, and AL carries no __restrict__.
//
// What bounds it: the FP64 pipe still (the rows' solves, one subtraction per
// product), then latency.  2048 x 128: 4.45 -> 1.46 ms with the factor stored,
// 6.27 -> 2.20 ms recomputing it; 4000 x 40: 0.71 -> 0.44 ms. At or below order 32 (two
// blocks) the shared-memory kernel above keeps the call.
// ---------------------------------------------------------------------------
constexpr int kAdjTcThreads = 128;
constexpr int kAdjTcMinOrder = 32;

constexpr size_t adj_tc_smem(int n) {
  const size_t slots = (size_t)(n + 15) / 16 * 16 + 8;
  return slots * (kSlices * kSliceRow + 4) + (size_t)(272 + 2 * ((n + 1) & ~1) + 16) * sizeof(double);
}

// One 16 x 8 tile of slice products added to (sign +) or subtracted from the
// destination p(i), i = 0..3 the fragment's elements (null: none); fresh: the
// destination starts at zero.
template <typename F>
__device__ __forceinline__ void adj_tile(const unsigned char* sa, const int* ea, const unsigned char* sc, const int* ec, int sb,
                                         int lane, bool add, bool fresh, F dest) {
  const int g = lane >> 2, t = lane & 3;
  double* p[4];
  double v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    p[i] = dest(g + (i >> 1) * 8, 2 * t + (i & 1));
    v[i] = (p[i] && !fresh) ? *p[i] : 0.0;
  }
  float acc[kSlices][4];
  slice_products(sa, sc, sb, lane, acc);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double x = slice_value(acc, i, ea[g + (i >> 1) * 8] + ec[2 * t + (i & 1)]);
    if (p[i]) *p[i] = v[i] + (add ? x : -x);
  }
}

template <bool RECOMPUTE>
__global__ void __launch_bounds__(kAdjTcThreads, 4)
    adj_tc_backward_kernel(int n, const double* AL, int64_t strideA, const double* __restrict__ X,
                           const double* __restrict__ Wt, const double* __restrict__ Glog, double* dA,
                           double* __restrict__ db, int32_t* __restrict__ info) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_info, s_next;
  __shared__ uint8_t s_packed[136];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int nw = kAdjTcThreads / 32;
  const int np = (n + 15) / 16 * 16, slots = np + 8, sb = slots * kSliceRow;
  unsigned char* SL = smem_raw;
  double* Hd = reinterpret_cast<double*>(SL + (size_t)kSlices * sb);
  double* z = Hd + 272;            // w, then L^-1 w block by block
  double* v = z + ((n + 1) & ~1);  // A^-1 w
  double* rd = v + ((n + 1) & ~1); // 1 / L_jj of the current block
  int* ex = reinterpret_cast<int*>(rd + 16);
  const int s = blockIdx.x;
  const double* al = AL + (size_t)s * strideA;
  double* g = dA + (size_t)s * strideA;
  for (int e = tid; e < 136; e += kAdjTcThreads) s_packed[e] = (uint8_t)tc_packed(e);
  if (tid == 0) s_info = 0;
  if (RECOMPUTE)
    for (int c = warp; c < n; c += nw)
      for (int r = c + lane; r < n; r += 32) g[(size_t)c * n + r] = al[(size_t)c * n + r];
  for (int i = tid; i < n; i += kAdjTcThreads) {
    z[i] = Wt[(size_t)s * n + i];
    v[i] = 0.0;
  }
  __syncthreads();
  // the head at J0: factored in place (recompute), or read from the stored factor
  auto head = [&](int J0) {
    if (RECOMPUTE) {
      tc_head(n, g, J0, Hd, rd - J0, s_packed, &s_info, 0, 0.0, lane);
    } else {
      const int w = min(16, n - J0);
      for (int e = lane; e < 256; e += 32) {
        const int c = e >> 4, r = e & 15;
        Hd[e] = (r < w && c <= r) ? al[(size_t)(J0 + c) * n + J0 + r] : 0.0;
      }
      if (lane < w) rd[lane] = 1.0 / al[(size_t)(J0 + lane) * (n + 1)];
    }
  };
  if (warp == 0) head(0);
  __syncthreads();
  for (int J0 = 0; J0 < n; J0 += 16) {
    if (RECOMPUTE && s_info != 0) break;
    const int j1 = J0 + 16, w = min(16, n - J0), blk = J0 >> 4;
    const int mp = np - j1, mt = mp >> 4;  // rows below, padded
    // rows: slots [0, mp) the factor's, [mp, np) X's, np: z; the solve against
    // the head, the slices
    for (int q = tid; q < slots; q += kAdjTcThreads) {
      unsigned char* s0 = SL + q * kSliceRow;
      const int c = q - mp;  // X's row
      if (q < mp ? j1 + q >= n : c < j1 ? c >= n : q > np) {
        slice_zero_row(s0, sb);
        ex[q] = 1;
        continue;
      }
      double x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (q < mp) x[j] = j < w ? (RECOMPUTE ? g : al)[(size_t)(J0 + j) * n + j1 + q] : 0.0;
        else if (q == np) x[j] = j < w ? z[J0 + j] : 0.0;
        else if (c >= J0) x[j] = c - J0 == j ? 1.0 : 0.0;
        else x[j] = j < w ? g[(size_t)(J0 + j) * n + c] : 0.0;
      }
      if (RECOMPUTE || q >= mp) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          x[j] *= j < w ? rd[j] : 0.0;
#pragma unroll
          for (int k = j + 1; k < 16; ++k) x[k] = fma(-x[j], Hd[j * 16 + k], x[k]);
        }
      }
      ex[q] = slice_row(x, s0, sb);
    }
    if (tid == 0) s_next = nw - 1;
    __syncthreads();
    auto lower = [&](int rt, int c0) {  // the factor's trailing columns
      adj_tile(SL + 16 * rt * kSliceRow, ex + 16 * rt, SL + c0 * kSliceRow, ex + c0, sb, lane, false, false,
               [&](int i, int k) -> double* {
                 const int r = j1 + 16 * rt + i, c = j1 + c0 + k;
                 return r < n && c <= r ? g + (size_t)c * n + r : nullptr;
               });
    };
    if (RECOMPUTE && mt > 0) {
      for (int rt = warp; rt < mt; rt += nw)
        for (int c0 = 0; c0 < 16; c0 += 8) lower(rt, c0);
      __syncthreads();
    }
    // units of 16 rows x 32 columns: X against the factor's rows, X against X
    // (row tile i: ceil((i + 1) / 2)), every row against z, the factor's rest
    const int ux = (blk + 1) * ((mt + 1) >> 1);
    const int k1 = (blk + 1) >> 1, us = (blk + 1) & 1 ? (k1 + 1) * (k1 + 1) : k1 * (k1 + 1);
    const int uz = np >> 4;
    const int ul = RECOMPUTE ? ((mt & 1) ? (mt >> 1) * ((mt >> 1) + 1) : (mt >> 1) * (mt >> 1)) : 0;
    const int units = ux + us + uz + ul;
    int u = warp - 1;
    if (warp == 0) {
      if (mt > 0) head(j1);
      if (lane == 0) u = atomicAdd(&s_next, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
    }
    while (u < units) {
      int q = u;
      if (q < ux) {
        const int rt = q % (blk + 1), c0 = 32 * (q / (blk + 1));
        for (int c = c0; c < min(c0 + 32, mp); c += 8)
          adj_tile(SL + (mp + 16 * rt) * kSliceRow, ex + mp + 16 * rt, SL + c * kSliceRow, ex + c, sb, lane, false, rt == blk,
                   [&](int i, int k) -> double* {
                     const int r = j1 + c + k;
                     return r < n ? g + (size_t)r * n + 16 * rt + i : nullptr;
                   });
      } else if ((q -= ux) < us) {
        // row tiles 2 k and 2 k + 1 have k + 1 units each: k (k + 1) before them
        int k = (int)((sqrtf(1.0f + 4.0f * (float)q) - 1.0f) * 0.5f);
        if (k * (k + 1) > q) --k;
        if ((k + 1) * (k + 2) <= q) ++k;
        const int rem = q - k * (k + 1);
        const int rt = rem <= k ? 2 * k : 2 * k + 1, c0 = 32 * (rem <= k ? rem : rem - k - 1);
        for (int c = c0; c < min(c0 + 32, 16 * rt + 16); c += 8)
          adj_tile(SL + (mp + 16 * rt) * kSliceRow, ex + mp + 16 * rt, SL + (mp + c) * kSliceRow, ex + mp + c, sb, lane, true,
                   rt == blk, [&](int i, int kk) -> double* {
                     const int r = 16 * rt + i, cc = c + kk;
                     return r < n && cc <= r ? g + (size_t)cc * n + r : nullptr;
                   });
      } else if ((q -= us) < uz) {
        const bool fac = 16 * q < mp;  // the factor's rows: z; X's: v
        adj_tile(SL + 16 * q * kSliceRow, ex + 16 * q, SL + np * kSliceRow, ex + np, sb, lane, !fac, false,
                 [&](int i, int kk) -> double* {
                   const int r = fac ? j1 + 16 * q + i : 16 * q - mp + i;
                   return kk == 0 && r < n ? (fac ? z : v) + r : nullptr;
                 });
      } else {
        q -= uz;
        int k = (int)((1.0f + sqrtf(1.0f + 4.0f * (float)q)) * 0.5f);
        if (k * (k - 1) > q) --k;
        if (k * (k + 1) <= q) ++k;
        const int rem = q - k * (k - 1);
        const int rt = rem < k ? 2 * k - 1 : 2 * k, c0 = 16 + 32 * (rem < k ? rem : rem - k);
        for (int c = c0; c < min(c0 + 32, 16 * rt + 16); c += 8) lower(rt, c);
      }
      if (lane == 0) u = atomicAdd(&s_next, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
    }
    __syncthreads();
  }
  const int inf = RECOMPUTE ? s_info : 0;
  if (inf == 0) {
    double* xs = Hd;  // the forward solution, over the head and z (both done)
    for (int i = tid; i < n; i += kAdjTcThreads) {
      xs[i] = X[(size_t)s * n + i];
      db[(size_t)s * n + i] = v[i];
    }
    __syncthreads();
    const double gl = Glog ? Glog[s] : 1.0, gl2 = 2.0 * gl;
    for (int c = warp; c < n; c += nw) {
      const double vc = v[c], xc = xs[c];
      double* col = g + (size_t)c * n;
      for (int r = lane; r < n; r += 32) {
        double val = 0.0;
        if (r > c) val = fma(-v[r], xc, fma(-vc, xs[r], gl2 * col[r]));
        else if (r == c) val = fma(-vc, xc, gl * col[r]);
        col[r] = val;
      }
    }
  }
  if (tid == 0 && info) info[s] = inf;
}

// ---------------------------------------------------------------------------
// FP32 in blocks of 16 columns, orders above kAdjF32MinOrder.
//
// The column-by-column kernels above take three barriers and an integer
// division per element for every column; FP32 itself is far from its limits.
// Here the matrix sits in shared memory as a square (odd leading dimension) and
// a block of 16 columns takes three barriers: warp 0 factors the 16 x 16 head in
// registers, a thread per row solves its 16 entries against it and leaves them
// k-major in S, and warps apply 16-deep products in 16 x 32 tiles of 4 x 4 per
// lane.  The backward pass is the FP64 one's sweep (adj_tc_backward_kernel): X =
// L^-T rides below the factor, A^-1 = X X^T accumulates in the lower triangle.
// 1000 x 97, factor recomputed: forward 385 -> 117, backward 615 -> 210 us.
// ---------------------------------------------------------------------------
constexpr int kAdjF32Threads = 128;
// At order 4 both take 95 us forward (20,000 matrices; 10,000 of order 6: 72
// against 59); below it the 16 x 16 head is mostly padding (order 1: 40 against 92).
constexpr int kAdjF32MinOrder = 4;

__host__ __device__ constexpr int adj_f32_slots(int n) { return (n + 15) / 16 * 16 + 4; }  // rows of S, and one vector
constexpr size_t adj_f32_smem(int n) {
  return ((size_t)((n * (n | 1) + 3) & ~3) + 16 * (size_t)adj_f32_slots(n) + 256 + 16 + 2 * (size_t)((n + 3) & ~3)) *
         sizeof(float);
}
struct AdjF32 {
  float *M, *S, *Hd, *rd, *z, *v;
  int n, ld, slots;
  __device__ AdjF32(int n_, unsigned char* smem) : n(n_), ld(n_ | 1), slots(adj_f32_slots(n_)) {
    M = reinterpret_cast<float*>(smem);
    S = M + ((n * ld + 3) & ~3);
    Hd = S + 16 * slots;
    rd = Hd + 256;
    z = rd + 16;
    v = z + ((n + 3) & ~3);
  }
  // the head at J0 of the matrix in M, factored in place by one warp: Hd[j * 16 + r], 1 / L_jj in rd
  __device__ void head(int J0, int* s_info, int lane) const {
    const int w = min(16, n - J0), r = lane & 15, h = lane >> 4;
    float a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = 2 * i + h;
      a[i] = (r < w && c <= r) ? M[(J0 + c) * ld + J0 + r] : (r == c ? 1.f : 0.f);
    }
    int fail = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int ij = j >> 1, hj = (j & 1) * 16;
      const float d = __shfl_sync(0xffffffffu, a[ij], j + hj);
      if (!pos_or_inf(d) && fail == 0) fail = J0 + j + 1;
      const float rcp = rsqrt(d);
      if (h == (j & 1)) a[ij] = r > j ? a[ij] * rcp : (r == j ? d * rcp : a[ij]);
      if (lane == 0) rd[j] = rcp;
      const float x = __shfl_sync(0xffffffffu, a[ij], r + hj);
#pragma unroll
      for (int i = ij; i < 8; ++i) {
        const int c = 2 * i + h;
        const float l = __shfl_sync(0xffffffffu, a[ij], (c & 15) + hj);
        if (c > j && r >= c) a[i] = fmaf(-x, l, a[i]);
      }
    }
    if (fail && lane == 0) *s_info = fail;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = 2 * i + h;
      Hd[c * 16 + r] = a[i];
      if (r < w && c <= r) M[(J0 + c) * ld + J0 + r] = a[i];
    }
  }
  // x against the head (w <= 16 columns)
  __device__ void solve(float (&x)[16], int w) const {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      x[j] *= j < w ? rd[j] : 0.f;
#pragma unroll
      for (int k = j + 1; k < 16; ++k) x[k] = fmaf(-x[j], Hd[j * 16 + k], x[k]);
    }
  }
  // One tile: slots r0 .. r0 + 15 times slots c0 .. c0 + 31 (multiples of 4),
  // dest(i, k) its elements' places.  A lane's rows are four apart and its
  // columns adjacent, so a warp's places lie in 32 different banks (odd ld).
  template <typename F>
  __device__ void tile(int r0, int c0, int lane, bool add, bool fresh, F dest) const {
    const int rg = r0 + (lane & 3), cg = c0 + 4 * (lane >> 2);
    float acc[4][4] = {};
    if (cg < slots) {
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float4 b = *reinterpret_cast<const float4*>(S + k * slots + cg);
        const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float a = S[k * slots + rg + 4 * i];
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(a, bv[q], acc[i][q]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float* p = dest((lane & 3) + 4 * i, cg - c0 + q);
        if (p) *p = (fresh ? 0.f : *p) + (add ? acc[i][q] : -acc[i][q]);
      }
  }
  // dot product of two slots' 16 entries
  __device__ float dot(int p, int q) const {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) s = fmaf(S[k * slots + p], S[k * slots + q], s);
    return s;
  }
  __device__ void keep(const float (&x)[16], int slot) const {
#pragma unroll
    for (int k = 0; k < 16; ++k) S[k * slots + slot] = x[k];
  }
};

__global__ void __launch_bounds__(kAdjF32Threads) adj_f32_forward_kernel(int n, const float* __restrict__ A, int64_t strideA,
                                                                         const float* __restrict__ B, float* __restrict__ X,
                                                                         float* __restrict__ Lout, float* __restrict__ logdet,
                                                                         int32_t* __restrict__ info) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_info;
  __shared__ float s_part[kAdjF32Threads / 32];
  const AdjF32 m(n, smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, s = blockIdx.x;
  constexpr int nw = kAdjF32Threads / 32;
  float* y = m.z;
  const float* a = A + (size_t)s * strideA;
  for (int c = warp; c < n; c += nw)
    for (int r = c + lane; r < n; r += 32) m.M[c * m.ld + r] = a[(size_t)c * n + r];
  for (int i = tid; i < n; i += kAdjF32Threads) y[i] = B[(size_t)s * n + i];
  if (tid == 0) s_info = 0;
  __syncthreads();
  for (int J0 = 0; J0 < n; J0 += 16) {
    if (warp == 0) m.head(J0, &s_info, lane);
    __syncthreads();
    if (s_info != 0) break;
    const int j1 = J0 + 16, w = min(16, n - J0), mp = max(0, (n - j1 + 15) / 16 * 16);
    for (int q = tid; q <= mp; q += kAdjF32Threads) {  // rows below, then y
      float x[16];
      const bool vec = q == mp, on = vec || j1 + q < n;
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = (on && j < w) ? (vec ? y[J0 + j] : m.M[(J0 + j) * m.ld + j1 + q]) : 0.f;
      m.solve(x, w);
      m.keep(x, q);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (on && j < w) (vec ? y[J0 + j] : m.M[(J0 + j) * m.ld + j1 + q]) = x[j];
    }
    __syncthreads();
    const int mt = mp >> 4;
    for (int u = warp, rt = 0; rt < mt; u -= rt / 2 + 1, ++rt) {  // row tile rt: rt / 2 + 1 groups of 32 columns
      for (; u < rt / 2 + 1; u += nw)
        m.tile(16 * rt, 32 * u, lane, false, false, [&](int i, int k) -> float* {
          const int r = j1 + 16 * rt + i, c = j1 + 32 * u + k;
          return r < n && c <= r ? m.M + c * m.ld + r : nullptr;
        });
    }
    for (int r = j1 + tid; r < n; r += kAdjF32Threads) y[r] -= m.dot(r - j1, mp);
    __syncthreads();
  }
  const int inf = s_info;
  if (inf == 0) {
    // x = L^-T y in blocks of 16 rows from the bottom
    for (int J0 = (n - 1) / 16 * 16; J0 >= 0; J0 -= 16) {
      const int w = min(16, n - J0);
      if (warp == 0) {
        float v = lane < w ? y[J0 + lane] : 0.f;
        for (int j = w - 1; j >= 0; --j) {
          const float xj = __shfl_sync(0xffffffffu, v, j) / m.M[(J0 + j) * m.ld + J0 + j];
          if (lane == j) v = xj;
          if (lane < j) v = fmaf(-xj, m.M[(J0 + lane) * m.ld + J0 + j], v);
        }
        if (lane < w) y[J0 + lane] = v;
      }
      __syncthreads();
      for (int i = tid; i < J0; i += kAdjF32Threads) {
        float v = y[i];
        for (int r = 0; r < w; ++r) v = fmaf(-m.M[i * m.ld + J0 + r], y[J0 + r], v);
        y[i] = v;
      }
      __syncthreads();
    }
    float part = 0.f;
    for (int i = tid; i < n; i += kAdjF32Threads) {
      X[(size_t)s * n + i] = y[i];
      const float d = m.M[i * m.ld + i];
      part += logf(d * d);
    }
    part = warp_sum(part);
    if (lane == 0) s_part[warp] = part;
    __syncthreads();
    if (tid == 0) {
      float sum = 0.f;
      for (int u = 0; u < nw; ++u) sum += s_part[u];
      logdet[s] = sum;
    }
    if (Lout)
      for (int c = warp; c < n; c += nw)
        for (int r = lane; r < n; r += 32) Lout[(size_t)s * strideA + (size_t)c * n + r] = r >= c ? m.M[c * m.ld + r] : 0.f;
  }
  if (tid == 0 && info) info[s] = inf;
}

template <bool RECOMPUTE>
__global__ void __launch_bounds__(kAdjF32Threads)
    adj_f32_backward_kernel(int n, const float* AL, int64_t strideA, const float* __restrict__ X,
                            const float* __restrict__ Wt, const float* __restrict__ Glog, float* dA,
                            float* __restrict__ db, int32_t* __restrict__ info) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_info;
  const AdjF32 m(n, smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, s = blockIdx.x;
  constexpr int nw = kAdjF32Threads / 32;
  const int np = (n + 15) / 16 * 16;
  const float* al = AL + (size_t)s * strideA;
  if (RECOMPUTE)
    for (int c = warp; c < n; c += nw) {
      // a column's loads ahead of its stores, which AL without __restrict__ might alias (one
      // by one, 1000 x 97 forward + backward took 632 us for 603)
      float v[kAdjMaxN / 32];
#pragma unroll
      for (int k = 0; k < kAdjMaxN / 32; ++k) v[k] = c + lane + 32 * k < n ? al[(size_t)c * n + c + lane + 32 * k] : 0.f;
#pragma unroll
      for (int k = 0; k < kAdjMaxN / 32; ++k)
        if (c + lane + 32 * k < n) m.M[c * m.ld + c + lane + 32 * k] = v[k];
    }
  for (int i = tid; i < n; i += kAdjF32Threads) {
    m.z[i] = Wt[(size_t)s * n + i];
    m.v[i] = 0.f;
  }
  if (tid == 0) s_info = 0;
  __syncthreads();
  for (int J0 = 0; J0 < n; J0 += 16) {
    const int j1 = J0 + 16, w = min(16, n - J0), blk = J0 >> 4, mp = np - j1, mt = mp >> 4;
    if (warp == 0) {
      if (RECOMPUTE) {
        m.head(J0, &s_info, lane);
      } else {
        for (int e = lane; e < 256; e += 32) {
          const int c = e >> 4, r = e & 15;
          m.Hd[e] = (r < w && c <= r) ? al[(size_t)(J0 + c) * n + J0 + r] : 0.f;
        }
        if (lane < w) m.rd[lane] = 1.f / al[(size_t)(J0 + lane) * (n + 1)];
      }
    }
    __syncthreads();
    if (RECOMPUTE && s_info != 0) break;
    // slots [0, mp): the factor's rows below; [mp, np): X's rows; np: z
    for (int q = tid; q <= np; q += kAdjF32Threads) {
      const int c = q - mp;
      float x[16];
      const bool on = q < mp ? j1 + q < n : q == np || c < n;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        x[j] = 0.f;
        if (on && j < w) {
          if (q < mp) x[j] = RECOMPUTE ? m.M[(J0 + j) * m.ld + j1 + q] : al[(size_t)(J0 + j) * n + j1 + q];
          else if (q == np) x[j] = m.z[J0 + j];
          else if (c >= J0) x[j] = c - J0 == j ? 1.f : 0.f;
          else x[j] = m.M[(J0 + j) * m.ld + c];
        }
      }
      if (RECOMPUTE || q >= mp) m.solve(x, w);
      m.keep(x, q);
    }
    __syncthreads();
    // X against the factor's rows; X against X; the factor's rest; z and v
    const int ux = (blk + 1) * ((mt + 1) >> 1);
    const int k1 = (blk + 1) >> 1, us = (blk + 1) & 1 ? (k1 + 1) * (k1 + 1) : k1 * (k1 + 1);
    const int k2 = mt >> 1, ul = !RECOMPUTE ? 0 : mt & 1 ? (k2 + 1) * (k2 + 1) : k2 * (k2 + 1);
    // tiles 2 k and 2 k + 1 of a triangle have k + 1 units each
    auto triangle = [](int q, int* rt, int* c0) {
      int k = (int)((sqrtf(1.0f + 4.0f * (float)q) - 1.0f) * 0.5f);
      if (k * (k + 1) > q) --k;
      if ((k + 1) * (k + 2) <= q) ++k;
      const int rem = q - k * (k + 1);
      *rt = rem <= k ? 2 * k : 2 * k + 1;
      *c0 = 32 * (rem <= k ? rem : rem - k - 1);
    };
    for (int u = warp; u < ux + us + ul; u += nw) {
      int rt, c0;
      if (u < ux) {
        rt = u % (blk + 1);
        c0 = 32 * (u / (blk + 1));
        m.tile(mp + 16 * rt, c0, lane, false, rt == blk, [&](int i, int k) -> float* {
          const int r = j1 + c0 + k, c = 16 * rt + i;
          return c0 + k < mp && r < n && c < n ? m.M + r * m.ld + c : nullptr;
        });
      } else if (u < ux + us) {
        triangle(u - ux, &rt, &c0);
        m.tile(mp + 16 * rt, mp + c0, lane, true, rt == blk, [&](int i, int k) -> float* {
          const int r = 16 * rt + i, c = c0 + k;
          return r < n && c <= r ? m.M + c * m.ld + r : nullptr;
        });
      } else {
        triangle(u - ux - us, &rt, &c0);
        m.tile(16 * rt, c0, lane, false, false, [&](int i, int k) -> float* {
          const int r = j1 + 16 * rt + i, c = j1 + c0 + k;
          return r < n && c <= r ? m.M + c * m.ld + r : nullptr;
        });
      }
    }
    for (int q = tid; q < np; q += kAdjF32Threads) {
      const int r = q < mp ? j1 + q : q - mp;
      if (r < n) {
        if (q < mp) m.z[r] -= m.dot(q, np);
        else m.v[r] += m.dot(q, np);
      }
    }
    __syncthreads();
  }
  const int inf = RECOMPUTE ? s_info : 0;
  if (inf == 0) {
    float* xs = m.z;
    for (int i = tid; i < n; i += kAdjF32Threads) {
      xs[i] = X[(size_t)s * n + i];
      db[(size_t)s * n + i] = m.v[i];
    }
    __syncthreads();
    const float gl = Glog ? Glog[s] : 1.f, gl2 = 2.f * gl;
    for (int c = warp; c < n; c += nw) {
      const float vc = m.v[c], xc = xs[c];
      const float* col = m.M + c * m.ld;
      float* out = dA + (size_t)s * strideA + (size_t)c * n;
      for (int r = lane; r < n; r += 32) {
        float val = 0.f;
        if (r > c) val = fmaf(-m.v[r], xc, fmaf(-vc, xs[r], gl2 * col[r]));
        else if (r == c) val = fmaf(-vc, xc, gl * col[r]);
        out[r] = val;
      }
    }
  }
  if (tid == 0 && info) info[s] = inf;
}

template <typename T>
int adj_launch_forward(int n, const T* A, int64_t strideA, const T* B, T* X, T* Lout, T* logdet, int32_t* info,
                       int batch, cudaStream_t stream, const char* name) {
  if (n < 1 || n > kAdjMaxN) return record_arg_error(-1, "posv_logdet_forward: n out of range [1, 128]");
  if (batch < 0) return record_arg_error(-9, "posv_logdet_forward: negative batch");
  if (batch == 0) return NACU_SUCCESS;
  if (!A || !B || !X || !logdet) return record_arg_error(-2, "posv_logdet_forward: null A, B, X or logdet");
  if (strideA < (int64_t)n * n) return record_arg_error(-3, "posv_logdet_forward: strideA < n*n");
  if constexpr (sizeof(T) == 4) {
    if (n > kAdjF32MinOrder) {
      const size_t bytes = adj_f32_smem(n);
      cudaError_t e = ensure_dynamic_smem(adj_f32_forward_kernel, bytes);
      if (e != cudaSuccess) return record_cuda_error(e, name);
      adj_f32_forward_kernel<<<batch, kAdjF32Threads, bytes, stream>>>(n, A, strideA, B, X, Lout, logdet, info);
      return check_launch(name);
    }
  }
  const size_t smem = ((size_t)n * (n + 1) / 2 + n) * sizeof(T);
  cudaError_t e = ensure_dynamic_smem(adj_forward_kernel<T>, smem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  adj_forward_kernel<T><<<batch, kAdjThreads, smem, stream>>>(n, A, strideA, B, X, Lout, logdet, info, batch);
  return check_launch(name);
}

template <typename T>
int adj_launch_backward(int n, const T* AL, int64_t strideA, int recompute, const T* X, const T* W, const T* G, T* dA,
                        T* db, int32_t* info, int batch, cudaStream_t stream, const char* name) {
  if (n < 1 || n > kAdjMaxN) return record_arg_error(-1, "posv_logdet_backward: n out of range [1, 128]");
  if (batch < 0) return record_arg_error(-10, "posv_logdet_backward: negative batch");
  if (batch == 0) return NACU_SUCCESS;
  if (!AL || !X || !W || !dA || !db) return record_arg_error(-2, "posv_logdet_backward: null argument");
  if (strideA < (int64_t)n * n) return record_arg_error(-3, "posv_logdet_backward: strideA < n*n");
  if constexpr (sizeof(T) == 4) {
    if (n > kAdjF32MinOrder) {
      const auto kern = recompute ? adj_f32_backward_kernel<true> : adj_f32_backward_kernel<false>;
      const size_t bytes = adj_f32_smem(n);
      cudaError_t e = ensure_dynamic_smem(kern, bytes);
      if (e != cudaSuccess) return record_cuda_error(e, name);
      kern<<<batch, kAdjF32Threads, bytes, stream>>>(n, AL, strideA, X, W, G, dA, db, info);
      return check_launch(name);
    }
  } else {
    if (n > kAdjTcMinOrder) {
      const auto kern = recompute ? adj_tc_backward_kernel<true> : adj_tc_backward_kernel<false>;
      const size_t bytes = adj_tc_smem(n);
      cudaError_t e = ensure_dynamic_smem(kern, bytes);
      if (e != cudaSuccess) return record_cuda_error(e, name);
      kern<<<batch, kAdjTcThreads, bytes, stream>>>(n, AL, strideA, X, W, G, dA, db, info);
      return check_launch(name);
    }
  }
  const size_t smem = ((size_t)n * (n + 1) / 2 + 5 * (size_t)n) * sizeof(T);
  cudaError_t e = ensure_dynamic_smem(adj_backward_kernel<T>, smem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  adj_backward_kernel<T><<<batch, kAdjThreads, smem, stream>>>(n, AL, strideA, recompute, X, W, G, dA, db, info,
                                                               batch);
  return check_launch(name);
}

}  // namespace
}  // namespace nacu

extern "C" {

int nacu_dposv_logdet_forward(int n, const double* A, int64_t strideA, const double* B, double* X, double* L,
                              double* logdet, int32_t* info, int batch, nacu_stream_t stream) {
  using namespace nacu;
  if (L == nullptr)  // recompute form: no factor buffer, the shared-memory kernel keeps nothing
    return adj_launch_forward<double>(n, A, strideA, B, X, L, logdet, info, batch, (cudaStream_t)stream,
                                      "nacu_dposv_logdet_forward");
  // store form: the factor is built in L by the FP64 batched Cholesky kernel
  // (factor + solve + log-det in place on copies of A and b)
  if (n < 1 || n > kAdjMaxN) return record_arg_error(-1, "posv_logdet_forward: n out of range [1, 128]");
  if (batch < 0) return record_arg_error(-9, "posv_logdet_forward: negative batch");
  if (batch == 0) return NACU_SUCCESS;
  if (!A || !B || !X || !logdet || !info)
    return record_arg_error(-2, "posv_logdet_forward: null A, B, X, logdet or info");
  if (strideA < (int64_t)n * n) return record_arg_error(-3, "posv_logdet_forward: strideA < n*n");
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemcpyAsync(L, A, (size_t)batch * strideA * sizeof(double), cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(X, B, (size_t)batch * n * sizeof(double), cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dposv_logdet_forward");
  return chol_uniform_posv(n, L, strideA, 1, X, n, info, logdet, batch, s, "nacu_dposv_logdet_forward");
}
int nacu_sposv_logdet_forward(int n, const float* A, int64_t strideA, const float* B, float* X, float* L,
                              float* logdet, int32_t* info, int batch, nacu_stream_t stream) {
  return nacu::adj_launch_forward<float>(n, A, strideA, B, X, L, logdet, info, batch, (cudaStream_t)stream,
                                         "nacu_sposv_logdet_forward");
}
int nacu_dposv_logdet_backward(int n, const double* AL, int64_t strideA, int recompute, const double* X,
                               const double* W, const double* G, double* dA, double* db, int32_t* info, int batch,
                               nacu_stream_t stream) {
  return nacu::adj_launch_backward<double>(n, AL, strideA, recompute, X, W, G, dA, db, info, batch,
                                           (cudaStream_t)stream, "nacu_dposv_logdet_backward");
}
int nacu_sposv_logdet_backward(int n, const float* AL, int64_t strideA, int recompute, const float* X,
                               const float* W, const float* G, float* dA, float* db, int32_t* info, int batch,
                               nacu_stream_t stream) {
  return nacu::adj_launch_backward<float>(n, AL, strideA, recompute, X, W, G, dA, db, info, batch,
                                          (cudaStream_t)stream, "nacu_sposv_logdet_backward");
}

}  // extern "C"
