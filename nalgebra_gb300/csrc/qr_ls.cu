// Batched Householder QR and least squares for tall-skinny systems
// (m >= n, n <= 128): the GPU form of nalgebra's `m.qr()`
// (src/linalg/qr.rs:55-76, householder.rs:19-85, geometry/reflection.rs:70-83),
// `q_tr_mul` (qr.rs:157-171) and the least-squares solve of nalgebra-lapack
// (nalgebra-lapack/src/qr_util.rs:167-239: Q^T b, then the upper-triangular
// solve with R[0:n, 0:n], dividing by |diag_i| as qr.rs:224-256 does).
//
// Sign convention.  nalgebra applies each reflection with a sign,
// c <- s_i * (I - 2 v v^T) c with s_i = signum(diag_i) (householder.rs:75-82).
// Writing D_i for the diagonal matrix that is s_i on rows >= i and 1 above,
// nalgebra's transform is D_{n-1} H_{n-1} ... D_0 H_0, and every D_i commutes
// with the later H_j (H_j touches rows >= j > i, where D_i is a scalar), so it
// equals D H_{n-1} ... H_0 with D = diag(d_r), d_r = prod_{i <= min(r, n-1)} s_i.
// The reflections themselves do not depend on the signs (a reflection axis is
// defined up to sign).  So the kernel runs plain Householder QR in compact-WY
// blocks, and each value takes its sign when it is final, which gives nalgebra's
// stored factors exactly:
//   diag_i  = P_i * diag_std_i   (P_i = prod_{j<i} s_j, s_i = signum(diag_i)),
//   axis_i  = P_i * v_i          (the stored unit axis),
//   R[r][c] = d_r * R_std[r][c]  (strict upper part), Q^T b rows likewise,
// and the least-squares solution does not change at all (D cancels).
//
// Design (GB300): one CTA (128 threads) per problem; problems are pulled from a
// work queue (largest first).  The matrix stays in global memory (L2-resident
// while the CTA works on it); each 8-column panel is factored in shared memory
// in FP64, then the trailing columns and the right-hand side take the block
// reflector I - V T^T V^T on the tensor cores (qr_trailing_tc), each FP64 value
// cut into digit slices in registers.
//
// What bounds it: the FP64 pipe, now mostly the panels (12.6k of the 16.4k
// warp-wide FP64 instructions of a 320 x 64 problem; 41k when the trailing
// update was dots and axpys), and the panels' serial steps.  Measured: 8192
// problems of 128..512 x 64 23.7 -> 12.7 ms (the launch; 13.5 the call), 4096 of 100 x 100 10.0 -> 5.2 ms, 8000 of
// 20..64 x 16 1.23 -> 1.06 ms, 384 of 261..936 x 124 12.2 -> 4.9 ms.
#include "householder.cuh"
#include "slices.cuh"

namespace nacu {
namespace {

constexpr int kQrThreads = 128;
constexpr int kQrNB = 8;
constexpr int kQrMaxN = 128;
// s_t layout: tau (NB) | scratch (128) | V^T V strict upper part (28, padded to 32)
constexpr int kTauOff = 0;
constexpr int kGOff = kTauOff + kQrNB;            // scratch (1 / |diag_i| of the back substitution)
constexpr int kGSumOff = kGOff + 4 * 32;           // 28 reduced pairs (i < j)
constexpr int kSTSize = kGSumOff + 32;

struct QrArgs {
  int count;
  int n;
  int m_max;
  const int32_t* ms;    // null: every problem is m_uni x n
  const int64_t* aoff;  // null: problem s at A + s * strideA
  double* A;
  const int64_t* boff;  // null with B set: b of problem s at B + s * strideB
  double* B;            // nullable: factor only
  double* X;      // n per problem, nullable
  double* diag;   // n per problem
  int32_t* info;
  const int32_t* order;
  int32_t* counter;     // null: problems taken grid-stride (no queue)
  int m_uni;
  int64_t strideA, strideB;
  int x_in_b;           // the square form: the solution overwrites b (QR::solve_mut)
};

// x with its sign bit flipped where mask has it: +-1 factors cost no FP64 slot.
__device__ __forceinline__ double qr_flip(double x, unsigned mask) {
  return __hiloint2double(__double2hiint(x) ^ (int)mask, __double2loint(x));
}

// Butterfly reduce-scatter of N (a power of two <= 32) per-lane values: lane L
// ends with the warp-wide sum of value (L mod N) in v[0]; N-1 adds per lane
// plus log2(32/N) more, instead of N separate 5-step warp reductions.
template <int N>
__device__ __forceinline__ void warp_reduce_scatter(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = N / 2; half >= 1; half >>= 1) {
    const bool up = (lane & half) != 0;
#pragma unroll
    for (int t = 0; t < half; ++t) {
      const double keep = up ? v[t + half] : v[t];
      const double give = up ? v[t] : v[t + half];
      v[t] = keep + __shfl_xor_sync(0xffffffffu, give, half);
    }
  }
#pragma unroll
  for (int off = N; off < 32; off <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
}

// Element j < k of the panel's V^T V.
__device__ __forceinline__ double qr_gram(const double* s_t, int j, int k) {
  return s_t[kGSumOff + j * kQrNB - j * (j + 1) / 2 + (k - j - 1)];
}

// The compact-WY factor T of the block reflector I - V T^T V^T has T^-1 =
// diag(1 / tau) + the strict upper part of V^T V (Puglisi 1992), so T^T w is a
// forward substitution with V^T V and T itself is never formed:
// w'_k = tau_k (w_k - sum_{j<k} (v_j . v_k) w'_j).

// c <- c - V T^T V^T c for one column by one warp (V: the panel's jb axes in
// shared memory, ld ldp, zero above their diagonal), rows 0..jb-1 times their
// signs (masks in row_sign).
__device__ __forceinline__ void qr_apply_reflector(double* col, int rows, const double* P, int ldp, int jb,
                                                   const double* s_t, const unsigned* row_sign, int lane) {
  double w[kQrNB];
#pragma unroll
  for (int e = 0; e < kQrNB; ++e) w[e] = 0.0;
  for (int r = lane; r < rows; r += 32) {
    const double x = col[r];
#pragma unroll
    for (int c = 0; c < kQrNB; ++c) w[c] = fma((c < jb && r >= c) ? P[(size_t)c * ldp + r] : 0.0, x, w[c]);
  }
  warp_reduce_scatter<kQrNB>(w);  // lane L holds the sum of axis L mod 8
  const int k = lane % kQrNB;
  double wp[kQrNB];
#pragma unroll
  for (int j = 0; j < kQrNB; ++j) {
    wp[j] = j < jb ? s_t[kTauOff + j] * __shfl_sync(0xffffffffu, w[0], j) : 0.0;
    if (j < jb && k > j && k < jb) w[0] = fma(-qr_gram(s_t, j, k), wp[j], w[0]);
  }
  for (int r = lane; r < rows; r += 32) {
    double x = col[r];
#pragma unroll
    for (int c = 0; c < kQrNB; ++c) x = fma(-((c < jb && r >= c) ? P[(size_t)c * ldp + r] : 0.0), wp[c], x);
    col[r] = r < jb ? qr_flip(x, row_sign[r]) : x;
  }
}

// ---- the trailing update on the tensor cores ----------------------------------------------------------------
// A CTA's scratch: a slot per trailing column (the right-hand side included,
// padded to 16).  A slot holds the column's partial sums V^T c of the two row
// halves, then in their place the slices of w' = T^T V^T c; 144 bytes apart, so
// a fragment's loads from eight slots hit different banks.  Two halves and one
// place for both keep four CTAs on an SM at m = 512 (three with four quarters:
// 8192 problems of 128..512 x 64 14.4 -> 12.6 ms).
constexpr int kQrParts = 2;
// Levels of digit products (slices.cuh).  With seven, rows of falling or rising scale
// (2^+-20) left 1.4 to 1.5 times the error of the FP64 update; with eight 0.7.  8192
// problems of 128..512 x 64 (the call) 13.3 -> 13.5 ms.
constexpr int kQrLevels = kSlices + 1;
constexpr int kQrSlot = kQrParts * kQrNB * 8 + 16;
__host__ __device__ constexpr int qr_tc_cols(int n) { return (n + 1 + 15) / 16 * 16; }
__host__ __device__ constexpr size_t qr_tc_bytes(int n) { return (size_t)qr_tc_cols(n) * (kQrSlot + 4); }
// Fewer trailing columns than this: a warp each in FP64, which has no second
// barrier; a 16-column tile would be mostly padding.
constexpr int kQrTcMinCols = 4;

// C <- C - V T^T V^T C for a full panel of kQrNB axes and ncol columns, by
// digit slices (slices.cuh).  Both products' fragments are cut from the FP64
// values in registers, so neither V nor C is kept in sliced form:
//   1. D[column][axis] = sum_r C[r][column] V[r][axis]: 16 columns x 8 axes,
//      32 rows per exact sum (exponents common to a column's / an axis' 32 rows);
//      a warp takes every other row block of a column group, the two partial
//      sums meet in shared memory;
//   2. W' = T^T D in FP64, a thread per column, cut into slices;
//   3. C[r][column] -= sum_k V[r][k] W'[k][column]: 16 rows x 8 columns, 8 deep.
// An element costs one FP64 subtraction per panel (and 1/8 of one in step 1)
// where the dot and axpy form issued sixteen multiply-adds.
template <typename ColPtr>
__device__ __forceinline__ void qr_trailing_tc(ColPtr colptr, int ncol, int rows, const double* P, int ldp, const double* s_t,
                                               const unsigned* row_sign, unsigned char* scratch, int n) {
  constexpr int NW = kQrThreads / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  int* ew = reinterpret_cast<int*>(scratch + (size_t)qr_tc_cols(n) * kQrSlot);
  const int groups = (ncol + 15) >> 4;
  auto axis = [&](int c, int r) { return (r >= c && r < rows) ? P[(size_t)c * ldp + r] : 0.0; };
  for (int unit = warp; unit < groups * kQrParts; unit += NW) {
    const int part = unit % kQrParts, c0 = unit / kQrParts * 16 + g, c1 = c0 + 8;
    const double* p0 = c0 < ncol ? colptr(c0) : nullptr;
    const double* p1 = c1 < ncol ? colptr(c1) : nullptr;
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    for (int rb = part * 32; rb < rows; rb += kQrParts * 32) {
      // rows rb + 16 h + 4 t + q, q = 0..3 of axis g and of the two columns
      double x[2][2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = rb + 16 * h + 4 * t + q;
          x[0][h][q] = (p0 && r < rows) ? p0[r] : 0.0;
          x[1][h][q] = (p1 && r < rows) ? p1[r] : 0.0;
        }
      uint32_t b[2][2][kSlices];
      int eb = 1;
      {
        double v[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            v[h][q] = axis(g, rb + 16 * h + 4 * t + q);
            eb = max(eb, slice_exponent(v[h][q]));
          }
        eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, 1));
        eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, 2));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          slice_pair(v[h][0], v[h][1], eb, b[h][0]);
          slice_pair(v[h][2], v[h][3], eb, b[h][1]);
        }
      }
      int ea[2] = {1, 1};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 4; ++q) ea[u] = max(ea[u], slice_exponent(x[u][h][q]));
        ea[u] = max(ea[u], __shfl_xor_sync(0xffffffffu, ea[u], 1));
        ea[u] = max(ea[u], __shfl_xor_sync(0xffffffffu, ea[u], 2));
      }
      float acc[kQrLevels][4];
      slice_sums_start(acc);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t a0[kSlices], a1[kSlices], a2[kSlices], a3[kSlices];
        slice_pair(x[0][h][0], x[0][h][1], ea[0], a0);
        slice_pair(x[1][h][0], x[1][h][1], ea[1], a1);
        slice_pair(x[0][h][2], x[0][h][3], ea[0], a2);
        slice_pair(x[1][h][2], x[1][h][3], ea[1], a3);
#pragma unroll
        for (int p = 0; p < kSlices; ++p) {
          const uint32_t a[4] = {a0[p], a1[p], a2[p], a3[p]};
#pragma unroll
          for (int q = 0; q < kSlices && p + q < kQrLevels; ++q) {
            const uint32_t bb[2] = {b[h][0][q], b[h][1][q]};
            mma_f16_16x8x16(acc[p + q], a, bb);
          }
        }
      }
      // lane's axes 2 t and 2 t + 1: their exponents are on the lanes of g = 2 t, 2 t + 1
      const int eb0 = slice_code(__shfl_sync(0xffffffffu, eb, 8 * t)), eb1 = slice_code(__shfl_sync(0xffffffffu, eb, 8 * t + 4));
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[i] += slice_value<32>(acc, i, slice_code(ea[i >> 1]) + (i & 1 ? eb1 : eb0));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      reinterpret_cast<double*>(scratch + (size_t)(i >> 1 ? c1 : c0) * kQrSlot)[part * kQrNB + 2 * t + (i & 1)] = sum[i];
  }
  __syncthreads();
  for (int c = tid; c < groups * 16; c += kQrThreads) {
    double w[kQrNB], o[kQrNB];
    int em = 1;
#pragma unroll
    for (int k = 0; k < kQrNB; ++k) {
      const double* p = reinterpret_cast<const double*>(scratch + (size_t)c * kQrSlot) + k;
      w[k] = p[0] + p[kQrNB];
    }
#pragma unroll
    for (int k = 0; k < kQrNB; ++k) {
#pragma unroll
      for (int j = 0; j < k; ++j) w[k] = fma(-qr_gram(s_t, j, k), o[j], w[k]);
      o[k] = s_t[kTauOff + k] * w[k];
      em = max(em, slice_exponent(o[k]));
    }
    uint32_t s0[kSlices], s1[kSlices], s2[kSlices], s3[kSlices];
    slice_pair(o[0], o[1], em, s0);
    slice_pair(o[2], o[3], em, s1);
    slice_pair(o[4], o[5], em, s2);
    slice_pair(o[6], o[7], em, s3);
#pragma unroll
    for (int p = 0; p < kSlices; ++p)
      *reinterpret_cast<uint4*>(scratch + (size_t)c * kQrSlot + 16 * p) = make_uint4(s0[p], s1[p], s2[p], s3[p]);
    ew[c] = slice_code(em);
  }
  __syncthreads();
  for (int rb = warp * 16; rb < rows; rb += NW * 16) {
    // rows rb + g and rb + g + 8, axes 2 t and 2 t + 1
    uint32_t a[2][kSlices];
    int ea[2];
    const int r0 = rb + g;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const double v0 = axis(2 * t, r0 + 8 * u), v1 = axis(2 * t + 1, r0 + 8 * u);
      ea[u] = max(slice_exponent(v0), slice_exponent(v1));
      ea[u] = max(ea[u], __shfl_xor_sync(0xffffffffu, ea[u], 1));
      ea[u] = max(ea[u], __shfl_xor_sync(0xffffffffu, ea[u], 2));
      slice_pair(v0, v1, ea[u], a[u]);
      ea[u] = slice_code(ea[u]);
    }
    for (int c = 0; c < ncol; c += 8) {
      double* p[4];
      double v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + (i >> 1) * 8, cc = c + 2 * t + (i & 1);
        p[i] = (r < rows && cc < ncol) ? colptr(cc) + r : nullptr;
        v[i] = p[i] ? *p[i] : 0.0;
      }
      float acc[kQrLevels][4];
      slice_sums_start(acc);
      uint32_t b[kSlices];
#pragma unroll
      for (int q = 0; q < kSlices; ++q)
        b[q] = *reinterpret_cast<const uint32_t*>(scratch + (size_t)(c + g) * kQrSlot + 16 * q + 4 * t);
#pragma unroll
      for (int p2 = 0; p2 < kSlices; ++p2)
#pragma unroll
        for (int q = 0; q < kSlices && p2 + q < kQrLevels; ++q) mma_f16_16x8x8(acc[p2 + q], a[0][p2], a[1][p2], b[q]);
      const int e0 = ew[c + 2 * t], e1 = ew[c + 2 * t + 1];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double x = slice_value(acc, i, ea[i >> 1] + (i & 1 ? e1 : e0));
        const double y = v[i] - x;  // rows 0..7 are final rows of R
        if (p[i]) *p[i] = (rb == 0 && i < 2) ? qr_flip(y, row_sign[g]) : y;
      }
    }
  }
}

// CTA sum, valid in thread 0 only (the one thread that uses it: the other
// threads add nothing, which saves the FP64 issue slots of 127 redundant sums).
__device__ __forceinline__ double block_sum_to0(double v, double* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
#pragma unroll
    for (int w = 0; w < kQrThreads / 32; ++w) s += red[w];
  return s;
}

// A full panel (kQrNB columns, rows x kQrNB in P) in kQrNB Householder steps,
// each ONE pass over the rows with ONE CTA reduction: the pass of step j
// scales axis j, updates the later columns and accumulates, from the updated
// values, the sums step j+1 needs (|x_{j+1}|^2 and x_{j+1} . P_c for every
// other column c, x_{j+1} unscaled and unmodified); step j+1 then corrects
// them for the modified diagonal entry and the axis scale by scalars.  The
// steps are unrolled, so each pass issues only the FMAs of its live columns:
// on this part an FP64 instruction with its lanes predicated off still costs
// its issue slot.  Same reflections as the generic steps (householder.rs:
// 19-53 without the sign step); the sums are formed in a different order.
__device__ void qr_panel_full(double* P, int ldp, int rows, int J0, double* s_t, double* s_dstd, double* s_red) {
  constexpr int NB = kQrNB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* s_sum = s_red + 4;           // 4 warps x NB partial sums
  double* s_par = s_red + 4 + 4 * NB;  // slot j: the axis scale; slots c > j: the column coefficients
  {
    double acc[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) acc[c] = 0.0;
    for (int r = tid; r < rows; r += kQrThreads) {
      const double x = P[r];
      acc[0] = fma(x, x, acc[0]);
#pragma unroll
      for (int c = 1; c < NB; ++c) acc[c] = fma(x, P[(size_t)c * ldp + r], acc[c]);
    }
    warp_reduce_scatter<NB>(acc);
    if (lane < NB) s_sum[warp * NB + lane] = acc[0];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    double* pj = P + (size_t)j * ldp;
    if (tid < NB) {  // lanes 0..NB-1 of warp 0: the scalars (redundantly), then column tid's term
      double sq = 0.0, dc = 0.0;
#pragma unroll
      for (int w = 0; w < kQrThreads / 32; ++w) {
        sq += s_sum[w * NB + j];
        dc += s_sum[w * NB + tid];
      }
      const double nrm = sqrt_halley(sq);
      const double x0 = pj[j];
      const bool pos = x0 >= 0.0;  // simba to_exp
      const double signed_norm = pos ? nrm : neg_bits(nrm);
      const double factor = 2.0 * fma(pos ? x0 : neg_bits(x0), nrm, sq);
      const bool nz = factor != 0.0;
      const double scale = nz ? rsqrt_halley(factor) : 0.0, tau = nz ? 2.0 : 0.0;
      // v . P_c with v = scale * x', x' = x but x'_j = x0 + signed_norm
      const double dv = fma(signed_norm, P[(size_t)tid * ldp + j], dc) * scale;
      if (tid == j) {
        s_dstd[J0 + j] = nz ? -signed_norm : signed_norm;  // R_std[j][j]
        s_t[kTauOff + j] = tau;
        s_par[j] = scale;
      } else if (tid > j) {
        s_par[tid] = -tau * dv;
      } else {
        s_t[kGSumOff + tid * NB - tid * (tid + 1) / 2 + (j - tid - 1)] = dv;  // G[tid][j] = v_tid . v_j
      }
      __syncwarp(0xffu);
      if (tid == j && nz) pj[j] = x0 + signed_norm;
    }
    __syncthreads();
    const double scale = s_par[j];
    double coef[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) coef[c] = (c > j) ? s_par[c] : 0.0;
    double acc[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) acc[c] = 0.0;
    for (int r = j + tid; r < rows; r += kQrThreads) {
      const double v = pj[r] * scale;
      pj[r] = v;
      double pc[NB];
#pragma unroll
      for (int c = j + 1; c < NB; ++c) {
        pc[c] = fma(coef[c], v, P[(size_t)c * ldp + r]);
        P[(size_t)c * ldp + r] = pc[c];
      }
      if (j + 1 < NB && r > j) {  // step j+1's sums over rows > j
        const double y = pc[j + 1];
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          if (c == j + 1) acc[c] = fma(y, y, acc[c]);
          else if (c == j) acc[c] = fma(y, v, acc[c]);
          else if (c < j) acc[c] = fma(y, P[(size_t)c * ldp + r], acc[c]);
          else acc[c] = fma(y, pc[c], acc[c]);
        }
      }
    }
    if (j + 1 < NB) {
      warp_reduce_scatter<NB>(acc);
      if (lane < NB) s_sum[warp * NB + lane] = acc[0];
    }
    __syncthreads();
  }
}

// One problem.  P: panel buffer (ldp x kQrNB), V^T V and T in s_t, per-column
// standard diagonals in s_dstd, reductions in s_red.
__device__ void qr_one(const QrArgs& g, int s, double* P, int ldp, unsigned char* scratch, double* s_t, double* s_dstd,
                       double* s_red, double* s_misc) {
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int n = g.n;
  const int m = g.ms ? g.ms[s] : g.m_uni;
  if (m < n || m > g.m_max) {
    if (tid == 0 && g.info) g.info[s] = -1;
    return;
  }
  double* a = g.A + (g.aoff ? g.aoff[s] : (int64_t)s * g.strideA);
  double* b = g.B ? g.B + (g.boff ? g.boff[s] : (int64_t)s * g.strideB) : nullptr;
  double* s_coef = s_red + 4 + 4 * kQrNB;
  unsigned* axis_sign = reinterpret_cast<unsigned*>(s_misc + 2);  // sign masks: P_i, then d_i
  unsigned* row_sign = axis_sign + kQrMaxN;
  for (int J0 = 0; J0 < n; J0 += kQrNB) {
    const int jb = min(kQrNB, n - J0);
    const int rows = m - J0;
    for (int e = tid; e < rows * jb; e += kQrThreads) {
      const int c = e / rows, r = e - c * rows;
      P[(size_t)c * ldp + r] = a[(size_t)(J0 + c) * m + J0 + r];
    }
    __syncthreads();
    // ---- panel: jb Householder steps in shared memory ----
    if (jb == kQrNB) qr_panel_full(P, ldp, rows, J0, s_t, s_dstd, s_red);
    else for (int j = 0; j < jb; ++j) {
      double* pj = P + (size_t)j * ldp;
      double part = 0.0;
      for (int r = j + tid; r < rows; r += kQrThreads) part = fma(pj[r], pj[r], part);
      const double sq = block_sum_to0(part, s_red);
      if (tid == 0) {
        // householder.rs:19-53 (reflection_axis_mut) without the sign step
        const double nrm = sqrt(sq);
        const double x0 = pj[j];
        const double mod = (x0 >= 0.0) ? x0 : -x0;
        const double sgn = (x0 >= 0.0) ? 1.0 : -1.0;  // simba to_exp
        const double signed_norm = sgn * nrm;
        const double factor = (sq + mod * nrm) * 2.0;
        if (factor != 0.0) {
          pj[j] = x0 + signed_norm;
          s_misc[0] = rsqrt(factor);
          s_misc[1] = 2.0;                // tau: v is unit length
          s_dstd[J0 + j] = -signed_norm;  // R_std[j][j]
        } else {
          s_misc[0] = 0.0;
          s_misc[1] = 0.0;  // no reflection (zero column)
          s_dstd[J0 + j] = signed_norm;
        }
        s_t[kTauOff + j] = s_misc[1];
      }
      __syncthreads();
      const double scale = s_misc[0], tau = s_misc[1];
      // v = x * scale; dots of v with the remaining panel columns (c > j) and
      // with the earlier reflection axes (c < j: the entries G[c][j] = v_c . v_j
      // of V^T V that the T factor needs, v_j being zero above row j)
      double dots[kQrNB];
#pragma unroll
      for (int c = 0; c < kQrNB; ++c) dots[c] = 0.0;
      for (int r = j + tid; r < rows; r += kQrThreads) {
        const double v = pj[r] * scale;
        pj[r] = v;
#pragma unroll
        for (int c = 0; c < kQrNB; ++c)
          if (c != j && c < jb) dots[c] = fma(v, P[(size_t)c * ldp + r], dots[c]);
      }
      // reduce the dots (at most 7) across the CTA
      warp_reduce_scatter<kQrNB>(dots);
      if (lane < kQrNB) s_red[4 + warp * kQrNB + lane] = dots[0];
      __syncthreads();
      // coef_c = -tau * (v^T P_c), formed once per column by kQrNB threads
      // (every thread forming all of them cost more FP64 issue slots than the
      // panel update itself); zero outside columns j+1..jb-1
      if (tid < kQrNB) {
        double d = 0.0;
#pragma unroll
        for (int w = 0; w < kQrThreads / 32; ++w) d += s_red[4 + w * kQrNB + tid];
        s_coef[tid] = (tid > j && tid < jb) ? -tau * d : 0.0;
        if (tid < j) s_t[kGSumOff + tid * kQrNB - tid * (tid + 1) / 2 + (j - tid - 1)] = d;  // G[tid][j]
      }
      __syncthreads();
      double coef[kQrNB];
#pragma unroll
      for (int c = 0; c < kQrNB; ++c) coef[c] = s_coef[c];
      for (int r = j + tid; r < rows; r += kQrThreads) {
        const double v = pj[r];
#pragma unroll
        for (int c = 0; c < kQrNB; ++c)
          if (c > j && c < jb) P[(size_t)c * ldp + r] = fma(coef[c], v, P[(size_t)c * ldp + r]);
      }
      __syncthreads();
    }
    // ---- the panel's signs: axis i is stored times P_i, row i of R times d_i = P_{i+1} ----
    if (tid == 0) {
      unsigned pi = J0 ? row_sign[J0 - 1] : 0u;
      for (int i = J0; i < J0 + jb; ++i) {
        axis_sign[i] = pi;
        s_dstd[i] = qr_flip(s_dstd[i], pi);  // diag_i = P_i diag_std_i
        pi ^= (unsigned)__double2hiint(s_dstd[i]) & 0x80000000u;
        row_sign[i] = pi;
      }
    }
    __syncthreads();
    // ---- trailing columns and the right-hand side: c <- c - V T^T V^T c ----
    // on the tensor cores; a few columns (or the last, narrower panel's) a warp
    // per column
    const int ntrail = n - J0 - jb;
    const int ncol = ntrail + (b ? 1 : 0);
    auto colptr = [&](int t) { return (t < ntrail) ? a + (size_t)(J0 + jb + t) * m + J0 : b + J0; };
    if (jb == kQrNB && ncol >= kQrTcMinCols) {
      qr_trailing_tc(colptr, ncol, rows, P, ldp, s_t, row_sign + J0, scratch, n);
    } else {
      for (int t = warp; t < ncol; t += kQrThreads / 32)
        qr_apply_reflector(colptr(t), rows, P, ldp, jb, s_t, row_sign + J0, lane);
    }
    __syncthreads();
    // ---- write the factored panel back ----
    for (int e = tid; e < rows * jb; e += kQrThreads) {
      const int c = e / rows, r = e - c * rows;
      a[(size_t)(J0 + c) * m + J0 + r] =
          qr_flip(P[(size_t)c * ldp + r], r >= c ? axis_sign[J0 + c] : row_sign[J0 + r]);
    }
    __syncthreads();
  }
  if (tid == 0) {
    int inf = 0;
    for (int i = n - 1; i >= 0; --i)
      if (is_zero_bits(s_dstd[i])) inf = i + 1;
    s_misc[1] = (double)inf;
  }
  // |diag_i|^-1 for the back substitution (computed in parallel, once).
  for (int i = tid; i < n; i += kQrThreads) s_t[kGOff + i] = 1.0 / fabs(s_dstd[i]);
  __syncthreads();
  const int inf = (int)s_misc[1];
  // The least-squares solution with nalgebra's R (rows times d_r, diagonal
  // |diag_i|) and Q^T b, as qr.rs:224-256 restricted to the top n rows; the
  // signs cancel.  R comes eight columns at a time through the panel buffer:
  // read straight from L2 each step waited for it.
  if (b && (g.X || g.x_in_b) && inf == 0) {
    constexpr int KR = kQrMaxN / 32;  // rows per lane
    double yv[KR];
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int r = lane + 32 * k;
      yv[k] = (warp == 0 && r < n) ? b[r] : 0.0;
    }
    for (int i0 = (n - 1) / kQrNB * kQrNB; i0 >= 0; i0 -= kQrNB) {
      const int w = min(kQrNB, n - i0);
      for (int e = tid; e < (i0 + w) * w; e += kQrThreads) {
        const int c = e / (i0 + w), r = e - c * (i0 + w);
        P[(size_t)c * ldp + r] = a[(size_t)(i0 + c) * m + r];
      }
      __syncthreads();
      if (warp == 0)
        for (int i = i0 + w - 1; i >= i0; --i) {
          const double* col = P + (size_t)(i - i0) * ldp;
          double own = yv[0];
#pragma unroll
          for (int k = 1; k < KR; ++k)
            if ((i >> 5) == k) own = yv[k];
          const double xi = __shfl_sync(0xffffffffu, own, i & 31) * s_t[kGOff + i];
#pragma unroll
          for (int k = 0; k < KR; ++k) {
            const int r = lane + 32 * k;
            if (r == i) yv[k] = xi;
            if (32 * k < i) yv[k] = r < i ? fma(-xi, col[r], yv[k]) : yv[k];
          }
        }
      __syncthreads();
    }
    double* x = g.x_in_b ? b : g.X + (size_t)s * n;
    if (warp == 0)
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        const int r = lane + 32 * k;
        if (r < n) x[r] = yv[k];
      }
  }
  if (b)  // the rows of Q^T b below R: the sign of all n reflections
    for (int r = n + tid; r < m; r += kQrThreads) b[r] = qr_flip(b[r], row_sign[n - 1]);
  for (int i = tid; i < n; i += kQrThreads) g.diag[(size_t)s * n + i] = s_dstd[i];
  if (tid == 0 && g.info) g.info[s] = inf;
  __syncthreads();
}

__host__ __device__ constexpr size_t qr_panel_bytes(int m_max) {
  return ((size_t)(m_max | 1) * kQrNB * sizeof(double) + 15) & ~(size_t)15;
}

__global__ void __launch_bounds__(kQrThreads, 4) qr_batched_kernel(QrArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_t[kSTSize];
  __shared__ double s_dstd[kQrMaxN];
  __shared__ double s_red[4 + 5 * kQrNB];  // block sums | 4 warps x NB dots | NB panel coefficients
  __shared__ double s_misc[2 + kQrMaxN];
  __shared__ int s_item;
  const int ldp = g.m_max | 1;
  double* P = reinterpret_cast<double*>(smem_raw);
  unsigned char* scratch = smem_raw + qr_panel_bytes(g.m_max);
  if (!g.counter) {  // uniform batch: problems grid-stride
    for (int s = blockIdx.x; s < g.count; s += gridDim.x) qr_one(g, s, P, ldp, scratch, s_t, s_dstd, s_red, s_misc);
    return;
  }
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(g.counter, 1);
    __syncthreads();
    const int idx = s_item;
    __syncthreads();
    if (idx >= g.count) break;
    const int s = g.order ? g.order[idx] : idx;
    qr_one(g, s, P, ldp, scratch, s_t, s_dstd, s_red, s_misc);
  }
}

}  // namespace

// The square QR's FMA form on this kernel: count uniform n x n problems
// (n <= kQrMaxN) at A + s * strideA, nalgebra's QR layout and signs in place,
// diag and info out; with B (one right-hand side per problem at B + s *
// strideB) QR::solve_mut overwrites b with x.
int qr_uniform_launch(int n, int count, double* A, int64_t strideA, double* diag, double* B, int64_t strideB,
                      int32_t* info, cudaStream_t s, const char* name) {
  QrArgs g{count, n, n, nullptr, nullptr, A, nullptr, B, nullptr, diag, info, nullptr, nullptr, n, strideA, strideB,
           1};
  const size_t smem = qr_panel_bytes(n) + qr_tc_bytes(n);
  cudaError_t e = ensure_dynamic_smem(qr_batched_kernel, smem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, qr_batched_kernel, kQrThreads, smem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  if (per_sm < 1) per_sm = 1;
  int grid = sm_count() * per_sm;
  if (grid > count) grid = count;
  qr_batched_kernel<<<grid, kQrThreads, smem, s>>>(g);
  return check_launch(name);
}

}  // namespace nacu

extern "C" {

size_t nacu_qr_workspace_bytes(int count) {
  (void)count;
  return 256;
}

int nacu_dgels_batched(int count, int n, int m_max, const int32_t* ms, const int64_t* a_offsets, double* A,
                       const int64_t* b_offsets, double* B, double* X, double* diag, int32_t* info,
                       const int32_t* order, void* workspace, size_t workspace_bytes, int flags,
                       nacu_stream_t stream) {
  using namespace nacu;
  if (count < 0) return record_arg_error(-1, "dgels_batched: negative count");
  if (n < 1 || n > kQrMaxN) return record_arg_error(-2, "dgels_batched: n out of range [1, 128]");
  if (m_max < n || m_max > NACU_QR_MAX_M) return record_arg_error(-3, "dgels_batched: m_max out of range [n, 2048]");
  if (count == 0) return NACU_SUCCESS;
  if (!ms || !a_offsets || !A) return record_arg_error(-4, "dgels_batched: null ms, a_offsets or A");
  if ((b_offsets == nullptr) != (B == nullptr)) return record_arg_error(-7, "dgels_batched: b_offsets and B must both be set or both null");
  if (!diag) return record_arg_error(-10, "dgels_batched: null diag");
  if (!workspace || workspace_bytes < nacu_qr_workspace_bytes(count))
    return record_arg_error(-14, "dgels_batched: workspace too small");
  if (flags & NACU_FLAG_EXACT) return record_arg_error(-15, "dgels_batched: NACU_FLAG_EXACT is not available for QR");
  QrArgs g{count, n, m_max, ms, a_offsets, A, b_offsets, B, X, diag, info, order,
           reinterpret_cast<int32_t*>(workspace), 0, 0, 0, 0};
  const size_t smem = qr_panel_bytes(m_max) + qr_tc_bytes(n);
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = ensure_dynamic_smem(qr_batched_kernel, smem);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgels_batched");
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, qr_batched_kernel, kQrThreads, smem);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgels_batched");
  if (per_sm < 1) per_sm = 1;
  int grid = sm_count() * per_sm;
  if (grid > count) grid = count;
  e = cudaMemsetAsync(workspace, 0, sizeof(int32_t), s);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgels_batched");
  qr_batched_kernel<<<grid, kQrThreads, smem, s>>>(g);
  return check_launch("nacu_dgels_batched");
}

}  // extern "C"
