// Large dense LU with partial pivoting (one matrix, n up to tens of
// thousands) and its solve, in FP64 (the plain form of nalgebra's `m.lu()` /
// `.solve(&b)`, src/linalg/lu.rs:93-122, 221-260) and in FP32 (the factor of
// the mixed-precision form, see gesv_mixed.cu).
//
// Blocked right-looking LU, panels of NB columns:
//   1. panel factorization, partial pivoting with nalgebra's icamax rule
//      (largest |x|, first index on ties, src/base/min_max.rs:221-240; an
//      all-zero column is skipped, lu.rs:107-110), by one cooperative kernel
//      whose CTAs own row blocks of the panel and meet at two grid barriers per
//      column (candidate pivots published; pivot row swapped);
//   2. the panel's row swaps applied to the columns left and right of it;
//   3. U12 = L11^-1 A12 (unit lower triangular solve, one thread per column);
//   4. A22 -= L21 U12 by the GEMM kernels: residues on the tensor cores for
//      FP64 (gemm_crt.cu), the BF16-split tensor-core GEMM for the FP32 factor.
// Orders up to 8192 take 128 columns per block, panels in registers and 32-deep
// updates inside the block; above, a block is one panel of 64 (FP64) or 128.
// Measured, the factorization alone, FP64, ms (all on the FP64 pipe -> residue updates with 64-wide panels ->
// register panels behind a cluster barrier -> as below): n = 8192 328 -> 114 -> 65 ->
// 56.0, 4096 50 -> 24.6 -> 20.0 -> 15.3, 2000 11.6 -> 9.4 -> 8.7 -> 5.5, 1000 4.62 ->
// 4.20 -> 4.08 -> 2.41 (the checks of the digit products are 0.5 to 1.5% of these).  FP32 factor with refinement, n = 4096: 15.8 -> 15.8 -> 14.2 -> 9.9.
// The chain of panels and inner updates bounds it: at n = 8192 50 ms were left of 67
// when the trailing update beyond the next panel cost nothing.
// The triangular solves for the right-hand side run as one cooperative kernel
// per triangle: the diagonal block of each step is solved by CTA 0 while all
// CTAs then apply it to the remaining rows (coalesced GEMV), one grid barrier
// per phase.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "slices.cuh"

namespace cg = cooperative_groups;

namespace nacu {

// ---------------------------------------------------------------------------
// panel factorization (cooperative, the panel resident in shared memory)
// ---------------------------------------------------------------------------
constexpr int kPanelThreads = 256;
constexpr int kPanelMaxG = 255;          // CTAs of one panel launch
constexpr int kPanelMaxNb = 128;         // panel width
constexpr int kPanelRowsPerCta = 64;     // rows per CTA aimed for
constexpr size_t kPanelMaxSmem = 200 * 1024;

// What each column step publishes to the other CTAs, double-buffered by the
// column's parity (a slot is rewritten two steps later, after every CTA has
// passed the barrier between): each CTA's pivot candidate (|x| key, row) and
// that row's panel values, and the current values of row c.
template <typename T>
struct PanelPub {
  unsigned long long key[2][kPanelMaxG];
  int idx[2][kPanelMaxG];
  T row[2][kPanelMaxG][kPanelMaxNb];
  T diag[2][kPanelMaxNb];
  // the panel's swaps as one row mapping: row pdst[k] takes old row psrc[k];
  // the register panels of an outer block one list each, in order
  int npairs;
  int nlist[kPanelMaxNb / 32];
  int pdst[2 * kPanelMaxNb];
  int psrc[2 * kPanelMaxNb];
  int balance[kPanelMaxNb];  // of the block's trailing updates (u_row_exponents)
};

template <typename T>
struct PanelArgs {
  int n;        // matrix order
  T* A;         // column-major, lda
  int64_t lda;
  int j0, nb;   // panel columns [j0, j0 + nb)
  int chunk;    // rows per CTA (CTA b owns rows j0 + b*chunk ...)
  int32_t* ipiv;   // per-step pivots (0-based rows)
  int32_t* info;   // first zero pivot (1-based), atomicMin
  PanelPub<T>* pub;
};

// The cluster form gives each CTA a copy of every CTA's publication slots in
// its own shared memory: each CTA pushes its candidate (key, row index, row)
// and, when it owns it, row c into all CTAs of the cluster with remote
// stores before the cluster barrier, so that after it the pivot decision and
// the pivot row are local reads.  The header is followed by
// T row[2][kClusterMaxCtas][nb] and T diag[2][nb].
constexpr int kClusterMaxCtas = 16;
struct ClusterPub {
  unsigned long long key[2][kClusterMaxCtas];
  int idx[2][kClusterMaxCtas];
};
constexpr size_t kClusterPubHead = (sizeof(ClusterPub) + 15) & ~(size_t)15;
// Rows are stored with a stride of nb rounded up to 16 bytes (vector pushes).
template <typename T>
__host__ __device__ constexpr int cpub_stride(int nb) {
  return (nb + (int)(16 / sizeof(T)) - 1) & ~((int)(16 / sizeof(T)) - 1);
}
template <typename T>
__host__ __device__ constexpr size_t cluster_pub_bytes(int nb) {
  return kClusterPubHead + (size_t)(2 * kClusterMaxCtas + 2) * cpub_stride<T>(nb) * sizeof(T);
}
template <typename T>
__device__ __forceinline__ T* cpub_row(ClusterPub* p, int nb, int par, int q) {
  return reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(p) + kClusterPubHead) +
         (size_t)(par * kClusterMaxCtas + q) * cpub_stride<T>(nb);
}
template <typename T>
__device__ __forceinline__ T* cpub_diag(ClusterPub* p, int nb, int par) {
  return reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(p) + kClusterPubHead) +
         (size_t)(2 * kClusterMaxCtas + par) * cpub_stride<T>(nb);
}
// Row r of the panel (columns 0..nb) into dst in 16-byte vectors: 16 threads
// per destination (sub = 0..15), the tail element by element.
template <typename T>
__device__ __forceinline__ void push_row(T* dst, const T* P, int ldp, int r, int nb, int sub) {
  constexpr int kV = 16 / sizeof(T);
  const int nv = nb / kV;
  for (int v = sub; v < nv; v += 16) {
    T x[kV];
#pragma unroll
    for (int i = 0; i < kV; ++i) x[i] = P[(v * kV + i) * ldp + r];
    if constexpr (kV == 4) {
      *reinterpret_cast<float4*>(dst + v * kV) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
      *reinterpret_cast<double2*>(dst + v * kV) = make_double2(x[0], x[1]);
    }
  }
  for (int t = nv * kV + sub; t < nb; t += 16) dst[t] = P[t * ldp + r];
}

// Composes the panel's swaps into one mapping for the columns outside it
// (one CTA): slots 0..nb-1 are rows j0.., slot nb + i the first swap partner
// ipiv[j0+i] below the panel.
template <typename T>
__device__ void panel_compose_swaps(const PanelArgs<T>& g, int nb, int tid) {
  PanelPub<T>* pub = g.pub;
  __shared__ int s_slot[kPanelMaxNb];
  __shared__ int s_row[2 * kPanelMaxNb];
  __shared__ int s_src[2 * kPanelMaxNb];
  for (int i = tid; i < nb; i += kPanelThreads) {
    const int p = g.ipiv[g.j0 + i];
    int slot = p - g.j0;
    if (p >= g.j0 + nb) {
      int f = i;
      for (int q = 0; q < i; ++q)
        if (g.ipiv[g.j0 + q] == p) {
          f = q;
          break;
        }
      slot = nb + f;
    }
    s_slot[i] = slot;
    s_row[i] = g.j0 + i;
    s_row[nb + i] = p;
  }
  for (int sl = tid; sl < 2 * nb; sl += kPanelThreads) s_src[sl] = sl;
  __syncthreads();
  if (tid == 0) {
    for (int i = 0; i < nb; ++i) {
      const int o = s_slot[i];
      const int t = s_src[i];
      s_src[i] = s_src[o];
      s_src[o] = t;
    }
    int k = 0;
    for (int sl = 0; sl < 2 * nb; ++sl)
      if (s_src[sl] != sl) {
        pub->pdst[k] = s_row[sl];
        pub->psrc[k] = s_row[s_src[sl]];
        ++k;
      }
    pub->npairs = k;
  }
}

// The grid form (the panel's rows spread over a cooperative grid, for panels
// too tall for one cluster's shared memory).  One grid barrier per column:
// the candidates and the candidate rows are published in global memory before
// it, so after it every CTA knows the pivot row's values without a second
// exchange; row c and the pivot row are swapped by their owners (nalgebra
// swaps whole rows, lu.rs:111-116; the columns outside the panel are swapped
// afterwards by lu_swap_kernel).
// The panel's pivot reciprocal, on its serial per-column path: the Newton
// form in FP64 (rcp_nr), a division in FP32.
__device__ __forceinline__ double pivot_rcp(double d) { return rcp_nr(d); }
__device__ __forceinline__ float pivot_rcp(float d) { return 1.0f / d; }

template <typename T>
__global__ void __launch_bounds__(kPanelThreads) lu_panel_grid_kernel(PanelArgs<T> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* P = reinterpret_cast<T*>(smem_raw);  // P[t * ldp + r]
  __shared__ uint64_t s_key[kPanelThreads / 32];
  __shared__ int s_idx[kPanelThreads / 32];
  __shared__ T s_prow[kPanelMaxNb];
  __shared__ T s_drow[kPanelMaxNb];
  __shared__ int s_win, s_piv, s_wcta;
  __shared__ T s_inv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, b = blockIdx.x;
  const int nb = g.nb, ldp = g.chunk | 1;  // odd: row walks (t varies) hit distinct banks
  const int rb = g.j0 + b * g.chunk;
  const int nr = max(0, min(g.n, rb + g.chunk) - rb);
  T* A = g.A;
  const int64_t lda = g.lda;
  PanelPub<T>* pub = g.pub;
  for (int e = tid; e < nb * nr; e += kPanelThreads) {
    const int t = e / nr, r = e - t * nr;
    P[t * ldp + r] = A[(size_t)(g.j0 + t) * lda + rb + r];
  }
  __syncthreads();
  for (int j = 0; j < nb; ++j) {
    const int c = g.j0 + j, par = j & 1;
    // 1. my candidate: the largest |x| of column j over my rows >= c
    //    (icamax, src/base/min_max.rs:221-240: first index on ties)
    uint64_t key = 0;
    int idx = 0x7fffffff;
    for (int r = max(0, c - rb) + tid; r < nr; r += kPanelThreads) {
      const uint64_t k = pivot_key(P[j * ldp + r], rb + r == c);
      if (idx == 0x7fffffff || k > key) {
        key = k;
        idx = rb + r;
      }
    }
    warp_argmax(key, idx);
    if (lane == 0) {
      s_key[warp] = key;
      s_idx[warp] = idx;
    }
    __syncthreads();
    if (warp == 0) {
      key = lane < kPanelThreads / 32 ? s_key[lane] : 0ull;
      idx = lane < kPanelThreads / 32 ? s_idx[lane] : 0x7fffffff;
      warp_argmax(key, idx);
      if (lane == 0) {
        s_win = idx;
        pub->key[par][b] = key;
        pub->idx[par][b] = (idx == 0x7fffffff) ? -1 : idx;
      }
    }
    __syncthreads();
    // 2. publish my candidate row and, if I own it, row c
    {
      const int w = s_win;
      T* prow_out = pub->row[par][b];
      T* diag_out = pub->diag[par];
      if (w != 0x7fffffff)
        for (int t = tid; t < nb; t += kPanelThreads) prow_out[t] = P[t * ldp + (w - rb)];
      if (c >= rb && c < rb + nr)
        for (int t = tid; t < nb; t += kPanelThreads) diag_out[t] = P[t * ldp + (c - rb)];
    }
    cg::this_grid().sync();
    // 3. the pivot: every CTA reduces the G candidates the same way
    if (warp == 0) {
      uint64_t bk = 0;
      int bi = 0x7fffffff, bw = 0;
      for (int q = lane; q < G; q += 32) {
        const int ri = pub->idx[par][q];
        const uint64_t kk = pub->key[par][q];
        if (ri < 0) continue;
        if (bi == 0x7fffffff || kk > bk || (kk == bk && ri < bi)) {
          bk = kk;
          bi = ri;
          bw = q;
        }
      }
      {  // the winner's CTA: the lane holding the winning row (rows have one owner)
        const int myi = bi;
        warp_argmax(bk, bi);
        const unsigned holder = __ballot_sync(0xffffffffu, myi == bi);
        bw = __shfl_sync(0xffffffffu, bw, __ffs(holder) - 1);
      }
      if (lane == 0) {
        const bool zero = (bi == 0x7fffffff || bk == 0);  // all |x| == 0: skipped, lu.rs:107-110
        s_piv = zero ? -1 : bi;
        s_wcta = bw;
        if (b == 0) {
          g.ipiv[c] = zero ? c : bi;
          if (zero) atomicMin(g.info, c + 1);
        }
      }
    }
    __syncthreads();
    const int piv = s_piv;
    if (piv < 0) continue;
    // 4. swap rows c and piv (their owners), from the published copies
    const bool own_c = (c >= rb && c < rb + nr), own_p = (piv >= rb && piv < rb + nr);
    {
      const T* win_row = pub->row[par][s_wcta];
      const T* c_row = pub->diag[par];
      for (int t = tid; t < nb; t += kPanelThreads) {
        s_prow[t] = win_row[t];
        if (own_p && piv != c) s_drow[t] = c_row[t];
      }
      if (tid == 0) s_inv = pivot_rcp(win_row[j]);
    }
    __syncthreads();
    if (piv != c) {
      for (int t = tid; t < nb; t += kPanelThreads) {
        if (own_c) P[t * ldp + (c - rb)] = s_prow[t];
        if (own_p) P[t * ldp + (piv - rb)] = s_drow[t];
      }
      __syncthreads();
    }
    // 5. multipliers of column j below row c; their elimination from the
    //    panel's remaining columns (gauss_step, lu.rs:340-357)
    const int r0 = max(0, c + 1 - rb);
    const T inv = s_inv;
    for (int r = r0 + tid; r < nr; r += kPanelThreads) P[j * ldp + r] *= inv;
    __syncthreads();
    if (j + 1 < nb && r0 < nr) {
      const int tr = tid & 63, tc = tid >> 6;  // rows r0 + tr + 64 i, columns j + 1 + tc + 4 k
      for (int r = r0 + tr; r < nr; r += 64) {
        const T l = P[j * ldp + r];
        int t = j + 1 + tc;
        for (; t + 12 < nb; t += 16) {
          const T p0 = P[t * ldp + r], p1 = P[(t + 4) * ldp + r], p2 = P[(t + 8) * ldp + r],
                  p3 = P[(t + 12) * ldp + r];
          const T q0 = s_prow[t], q1 = s_prow[t + 4], q2 = s_prow[t + 8], q3 = s_prow[t + 12];
          P[t * ldp + r] = axpy1<false>(p0, -q0, l);
          P[(t + 4) * ldp + r] = axpy1<false>(p1, -q1, l);
          P[(t + 8) * ldp + r] = axpy1<false>(p2, -q2, l);
          P[(t + 12) * ldp + r] = axpy1<false>(p3, -q3, l);
        }
        for (; t < nb; t += 4) P[t * ldp + r] = axpy1<false>(P[t * ldp + r], -s_prow[t], l);
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < nb * nr; e += kPanelThreads) {
    const int t = e / nr, r = e - t * nr;
    A[(size_t)(g.j0 + t) * lda + rb + r] = P[t * ldp + r];
  }
  __syncthreads();  // the pivots thread 0 wrote, for the composition
  if (b == 0) panel_compose_swaps(g, nb, tid);
}

__device__ __forceinline__ void cluster_arrive_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait_acquire() {
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// The cluster form with look-ahead inside the panel.  Column j's rank-1
// update is split: the next column (j+1) is updated at once, so that its
// pivot search can start, and the rest (columns j+2..) is deferred into the
// next column's exchange, between the cluster barrier's arrive and wait, where
// it hides the barrier's latency.  The candidate rows pushed for column j+1
// therefore still lack column j's update of columns j+2..; every CTA applies
// it to its copies with the same operands (fma(-u_t, l, x)), so the copies
// stay bit-identical to the rows their owners update.  The pivot decision and
// the pivot row are local reads (rows pushed into every CTA before the
// barrier: no remote reads).
template <typename T>
__global__ void __launch_bounds__(kPanelThreads) lu_panel_cluster_kernel(PanelArgs<T> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ClusterPub* cpub = reinterpret_cast<ClusterPub*>(smem_raw);
  T* P = reinterpret_cast<T*>(smem_raw + cluster_pub_bytes<T>(g.nb));  // P[t * ldp + r]
  constexpr int kWarps = kPanelThreads / 32;
  __shared__ uint64_t s_key[kWarps];
  __shared__ int s_idx[kWarps];
  __shared__ T s_prev[kPanelMaxNb];  // the last eliminated column's pivot row (complete)
  __shared__ uint64_t s_ckey;
  __shared__ int s_win, s_piv, s_wcta;
  __shared__ T s_inv;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)cl.num_blocks(), b = (int)cl.block_rank();
  const int nb = g.nb, ldp = g.chunk | 1;
  const int rb = g.j0 + b * g.chunk;
  const int nr = max(0, min(g.n, rb + g.chunk) - rb);
  T* A = g.A;
  const int64_t lda = g.lda;
  for (int e = tid; e < nb * nr; e += kPanelThreads) {
    const int t = e / nr, r = e - t * nr;
    P[t * ldp + r] = A[(size_t)(g.j0 + t) * lda + rb + r];
  }
  __syncthreads();
  bool pend = false;  // column j-1 was eliminated and its update of columns j+1.. is pending
  for (int j = 0; j < nb; ++j) {
    const int c = g.j0 + j, par = j & 1;
    // 1. my candidate: the largest |x| of column j over my rows >= c
    //    (icamax, src/base/min_max.rs:221-240: first index on ties)
    uint64_t key = 0;
    int idx = 0x7fffffff;
    for (int r = max(0, c - rb) + tid; r < nr; r += kPanelThreads) {
      const uint64_t k = pivot_key(P[j * ldp + r], rb + r == c);
      if (idx == 0x7fffffff || k > key) {
        key = k;
        idx = rb + r;
      }
    }
    warp_argmax(key, idx);
    if (lane == 0) {
      s_key[warp] = key;
      s_idx[warp] = idx;
    }
    __syncthreads();
    if (warp == 0) {
      key = lane < kWarps ? s_key[lane] : 0ull;
      idx = lane < kWarps ? s_idx[lane] : 0x7fffffff;
      warp_argmax(key, idx);
      if (lane == 0) {
        s_win = idx;
        s_ckey = key;
      }
    }
    __syncthreads();
    // 2. push my candidate (key, row index, row) and, if I own it, row c into
    //    every CTA of the cluster
    {
      const int w = s_win;
      if (tid < G) {
        ClusterPub* dst = cl.map_shared_rank(cpub, tid);
        dst->key[par][b] = s_ckey;
        dst->idx[par][b] = (w == 0x7fffffff) ? -1 : w;
      }
      const int q = tid >> 4;  // 16 threads per destination CTA
      if (q < G) {
        ClusterPub* dst = cl.map_shared_rank(cpub, q);
        if (w != 0x7fffffff) push_row<T>(cpub_row<T>(dst, nb, par, b), P, ldp, w - rb, nb, tid & 15);
        if (c >= rb && c < rb + nr) push_row<T>(cpub_diag<T>(dst, nb, par), P, ldp, c - rb, nb, tid & 15);
      }
    }
    __syncthreads();  // the rows are read out before the deferred update changes them
    cluster_arrive_release();
    // 3. deferred: column j-1's update of columns j+1.. (rows >= c; gauss_step,
    //    lu.rs:340-357), while the other CTAs arrive
    if (pend && j + 1 < nb) {
      const int tr = tid & 63, tc = tid >> 6;  // rows r0 + tr + 64 i, columns j + 1 + tc + 4 k
      for (int r = max(0, c - rb) + tr; r < nr; r += 64) {
        const T l = P[(j - 1) * ldp + r];
        int t = j + 1 + tc;
        for (; t + 12 < nb; t += 16) {
          const T p0 = P[t * ldp + r], p1 = P[(t + 4) * ldp + r], p2 = P[(t + 8) * ldp + r],
                  p3 = P[(t + 12) * ldp + r];
          const T q0 = s_prev[t], q1 = s_prev[t + 4], q2 = s_prev[t + 8], q3 = s_prev[t + 12];
          P[t * ldp + r] = axpy1<false>(p0, -q0, l);
          P[(t + 4) * ldp + r] = axpy1<false>(p1, -q1, l);
          P[(t + 8) * ldp + r] = axpy1<false>(p2, -q2, l);
          P[(t + 12) * ldp + r] = axpy1<false>(p3, -q3, l);
        }
        for (; t < nb; t += 4) P[t * ldp + r] = axpy1<false>(P[t * ldp + r], -s_prev[t], l);
      }
    }
    cluster_wait_acquire();
    // 4. the pivot, from the local copies of the G candidates
    if (warp == 0) {
      uint64_t bk = 0;
      int bi = 0x7fffffff, bw = 0;
      if (lane < G) {
        const int ri = cpub->idx[par][lane];
        if (ri >= 0) {
          bk = cpub->key[par][lane];
          bi = ri;
          bw = lane;
        }
      }
      const int myi = bi;
      warp_argmax(bk, bi);
      const unsigned holder = __ballot_sync(0xffffffffu, myi == bi);
      bw = __shfl_sync(0xffffffffu, bw, __ffs(holder) - 1);
      if (lane == 0) {
        const bool zero = (bi == 0x7fffffff || bk == 0);  // all |x| == 0: skipped, lu.rs:107-110
        s_piv = zero ? -1 : bi;
        s_wcta = bw;
        if (b == 0) {
          g.ipiv[c] = zero ? c : bi;
          if (zero) atomicMin(g.info, c + 1);
        }
        if (!zero) s_inv = pivot_rcp(cpub_row<T>(cpub, nb, par, bw)[j]);  // column j: complete in the copy
      }
    }
    __syncthreads();
    const int piv = s_piv;
    if (piv < 0) {  // nothing to eliminate; column j+1 already has every earlier update
      pend = false;
      continue;
    }
    // 5. complete the copies (column j-1's pending update), keep the pivot row
    //    for the next column, and swap rows c and piv (their owners)
    {
      const T* prow = cpub_row<T>(cpub, nb, par, s_wcta);
      const T* crow = cpub_diag<T>(cpub, nb, par);
      const bool own_c = (c >= rb && c < rb + nr), own_p = (piv >= rb && piv < rb + nr);
      const bool swap = (piv != c);
      const bool need_c = swap && own_p;
      const T lp = pend ? prow[j - 1] : T(0);
      const T lc = (pend && need_c) ? crow[j - 1] : T(0);
      for (int t = tid; t < nb; t += kPanelThreads) {
        T pv = prow[t];
        T cv = need_c ? crow[t] : T(0);
        if (pend && t > j) {
          const T u = s_prev[t];
          pv = axpy1<false>(pv, -u, lp);
          if (need_c) cv = axpy1<false>(cv, -u, lc);
        }
        s_prev[t] = pv;
        if (swap) {
          if (own_c) P[t * ldp + (c - rb)] = pv;
          if (own_p) P[t * ldp + (piv - rb)] = cv;
        }
      }
    }
    __syncthreads();
    // 6. multipliers of column j below row c, and their update of column j+1
    //    (the look-ahead column); the rest of the update is deferred
    {
      const T inv = s_inv;
      const T u = (j + 1 < nb) ? s_prev[j + 1] : T(0);
      for (int r = max(0, c + 1 - rb) + tid; r < nr; r += kPanelThreads) {
        const T l = P[j * ldp + r] * inv;
        P[j * ldp + r] = l;
        if (j + 1 < nb) P[(j + 1) * ldp + r] = axpy1<false>(P[(j + 1) * ldp + r], -u, l);
      }
    }
    pend = true;
    __syncthreads();
  }
  for (int e = tid; e < nb * nr; e += kPanelThreads) {
    const int t = e / nr, r = e - t * nr;
    A[(size_t)(g.j0 + t) * lda + rb + r] = P[t * ldp + r];
  }
  __syncthreads();  // the pivots thread 0 wrote, for the composition
  if (b == 0) panel_compose_swaps(g, nb, tid);
  cl.sync();  // every remote access to this CTA's shared memory is over
}

// ---------------------------------------------------------------------------
// narrow panels in registers
//
// The cluster form above pays about six CTA barriers and one cluster barrier
// per column (2.5 us, 4.2 us for FP64 at 6000 rows, where 64-wide panels also
// hold the FP64 pipe).  Here a panel is 32 columns wide and each row lives in the
// registers of TPR threads, so a column costs one CTA barrier (the warps' pivot
// candidates) and one exchange between the CTAs: the warp that holds a CTA's
// candidate stores its row into every CTA's shared memory, and the stores
// themselves count on the barrier there that the reader waits for.
//   - Rows never move.  Each thread tracks the position its row has under
//     nalgebra's swaps (icamax compares positions, src/base/min_max.rs:221-240;
//     a pivot's row takes position c, the row that was there the pivot's old
//     one) and writes its row there at the end.
//   - A warp-wide FP64 FMA holds its quarter of an SM for 64 cycles, whatever the
//     lanes in use, and the chain through a column is all there is to hide it
//     under.  So a row's columns are dealt to TPR threads (column j to thread j mod
//     TPR) as long as the CTA has threads left, and a pivot's update of the columns
//     beyond the next one is put off until the next column's candidates are under
//     way.  The candidate's own row is brought up to date first, a lane per column.
//   - The registers shift as columns finish, so the loop over columns stays
//     rolled; finished multipliers and pivot rows wait in shared memory.
//   - The cluster then applies the swaps to the outer block's other columns and
//     solves their 32 rows of U, a warp per column.
// Panels of 128 columns are made of four of these, each followed by the 32-deep
// update of the block's remaining columns.  Cycles a column, FP64, before (a
// cluster barrier, one thread a row, the whole update at once) and now: n = 1000
// 4870 and 2770 (search 580, send 250, deferred update 700, wait 260, select 530,
// next column 450); n = 8192 6400 and 6300, of them 4250 the update: there the 16
// SMs' FP64 pipes bound it.
// ---------------------------------------------------------------------------
constexpr int kRegThreads = 512;
constexpr int kRegNb = 32;
constexpr int kRegMaxRows = kRegThreads * kClusterMaxCtas;  // 8192
constexpr int kRegInfoTimeout = -1000;                      // info when a wait ran out
constexpr int kRegPollLimit = 1 << 20;

struct alignas(16) RegMeta {
  unsigned long long key;  // |pivot candidate|'s bit image
  int pos, pad;
  double rcp;  // its reciprocal (of the panel's type)
  double pad2;
};
template <typename T>
struct RegPanelArgs {
  int n;
  T* A;
  int64_t lda;
  int j0, nb, chunk;  // panel columns, rows per CTA
  int c_lo, c_hi;     // the outer block's columns
  int list;           // this panel's place in the block
  int32_t* ipiv;
  int32_t* info;
  PanelPub<T>* pub;
  int poll_limit;  // polls of one wait
};
// Three slots: a CTA's stores for column j + 1 may arrive while this one still
// reads column j - 1's pivot row, but not those for j + 2 (they follow this CTA's
// own for j + 1).
template <typename T>
struct RegPanelSmem {
  RegMeta meta[3][kClusterMaxCtas];
  T slot[3][kClusterMaxCtas][kRegNb];
  T stage[kRegNb];
  T rows[kRegNb][kRegThreads];
  T l11[kRegNb][kRegNb + 1];
  unsigned long long bar[3];
  unsigned long long wkey[2][kRegThreads / 32];
  int wpos[2][kRegThreads / 32];
  int dst[2 * kRegNb], src[2 * kRegNb];
};

// |x| from its bit image, and a reciprocal of |x| given x's sign
template <typename T>
__device__ __forceinline__ T from_bits(unsigned long long key) {
  if constexpr (sizeof(T) == 8) return __longlong_as_double((long long)key);
  else return __uint_as_float((unsigned)key);
}
__device__ __forceinline__ double with_sign(double r, double x) {
  return __hiloint2double(__double2hiint(r) ^ (__double2hiint(x) & 0x80000000), __double2loint(r));
}
__device__ __forceinline__ float with_sign(float r, float x) {
  return __uint_as_float(__float_as_uint(r) ^ (__float_as_uint(x) & 0x80000000u));
}
// warp_argmax, cut short where one lane alone holds the largest leading word
template <typename T>
__device__ __forceinline__ void panel_argmax(uint64_t& key, int& idx) {
  const unsigned lead = sizeof(T) == 8 ? (unsigned)(key >> 32) : (unsigned)key;
  const unsigned m = __reduce_max_sync(0xffffffffu, lead);
  const unsigned who = __ballot_sync(0xffffffffu, lead == m);
  if (__popc(who) == 1) {
    const int from = __ffs(who) - 1;
    key = __shfl_sync(0xffffffffu, key, from);
    idx = __shfl_sync(0xffffffffu, idx, from);
  } else {
    warp_argmax(key, idx);
  }
}
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void store_async(unsigned dst, float4 v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)),
               "r"(bar)
               : "memory");
}
// false when the limit is reached
__device__ __forceinline__ bool bar_wait(const void* bar, unsigned parity, int limit) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  for (int it = 0; it < limit; ++it) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// The chain of small kernels between two trailing updates is launched ahead of its
// predecessors' ends (launch_chained); the panel lets the next one in only in its
// tail, so that nothing idle holds the SMs which the trailing update runs on.
// n = 1000 2.75 -> 2.55 ms, 4096 16.8 -> 16.0; FP32 with refinement, 4096 10.6 -> 10.2.
template <typename T, int TPR>
__global__ void __launch_bounds__(kRegThreads, 1) lu_panel_reg_kernel(RegPanelArgs<T> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RegPanelSmem<T>& sm = *reinterpret_cast<RegPanelSmem<T>*>(smem_raw);
  constexpr int kWarps = kRegThreads / 32, kPer = kRegNb / TPR;
  constexpr int kV = 16 / (int)sizeof(T), kVecs = kRegNb / kV;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)cl.num_blocks(), b = (int)cl.block_rank();
  const int rb = g.j0 + b * g.chunk;
  const int nr = max(0, min(g.n - rb, g.chunk));
  const int rl = tid / TPR, sub = tid % TPR;  // the row's place in the CTA, and which of its threads
  const bool valid = rl < nr;
  const int row = rb + rl;
  int pos = row;
  bool done = !valid;
  wait_for_predecessor();
  T x[kPer];  // columns j + ((sub - j) mod TPR) + TPR k at step j
#pragma unroll
  for (int k = 0; k < kPer; ++k)
    x[k] = (valid && sub + TPR * k < g.nb) ? g.A[(size_t)(g.j0 + sub + TPR * k) * g.lda + row] : T(0);
  int* const npairs = &g.pub->nlist[g.list];
  int *const pdst = g.pub->pdst + 2 * kRegNb * g.list, *const psrc = g.pub->psrc + 2 * kRegNb * g.list;
  if (b == 0 && tid == 0) *npairs = 0;
  if (tid == 0) {
    for (int q = 0; q < 3; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&sm.bar[q])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cl.sync();  // every CTA of the cluster runs, its barriers ready, before anything is stored to it
  int w = 0;          // the CTA that held the last pivot
  bool pend = false;  // column j - 1's update of columns j + 1.. is still to come
  T lp = T(0);        // with this row's multiplier
  // This thread's wait ran out: an error; it waits no more and writes no row, and the
  // barriers, whose phases may still be open, are armed no more (so the other waits run
  // out too).  What is read meanwhile is any column's: pivots stay rows of the matrix.
  bool late = false;
  for (int j = 0, now = 0, last = 2, phase = 0; j < g.nb; ++j) {
    const int c = g.j0 + j, par = j & 1, left = g.nb - j;
    const int s0 = j % TPR, d = (sub - s0) & (TPR - 1);  // x[k] is column j + d + TPR k
    if (tid == 0 && !late)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(&sm.bar[now])),
                   "r"(G * ((left + kV - 1) / kV * 16 + (int)sizeof(RegMeta)))
                   : "memory");
    uint64_t key = done || d != 0 ? 0ull : pivot_key(x[0], pos == c);
    int idx = done || d != 0 ? 0x7fffffff : pos;
    panel_argmax<T>(key, idx);
    if (lane == 0) {
      sm.wkey[par][warp] = key;
      sm.wpos[par][warp] = idx;
    }
    __syncthreads();
    key = lane < kWarps ? sm.wkey[par][lane] : 0ull;
    idx = lane < kWarps ? sm.wpos[par][lane] : 0x7fffffff;
    const int wp = idx;
    panel_argmax<T>(key, idx);
    const bool none = idx == 0x7fffffff;
    const int holder = none ? 0 : __ffs(__ballot_sync(0xffffffffu, wp == idx)) - 1;
    const T* const up = sm.slot[last][w];
    // the warp that holds this CTA's candidate sends its row, brought up to date
    // a lane per column; another warp takes the reciprocal and sends the rest
    if (warp == holder) {
      const bool cand = !done && pos == idx;
      if (cand) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) sm.stage[(d + TPR * k) & (kRegNb - 1)] = x[k];
      }
      const unsigned who = __ballot_sync(0xffffffffu, cand);
      const T l = __shfl_sync(0xffffffffu, lp, who ? __ffs(who) - 1 : 0);
      __syncwarp();
      if (pend && lane > 0 && lane < left) sm.stage[lane] = axpy1<false>(sm.stage[lane], -up[lane + 1], l);
      __syncwarp();
      const int v = lane % kVecs;
      const float4 val = reinterpret_cast<const float4*>(sm.stage)[v];
      if (v * kV < left)
        for (int q = lane / kVecs; q < G; q += 32 / kVecs)
          store_async(cluster_addr(&sm.slot[now][b][v * kV], q), val, cluster_addr(&sm.bar[now], q));
    } else if (warp == (holder ^ 1)) {
      union {
        RegMeta m;
        float4 f[2];
      } u;
      u.m.key = key;
      u.m.pos = none ? -1 : idx;
      *reinterpret_cast<T*>(&u.m.rcp) = pivot_rcp(from_bits<T>(key));
      if ((lane >> 1) < G)
        store_async(cluster_addr(reinterpret_cast<const float4*>(&sm.meta[now][b]) + (lane & 1), lane >> 1),
                    lane & 1 ? u.f[1] : u.f[0], cluster_addr(&sm.bar[now], lane >> 1));
    }
    // on the way meanwhile: the rest of column j - 1's update
    if (pend && !done) {
#pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (TPR * k < left && (TPR > 1 || (k > 0 && k + 1 < kPer))) {  // past the panel's end the values are never used
          if (TPR == 1 || k > 0 || d > 0) x[k] = axpy1<false>(x[k], -up[(d + TPR * k + 1) & (kRegNb - 1)], lp);
        }
    }
    if (!late) late = !bar_wait(&sm.bar[now], phase, g.poll_limit);
    // the pivot, the same in every warp
    {
      const RegMeta* m = &sm.meta[now][lane < G ? lane : 0];
      const int p = lane < G && m->pos >= c && m->pos < g.n ? m->pos : -1;
      key = p >= 0 ? m->key : 0ull;
      idx = p >= 0 ? p : 0x7fffffff;
      panel_argmax<T>(key, idx);
      const unsigned from = __ballot_sync(0xffffffffu, p >= 0 && p == idx);
      w = from ? __ffs(from) - 1 : 0;
    }
    const bool zero = idx == 0x7fffffff || key == 0;  // all |x| == 0: skipped, lu.rs:107-110
    if (b == 0 && tid == 0) {
      g.ipiv[c] = zero ? c : idx;
      if (zero) atomicMin(g.info, c + 1);
    }
    if (!__all_sync(0xffffffffu, done)) {
      const T* u = sm.slot[now][w];
      const bool mine = !done && pos == (zero ? c : idx);  // this row is row c of U
      if (mine) {
        done = true;
        pos = c;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
          if (d + TPR * k < left) sm.rows[j + d + TPR * k][rl] = x[k];
      }
      T l = x[0];
      if (!zero) l *= with_sign(*reinterpret_cast<const T*>(&sm.meta[now][w].rcp), u[0]);
      if (TPR > 1) l = __shfl_sync(0xffffffffu, l, (lane & ~(TPR - 1)) | s0);
      lp = l;
      if (!done) {
        if (!zero && pos == c) pos = idx;
        if (d == 0) {
          sm.rows[j][rl] = l;
#pragma unroll
          for (int k = 0; k + 1 < kPer; ++k) x[k] = x[k + 1];
        }
        if (!zero && d == (TPR > 1 ? 1 : 0)) x[0] = axpy1<false>(x[0], -u[1], l);
      }
    }
    pend = !zero;
    last = now;
    now = now == 2 ? 0 : now + 1;
    if (now == 0) phase ^= 1;
  }
  let_successor_in();
  if (late) atomicMin(g.info, kRegInfoTimeout);
  __syncwarp();
  if (valid && !late) {
    for (int k = sub; k < g.nb; k += TPR) g.A[(size_t)(g.j0 + k) * g.lda + pos] = sm.rows[k][rl];
    if (pos != row && sub == 0) {
      const int q = atomicAdd(npairs, 1);
      if (q < 2 * kRegNb) {
        pdst[q] = pos;
        psrc[q] = row;
      }
    }
  }
  __threadfence();
  cl.sync();
  const int np = min(__ldcg(npairs), 2 * kRegNb);
  for (int k = tid; k < np; k += kRegThreads) {
    sm.dst[k] = __ldcg(&pdst[k]);
    sm.src[k] = __ldcg(&psrc[k]);
  }
  for (int e = tid; e < g.nb * g.nb; e += kRegThreads) {
    const int k = e / g.nb, i = e - k * g.nb;
    sm.l11[k][i] = __ldcg(&g.A[(size_t)(g.j0 + k) * g.lda + g.j0 + i]);
  }
  __syncthreads();
  const int others = g.c_hi - g.c_lo - g.nb;
  for (int q = b * kWarps + warp; q < others; q += G * kWarps) {
    const int cc = g.c_lo + q < g.j0 ? g.c_lo + q : g.c_lo + q + g.nb;
    T* col = g.A + (size_t)cc * g.lda;
    T v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (lane + 32 * u < np) v[u] = col[sm.src[lane + 32 * u]];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (lane + 32 * u < np) col[sm.dst[lane + 32 * u]] = v[u];
    __syncwarp();
    if (cc > g.j0) {  // U12 = L11^-1 A12
      T y = lane < g.nb ? col[g.j0 + lane] : T(0);
      for (int k = 0; k + 1 < g.nb; ++k) {
        const T yk = __shfl_sync(0xffffffffu, y, k);
        if (lane > k && lane < g.nb) y = axpy1<false>(y, -sm.l11[k][lane], yk);
      }
      if (lane < g.nb) col[g.j0 + lane] = y;
    }
  }
}

// A22 -= L21 U12 for the outer block's remaining columns (at most 96), 32 deep:
// FP32, a thread per row with its 32 multipliers in registers, four column
// phases; U in shared memory.
__global__ void __launch_bounds__(256) lu_inner_update_kernel(int n, float* __restrict__ A, int64_t lda, int j0, int nb,
                                                              int c_hi) {
  __shared__ __align__(16) float U[96][kRegNb];
  wait_for_predecessor();
  let_successor_in();
  const int j1 = j0 + nb, w = c_hi - j1;
  for (int e = threadIdx.x; e < w * kRegNb; e += 256) {
    const int c = e >> 5, k = e & 31;
    U[c][k] = k < nb ? A[(size_t)(j1 + c) * lda + j0 + k] : 0.f;
  }
  __syncthreads();
  const int r = j1 + blockIdx.x * 64 + (threadIdx.x & 63);
  if (r >= n) return;
  float l[kRegNb];
#pragma unroll
  for (int k = 0; k < kRegNb; ++k) l[k] = k < nb ? A[(size_t)(j0 + k) * lda + r] : 0.f;
  for (int c = threadIdx.x >> 6; c < w; c += 4) {
    float* p = A + (size_t)(j1 + c) * lda + r;
    float acc = *p;
#pragma unroll
    for (int k = 0; k < kRegNb; ++k) acc = fmaf(-l[k], U[c][k], acc);
    *p = acc;
  }
}

// The scales of 32 rows of U, for the balance of the products L U: a CTA's warps hold
// a column each (lane: row), the first eight right of the block.  The mean of a row's
// exponents is blind to column scaling, which moves all rows' alike; the pivots' are
// not.  A row without a sample counts for little: where it is not zero further right,
// the products' checks send the outputs to the FP64 loop.
constexpr int kBalanceMax = 400;
__device__ __forceinline__ int packed_exponent(double x) {  // sum and count in one word, up to 255 of them
  const int ex = (__double2hiint(x) >> 20) & 0x7ff;
  return ex == 0x7ff || is_zero_bits(x) ? 0 : ex << 8 | 1;
}
__device__ __forceinline__ int mean_exponent(int packed) {
  if ((packed & 255) == 32) return packed >> 13;
  return __float2int_rn(__fdividef((float)(packed >> 8), (float)(packed & 255)));
}
__device__ __forceinline__ void u_row_exponents(double y, bool on, int nb, int* balance) {
  __shared__ int s_e[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  s_e[warp][lane] = on ? packed_exponent(y) : 0;
  __syncthreads();
  if (warp == 0 && lane < nb) {
    int e = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) e += s_e[w][lane];
    balance[lane] = e == 0 ? -kBalanceMax : max(-kBalanceMax, min(kBalanceMax, mean_exponent(e) - 1023));
  }
}

// The same in FP64 by digit slices (slices.cuh): rows j0 + nb .. r_hi - 1 times
// columns c_lo .. c_hi - 1, 64 x 32 of them per CTA, the 32 products of an
// output in one exact sum.  Where A's rows and columns have scales r_i and c_j, L_ik
// goes as r_i / r_k and U_kj as r_k c_j; so row k of U is cut against its mean
// exponent over the CTA's columns and column k of L the other way, which leaves r_i
// in every term of a row of L and c_j in every one of a column of U: both kinds of
// scaling keep their precision, as they do in the FP64 loop.  (The exponent of the
// pivot, r_k c_k, serves rows only: columns scaled by 2^+-20 lost 40 bits.)  What
// grading is left the meeting test finds, and those outputs take the FP64 loop.
// Eight levels of digit products and not seven: the solution's error is half that of
// the FP64 loop (orders 200 to 700, geometric means; seven levels 0.8 to 1.2 of it), at
// no time that shows.
// It sits between two panels, so its own latency counts and little else: four
// threads cut a row, a warp has one 16 x 8 tile, its 4 elements loaded first.  With
// 128 threads on 64 x 96 it took 17 us (3500 instructions in a row) at 1900 rows;
// the factorization at n = 2000 7.1 ms, so 6.1.
constexpr int kInnerRows = 64, kInnerCols = 32, kInnerThreads = 512;
constexpr int kInnerSlots = kInnerRows + kInnerCols;
constexpr int kInnerUWarps = 4 * kInnerCols / 32;  // the warps that hold U
constexpr size_t kInnerSmem = (size_t)2 * kSlices * kInnerSlots * kSliceRow + (kRegNb * kInnerUWarps + kInnerSlots) * 4;
// One output by the FP64 loop; out of line, its code would be fetched in vain.
__device__ __noinline__ void lu_inner_fp64(double* A, int64_t lda, int j0, int nb, int r, int c) {
  double v = A[(size_t)c * lda + r];
  for (int k = 0; k < nb; ++k) v = axpy1<false>(v, -A[(size_t)c * lda + j0 + k], A[(size_t)(j0 + k) * lda + r]);
  A[(size_t)c * lda + r] = v;
}
__global__ void __launch_bounds__(kInnerThreads) lu_inner_update_kernel(int r_hi, double* __restrict__ A, int64_t lda, int j0,
                                                                        int nb, int c_lo, int c_hi) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int sb = kInnerSlots * kSliceRow;
  unsigned char* SL = smem_raw;  // [half][slice][slot]
  int* uexp = reinterpret_cast<int*>(smem_raw + (size_t)2 * kSlices * sb);  // [row of U][warp]
  int* ex = uexp + kRegNb * kInnerUWarps;
  static_assert(kInnerUWarps == 4, "a row's exponents are read as one int4");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int r0 = j0 + nb + blockIdx.x * kInnerRows, cb = c_lo + blockIdx.y * kInnerCols;
  const int w = min(kInnerCols, c_hi - cb);
  const int rt = (warp & 3) * 16, c = (warp >> 2) * 8;  // this warp's tile
  wait_for_predecessor();
  let_successor_in();
  const int rg = r0 + rt + g, cg = c + 2 * t;  // the element's place: row rg (+ 8), column cb + cg (+ 1)
  const auto on = [&](int i) { return rg + (i >> 1) * 8 < r_hi && cg + (i & 1) < w; };
  double v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = on(i) ? A[(size_t)(cb + cg + (i & 1)) * lda + rg + (i >> 1) * 8] : 0.0;
  constexpr int kPart = kRegNb / 4;  // a thread's elements of its slot
  const int s = tid >> 2, k0 = (tid & 3) * kPart;
  const bool lrow = s < kInnerRows;
  double x[kPart];
  if (s < kInnerSlots) {
    const int r = r0 + s, cc = s - kInnerRows;
    const bool in = lrow ? r < r_hi : cc < w;
    const double* src = lrow ? A + (size_t)j0 * lda + r : A + (size_t)(cb + cc) * lda + j0;
    const int64_t st = lrow ? lda : 1;
#pragma unroll
    for (int k = 0; k < kPart; ++k) x[k] = in && k0 + k < nb ? src[(k0 + k) * st] : 0.0;
    if (!lrow) {
#pragma unroll
      for (int k = 0; k < kPart; ++k) {
        int e = packed_exponent(x[k]);
        e += __shfl_xor_sync(0xffffffffu, e, 4);
        e += __shfl_xor_sync(0xffffffffu, e, 8);
        e += __shfl_xor_sync(0xffffffffu, e, 16);
        if (lane < 4) uexp[(k0 + k) * kInnerUWarps + (s - kInnerRows) / 8] = e;
      }
    }
  }
  __syncthreads();
  if (s < kInnerSlots) {
    int shift[kPart];  // kNoExponent: the row of U is zero, L's entry does not count
    int em = kNoExponent;
#pragma unroll
    for (int k = 0; k < kPart; ++k) {
      const int4 u = *reinterpret_cast<const int4*>(uexp + (k0 + k) * kInnerUWarps);
      const int sum = u.x + u.y + u.z + u.w, e = sum ? mean_exponent(sum) : kNoExponent;
      shift[k] = lrow ? e : -e;
      em = max(em, shifted_exponent(x[k], shift[k]));
    }
    em = max(em, __shfl_xor_sync(0xffffffffu, em, 1));
    em = max(em, __shfl_xor_sync(0xffffffffu, em, 2));
#pragma unroll
    for (int k = 0; k < kPart; k += 4) {
      uint32_t w0[kSlices], w1[kSlices];
      slice_digits(x[k], x[k + 1], em - shift[k], em - shift[k + 1], w0);
      slice_digits(x[k + 2], x[k + 3], em - shift[k + 2], em - shift[k + 3], w1);
      const int kk = k0 + k;
#pragma unroll
      for (int q = 0; q < kSlices; ++q)
        *reinterpret_cast<uint2*>(SL + (size_t)((kk >> 4) * kSlices + q) * sb + s * kSliceRow + (kk & 15) * 2) =
            make_uint2(w0[q], w1[q]);
    }
    if (k0 == 0) ex[s] = graded_code(em);
  }
  __syncthreads();
  if (c >= w) return;
  float acc[kSlices + 1][4], met[4] = {0.f, 0.f, 0.f, 0.f};
  slice_sums_start(acc);
#pragma unroll
  for (int h = 0; h < 2; ++h)
    slice_products_met(SL + (size_t)h * kSlices * sb + rt * kSliceRow,
                       SL + (size_t)h * kSlices * sb + (kInnerRows + c) * kSliceRow, sb, lane, acc, met);
  const int e0 = ex[rt + g], e1 = ex[rt + g + 8];
  const int f0 = ex[kInnerRows + c + 2 * t], f1 = ex[kInnerRows + c + 2 * t + 1];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int er = i >> 1 ? e1 : e0, ec = i & 1 ? f1 : f0;
    const bool bad = er == kBadRow || ec == kBadRow, zero = er == kNoExponent || ec == kNoExponent;
    const double y = slice_value<32>(acc, i, er + ec);
    if (!on(i)) continue;
    if (bad || (!zero && met[i] < kMeet)) lu_inner_fp64(A, lda, j0, nb, rg + (i >> 1) * 8, cb + cg + (i & 1));
    else A[(size_t)(cb + cg + (i & 1)) * lda + rg + (i >> 1) * 8] = v[i] - y;
  }
}

// The outer block's swaps on the columns outside it: the panels' lists in
// order, a warp per column.
template <typename T>
__global__ void __launch_bounds__(256) lu_swap_lists_kernel(int n, T* A, int64_t lda, const PanelPub<T>* __restrict__ pub,
                                                            int lists, int j0, int nb) {
  __shared__ int s_dst[2 * kPanelMaxNb], s_src[2 * kPanelMaxNb], s_np[kPanelMaxNb / kRegNb];
  for (int k = threadIdx.x; k < 2 * kRegNb * lists; k += blockDim.x) {
    s_dst[k] = pub->pdst[k];
    s_src[k] = pub->psrc[k];
  }
  if (threadIdx.x < (unsigned)lists) s_np[threadIdx.x] = pub->nlist[threadIdx.x];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int c = blockIdx.x * 8 + warp;
  if (c >= j0) c += nb;
  if (c >= n) return;
  T* col = A + (size_t)c * lda;
  for (int l = 0; l < lists; ++l) {
    const int np = s_np[l], o = 2 * kRegNb * l;
    T v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (lane + 32 * u < np) v[u] = col[s_src[o + lane + 32 * u]];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (lane + 32 * u < np) col[s_dst[o + lane + 32 * u]] = v[u];
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// row swaps of the panel applied to the other columns; unit-lower TRSM
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) lu_swap_kernel(int n, T* A, int64_t lda, const PanelPub<T>* __restrict__ pub,
                                                      int j0, int nb) {
  __shared__ int s_dst[2 * kPanelMaxNb], s_src[2 * kPanelMaxNb];
  const int np = pub->npairs;
  for (int k = threadIdx.x; k < np; k += blockDim.x) {
    s_dst[k] = pub->pdst[k];
    s_src[k] = pub->psrc[k];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int c = blockIdx.x * 8 + warp;  // a warp per column outside the panel
  if (c >= j0) c += nb;
  if (np == 0 || c >= n) return;
  T* col = A + (size_t)c * lda;
  constexpr int U = 2 * kPanelMaxNb / 32;
  T v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int k = lane + 32 * u;
    if (k < np) v[u] = col[s_src[k]];
  }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int k = lane + 32 * u;
    if (k < np) col[s_dst[k]] = v[u];
  }
}

// U12 = L11^-1 A12 (unit lower L11, NB x NB, in shared memory) for the columns
// right of the panel: a warp owns kTrsmCols columns, lane l holding rows
// l, l + 32, ... of each in registers; row k's final value is broadcast by a
// shuffle and eliminated from the rows below (solve_lower_triangular_with_diag,
// src/linalg/solve.rs:106-133, column-oriented).
constexpr int kTrsmCols = 4;
template <typename T, int NB>
__global__ void __launch_bounds__(256) lu_trsm_kernel(int n, T* A, int64_t lda, int j0) {
  constexpr int M = NB / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* L = reinterpret_cast<T*>(smem_raw);  // L[k * NB + i] = A[j0 + i][j0 + k]
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    const int k = e / NB, i = e - k * NB;
    L[e] = A[(size_t)(j0 + k) * lda + j0 + i];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cbase = j0 + NB + (blockIdx.x * 8 + warp) * kTrsmCols;
  if (cbase >= n) return;
  T v[kTrsmCols][M];
#pragma unroll
  for (int c = 0; c < kTrsmCols; ++c) {
    const int col = min(cbase + c, n - 1);
#pragma unroll
    for (int m = 0; m < M; ++m) v[c][m] = A[(size_t)col * lda + j0 + m * 32 + lane];
  }
#pragma unroll
  for (int mb = 0; mb < M; ++mb) {
#pragma unroll 4
    for (int kk = 0; kk < 32; ++kk) {
      const int k = mb * 32 + kk;
      T lk[M];
#pragma unroll
      for (int m = mb; m < M; ++m) lk[m] = L[k * NB + m * 32 + lane];
#pragma unroll
      for (int c = 0; c < kTrsmCols; ++c) {
        const T xk = __shfl_sync(0xffffffffu, v[c][mb], kk);
#pragma unroll
        for (int m = mb; m < M; ++m)
          if (m > mb || lane > kk) v[c][m] = axpy1<false>(v[c][m], -lk[m], xk);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kTrsmCols; ++c) {
    const int col = cbase + c;
    if (col < n)
#pragma unroll
      for (int m = 0; m < M; ++m) A[(size_t)col * lda + j0 + m * 32 + lane] = v[c][m];
  }
}

__global__ void __launch_bounds__(256) lu_balance_kernel(int n, const double* A, int64_t lda, int p0, int nb, int c0,
                                                         int* balance) {
  const int lane = threadIdx.x & 31, c = c0 + (threadIdx.x >> 5);
  const bool on = c < n && lane < nb;
  u_row_exponents(on ? A[(size_t)c * lda + p0 + lane] : 0.0, on, nb, balance);
}

// The solve with one unit lower triangle of at most 32 rows at p0 for columns
// c0 .. n - 1: a warp per column, a row per lane.  The first CTA leaves the rows' scales.
__global__ void __launch_bounds__(256) lu_trsm_piece_kernel(int n, double* __restrict__ A, int64_t lda, int p0, int nb,
                                                            int c0, int* balance) {
  __shared__ double L[32][33];
  wait_for_predecessor();
  let_successor_in();
  for (int e = threadIdx.x; e < nb * nb; e += 256) {
    const int k = e / nb, i = e - k * nb;
    L[k][i] = A[(size_t)(p0 + k) * lda + p0 + i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, c = c0 + blockIdx.x * 8 + (threadIdx.x >> 5);
  const bool on = c < n && lane < nb;
  double* col = A + (size_t)c * lda + p0;
  double y = on ? col[lane] : 0.0;
  for (int k = 0; k + 1 < nb; ++k) {
    const double yk = __shfl_sync(0xffffffffu, y, k);
    if (lane > k && lane < nb) y = axpy1<false>(y, -L[k][lane], yk);
  }
  if (on) col[lane] = y;
  if (blockIdx.x == 0) u_row_exponents(y, on, nb, balance);
}

// The same for a panel width without a register-tiled instance: L11 in shared
// memory, one thread per column, the column kept in shared memory.
template <typename T>
__global__ void __launch_bounds__(64) lu_trsm_generic_kernel(int n, T* A, int64_t lda, int j0, int nb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* L = reinterpret_cast<T*>(smem_raw);  // nb x nb
  T* X = L + (size_t)nb * nb;             // nb x 64 (column-major per thread)
  const int tid = threadIdx.x;
  for (int e = tid; e < nb * nb; e += blockDim.x) {
    const int cc = e / nb, r = e - cc * nb;
    L[e] = A[(size_t)(j0 + cc) * lda + j0 + r];
  }
  const int c = j0 + nb + blockIdx.x * 64 + tid;
  const bool valid = c < n;
  T* col = A + (size_t)(valid ? c : j0) * lda + j0;
  for (int i = 0; i < nb; ++i) X[(size_t)i * 64 + tid] = valid ? col[i] : T(0);
  __syncthreads();
  for (int i = 1; i < nb; ++i) {
    T x = X[(size_t)i * 64 + tid];
    for (int k = 0; k < i; ++k) x = axpy1<false>(x, -L[(size_t)k * nb + i], X[(size_t)k * 64 + tid]);
    X[(size_t)i * 64 + tid] = x;
  }
  if (valid)
    for (int i = 0; i < nb; ++i) col[i] = X[(size_t)i * 64 + tid];
}

template <typename T, int NB>
cudaError_t launch_trsm_tiled(int n, T* A, int64_t lda, int j0, int rest, cudaStream_t s) {
  const size_t smem = (size_t)NB * NB * sizeof(T);
  cudaError_t e = ensure_dynamic_smem(lu_trsm_kernel<T, NB>, smem);
  if (e != cudaSuccess) return e;
  const int per_cta = 8 * kTrsmCols;
  lu_trsm_kernel<T, NB><<<(rest + per_cta - 1) / per_cta, 256, smem, s>>>(n, A, lda, j0);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_trsm(int n, T* A, int64_t lda, int j0, int jb, int rest, cudaStream_t s) {
  if (jb == 64) return launch_trsm_tiled<T, 64>(n, A, lda, j0, rest, s);
  if constexpr (sizeof(T) == 4)  // FP64 blocks of 128 go by pieces
    if (jb == 128) return launch_trsm_tiled<T, 128>(n, A, lda, j0, rest, s);
  const size_t smem = (size_t)jb * jb * sizeof(T) + (size_t)jb * 64 * sizeof(T);
  if (smem > 48 * 1024) {
    cudaError_t e = ensure_dynamic_smem(lu_trsm_generic_kernel<T>, smem);
    if (e != cudaSuccess) return e;
  }
  lu_trsm_generic_kernel<T><<<(rest + 63) / 64, 64, smem, s>>>(n, A, lda, j0, jb);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// triangular solves for one right-hand side (one CTA per row block, ready flags)
// ---------------------------------------------------------------------------
constexpr int kTrsvThreads = 256;
constexpr int kTrsvInfoTimeout = -1000;  // info value when a wait ran out
template <typename T>
struct TrsvTile {
  static constexpr int BS = sizeof(T) == 4 ? 128 : 64;  // rows per block
  static constexpr int NC = kTrsvThreads / BS;          // column parts per row
  static constexpr int CW = BS / NC;                    // columns per part
};

template <typename T>
struct TrsvArgs {
  int n;
  const T* A;
  int64_t lda;
  T* x;
  int lower;
  int32_t* info;
  int* sync;  // [0] ticket, [1] timeout flag, [2 + b] block b solved (zeroed before the launch)
  int poll_limit;  // polls of one flag before the wait gives up
  int skip_flag;   // a block that never raises its flag (test hook only; -1 otherwise)
};
constexpr int kTrsvPollLimit = 1 << 22;  // with the 64 ns back-off: seconds, far above any block's solve

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// lower = 1: x <- L^-1 x (unit diagonal, blocks top-down); lower = 0:
// x <- U^-1 x (bottom-up; a zero U_ii is reported in info, as
// solve_upper_triangular_mut returns false, src/linalg/solve.rs:137-182).
// CTAs take row blocks in ticket order, so a CTA only ever waits for blocks
// whose CTAs have started: for each solved block it prefetches its tile of the
// triangle into registers, waits for the block's flag (bounded), and applies
// it; then it solves its diagonal block in shared memory, stores it and raises
// its own flag.  Every wait gives up after a fixed number of polls, sets the
// timeout flag and info = kTrsvInfoTimeout, and the CTA returns.
template <typename T>
__global__ void __launch_bounds__(kTrsvThreads) trsv_kernel(TrsvArgs<T> g) {
  constexpr int BS = TrsvTile<T>::BS, NC = TrsvTile<T>::NC, CW = TrsvTile<T>::CW, LD = BS + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ts = reinterpret_cast<T*>(smem_raw);  // Ts[k * LD + i] = A[r0 + i][r0 + k]
  __shared__ T xs[BS];
  __shared__ T rd[BS];
  __shared__ T part[NC][BS];
  constexpr int kW = kTrsvThreads / 32, kPer = 32 / kW;  // row update: warps, terms per warp
  constexpr int kH = (BS - 32 + 31) / 32;                 // 32-row groups on the far side of a piece
  __shared__ T pp[kW * kH * 32];
  __shared__ int s_ticket, s_abort;
  const int tid = threadIdx.x, tr = tid % BS, tc = tid / BS;
  const int n = g.n, lower = g.lower;
  static_assert(kTrsvThreads % 32 == 0, "warps");
  const int nblk = (n + BS - 1) / BS;
  if (tid == 0) {
    s_ticket = atomicAdd(&g.sync[0], 1);
    s_abort = 0;
  }
  __syncthreads();
  const int t = s_ticket;
  if (t >= nblk) return;
  const int kb = lower ? t : nblk - 1 - t;
  const int r0 = kb * BS, bs = min(BS, n - r0);
  const T* A = g.A;
  const int64_t lda = g.lda;
  // U's columns are pre-scaled by 1 / U_kk, so the diagonal solve takes one
  // FMA per step on the unscaled values (scaled once when the block is
  // stored); L has a unit diagonal
  if (!lower) {
    for (int i = tid; i < bs; i += kTrsvThreads) {
      const T d = A[(size_t)(r0 + i) * lda + r0 + i];
      if (d == T(0)) atomicMin(g.info, r0 + i + 1);
      rd[i] = T(1) / d;
    }
    __syncthreads();
  }
  for (int e = tid; e < bs * bs; e += kTrsvThreads) {
    const int k = e / bs, i = e - k * bs;
    if (lower ? (i > k) : (i < k)) {
      const T v = A[(size_t)(r0 + k) * lda + r0 + i];
      Ts[k * LD + i] = lower ? v : v * rd[k];
    }
  }
  T acc = (tc == 0 && tr < bs) ? g.x[r0 + tr] : T(0);
  for (int q = 0; q < t; ++q) {
    const int jb = lower ? q : nblk - 1 - q;
    const int c0 = jb * BS, cs = min(BS, n - c0);
    T a[CW];
#pragma unroll
    for (int u = 0; u < CW; ++u) {
      const int col = tc * CW + u;
      a[u] = (tr < bs && col < cs) ? A[(size_t)(c0 + col) * lda + r0 + tr] : T(0);
    }
    if (tid == 0) {
      int polls = 0;
      while (ld_acquire(&g.sync[2 + jb]) == 0) {
        if (++polls > g.poll_limit) {
          s_abort = 1;
          atomicExch(&g.sync[1], 1);
          atomicMin(g.info, kTrsvInfoTimeout);
          break;
        }
        __nanosleep(64);
      }
    }
    __syncthreads();
    if (s_abort) return;
    // all of xs: past cs it meets zero tile entries, and shared memory may
    // still hold an earlier kernel's inf or NaN there (NaN * 0)
    if (tid < BS) xs[tid] = tid < cs ? __ldcg(&g.x[c0 + tid]) : T(0);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < CW; ++u) acc = axpy1<false>(acc, -xs[tc * CW + u], a[u]);
    __syncthreads();
  }
  part[tc][tr] = acc;
  __syncthreads();
  if (tid < bs) {
    T y = part[0][tid];
#pragma unroll
    for (int c = 1; c < NC; ++c) y += part[c][tid];
    xs[tid] = y;
  }
  __syncthreads();
  // the diagonal block, 32 rows at a time: one warp solves the 32 x 32
  // diagonal piece with shuffles, then all threads apply it to the block's
  // remaining rows
  const int warp = tid >> 5, lane = tid & 31;
  const int nsub = (bs + 31) / 32;
  for (int q = 0; q < nsub; ++q) {
    const int sb = lower ? q * 32 : (nsub - 1 - q) * 32;
    const int sw = min(32, bs - sb);
    if (warp == 0) {
      T v = lane < sw ? xs[sb + lane] : T(0);
      if (lower) {
#pragma unroll
        for (int kk = 0; kk < 32; ++kk) {
          const T xk = __shfl_sync(0xffffffffu, v, kk);
          if (lane > kk && lane < sw) v = axpy1<false>(v, -Ts[(sb + kk) * LD + sb + lane], xk);
        }
      } else {
#pragma unroll
        for (int kk = 31; kk >= 0; --kk) {
          const T xk = __shfl_sync(0xffffffffu, v, kk);
          if (lane < kk && kk < sw) v = axpy1<false>(v, -Ts[(sb + kk) * LD + sb + lane], xk);
        }
      }
      if (lane < sw) xs[sb + lane] = v;  // U: unscaled
    }
    __syncthreads();
    // the block's rows on the far side of the piece (at most BS - 32) take its
    // contribution: warp w sums its share of the piece's terms for row i0 +
    // lane (+ 32h), then one thread per row adds the partial sums (a short
    // chain instead of sw dependent FMAs on one warp)
    const int i0 = lower ? sb + sw : 0, i1 = lower ? bs : sb;
    if (i1 > i0) {
#pragma unroll
      for (int h = 0; h < kH; ++h) {
        const int i = i0 + lane + 32 * h;
        T acc = T(0);
        if (i < i1)
#pragma unroll
          for (int u = 0; u < kPer; ++u) {
            const int k = kPer * warp + u;
            if (k < sw) acc = axpy1<false>(acc, -Ts[(sb + k) * LD + i], xs[sb + k]);
          }
        pp[(warp * kH + h) * 32 + lane] = acc;
      }
      __syncthreads();
      for (int r = tid; r < i1 - i0; r += kTrsvThreads) {
        T y = xs[i0 + r];
#pragma unroll
        for (int w = 0; w < kW; ++w) y += pp[(w * kH + (r >> 5)) * 32 + (r & 31)];
        xs[i0 + r] = y;
      }
    }
    __syncthreads();
  }
  if (tid < bs) g.x[r0 + tid] = lower ? xs[tid] : xs[tid] * rd[tid];
  // the barrier orders the block's stores before thread 0's release, which is
  // cumulative over them: a CTA that acquires the flag sees x (no fence needed)
  __syncthreads();
  if (tid == 0 && kb != g.skip_flag) st_release(&g.sync[2 + kb], 1);
}

// info holds a large sentinel until some pivot fails; 0 afterwards means "ok".
__global__ void info_init_kernel(int32_t* info) { *info = 0x7fffffff; }
__global__ void info_finalize_kernel(int32_t* info) {
  if (*info == 0x7fffffff) *info = 0;
}

// x <- P x: nalgebra's row swaps in order (PermutationSequence::permute_rows,
// src/linalg/permutation_sequence.rs), one thread, the vector and the swap
// list staged in shared memory when they fit.
template <typename T>
__global__ void apply_pivots_kernel(int n, const int32_t* __restrict__ ipiv, T* x, int staged) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* xs = reinterpret_cast<T*>(smem_raw);
  int32_t* ps = reinterpret_cast<int32_t*>(xs + (staged ? n : 0));
  if (!staged) {
    if (threadIdx.x == 0)
      for (int i = 0; i < n; ++i) {
        const int p = ipiv[i];
        if (p != i) {
          const T t = x[i];
          x[i] = x[p];
          x[p] = t;
        }
      }
    return;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    xs[i] = x[i];
    ps[i] = ipiv[i];
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 0; i < n; ++i) {
      const int p = ps[i];
      if (p != i) {
        const T t = xs[i];
        xs[i] = xs[p];
        xs[p] = t;
      }
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] = xs[i];
}

// perm[i] = the source row of row i after the swaps (gathers replace them).
__global__ void pivots_to_perm_kernel(int n, const int32_t* __restrict__ ipiv, int32_t* perm, int staged) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int32_t* pm = staged ? reinterpret_cast<int32_t*>(smem_raw) : perm;
  int32_t* ps = staged ? pm + n : nullptr;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    pm[i] = i;
    if (staged) ps[i] = ipiv[i];
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 0; i < n; ++i) {
      const int p = staged ? ps[i] : ipiv[i];
      if (p != i) {
        const int32_t t = pm[i];
        pm[i] = pm[p];
        pm[p] = t;
      }
    }
  __syncthreads();
  if (staged)
    for (int i = threadIdx.x; i < n; i += blockDim.x) perm[i] = pm[i];
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
int coop_grid(const void* kern, int threads, size_t smem) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (per_sm < 1) per_sm = 1;
  return sm_count() * per_sm;
}

// The panel's exchange area (sized for FP64 and the widest panel).
size_t getrf_ws_bytes() { return (sizeof(PanelPub<double>) + 255) & ~(size_t)255; }

// slot 0: the next panel's columns (on the panel stream), slot 1: the rest of
// the trailing update (on the update stream, concurrently)
typedef int (*UpdateFn)(int m, int n, int k, const void* L21, const void* U12, void* A22, int64_t lda, void* ctx,
                        int slot, cudaStream_t s);

// Internal streams of the look-ahead schedule (per device, created on first
// use): the panel chain runs at the highest stream priority, the bulk of each
// trailing update at the lowest, so the next panel's CTAs are dispatched as
// soon as SMs free up.
struct LookaheadStreams {
  cudaStream_t panel = nullptr, rest = nullptr;
  cudaEvent_t fork = nullptr, trsm_done = nullptr, rest_done = nullptr, join = nullptr;
  bool ready = false;
};
LookaheadStreams g_lookahead[64];

int lookahead_streams(LookaheadStreams** out, const char* name) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  if (dev < 0 || dev >= 64) return record_arg_error(-99, "getrf: device index >= 64");
  LookaheadStreams& L = g_lookahead[dev];
  if (!L.ready) {
    int least = 0, greatest = 0;
    e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&L.panel, cudaStreamNonBlocking, greatest);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&L.rest, cudaStreamNonBlocking, least);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&L.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&L.trsm_done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&L.rest_done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&L.join, cudaEventDisableTiming);
    if (e != cudaSuccess) return record_cuda_error(e, name);
    L.ready = true;
  }
  *out = &L;
  return NACU_SUCCESS;
}

// CTAs per cluster for the cluster-form panel (16, else 8, else 0 = grid
// form only), from the occupancy API with the largest panel's shared memory;
// queried once per scalar type.
template <typename T>
int panel_cluster_ctas() {
  static int ctas = -1;
  if (ctas >= 0) return ctas;
  ctas = 0;
  auto kern = lu_panel_cluster_kernel<T>;
  if (ensure_dynamic_smem(kern, kPanelMaxSmem) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return ctas;
  }
  for (int c = kClusterMaxCtas; c >= 8; c /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kPanelThreads);
    cfg.dynamicSmemBytes = kPanelMaxSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters >= 1) {
      ctas = c;
      break;
    }
    cudaGetLastError();
  }
  return ctas;
}

// CTAs of a register panel's cluster: rows spread over as many as there are 64
// rows for (an FP64 update is bound by its SMs' FP64 pipes), at most 16.
inline int reg_panel_ctas(int rows) {
  int g = 1;
  while (g < kClusterMaxCtas && rows > 64 * g) g *= 2;
  return g;
}

using InnerUpdate32 = void (*)(int, float*, int64_t, int, int, int);
using InnerUpdate64 = void (*)(int, double*, int64_t, int, int, int, int);

// The kernel with as many threads to a row as a CTA of `chunk` rows has.
template <typename T>
void (*reg_panel_kernel(int chunk))(RegPanelArgs<T>) {
  if (chunk <= kRegThreads / 8) return lu_panel_reg_kernel<T, 8>;
  if (chunk <= kRegThreads / 4) return lu_panel_reg_kernel<T, 4>;
  if (chunk <= kRegThreads / 2) return lu_panel_reg_kernel<T, 2>;
  return lu_panel_reg_kernel<T, 1>;
}

// An outer block of jb columns at j0 by panels of kRegNb (swaps and U inside
// the block included); the panels' swap lists stay in pub.
template <typename T>
int reg_block(int n, T* A, int64_t lda, int j0, int jb, int32_t* ipiv, int32_t* info, PanelPub<T>* pub, int poll_limit,
              cudaStream_t s, const char* name) {
  for (int p0 = j0; p0 < j0 + jb; p0 += kRegNb) {
    const int nb = std::min(kRegNb, j0 + jb - p0), rows = n - p0;
    const int G = reg_panel_ctas(rows);
    RegPanelArgs<T> pa{n, A, lda, p0, nb, (rows + G - 1) / G, j0, j0 + jb, (p0 - j0) / kRegNb, ipiv, info, pub,
                       poll_limit};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(kRegThreads);
    cfg.dynamicSmemBytes = sizeof(RegPanelSmem<T>);
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, reg_panel_kernel<T>(pa.chunk), pa);
    if (e != cudaSuccess) return record_cuda_error(e, name);
    const int below = rows - nb;
    if (p0 + nb < j0 + jb && below > 0) {
      if constexpr (sizeof(T) == 8)
        e = launch_chained(static_cast<InnerUpdate64>(lu_inner_update_kernel),
                           dim3((below + kInnerRows - 1) / kInnerRows, (j0 + jb - p0 - nb + kInnerCols - 1) / kInnerCols),
                           kInnerThreads, kInnerSmem, s, n, A, lda, p0, nb, p0 + nb, j0 + jb);
      else
        e = launch_chained(static_cast<InnerUpdate32>(lu_inner_update_kernel), dim3((below + 63) / 64), 256, 0, s, n, A, lda,
                           p0, nb, j0 + jb);
      if (e != cudaSuccess) return record_cuda_error(e, name);
    }
  }
  return check_launch(name);
}

// Whether this device runs the register panels for order n: a cluster of 16
// with their shared memory, and no more rows than its threads.
template <typename T>
bool reg_panels(int n) {
  static int ok = -1;
  if (ok < 0) {
    ok = 0;
    bool good = true;
    for (int chunk = kRegThreads; chunk >= kRegThreads / 8 && good; chunk /= 2) {
      const auto kern = reg_panel_kernel<T>(chunk);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(kClusterMaxCtas);
      cfg.blockDim = dim3(kRegThreads);
      cfg.dynamicSmemBytes = sizeof(RegPanelSmem<T>);
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = kClusterMaxCtas;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nclusters = 0;
      good = ensure_dynamic_smem(kern, sizeof(RegPanelSmem<T>)) == cudaSuccess &&
             cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
             cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters >= 1;
    }
    if constexpr (sizeof(T) == 8) {
      good = good && ensure_dynamic_smem(static_cast<InnerUpdate64>(lu_inner_update_kernel), kInnerSmem) == cudaSuccess;
    }
    if (!good) cudaGetLastError();
    ok = good ? 1 : 0;
  }
  return ok == 1 && n <= kRegMaxRows;
}

// U12 = L11^-1 A12 in FP64 for an outer block, 32 rows at a time: the solve with
// the piece's triangle, then its update of the block's rows below by digit
// slices.  A quarter of the solve's FP64 instructions (2048 columns: 94 us in one
// kernel; seven launches of 6 to 10 us here).
cudaError_t trsm_by_pieces(int n, double* A, int64_t lda, int j0, int jb, int* balance, cudaStream_t s) {
  const int c0 = j0 + jb, rest = n - c0;
  for (int p0 = j0; p0 < c0; p0 += kRegNb) {
    const int nb = std::min(kRegNb, c0 - p0);
    cudaError_t e = launch_chained(lu_trsm_piece_kernel, dim3((rest + 7) / 8), 256, 0, s, n, A, lda, p0, nb, c0,
                                   balance + (p0 - j0));
    const int below = c0 - p0 - nb;
    if (e == cudaSuccess && below > 0)
      e = launch_chained(static_cast<InnerUpdate64>(lu_inner_update_kernel),
                         dim3((below + kInnerRows - 1) / kInnerRows, (rest + kInnerCols - 1) / kInnerCols), kInnerThreads,
                         kInnerSmem, s, c0, A, lda, p0, nb, c0, n);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Blocked LU with look-ahead: step k's panel chain (panel, row swaps, TRSM,
// and the update of the next panel's columns) runs on the panel stream; the
// rest of step k's trailing update runs on the update stream while panel k+1
// is factored.  Step k+1's row swaps wait for that update.  Forks from and
// joins to the caller's stream.
template <typename T>
int getrf_blocked(int n, T* A, int64_t lda, int32_t* ipiv, int32_t* info, void* ws, int nb, UpdateFn update,
                  void* ctx, cudaStream_t s, const char* name, int poll_limit = kRegPollLimit) {
  cudaError_t e;
  const bool by_registers = reg_panels<T>(n);
  nb = by_registers ? kPanelMaxNb : std::min(nb, kPanelMaxNb);
  const void* pk = reinterpret_cast<const void*>(lu_panel_grid_kernel<T>);
  e = ensure_dynamic_smem(pk, kPanelMaxSmem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  const int cluster = panel_cluster_ctas<T>();
  const int gmax = std::min(kPanelMaxG, sm_count());
  LookaheadStreams* la = nullptr;
  int rc = lookahead_streams(&la, name);
  if (rc != NACU_SUCCESS) return rc;
  const cudaStream_t sp = la->panel, su = la->rest;
  e = cudaEventRecord(la->fork, s);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(sp, la->fork, 0);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(su, la->fork, 0);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  info_init_kernel<<<1, 1, 0, sp>>>(info);
  bool rest_pending = false;
  for (int j0 = 0; j0 < n; j0 += nb) {
    const int jb = std::min(nb, n - j0);
    const int rows = n - j0;
    PanelArgs<T> pa{n, A, lda, j0, jb, 0, ipiv, info, reinterpret_cast<PanelPub<T>*>(ws)};
    if (by_registers) {
      rc = reg_block<T>(n, A, lda, j0, jb, ipiv, info, pa.pub, poll_limit, sp, name);
      if (rc != NACU_SUCCESS) return rc;
    } else {
      const int cchunk = cluster ? (rows + cluster - 1) / cluster : 0;
      const size_t csmem = cluster_pub_bytes<T>(jb) + (size_t)(cchunk | 1) * jb * sizeof(T);
      if (cluster && csmem <= kPanelMaxSmem) {
        pa.chunk = cchunk;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cluster);
        cfg.blockDim = dim3(kPanelThreads);
        cfg.dynamicSmemBytes = csmem;
        cfg.stream = sp;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, lu_panel_cluster_kernel<T>, pa);
        if (e != cudaSuccess) return record_cuda_error(e, name);
      } else {
        const int max_rows = (int)(kPanelMaxSmem / ((size_t)jb * sizeof(T))) - 1;  // leading dimension chunk | 1
        int G = std::max((rows + kPanelRowsPerCta - 1) / kPanelRowsPerCta, (rows + max_rows - 1) / max_rows);
        G = std::max(1, std::min(G, gmax));
        const int chunk = (rows + G - 1) / G;
        if (chunk > max_rows) return record_arg_error(-1, "getrf: n too large for the shared-memory panel");
        pa.chunk = chunk;
        void* args[] = {&pa};
        e = cudaLaunchCooperativeKernel(pk, G, kPanelThreads, args, (size_t)(chunk | 1) * jb * sizeof(T), sp);
        if (e != cudaSuccess) return record_cuda_error(e, name);
      }
    }
    if (rest_pending) {  // the swaps below touch the columns the previous update is still writing
      e = cudaStreamWaitEvent(sp, la->rest_done, 0);
      if (e != cudaSuccess) return record_cuda_error(e, name);
      rest_pending = false;
    }
    if (n > jb && by_registers)
      lu_swap_lists_kernel<T><<<(n - jb + 7) / 8, 256, 0, sp>>>(n, A, lda, pa.pub, (jb + kRegNb - 1) / kRegNb, j0, jb);
    else if (n > jb)
      lu_swap_kernel<T><<<(n - jb + 7) / 8, 256, 0, sp>>>(n, A, lda, pa.pub, j0, jb);
    const int rest = n - j0 - jb;
    if (rest > 0) {
      if constexpr (sizeof(T) == 8) {
        if (by_registers) {
          e = trsm_by_pieces(n, A, lda, j0, jb, pa.pub->balance, sp);
        } else {
          e = launch_trsm<T>(n, A, lda, j0, jb, rest, sp);
          for (int p0 = 0; p0 < jb; p0 += kRegNb)
            lu_balance_kernel<<<1, 256, 0, sp>>>(n, A, lda, j0 + p0, std::min(kRegNb, jb - p0), j0 + jb,
                                                 pa.pub->balance + p0);
        }
      } else {
        e = launch_trsm<T>(n, A, lda, j0, jb, rest, sp);
      }
      if (e != cudaSuccess) return record_cuda_error(e, name);
      const T* L21 = A + (size_t)j0 * lda + j0 + jb;
      const T* U12 = A + (size_t)(j0 + jb) * lda + j0;
      T* A22 = A + (size_t)(j0 + jb) * lda + j0 + jb;
      const int nn = std::min(nb, rest);  // the next panel's columns
      rc = update(rest, nn, jb, L21, U12, A22, lda, ctx, 0, sp);
      if (rc != NACU_SUCCESS) return rc;
      if (rest > nn) {
        e = cudaEventRecord(la->trsm_done, sp);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(su, la->trsm_done, 0);
        if (e != cudaSuccess) return record_cuda_error(e, name);
        rc = update(rest, rest - nn, jb, L21, U12 + (size_t)nn * lda, A22 + (size_t)nn * lda, lda, ctx, 1, su);
        if (rc != NACU_SUCCESS) return rc;
        e = cudaEventRecord(la->rest_done, su);
        if (e != cudaSuccess) return record_cuda_error(e, name);
        rest_pending = true;
      }
    }
    rc = check_launch(name);
    if (rc != NACU_SUCCESS) return rc;
  }
  if (rest_pending) {
    e = cudaStreamWaitEvent(sp, la->rest_done, 0);
    if (e != cudaSuccess) return record_cuda_error(e, name);
  }
  info_finalize_kernel<<<1, 1, 0, sp>>>(info);
  e = cudaEventRecord(la->join, sp);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(s, la->join, 0);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  return check_launch(name);
}

// x <- U^-1 L^-1 x (the permutation already applied); sync: 2 + n/64 + 1 ints.
size_t trsv_sync_bytes(int n) { return ((size_t)n / 64 + 4) * sizeof(int); }

template <typename T>
int trsv_pair(int n, const T* LU, int64_t lda, T* x, int32_t* info, int* sync, cudaStream_t s, const char* name,
              int poll_limit = kTrsvPollLimit, int skip_lower_flag = -1) {
  const void* tk = reinterpret_cast<const void*>(trsv_kernel<T>);
  constexpr int BS = TrsvTile<T>::BS;
  const size_t smem = (size_t)BS * (BS + 1) * sizeof(T);
  cudaError_t e = ensure_dynamic_smem(tk, smem);
  if (e != cudaSuccess) return record_cuda_error(e, name);
  const int nblk = (n + BS - 1) / BS;
  for (int lower = 1; lower >= 0; --lower) {
    e = cudaMemsetAsync(sync, 0, (size_t)(nblk + 2) * sizeof(int), s);
    if (e != cudaSuccess) return record_cuda_error(e, name);
    TrsvArgs<T> ta{n, LU, lda, x, lower, info, sync, poll_limit, lower ? skip_lower_flag : -1};
    trsv_kernel<T><<<nblk, kTrsvThreads, smem, s>>>(ta);
  }
  return check_launch(name);
}

constexpr size_t kStageLimit = 160 * 1024;

template <typename T>
int getrs_one(int n, const T* LU, int64_t lda, const int32_t* ipiv, T* x, int32_t* info, int* sync, cudaStream_t s,
              const char* name, int poll_limit = kTrsvPollLimit, int skip_lower_flag = -1) {
  info_init_kernel<<<1, 1, 0, s>>>(info);
  const size_t stage = (size_t)n * (sizeof(T) + sizeof(int32_t));
  const int staged = stage <= kStageLimit;
  if (staged && stage > 48 * 1024) {
    cudaError_t e = ensure_dynamic_smem(apply_pivots_kernel<T>, kStageLimit);
    if (e != cudaSuccess) return record_cuda_error(e, name);
  }
  apply_pivots_kernel<T><<<1, 256, staged ? stage : 0, s>>>(n, ipiv, x, staged);
  int rc = trsv_pair<T>(n, LU, lda, x, info, sync, s, name, poll_limit, skip_lower_flag);
  if (rc != NACU_SUCCESS) return rc;
  info_finalize_kernel<<<1, 1, 0, s>>>(info);
  return check_launch(name);
}

struct Update64Ctx {
  const int* balance;  // PanelPub's
  void* ws[2];  // scratch of the tensor-core product, one per concurrent update (slot); null: the FP64 kernel
  size_t ws_bytes[2];
};

int update_fp64(int m, int n, int k, const void* L21, const void* U12, void* A22, int64_t lda, void* ctx, int slot,
                cudaStream_t s) {
  const Update64Ctx* c = static_cast<const Update64Ctx*>(ctx);
  const double *a = static_cast<const double*>(L21), *b = static_cast<const double*>(U12);
  double* d = static_cast<double*>(A22);
  if (c && c->ws[slot] && c->ws_bytes[slot] >= crt_gemm_workspace_bytes(m, n, k))
    return crt_gemm_run(m, n, k, -1.0, a, lda, b, lda, 1.0, d, lda, c->ws[slot], c->ws_bytes[slot], s, "nacu_dgetrf",
                        c->balance);
  return nacu_dgemm(m, n, k, -1.0, a, lda, b, lda, 1.0, d, lda, s);
}

constexpr int kNb64 = 64;  // panel width of the FP64 factorization past the register panels

// The FP64 factorization's workspace: the panel's exchange area, then the
// scratch of the two concurrent updates.
struct Getrf64Layout {
  size_t slot[2], bytes[2], total;
};
Getrf64Layout getrf64_layout(int n) {
  Getrf64Layout L;
  // either panel width: the device decides between them
  const int nb = kPanelMaxNb;
  L.bytes[0] = crt_gemm_workspace_bytes(n, nb, nb);
  L.bytes[1] = crt_gemm_workspace_bytes(n, n, nb);
  L.slot[0] = getrf_ws_bytes();
  L.slot[1] = L.slot[0] + L.bytes[0];
  L.total = L.slot[1] + L.bytes[1];
  return L;
}

// ---------------------------------------------------------------------------
// mixed precision: FP32 factor (tensor-core trailing updates), FP64 refinement
// ---------------------------------------------------------------------------
struct Update32Ctx {
  void* ws[2];  // one split-GEMM workspace per concurrent update (slot)
  size_t ws_bytes[2];
};

int update_fp32_split(int m, int n, int k, const void* L21, const void* U12, void* A22, int64_t lda, void* ctx,
                      int slot, cudaStream_t s) {
  const Update32Ctx* c = static_cast<const Update32Ctx*>(ctx);
  return split_gemm_run<float, float>(m, n, k, -1.0, static_cast<const float*>(L21), lda,
                                      static_cast<const float*>(U12), lda, 1.0, static_cast<float*>(A22), lda, 3,
                                      c->ws[slot], c->ws_bytes[slot], s);
}

__global__ void to_fp32_kernel(int n, const double* __restrict__ A, int64_t lda, float* __restrict__ A32) {
  const int64_t total = (int64_t)n * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = e / n, r = e - c * n;
    A32[e] = (float)A[c * lda + r];
  }
}

__device__ __forceinline__ unsigned long long dabs_bits(double x) { return abs_bits_f64(x); }

// part[cb * n + i] = sum over the column chunk cb of A[i][j] * x[j] (or |A[i][j]| when abs_mode).
constexpr int kGemvChunks = 16;
__global__ void gemv_partial_kernel(int n, const double* __restrict__ A, int64_t lda, const double* __restrict__ x,
                                    double* __restrict__ part, int abs_mode) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int chunk = (n + kGemvChunks - 1) / kGemvChunks;
  const int j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
  double acc = 0.0;
  int j = j0;
  for (; j + 4 <= j1; j += 4) {
    const double a0 = A[(size_t)j * lda + i], a1 = A[(size_t)(j + 1) * lda + i];
    const double a2 = A[(size_t)(j + 2) * lda + i], a3 = A[(size_t)(j + 3) * lda + i];
    if (abs_mode) acc += fabs(a0) + fabs(a1) + fabs(a2) + fabs(a3);
    else acc = fma(a3, x[j + 3], fma(a2, x[j + 2], fma(a1, x[j + 1], fma(a0, x[j], acc))));
  }
  for (; j < j1; ++j) acc = abs_mode ? acc + fabs(A[(size_t)j * lda + i]) : fma(A[(size_t)j * lda + i], x[j], acc);
  part[(size_t)blockIdx.y * n + i] = acc;
}

// r = b - sum(part) (or the row sums when abs_mode); norms (max |.|, as bits) of
// r, x and b into nrm[0..2] (atomicMax on non-negative doubles' bit images).
__global__ void residual_finish_kernel(int n, const double* __restrict__ b, const double* __restrict__ x,
                                       const double* __restrict__ part, double* __restrict__ r,
                                       unsigned long long* nrm, int abs_mode) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long rn = 0, xn = 0, bn = 0;
  if (i < n) {
    double s = 0.0;
    for (int cb = 0; cb < kGemvChunks; ++cb) s += part[(size_t)cb * n + i];
    const double v = abs_mode ? s : b[i] - s;
    if (!abs_mode) r[i] = v;
    rn = dabs_bits(v);
    xn = dabs_bits(x[i]);
    bn = dabs_bits(b[i]);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    rn = max(rn, __shfl_xor_sync(0xffffffffu, rn, off));
    xn = max(xn, __shfl_xor_sync(0xffffffffu, xn, off));
    bn = max(bn, __shfl_xor_sync(0xffffffffu, bn, off));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&nrm[0], rn);
    atomicMax(&nrm[1], xn);
    atomicMax(&nrm[2], bn);
  }
}

// d32 = (float)(P src * 2^-e): the row permutation of the factor fused as a gather
__global__ void scale_to_fp32_kernel(int n, const double* __restrict__ src, const int32_t* __restrict__ perm, int e,
                                     float* __restrict__ d32) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d32[i] = (float)(src[perm[i]] * __longlong_as_double((long long)(1023 - e) << 52));
}
// x += (double)d32 * 2^e; max |d| into nrm[3]
__global__ void accumulate_kernel(int n, const float* __restrict__ d32, int e, double* __restrict__ x,
                                  unsigned long long* nrm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long dn = 0;
  if (i < n) {
    const double d = (double)d32[i] * __longlong_as_double((long long)(1023 + e) << 52);
    x[i] += d;
    dn = dabs_bits(d);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) dn = max(dn, __shfl_xor_sync(0xffffffffu, dn, off));
  if ((threadIdx.x & 31) == 0) atomicMax(&nrm[3], dn);
}

// ---- GMRES refinement (Carson & Higham 2018, "Accelerating the solution of
// linear systems by iterative refinement in three precisions", GMRES-IR) ----
// When u32 * cond(A) approaches 1 the FP32 correction (LU)^-1 r no longer
// contracts and classical refinement stalls.  GMRES-IR keeps the FP32 factors
// as a preconditioner instead: each outer step solves the correction equation
// M^-1 A d = M^-1 r (M = P^T L U, FP32) by restarted GMRES with FP64 vectors --
// the product A v in FP64, the preconditioner applied with the FP32 triangular
// solves (the vector scaled by a power of two into FP32 and back) -- and then
// forms the new FP64 residual.  The preconditioner is applied in FP64 with the
// FP32 factors promoted exactly to FP64 (applying it in FP32 inflated the
// first correction's error by the FP32 solve's own rounding, ~1e5x at cond
// 1e8 in a CPU study).  The Krylov basis is orthogonalised by
// classical Gram-Schmidt applied twice (one multi-dot and one update kernel
// per pass), the small Hessenberg least-squares problem is solved on the host
// with Givens rotations.
// When classical refinement diverges outright (the correction grows by more
// than kGmresMaxRho per step, u32 * cond well above 1), the FP32 preconditioner
// is too weak for GMRES to pay: measured at n = 4096, 100 GMRES iterations
// reduced the preconditioned residual only to 6e-2 at cond 1e8 (ratio 68)
// and 3e7 (ratio 15), against 29 iterations at cond 1e7 (ratio 1.4).  Those
// systems go to the FP64 refactorization at once, and so does a GMRES cycle
// that ends above kGmresGiveUp.
constexpr int kGmresM = 64;           // restart length (basis vectors)
constexpr double kGmresTol = 1e-6;    // relative reduction of the preconditioned residual per outer step
constexpr int kGmresOuter = 8;        // outer steps (FP64 residuals) before the FP64 fallback
constexpr double kGmresMaxRho = 2.5;  // correction growth per classical step above which GMRES is skipped
constexpr double kGmresGiveUp = 1e-2; // relative residual after a full cycle above which GMRES is abandoned

// y = sum of the GEMV partials; max |y| (bits) into *nrm
__global__ void gemv_finish_kernel(int n, const double* __restrict__ part, double* __restrict__ y,
                                   unsigned long long* nrm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long yn = 0;
  if (i < n) {
    double acc = 0.0;
    for (int cb = 0; cb < kGemvChunks; ++cb) acc += part[(size_t)cb * n + i];
    y[i] = acc;
    yn = abs_bits_f64(acc);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) yn = max(yn, __shfl_xor_sync(0xffffffffu, yn, off));
  if ((threadIdx.x & 31) == 0) atomicMax(nrm, yn);
}
// out[c] = V[:, c] . w for c < cols (one block per column, fixed reduction order)
__global__ void __launch_bounds__(256) block_dots_kernel(int n, const double* __restrict__ V, int64_t ldv,
                                                         const double* __restrict__ w, double* __restrict__ out) {
  __shared__ double red[8];
  const double* v = V + (size_t)blockIdx.x * ldv;
  double acc = 0.0;
  for (int t = threadIdx.x; t < n; t += 256) acc = fma(v[t], w[t], acc);
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int k = 0; k < 8; ++k) sum += red[k];
    out[blockIdx.x] = sum;
  }
}
// w += sign * V[:, 0..cols) h
__global__ void combo_kernel(int n, const double* __restrict__ V, int64_t ldv, int cols, const double* __restrict__ h,
                             double sign, double* __restrict__ w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double acc = 0.0;
  for (int c = 0; c < cols; ++c) acc = fma(V[(size_t)c * ldv + t], h[c], acc);
  w[t] = fma(sign, acc, w[t]);
}
// dst = P src (the factors' row permutation as a gather)
__global__ void permute_kernel(int n, const double* __restrict__ src, const int32_t* __restrict__ perm,
                               double* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[perm[i]];
}
// A64 = (double)A32, exact
__global__ void to_fp64_kernel(int64_t total, const float* __restrict__ A32, double* __restrict__ A64) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x)
    A64[e] = (double)A32[e];
}
// v = w * s
__global__ void scale_kernel(int n, const double* __restrict__ w, double s, double* __restrict__ v) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) v[t] = w[t] * s;
}

struct MixedLuLayout {
  size_t a32, ipiv, perm, info, cand, split, split2, r, d32, part, nrm, a64, vk, wv, yv, hv, total;
};
inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }
MixedLuLayout mixed_lu_layout(int n, int nb) {
  MixedLuLayout L;
  size_t o = 0;
  // the FP64 fallback's updates keep their residues where the FP32 factor was
  const Getrf64Layout F = getrf64_layout(n);
  L.a32 = o;   o = up256(o + std::max((size_t)n * n * 4, F.bytes[0] + F.bytes[1]));
  L.ipiv = o;  o = up256(o + (size_t)n * 4);
  L.perm = o;  o = up256(o + (size_t)n * 4);
  L.info = o;  o = up256(o + 16);
  L.cand = o;  o = up256(o + getrf_ws_bytes());
  o = (o + 1023) & ~(size_t)1023;
  L.split = o; o = up256(o + nacu_gemm_split_workspace_bytes(n, n, nb));
  o = (o + 1023) & ~(size_t)1023;
  L.split2 = o; o = up256(o + nacu_gemm_split_workspace_bytes(n, nb, nb));
  L.r = o;     o = up256(o + (size_t)n * 8);
  L.d32 = o;   o = up256(o + (size_t)n * 4);
  L.part = o;  o = up256(o + (size_t)kGemvChunks * n * 8);
  L.nrm = o;   o = up256(o + 8 * 8);
  L.a64 = o;   o = up256(o + (size_t)n * n * 8);
  L.vk = o;    o = up256(o + (size_t)n * (kGmresM + 1) * 8);  // GMRES basis
  L.wv = o;    o = up256(o + (size_t)n * 8);
  L.yv = o;    o = up256(o + (size_t)n * 8);
  L.hv = o;    o = up256(o + (size_t)(2 * kGmresM + 4) * 8);  // two Gram-Schmidt passes' coefficients
  L.total = o + 1024;  // the caller's base may need aligning to 1024
  return L;
}

int exp_of_bits(unsigned long long b) {
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex == 0 || ex == 0x7ff) return 0;
  const int e = ex - 1023;
  return e < -1000 ? -1000 : (e > 1000 ? 1000 : e);
}

// The buffers of one GMRES correction solve.
struct GmresBufs {
  int n;
  const double* A;
  int64_t lda;
  const double* LU;       // the FP32 LU factors promoted to FP64 (packed, lda = n)
  const int32_t* perm;    // row permutation of the factors as a gather
  int32_t* info;          // trsv info slot
  void* trsv_sync;
  double* part;
  unsigned long long* nrm;  // [4]: max |y| of the last product
  double *V, *w, *y, *h;
};

// z = M^-1 src (M = P^T L U, the FP32 factors applied in FP64).
int gmres_precond(const GmresBufs& g, const double* src, double* z, cudaStream_t s) {
  const int nblk = (g.n + 255) / 256;
  permute_kernel<<<nblk, 256, 0, s>>>(g.n, src, g.perm, z);
  int rc = trsv_pair<double>(g.n, g.LU, g.n, z, g.info, static_cast<int*>(g.trsv_sync), s,
                             "nacu_dgesv_mixed_ir: gmres");
  if (rc != NACU_SUCCESS) return rc;
  return check_launch("nacu_dgesv_mixed_ir: gmres");
}

// d = approximate solution of M^-1 A d = M^-1 r by GMRES(kGmresM) from d = 0,
// the preconditioned residual reduced by kGmresTol (or the basis exhausted);
// d is added to x.  *inner counts the basis vectors used.
int gmres_correction(const GmresBufs& g, const double* r, double* x, int* inner, double* rel, cudaStream_t s) {
  const int n = g.n, nblk = (n + 255) / 256;
  double* V = g.V;
  // v0 = M^-1 r / ||M^-1 r||
  int rc = gmres_precond(g, r, g.w, s);
  if (rc != NACU_SUCCESS) return rc;
  block_dots_kernel<<<1, 256, 0, s>>>(n, g.w, n, g.w, g.h);
  double hb[kGmresM + 2];
  cudaMemcpyAsync(hb, g.h, 8, cudaMemcpyDeviceToHost, s);
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir: gmres");
  const double beta = std::sqrt(hb[0]);
  *inner = 0;
  *rel = 0.0;
  if (!(beta > 0.0) || !std::isfinite(beta)) return NACU_SUCCESS;
  scale_kernel<<<nblk, 256, 0, s>>>(n, g.w, 1.0 / beta, V);
  static thread_local double H[kGmresM + 1][kGmresM];  // column j: H[0..j+1][j]
  double cs[kGmresM], sn[kGmresM], gv[kGmresM + 1];
  for (int i = 0; i <= kGmresM; ++i) gv[i] = 0.0;
  gv[0] = beta;
  int k = 0;
  for (int j = 0; j < kGmresM; ++j) {
    // w = M^-1 A v_j
    cudaMemsetAsync(g.nrm + 4, 0, 8, s);
    gemv_partial_kernel<<<dim3(nblk, kGemvChunks), 256, 0, s>>>(n, g.A, g.lda, V + (size_t)j * n, g.part, 0);
    gemv_finish_kernel<<<nblk, 256, 0, s>>>(n, g.part, g.y, g.nrm + 4);
    rc = gmres_precond(g, g.y, g.w, s);
    if (rc != NACU_SUCCESS) return rc;
    // classical Gram-Schmidt, twice: h = V^T w, w -= V h
    block_dots_kernel<<<j + 1, 256, 0, s>>>(n, V, n, g.w, g.h);
    combo_kernel<<<nblk, 256, 0, s>>>(n, V, n, j + 1, g.h, -1.0, g.w);
    double* h2d = g.h + kGmresM + 2;
    block_dots_kernel<<<j + 1, 256, 0, s>>>(n, V, n, g.w, h2d);
    combo_kernel<<<nblk, 256, 0, s>>>(n, V, n, j + 1, h2d, -1.0, g.w);
    block_dots_kernel<<<1, 256, 0, s>>>(n, g.w, n, g.w, g.y);  // ||w||^2 (y is free here)
    double h1[kGmresM + 1], h2[kGmresM + 1], hn2 = 0.0;
    cudaMemcpyAsync(h1, g.h, (size_t)(j + 1) * 8, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h2, h2d, (size_t)(j + 1) * 8, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&hn2, g.y, 8, cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir: gmres");
    const double hn = std::sqrt(hn2);
    for (int i = 0; i <= j; ++i) H[i][j] = h1[i] + h2[i];
    H[j + 1][j] = hn;
    // previous rotations, then the one that zeroes H[j+1][j]
    for (int i = 0; i < j; ++i) {
      const double t = cs[i] * H[i][j] + sn[i] * H[i + 1][j];
      H[i + 1][j] = -sn[i] * H[i][j] + cs[i] * H[i + 1][j];
      H[i][j] = t;
    }
    const double den = std::hypot(H[j][j], H[j + 1][j]);
    cs[j] = den > 0.0 ? H[j][j] / den : 1.0;
    sn[j] = den > 0.0 ? H[j + 1][j] / den : 0.0;
    H[j][j] = den;
    H[j + 1][j] = 0.0;
    gv[j + 1] = -sn[j] * gv[j];
    gv[j] = cs[j] * gv[j];
    k = j + 1;
    if (!std::isfinite(gv[j + 1]) || std::fabs(gv[j + 1]) <= kGmresTol * beta || !(hn > 0.0)) break;
    if (j + 1 < kGmresM) scale_kernel<<<nblk, 256, 0, s>>>(n, g.w, 1.0 / hn, V + (size_t)(j + 1) * n);
  }
  // y = H^-1 g (upper triangular k x k), then x += V y
  double yk[kGmresM];
  for (int i = k - 1; i >= 0; --i) {
    double acc = gv[i];
    for (int c = i + 1; c < k; ++c) acc -= H[i][c] * yk[c];
    yk[i] = (H[i][i] != 0.0) ? acc / H[i][i] : 0.0;
  }
  cudaMemcpyAsync(g.h, yk, (size_t)k * 8, cudaMemcpyHostToDevice, s);
  combo_kernel<<<nblk, 256, 0, s>>>(n, V, n, k, g.h, 1.0, x);
  e = cudaStreamSynchronize(s);  // yk lives on the host stack
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir: gmres");
  *inner = k;
  *rel = (k > 0) ? std::fabs(gv[k]) / beta : 1.0;
  return check_launch("nacu_dgesv_mixed_ir: gmres");
}

int getrf_run(int n, double* A, int64_t lda, int32_t* ipiv, int32_t* info, void* workspace, size_t workspace_bytes,
              cudaStream_t stream, int poll_limit, const char* name) {
  if (n < 0) return record_arg_error(-1, "dgetrf: n < 0");
  if (n == 0) return NACU_SUCCESS;
  if (!A) return record_arg_error(-2, "dgetrf: null A");
  if (lda < n) return record_arg_error(-3, "dgetrf: lda < n");
  if (!ipiv || !info) return record_arg_error(-4, "dgetrf: null ipiv or info");
  if (!workspace || workspace_bytes < getrf_ws_bytes()) return record_arg_error(-6, "dgetrf: workspace too small");
  const Getrf64Layout L = getrf64_layout(n);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  Update64Ctx ctx{reinterpret_cast<PanelPub<double>*>(workspace)->balance,
                  {ws + L.slot[0], ws + L.slot[1]},
                  {L.bytes[0], L.bytes[1]}};
  if (workspace_bytes < L.total) ctx.ws[0] = ctx.ws[1] = nullptr;  // the updates on the FP64 pipe
  return getrf_blocked<double>(n, A, lda, ipiv, info, workspace, kNb64, update_fp64, &ctx, stream, name, poll_limit);
}

}  // namespace nacu

extern "C" {

size_t nacu_gesv_mixed_workspace_bytes(int n) { return nacu::mixed_lu_layout(n, 128).total; }

int nacu_dgesv_mixed_ir(int n, const double* A, int64_t lda, const double* b, double* x, double tol_units,
                        int max_iter, int* iters_out, double* berr_out, int* fallback_out, void* workspace,
                        size_t workspace_bytes, nacu_stream_t stream) {
  using namespace nacu;
  if (n < 0) return record_arg_error(-1, "dgesv_mixed_ir: n < 0");
  if (n == 0) return NACU_SUCCESS;
  if (!A || lda < n) return record_arg_error(-2, "dgesv_mixed_ir: bad A / lda");
  if (!b || !x) return record_arg_error(-4, "dgesv_mixed_ir: null b or x");
  const int nb = 128;
  MixedLuLayout L = mixed_lu_layout(n, nb);
  if (!workspace || workspace_bytes < L.total) return record_arg_error(-11, "dgesv_mixed_ir: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)workspace + 1023) & ~(uintptr_t)1023);
  float* A32 = reinterpret_cast<float*>(base + L.a32);
  int32_t* ipiv = reinterpret_cast<int32_t*>(base + L.ipiv);
  int32_t* perm = reinterpret_cast<int32_t*>(base + L.perm);
  int32_t* info = reinterpret_cast<int32_t*>(base + L.info);
  void* cand = base + L.cand;
  void* split_ws = base + L.split;
  double* r = reinterpret_cast<double*>(base + L.r);
  float* d32 = reinterpret_cast<float*>(base + L.d32);
  double* part = reinterpret_cast<double*>(base + L.part);
  unsigned long long* nrm = reinterpret_cast<unsigned long long*>(base + L.nrm);
  double* A64 = reinterpret_cast<double*>(base + L.a64);
  const double tol = (tol_units > 0 ? tol_units : 1.0) * n * 2.220446049250313e-16;
  if (max_iter <= 0) max_iter = 30;
  const int nblk = (n + 255) / 256;
  int iters = 0, fallback = 0;
  double berr = INFINITY;
  unsigned long long h[4];
  // ||A||_inf (FP64 row sums of |A|)
  cudaMemsetAsync(nrm, 0, 64, s);
  gemv_partial_kernel<<<dim3(nblk, kGemvChunks), 256, 0, s>>>(n, A, lda, x, part, 1);
  residual_finish_kernel<<<nblk, 256, 0, s>>>(n, b, b, part, r, nrm, 1);
  cudaMemcpyAsync(h, nrm, 32, cudaMemcpyDeviceToHost, s);
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir");
  const double anorm = __builtin_bit_cast(double, h[0]);
  const double bnorm = __builtin_bit_cast(double, h[2]);
  // FP32 factor
  to_fp32_kernel<<<sm_count() * 8, 256, 0, s>>>(n, A, lda, A32);
  Update32Ctx uctx{{base + L.split2, split_ws},
                   {nacu_gemm_split_workspace_bytes(n, nb, nb), nacu_gemm_split_workspace_bytes(n, n, nb)}};
  int rc = getrf_blocked<float>(n, A32, n, ipiv, info, cand, nb, update_fp32_split, &uctx, s, "nacu_dgesv_mixed_ir");
  if (rc != NACU_SUCCESS) return rc;
  int32_t hinfo = 0;
  cudaMemcpyAsync(&hinfo, info, 4, cudaMemcpyDeviceToHost, s);
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir");
  bool converged = false;
  double last_rho = INFINITY;  // growth of the correction over the last classical step
  if (hinfo == 0) {
    const int staged = (size_t)n * 8 <= kStageLimit;
    if (staged && (size_t)n * 8 > 48 * 1024) {
      e = ensure_dynamic_smem(pivots_to_perm_kernel, kStageLimit);
      if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir");
    }
    pivots_to_perm_kernel<<<1, 256, staged ? (size_t)n * 8 : 0, s>>>(n, ipiv, perm, staged);
    // refinement: x0 = 0, r0 = b
    cudaMemsetAsync(x, 0, (size_t)n * 8, s);
    cudaMemcpyAsync(r, b, (size_t)n * 8, cudaMemcpyDeviceToDevice, s);
    double rnorm = bnorm, dprev = 0.0;
    last_rho = 0.0;
    for (int it = 0; it < max_iter; ++it) {
      // d = (LU)^-1 P r in FP32, scaled by the exponent of ||r||
      int er = 0;
      {
        const double m = rnorm;
        er = (m > 0.0 && std::isfinite(m)) ? exp_of_bits(__builtin_bit_cast(unsigned long long, m)) : 0;
      }
      scale_to_fp32_kernel<<<nblk, 256, 0, s>>>(n, r, perm, er, d32);
      rc = trsv_pair<float>(n, A32, n, d32, info + 1, reinterpret_cast<int*>(cand), s, "nacu_dgesv_mixed_ir");
      if (rc != NACU_SUCCESS) return rc;
      cudaMemsetAsync(nrm, 0, 64, s);
      accumulate_kernel<<<nblk, 256, 0, s>>>(n, d32, er, x, nrm);
      gemv_partial_kernel<<<dim3(nblk, kGemvChunks), 256, 0, s>>>(n, A, lda, x, part, 0);
      residual_finish_kernel<<<nblk, 256, 0, s>>>(n, b, x, part, r, nrm, 0);
      cudaMemcpyAsync(h, nrm, 32, cudaMemcpyDeviceToHost, s);
      e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir");
      ++iters;
      rnorm = __builtin_bit_cast(double, h[0]);
      const double xnorm = __builtin_bit_cast(double, h[1]);
      const double dnorm = __builtin_bit_cast(double, h[3]);
      berr = rnorm / (anorm * xnorm + bnorm);
      if (berr <= tol) {
        converged = true;
        break;
      }
      if (it >= 1 && dprev > 0.0) last_rho = dnorm / dprev;
      if (!std::isfinite(berr)) last_rho = INFINITY;
      if (!std::isfinite(berr) || (it >= 1 && dprev > 0.0 && dnorm > 0.5 * dprev)) break;  // stagnation
      dprev = dnorm;
    }
  }
  if (!converged && hinfo == 0 && last_rho <= kGmresMaxRho) {
    // GMRES-IR with the FP32 factors as the preconditioner, from x = 0
    to_fp64_kernel<<<sm_count() * 8, 256, 0, s>>>((int64_t)n * n, A32, A64);
    GmresBufs gb{n, A, lda, A64, perm, info + 1, cand, part, nrm,
                 reinterpret_cast<double*>(base + L.vk), reinterpret_cast<double*>(base + L.wv),
                 reinterpret_cast<double*>(base + L.yv), reinterpret_cast<double*>(base + L.hv)};
    cudaMemsetAsync(x, 0, (size_t)n * 8, s);
    cudaMemcpyAsync(r, b, (size_t)n * 8, cudaMemcpyDeviceToDevice, s);
    double best = INFINITY;
    for (int outer = 0; outer < kGmresOuter; ++outer) {
      int inner = 0;
      double rel = 1.0;
      rc = gmres_correction(gb, r, x, &inner, &rel, s);
      if (rc != NACU_SUCCESS) return rc;
      if (!(rel <= kGmresGiveUp)) break;  // the preconditioner is too weak: FP64
      cudaMemsetAsync(nrm, 0, 64, s);
      gemv_partial_kernel<<<dim3(nblk, kGemvChunks), 256, 0, s>>>(n, A, lda, x, part, 0);
      residual_finish_kernel<<<nblk, 256, 0, s>>>(n, b, x, part, r, nrm, 0);
      cudaMemcpyAsync(h, nrm, 32, cudaMemcpyDeviceToHost, s);
      e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir");
      ++iters;
      berr = __builtin_bit_cast(double, h[0]) / (anorm * __builtin_bit_cast(double, h[1]) + bnorm);
      if (berr <= tol) {
        converged = true;
        fallback = 2;
        break;
      }
      if (!std::isfinite(berr) || !(berr < 0.5 * best) || inner == 0) break;  // no progress: FP64 fallback
      best = berr;
    }
  }
  if (!converged) {
    // FP64 fallback on a copy of A
    fallback = 1;
    cudaMemcpy2DAsync(A64, (size_t)n * 8, A, (size_t)lda * 8, (size_t)n * 8, n, cudaMemcpyDeviceToDevice, s);
    const Getrf64Layout F = getrf64_layout(n);
    Update64Ctx fctx{reinterpret_cast<PanelPub<double>*>(cand)->balance,
                     {base + L.a32, base + L.a32 + F.bytes[0]},
                     {F.bytes[0], F.bytes[1]}};
    rc = getrf_blocked<double>(n, A64, n, ipiv, info, cand, kNb64, update_fp64, &fctx, s, "nacu_dgesv_mixed_ir");
    if (rc != NACU_SUCCESS) return rc;
    cudaMemcpyAsync(x, b, (size_t)n * 8, cudaMemcpyDeviceToDevice, s);
    rc = nacu_dgetrs(n, A64, n, ipiv, x, info + 1, cand, getrf_ws_bytes(), stream);
    if (rc != NACU_SUCCESS) return rc;
    cudaMemsetAsync(nrm, 0, 64, s);
    gemv_partial_kernel<<<dim3(nblk, kGemvChunks), 256, 0, s>>>(n, A, lda, x, part, 0);
    residual_finish_kernel<<<nblk, 256, 0, s>>>(n, b, x, part, r, nrm, 0);
    cudaMemcpyAsync(h, nrm, 32, cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return record_cuda_error(e, "nacu_dgesv_mixed_ir");
    berr = __builtin_bit_cast(double, h[0]) / (anorm * __builtin_bit_cast(double, h[1]) + bnorm);
  }
  if (iters_out) *iters_out = iters;
  if (berr_out) *berr_out = berr;
  if (fallback_out) *fallback_out = fallback;
  return check_launch("nacu_dgesv_mixed_ir");
}

size_t nacu_getrf_workspace_bytes(int n) {
  return std::max(nacu::getrf64_layout(n < 0 ? 0 : n).total, nacu::trsv_sync_bytes(n < 0 ? 0 : n));
}

int nacu_dgetrf(int n, double* A, int64_t lda, int32_t* ipiv, int32_t* info, void* workspace, size_t workspace_bytes,
                nacu_stream_t stream) {
  return nacu::getrf_run(n, A, lda, ipiv, info, workspace, workspace_bytes, (cudaStream_t)stream, nacu::kRegPollLimit,
                         "nacu_dgetrf");
}

int nacu_test_dgetrf_wait_limit(int n, double* A, int64_t lda, int32_t* ipiv, int32_t* info, int poll_limit,
                                void* workspace, size_t workspace_bytes, nacu_stream_t stream) {
  using namespace nacu;
  if (n < 0) return record_arg_error(-1, "test_dgetrf_wait_limit: n < 0");
  if (poll_limit < 0 || poll_limit > kRegPollLimit)
    return record_arg_error(-6, "test_dgetrf_wait_limit: poll_limit outside [0, 2^20]");
  return getrf_run(n, A, lda, ipiv, info, workspace, workspace_bytes, (cudaStream_t)stream, poll_limit,
                   "nacu_test_dgetrf_wait_limit");
}

int nacu_dgetrs(int n, const double* LU, int64_t lda, const int32_t* ipiv, double* b, int32_t* info, void* workspace,
                size_t workspace_bytes, nacu_stream_t stream) {
  using namespace nacu;
  if (n < 0) return record_arg_error(-1, "dgetrs: n < 0");
  if (n == 0) return NACU_SUCCESS;
  if (!LU || !ipiv || !b || !info) return record_arg_error(-2, "dgetrs: null argument");
  if (lda < n) return record_arg_error(-3, "dgetrs: lda < n");
  if (!workspace || workspace_bytes < nacu::trsv_sync_bytes(n))
    return record_arg_error(-7, "dgetrs: workspace too small");
  return getrs_one<double>(n, LU, lda, ipiv, b, info, static_cast<int*>(workspace), (cudaStream_t)stream,
                           "nacu_dgetrs");
}

int nacu_test_dgetrs_flag_timeout(int n, const double* LU, int64_t lda, const int32_t* ipiv, double* b,
                                  int32_t* info, int skip_block, int poll_limit, void* workspace,
                                  size_t workspace_bytes, nacu_stream_t stream) {
  using namespace nacu;
  if (n <= 0) return record_arg_error(-1, "test_dgetrs_flag_timeout: n <= 0");
  if (!LU || !ipiv || !b || !info) return record_arg_error(-2, "test_dgetrs_flag_timeout: null argument");
  if (lda < n) return record_arg_error(-3, "test_dgetrs_flag_timeout: lda < n");
  const int nblk = (n + TrsvTile<double>::BS - 1) / TrsvTile<double>::BS;
  if (skip_block < 0 || skip_block >= nblk)
    return record_arg_error(-7, "test_dgetrs_flag_timeout: skip_block outside the row blocks");
  if (poll_limit < 1 || poll_limit > kTrsvPollLimit)
    return record_arg_error(-8, "test_dgetrs_flag_timeout: poll_limit outside [1, 2^22]");
  if (!workspace || workspace_bytes < nacu::trsv_sync_bytes(n))
    return record_arg_error(-10, "test_dgetrs_flag_timeout: workspace too small");
  return getrs_one<double>(n, LU, lda, ipiv, b, info, static_cast<int*>(workspace), (cudaStream_t)stream,
                           "nacu_test_dgetrs_flag_timeout", poll_limit, skip_block);
}

}  // extern "C"
