// Plain FP64 GEMM: C = alpha * A * B + beta * C, column-major, the GPU form of
// nalgebra's `Matrix::gemm` (src/base/blas.rs:729-746 -> gemm_uninit,
// src/base/blas_uninit.rs:187-333, which hands Dyn f64 matrices to
// matrixmultiply::dgemm).  As in nalgebra, beta == 0 means C is never read.
//
// Design (GB300): FP64 is bound by the FP64 pipe (~1 TFLOP/s), so the kernel
// only has to keep that pipe fed: 64 x 64 CTA tiles, 256 threads, a 4 x 4
// register tile per thread (16 independent DFMA chains), 16-deep K slices
// staged in shared memory with the next slice prefetched into registers while
// the current one is consumed.  Loads of A (column-major: rows contiguous) and
// B (columns contiguous along K) are coalesced; edges are zero-filled.  It
// reaches 1.25 TFLOP/s, all the pipe has; with scratch, products large enough
// go to the tensor cores instead (nacu_dgemm_ws, gemm_crt.cu).
#include "common.cuh"

namespace nacu {
namespace {

constexpr int kBK = 16, kGemmThreads = 256;

// Tiles of 16 T x 16 T, T x T per thread; the smaller ones for the tiles the modular
// form leaves over, the same sums in the same order.
template <int T>
__global__ void __launch_bounds__(kGemmThreads, T == 4 ? 3 : 4)
    dgemm_kernel(int M, int N, int K, double alpha, const double* __restrict__ A, int64_t lda,
                 const double* __restrict__ B, int64_t ldb, double beta, double* __restrict__ C, int64_t ldc,
                 const int* __restrict__ tile_flags, int flag_ld) {
  constexpr int kTile = 16 * T, kPerFlag = 128 / kTile;
  // with flags, only the 128 x 128 tiles the modular form (gemm_crt.cu) left to this kernel
  if (tile_flags && !tile_flags[(blockIdx.y / kPerFlag) * flag_ld + blockIdx.x / kPerFlag]) return;
  __shared__ __align__(16) double As[2][kBK][kTile];
  __shared__ __align__(16) double Bs[2][kBK][kTile + 2];  // +2: conflict-free column writes
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * kTile, n0 = blockIdx.y * kTile;
  // loader mapping: A slice (16 T x 16): T elements per thread, rows contiguous
  constexpr int kStep = kGemmThreads / kTile;
  const int ar = tid % kTile, ak = tid / kTile;  // rows ar, k = ak + kStep*u
  // B slice (16 x 16 T): k contiguous within a column
  const int bk = tid & 15, bc = tid >> 4;   // k = bk, columns bc + 16*u
  double ra[T], rb[T];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < T; ++u) {
      const int k = k0 + ak + kStep * u, r = m0 + ar;
      ra[u] = (r < M && k < K) ? A[(size_t)k * lda + r] : 0.0;
      const int c = n0 + bc + 16 * u, kb = k0 + bk;
      rb[u] = (c < N && kb < K) ? B[(size_t)c * ldb + kb] : 0.0;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int u = 0; u < T; ++u) {
      As[buf][ak + kStep * u][ar] = ra[u];
      Bs[buf][bk][bc + 16 * u] = rb[u];
    }
  };
  double acc[T][T];
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) acc[i][j] = 0.0;
  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += kBK) {
    const bool more = k0 + kBK < K;
    if (more) load(k0 + kBK);  // prefetch the next slice into registers
#pragma unroll
    for (int k = 0; k < kBK; ++k) {
      double a[T], b[T];
      if constexpr (T > 1) {
#pragma unroll
        for (int i = 0; i < T; i += 2) {
          const double2 p = *reinterpret_cast<const double2*>(&As[buf][k][ty * T + i]);
          a[i] = p.x, a[i + 1] = p.y;
        }
      } else {
        a[0] = As[buf][k][ty];
      }
#pragma unroll
      for (int j = 0; j < T; ++j) b[j] = Bs[buf][k][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    if (more) {
      store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
  // epilogue: thread (ty, tx) owns rows m0 + T ty + i, columns n0 + tx + 16j
#pragma unroll
  for (int j = 0; j < T; ++j) {
    const int c = n0 + tx + 16 * j;
    if (c >= N) continue;
#pragma unroll
    for (int i = 0; i < T; ++i) {
      const int r = m0 + ty * T + i;
      if (r >= M) continue;
      double* cp = C + (size_t)c * ldc + r;
      *cp = (beta == 0.0) ? alpha * acc[i][j] : fma(alpha, acc[i][j], beta * *cp);
    }
  }
}

}  // namespace

int dgemm_fp64_run(int m, int n, int k, double alpha, const double* A, int64_t lda, const double* B, int64_t ldb,
                   double beta, double* C, int64_t ldc, const int* tile_flags, int flag_ld, cudaStream_t stream) {
  const auto grid = [&](int t) { return dim3((m + 16 * t - 1) / (16 * t), (n + 16 * t - 1) / (16 * t)); };
  const auto tiles = [&](int t) { return (int64_t)grid(t).x * grid(t).y; };
  if (grid(4).y > 65535) return record_arg_error(-2, "dgemm: n too large for one launch");
  // Left-over tiles have paid for the modular form already; a product too small for
  // its 64 x 64 tiles to fill the chip takes smaller ones, so that diagonal, permutation
  // and banded operands, which leave every tile, come out no later than by this kernel
  // alone.  Whole call in us, this kernel alone, modular form and 64 x 64, and as here:
  // 256^3 266, 298, 68; 64^3 71, 97, 35; 1000 x 777 x 1333 2697, 2817, 2136.  Products
  // that fill the chip pay 2 to 5% (2048^3 14.29 and 14.65 ms), 3000 x 300 x 64 136 and 160.
  const int64_t enough = 4 * sm_count();
  if (tile_flags && tiles(4) < enough && tiles(2) < enough)
    dgemm_kernel<1><<<grid(1), kGemmThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, tile_flags, flag_ld);
  else if (tile_flags && tiles(4) < enough)
    dgemm_kernel<2><<<grid(2), kGemmThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, tile_flags, flag_ld);
  else
    dgemm_kernel<4><<<grid(4), kGemmThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, tile_flags, flag_ld);
  return check_launch("nacu_dgemm");
}

namespace {

int dgemm_args(int m, int n, int k, const double* A, int64_t lda, const double* B, int64_t ldb, const double* C,
               int64_t ldc) {
  if (m < 0) return record_arg_error(-1, "dgemm: m < 0");
  if (n < 0) return record_arg_error(-2, "dgemm: n < 0");
  if (k < 0) return record_arg_error(-3, "dgemm: k < 0");
  if (m == 0 || n == 0) return NACU_SUCCESS;
  if (k > 0 && !A) return record_arg_error(-5, "dgemm: null A");
  if (lda < (m > 1 ? m : 1)) return record_arg_error(-6, "dgemm: lda < max(1, m)");
  if (k > 0 && !B) return record_arg_error(-7, "dgemm: null B");
  if (ldb < (k > 1 ? k : 1)) return record_arg_error(-8, "dgemm: ldb < max(1, k)");
  if (!C) return record_arg_error(-10, "dgemm: null C");
  if (ldc < (m > 1 ? m : 1)) return record_arg_error(-11, "dgemm: ldc < max(1, m)");
  return NACU_SUCCESS;
}

}  // namespace
}  // namespace nacu

extern "C" int nacu_dgemm(int m, int n, int k, double alpha, const double* A, int64_t lda, const double* B,
                          int64_t ldb, double beta, double* C, int64_t ldc, nacu_stream_t stream) {
  using namespace nacu;
  const int rc = dgemm_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != NACU_SUCCESS || m == 0 || n == 0) return rc;
  return dgemm_fp64_run(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, nullptr, 0, (cudaStream_t)stream);
}

extern "C" size_t nacu_dgemm_workspace_bytes(int m, int n, int k) {
  return nacu::crt_gemm_pays(m, n, k) ? nacu::crt_gemm_workspace_bytes(m, n, k) : 0;
}

extern "C" int nacu_dgemm_ws(int m, int n, int k, double alpha, const double* A, int64_t lda, const double* B,
                             int64_t ldb, double beta, double* C, int64_t ldc, void* workspace,
                             size_t workspace_bytes, nacu_stream_t stream) {
  using namespace nacu;
  const int rc = dgemm_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != NACU_SUCCESS || m == 0 || n == 0) return rc;
  const size_t need = nacu_dgemm_workspace_bytes(m, n, k);
  if (need == 0)
    return dgemm_fp64_run(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, nullptr, 0, (cudaStream_t)stream);
  if (!workspace || workspace_bytes < need)
    return record_arg_error(-13, "dgemm_ws: workspace smaller than nacu_dgemm_workspace_bytes (argument 13)");
  return crt_gemm_run(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, workspace, workspace_bytes, (cudaStream_t)stream,
                      "nacu_dgemm_ws");
}
