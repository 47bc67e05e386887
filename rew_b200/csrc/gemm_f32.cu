// f32 matmul for the f32 parity path: C[M,N] = A[M,K] @ B[K,N] (+ bias[N]),
// the math of dotGeneral/matmul (src/rew/ops/linalg.nim:204-252) followed by
// Linear's bias add (src/rew/nn/linear.nim:43-49).  Plain FMA on CUDA cores, f32 accumulation: 64x64 tiles
// for large steps, rows against a strip of columns for small ones.
#include "common.cuh"
#include "ptx.cuh"

namespace rewb {
namespace {

constexpr int TM = 64, TN = 64, TK = 16;

__global__ void __launch_bounds__(256) gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                        const float* __restrict__ bias, float* __restrict__ C,
                                                        int64_t M, int64_t K, int64_t N, int64_t lda, int64_t ldb, int64_t ldc) {
  __shared__ float As[TK][TM + 1];
  __shared__ float Bs[TK][TN];
  pdl_launch_dependents();
  pdl_wait();
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int64_t m0 = (int64_t)blockIdx.y * TM, n0 = (int64_t)blockIdx.x * TN;
  float acc[4][4] = {};
  for (int64_t k0 = 0; k0 < K; k0 += TK) {
    for (int i = threadIdx.x; i < TM * TK; i += 256) {
      const int r = i / TK, c = i % TK;
      const int64_t gm = m0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? A[gm * lda + gk] : 0.f;
    }
    for (int i = threadIdx.x; i < TK * TN; i += 256) {
      const int r = i / TN, c = i % TN;
      const int64_t gk = k0 + r, gn = n0 + c;
      Bs[r][c] = (gk < K && gn < N) ? B[gk * ldb + gn] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t gn = n0 + tx * 4 + j;
      if (gn < N) C[gm * ldc + gn] = acc[i][j] + (bias ? bias[gn] : 0.f);
    }
  }
}

// Few rows: a launch is a latency chain (or a stream of B), not a contraction.  A CTA takes MR rows and a strip of COLS
// columns; its 256 threads are COLS columns x KL = 256 / COLS places along K, so that a strip 256 deep is in flight at once
// where the 64x64 tile walks K sixteen at a time behind two barriers.  The rows of A are staged KC at a time and read four
// k at a time by broadcast.  Partial sums meet in shared memory and are added pairwise in a fixed order, which also leaves
// less rounding than one long chain (2048 deep: 1.6e-7 relative against 8e-7 of the tiles).  The order is that of the strip's
// width, 8 or 32 columns, and so follows the rows of the call.  256 x 384, 1 row: 2.9 us (91 us in 64x64 tiles), 768 x 4128,
// 8 rows: 10.7 us (381 us).
constexpr int KC = 512;

template <int MR, int COLS>
__global__ void __launch_bounds__(256) gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                             const float* __restrict__ bias, float* __restrict__ C,
                                                             int64_t M, int64_t K, int64_t N, int64_t lda, int64_t ldb, int64_t ldc) {
  constexpr int KL = 256 / COLS;
  constexpr int STAGE = MR * KC, SUMS = MR * 256;
  __shared__ __align__(16) float sm[STAGE > SUMS ? STAGE : SUMS];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, col = tid % COLS, kl = tid / COLS;
  const int64_t n = (int64_t)blockIdx.x * COLS + col, m0 = (int64_t)blockIdx.y * MR;
  const bool live = n < N;
  float acc[MR] = {};
  for (int64_t k0 = 0; k0 < K; k0 += KC) {
    const int kc = (int)min((int64_t)KC, K - k0);
    if (k0 > 0) __syncthreads();
    for (int i = tid; i < MR * KC; i += 256) {
      const int r = i / KC, k = i % KC;
      sm[i] = (k < kc && m0 + r < M) ? A[(m0 + r) * lda + k0 + k] : 0.f;
    }
    __syncthreads();
    const float* b = B + k0 * ldb + n;
#pragma unroll 4
    for (int k = 4 * kl; k < kc; k += 4 * KL) {
      float w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = (live && k + j < kc) ? b[(int64_t)(k + j) * ldb] : 0.f;
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        const float4 x = *reinterpret_cast<const float4*>(sm + r * KC + k);
        acc[r] = fmaf(x.x, w[0], acc[r]);
        acc[r] = fmaf(x.y, w[1], acc[r]);
        acc[r] = fmaf(x.z, w[2], acc[r]);
        acc[r] = fmaf(x.w, w[3], acc[r]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < MR; ++r) sm[(r * KL + kl) * COLS + col] = acc[r];
  __syncthreads();
  for (int i = tid; i < MR * COLS; i += 256) {
    const int r = i / COLS, c = i % COLS;
    const int64_t gn = (int64_t)blockIdx.x * COLS + c;
    if (m0 + r >= M || gn >= N) continue;
    float part[KL / 4];   // four sums side by side, then their sum: a short chain
#pragma unroll
    for (int q = 0; q < KL / 4; ++q) {
      const float* p = sm + (r * KL + 4 * q) * COLS + c;
      part[q] = (p[0] + p[COLS]) + (p[2 * COLS] + p[3 * COLS]);
    }
#pragma unroll
    for (int w = KL / 8; w > 0; w /= 2)
#pragma unroll
      for (int q = 0; q < w; ++q) part[q] += part[q + w];
    C[(m0 + r) * ldc + gn] = part[0] + (bias ? bias[gn] : 0.f);
  }
}

template <int COLS>
int launch_rows(Ctx* c, const float* A, int64_t lda, const float* B, int64_t ldb, const float* bias, float* C, int64_t ldc, int64_t M, int64_t K,
                int64_t N) {
  auto go = [&](auto kernel, int mr) -> int {
    const dim3 grid((unsigned)((N + COLS - 1) / COLS), (unsigned)((M + mr - 1) / mr));
    RB_CUDA(launch_k(kernel, grid, dim3(256), 0, c->stream, c->use_pdl, A, B, bias, C, M, K, N, lda, ldb, ldc));
    ++g_launch_total;
    ++g_route_launches[ROUTE_F32_ROWS];
    return REWB200_OK;
  };
  if (M == 1) return go(gemm_f32_rows_kernel<1, COLS>, 1);
  if (M == 2) return go(gemm_f32_rows_kernel<2, COLS>, 2);
  if (M <= 4) return go(gemm_f32_rows_kernel<4, COLS>, 4);
  if (M <= 8) return go(gemm_f32_rows_kernel<8, COLS>, 8);
  return go(gemm_f32_rows_kernel<16, COLS>, 16);
}

}  // namespace

int gemm_f32_ld_launch(Ctx* c, const float* A, int64_t lda, const float* B, int64_t ldb, const float* bias, float* C, int64_t ldc,
                       int64_t M, int64_t K, int64_t N) {
  if (M == 0 || N == 0) return REWB200_OK;
  // Up to 512 rows, unless 64x64 tiles give every SM eleven or more, which hide one another's barriers: us, rows / tiles,
  // 1024 x 16384: 384 rows (1536 tiles) 855 / 885, 512 rows (2048) 1129 / 1030; 512 rows of 768 x 4128 (520) 232 / 415, of
  // 2048 x 6144 (768) 815 / 1153, of 4096 x 4096 (512) 1216 / 2209, of 64 x 96 (16) 6 / 14.  Above 512 rows 768 x 4128 is even at 1024
  // (444 / 453).
  if (M <= 512 && ((M + TM - 1) / TM) * ((N + TN - 1) / TN) < 11 * (int64_t)c->sm_count) {
    const int64_t groups = (M + 15) / 16, strips = (N + 31) / 32;
    // Narrow strips while one group of rows, or fewer wide strips than two thirds of the SMs, would leave the chip idle:
    // 4096 x 4096, 1 row 57 against 161 us; 2064 x 768, 64 rows 61 against 106 us; 256 x 1376, 33 rows (129 strips) 8.9 against 6.9 us.
    if (groups == 1 || 3 * strips * groups < 2 * (int64_t)c->sm_count) return launch_rows<8>(c, A, lda, B, ldb, bias, C, ldc, M, K, N);
    return launch_rows<32>(c, A, lda, B, ldb, bias, C, ldc, M, K, N);
  }
  dim3 grid((unsigned)((N + TN - 1) / TN), (unsigned)((M + TM - 1) / TM));
  RB_CUDA(launch_k(gemm_f32_kernel, grid, dim3(256), 0, c->stream, c->use_pdl, A, B, bias, C, M, K, N, lda, ldb, ldc));
  ++g_launch_total;
  ++g_route_launches[ROUTE_F32_TILES];
  return REWB200_OK;
}

int gemm_f32_launch(Ctx* c, const float* A, const float* B, const float* bias, float* C, int64_t M, int64_t K,
                    int64_t N) {
  return gemm_f32_ld_launch(c, A, K, B, N, bias, C, N, M, K, N);
}

}  // namespace rewb
