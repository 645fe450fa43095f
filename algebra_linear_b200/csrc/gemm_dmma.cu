// FP64 C -= A B on the FP64 tensor cores (DMMA, mma.sync m8n8k4 .f64) for the
// fused (non bit-exact) forms: the FP64 LU with fused updates and the sparse
// fronts' Schur complements.
//
// CTA tile 64 x 64 or 64 x 32 (four warps in a 2 x 2 grid, three or four CTAs
// per SM), each warp 4 x 4 or 4 x 2 m8n8 accumulators (two doubles per lane
// each); K in chunks of 16 staged in shared memory by cp.async through a
// three-stage ring: 16-byte copies of two consecutive doubles when the
// operands allow, 8-byte copies otherwise (any leading dimension and offset);
// out-of-range elements are zero-filled. The accumulators start as C and each
// MMA subtracts A B, so every partial sum is one fused multiply-add chain into
// C, as the CUDA-core fused kernel does. Bound by the FP64 tensor cores for
// K >= 128 (30.1 of cuBLAS's 35.4 TFLOP/s on a square GEMM), by C's traffic
// beside them for K = 64.
// Shared-memory rows are padded by 4 doubles so that a half-warp's fragment
// loads (4 k-rows x 4 m-columns) fall in 32 distinct banks.
#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "dense.cuh"

namespace alg {
namespace {

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = valid ? 8 : 0;  // src-size 0: fill with zeros
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// Two consecutive doubles; src_bytes 16, 8 (the second is zero-filled) or 0.
__device__ __forceinline__ void cp_async16(double* dst, const double* src, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Tile shape: four warps in a 2 x 2 grid, each warp 8 MI x 8 NJ (MI x NJ m8n8
// accumulators, two doubles per lane each). K in chunks of 16 through a
// three-stage cp.async ring. VEC: 16-byte copies of two consecutive doubles
// (A's rows / B's k entries), when both operands and their leading dimensions
// allow it; 8-byte copies otherwise.
template <int MI, int NJ>
struct DmmaCfg {
  static constexpr int kBM = 16 * MI, kBN = 16 * NJ, kBK = 16, kThreads = 128, kStages = 3;
  static constexpr int kAS = kBM + 4;  // As[k][m] row stride (doubles)
  static constexpr int kBS = kBK + 4;  // Bs[n][k] row stride
  static constexpr int kStage = kBK * kAS + kBN * kBS;
  static constexpr size_t kSmem = sizeof(double) * kStages * kStage;
};

// `ahead`: a CTA also asks L2 for the C tile that its slot takes next (linear
// tile index + ahead), so that DRAM works during the MMAs instead of between
// them.
template <int MI, int NJ, bool VEC>
__global__ void __launch_bounds__(128, NJ == 4 ? 3 : 4)
    dmma_gemm_sub_kernel(int M, int N, int K, const double* __restrict__ A, int lda, const double* __restrict__ B,
                         int ldb, double* __restrict__ C, int ldc, int ahead) {
  using Cfg = DmmaCfg<MI, NJ>;
  constexpr int kBM = Cfg::kBM, kBN = Cfg::kBN, kBK = Cfg::kBK, kThreads = Cfg::kThreads, STAGES = Cfg::kStages;
  constexpr int kAS = Cfg::kAS, kBS = Cfg::kBS, kStage = Cfg::kStage;
  extern __shared__ __align__(16) double smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp & 1) * (kBM / 2), wn = (warp >> 1) * (kBN / 2);
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;

  auto load_stage = [&](int stage, int k0) {
    double* As = smem + stage * kStage;
    double* Bs = As + kBK * kAS;
    if constexpr (VEC) {
#pragma unroll
      for (int r = 0; r < (kBM * kBK) / (2 * kThreads); ++r) {
        const int e = tid + r * kThreads;
        const int mm = 2 * (e % (kBM / 2)), kk = e / (kBM / 2);
        const int gm = m0 + mm, gk = k0 + kk;
        const int bytes = (gk < K && gm < M) ? (gm + 1 < M ? 16 : 8) : 0;
        cp_async16(As + kk * kAS + mm, bytes ? A + (size_t)gm + (size_t)gk * lda : A, bytes);
      }
#pragma unroll
      for (int r = 0; r < (kBN * kBK) / (2 * kThreads); ++r) {
        const int e = tid + r * kThreads;
        const int kk = 2 * (e % (kBK / 2)), nn = e / (kBK / 2);
        const int gn = n0 + nn, gk = k0 + kk;
        const int bytes = (gn < N && gk < K) ? (gk + 1 < K ? 16 : 8) : 0;
        cp_async16(Bs + nn * kBS + kk, bytes ? B + (size_t)gk + (size_t)gn * ldb : B, bytes);
      }
    } else {
#pragma unroll
      for (int r = 0; r < (kBM * kBK) / kThreads; ++r) {
        const int e = tid + r * kThreads;
        const int mm = e % kBM, kk = e / kBM;
        const int gm = m0 + mm, gk = k0 + kk;
        const bool ok = gm < M && gk < K;
        cp_async8(As + kk * kAS + mm, ok ? A + (size_t)gm + (size_t)gk * lda : A, ok);
      }
#pragma unroll
      for (int r = 0; r < (kBN * kBK) / kThreads; ++r) {
        const int e = tid + r * kThreads;
        const int kk = e % kBK, nn = e / kBK;
        const int gn = n0 + nn, gk = k0 + kk;
        const bool ok = gn < N && gk < K;
        cp_async8(Bs + nn * kBS + kk, ok ? B + (size_t)gk + (size_t)gn * ldb : B, ok);
      }
    }
  };

  const int nch = (K + kBK - 1) / kBK;
  // the ring fills while the accumulators load C
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < nch) load_stage(st, st * kBK);
    cp_async_commit();
  }

  // accumulators = C (fragment layout: row g, columns 2t and 2t + 1 of each
  // m8n8 tile); B's fragments are negated, so no instruction waits for a C
  // entry before the first MMA that takes it
  double acc[MI][NJ][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gm = m0 + wm + i * 8 + g, gn = n0 + wn + j * 8 + 2 * t + h;
        acc[i][j][h] = (gm < M && gn < N) ? C[(size_t)gm + (size_t)gn * ldc] : 0.0;
      }
  {
    const int nxt = (int)(blockIdx.x + blockIdx.y * gridDim.x) + ahead;
    if (nxt < (int)(gridDim.x * gridDim.y)) {
      const int pm = (nxt % (int)gridDim.x) * kBM, pn = (nxt / (int)gridDim.x) * kBN;
#pragma unroll
      for (int e = tid; e < kBN * (kBM / 16); e += kThreads) {  // a 128-byte line each
        const int r = pm + 16 * (e % (kBM / 16)), c = pn + e / (kBM / 16);
        if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (size_t)r + (size_t)c * ldc));
      }
    }
  }

  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<STAGES - 2>();  // chunk ch has landed
    __syncthreads();              // ... for every thread; the slot refilled below is free
    const int nx = ch + STAGES - 1;
    if (nx < nch) load_stage(nx % STAGES, nx * kBK);
    cp_async_commit();
    const double* As = smem + (ch % STAGES) * kStage;
    const double* Bs = As + kBK * kAS;
#pragma unroll
    for (int k4 = 0; k4 < kBK; k4 += 4) {
      double af[MI], bf[NJ];
#pragma unroll
      for (int i = 0; i < MI; ++i) af[i] = As[(k4 + t) * kAS + wm + i * 8 + g];
#pragma unroll
      for (int j = 0; j < NJ; ++j) bf[j] = -Bs[(wn + j * 8 + g) * kBS + k4 + t];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
    }
  }
  cp_async_wait<0>();

#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gm = m0 + wm + i * 8 + g, gn = n0 + wn + j * 8 + 2 * t + h;
        if (gm < M && gn < N) C[(size_t)gm + (size_t)gn * ldc] = acc[i][j][h];
      }
}

template <int MI, int NJ, bool VEC>
int launch_dmma(alg_ctx* ctx, int M, int N, int K, const double* A, int lda, const double* B, int ldb, double* C,
                int ldc) {
  using Cfg = DmmaCfg<MI, NJ>;
  static PerDevice configured;
  ALG_CUDA_TRY(once_per_device(configured, [] {
    return cudaFuncSetAttribute(dmma_gemm_sub_kernel<MI, NJ, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)Cfg::kSmem);
  }));
  dim3 grid((M + Cfg::kBM - 1) / Cfg::kBM, (N + Cfg::kBN - 1) / Cfg::kBN);
  dmma_gemm_sub_kernel<MI, NJ, VEC><<<grid, Cfg::kThreads, Cfg::kSmem, ctx->stream>>>(
      M, N, K, A, lda, B, ldb, C, ldc, (NJ == 4 ? 3 : 4) * ctx->sm_count);
  return ALG_OK;
}

}  // namespace

// 64 x 64 tiles, three CTAs per SM (one tile's C load and store overlap the
// others' MMAs); 64 x 32 tiles, four per SM, while there are few tiles: the
// last wave is shorter and a tile's own latency, which the look-ahead chain's
// narrow updates wait for, is halved. 16-byte copies when A, B are 16-byte
// aligned with even leading dimensions. Measured (M x N x K, us; 128 x 64
// tiles two to an SM before, 64 x 32, 64 x 64):
//   8192 x 8192 x 128    642   600   570  (cuBLAS's C - A B: 577)
//   4096 x 4096 x 64     106    92    91
//   2000 x 2000 x 64      30    25    25
//   1000 x 1000 x 64      10.5   8.5   8.8
//   16000 x 128 x 128     26    23    26
//   3000 x 64 x 64        10.2   4.0   5.9
constexpr long long kNarrowTiles = 1024;  // 64 x 64 tiles

int gemm_dmma_sub_dev(alg_ctx* ctx, int M, int N, int K, const double* A, int lda, const double* B, int ldb,
                      double* C, int ldc) {
  if (M <= 0 || N <= 0 || K <= 0) return ALG_OK;
  const bool vec = ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0 &&
                   (lda % 2) == 0 && (ldb % 2) == 0;
  const int tok = prof_begin(ctx, ALG_K_GEMM);
  int rc;
  const long long tiles = (long long)((M + 63) / 64) * ((N + 63) / 64);
  if (tiles <= kNarrowTiles) {
    rc = vec ? launch_dmma<4, 2, true>(ctx, M, N, K, A, lda, B, ldb, C, ldc)
             : launch_dmma<4, 2, false>(ctx, M, N, K, A, lda, B, ldb, C, ldc);
  } else {
    rc = vec ? launch_dmma<4, 4, true>(ctx, M, N, K, A, lda, B, ldb, C, ldc)
             : launch_dmma<4, 4, false>(ctx, M, N, K, A, lda, B, ldb, C, ldc);
  }
  count_launches();
  prof_end(ctx, tok, 2.0 * M * N * K, 8.0 * (2.0 * M * N + double(M) * K + double(K) * N));
  ALG_TRY(rc);
  ALG_CUDA_TRY(cudaGetLastError());
  return ALG_OK;
}

}  // namespace alg

extern "C" int alg_gemm_dmma_sub_dev(alg_ctx* ctx, int M, int N, int K, const double* A, int lda, const double* B,
                                     int ldb, double* C, int ldc) {
  if (ctx == nullptr || (M > 0 && N > 0 && K > 0 && (A == nullptr || B == nullptr || C == nullptr)))
    return ALG_INVALID_ARGUMENT;
  if (M < 0 || N < 0 || K < 0 || lda < std::max(1, M) || ldb < std::max(1, K) || ldc < std::max(1, M))
    return ALG_BAD_SHAPE;
  const int rc = alg::gemm_dmma_sub_dev(ctx, M, N, K, A, lda, B, ldb, C, ldc);
  if (rc != ALG_OK) return rc;
  ALG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return ALG_OK;
}
