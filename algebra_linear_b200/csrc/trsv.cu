// Triangular solves with the packed LU factors in one launch (dataflow).
//
// Forward (unit lower L) and backward (upper U) sweeps over column-major
// factors, nrhs right-hand sides. The rows are cut into blocks of kTB; CTA c
// of a cooperative grid owns block rows c, c+G, c+2G, ... in sweep order. For
// its block row i it subtracts L_ij x_j for every earlier block j as soon as
// block j's ready flag is set (acquire load, bounded spin), solves the
// diagonal block, stores x_i and releases its own flag. Block 0 needs
// nothing, and a CTA only waits on blocks that come earlier in the sweep, each
// owned by a co-resident CTA that reaches it before any later block of its
// own, so the chain always progresses.
//
// EXACT: each entry takes its terms in increasing column order with rounded
// products and differences — the row-dot order of the reference's forward
// sweep (src/lapack/mod.rs:341-347), bit for bit. Otherwise a block's 64
// terms are split over four threads and their partial sums are combined in a
// fixed order (deterministic, not the reference's rounding).
#include <algorithm>
#include <climits>

#include "dense.cuh"
#include "pivot.cuh"

namespace alg {
namespace {

constexpr int kTB = 64;         // block rows
constexpr int kTThreads = 256;  // 64 rows x 4 column quarters
constexpr int kMaxRhs = 4;      // right-hand sides handled per pass
template <typename T>
constexpr size_t kTSmem = 4 * kTB * kTB * sizeof(T);  // two factor tiles, the diagonal block, its inverse

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void cp_async_elem(void* dst, const void* src, int bytes) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if (bytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Tile (rows x cols) of the factor at (i0, j0) into smem [col][row], asynchronously.
template <typename T>
__device__ __forceinline__ void prefetch_tile(T* tile, const T* lu, int lda, int i0, int j0, int rows, int cols) {
  for (int idx = threadIdx.x; idx < kTB * kTB; idx += kTThreads) {
    const int rr = idx % kTB, cc = idx / kTB;
    if (rr < rows && cc < cols)
      cp_async_elem(&tile[cc * kTB + rr], lu + (size_t)(i0 + rr) + (size_t)(j0 + cc) * lda, (int)sizeof(T));
  }
}

// Thread 0's bounded wait for a block's ready flag: 1 when it is set, 0 when
// another CTA aborted or the limit ran out (then this CTA raises the abort
// flag and the status block's timeout, so every CTA of the launch returns).
__device__ __forceinline__ int wait_ready(const int* flag, int* abort_flag, DevStatus* status, uint64_t limit_ns) {
  // (the abort flag and the timer are looked at every 16th poll only: a poll
  // is a round trip to L2, and most waits end within a few)
  uint64_t t0 = 0;
  for (int it = 1;; ++it) {
    if (ld_acquire(flag) != 0) return 1;
    if ((it & 15) == 0) {
      if (ld_acquire(abort_flag) != 0) return 0;
      const uint64_t now = global_timer_ns();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > limit_ns) {
        atomicExch(abort_flag, 1);
        atomicExch(&status->timeout, 1);
        return 0;
      }
    }
  }
}

// The diagonal block of an exact sweep by one warp: lane l holds rows l and
// l + 32 of every right-hand side; step c's solved entry is broadcast by a
// shuffle and subtracted as a rounded product from the rows that follow (the
// reference's order, mod.rs:341-353), the upper sweep's quotient correctly
// rounded from the reciprocal formed beforehand. About 50 (lower) and 75
// (upper) cycles a step; through shared memory with a division per step it
// was 150 and 330.
template <typename T, bool UPPER>
__device__ __forceinline__ void exact_diag(const T* dtile, const T* drec, T (*acc_s)[kMaxRhs], int rows, int nrhs) {
  const int lane = threadIdx.x & 31;
  for (int k = 0; k < nrhs; ++k) {
    T v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) v[h] = lane + 32 * h < rows ? acc_s[lane + 32 * h][k] : T(0);
    if constexpr (!UPPER) {
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        const int ce = min(32, rows - 32 * hc);
#pragma unroll 8
        for (int c = 0; c < ce; ++c) {
          const T* col = dtile + (32 * hc + c) * kTB + lane;
          const T u = __shfl_sync(0xffffffffu, v[hc], c);
          if (lane > c) v[hc] = msub<true>(v[hc], col[32 * hc], u);
          if (hc == 0) v[1] = msub<true>(v[1], col[32], u);
        }
      }
    } else {
#pragma unroll
      for (int hc = 1; hc >= 0; --hc) {
        const int ce = min(32, rows - 32 * hc);
        const T y = 32 * hc + lane < rows ? drec[32 * hc + lane] : T(0);
        const T d = 32 * hc + lane < rows ? dtile[(32 * hc + lane) * (kTB + 1)] : T(1);
#pragma unroll 8
        for (int c = ce - 1; c >= 0; --c) {
          const T* col = dtile + (32 * hc + c) * kTB + lane;
          const T qv = mul_rn(v[hc], y);
          T q = fma_rn(fma_rn(-qv, d, v[hc]), y, qv);
          if (lane == c && !(y != T(0) && exp_fast_ok(v[hc]))) q = div_rn(v[hc], d);
          if (lane == c) v[hc] = q;
          const T u = __shfl_sync(0xffffffffu, v[hc], c);
          if (lane < c) v[hc] = msub<true>(v[hc], col[32 * hc], u);
          if (hc == 1) v[0] = msub<true>(v[0], col[0], u);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (lane + 32 * h < rows) acc_s[lane + 32 * h][k] = v[h];
  }
}

// stuck_wait != 0: the CTA of the sweep's first block waits on flags[nb], a
// slot cleared before the launch that nothing sets, so the wait runs out
// (the timeout path, exercised by tests without any fault).
template <typename T, bool EXACT, bool UPPER>
__global__ void __launch_bounds__(kTThreads) trsv_dataflow_kernel(const T* __restrict__ lu, int lda, int n, T* x,
                                                                  int ldx, int nrhs, int* flags, int* abort_flag,
                                                                  DevStatus* status, uint64_t wait_limit_ns,
                                                                  int stuck_wait) {
  extern __shared__ __align__(16) unsigned char tsm[];
  T* tiles = reinterpret_cast<T*>(tsm);                 // [2][kTB*kTB] factor tiles, [col][row]
  T* dtile = tiles + 2 * kTB * kTB;                      // diagonal block, [col][row]
  T* dinv = tiles + 3 * kTB * kTB;                       // its inverse (non-EXACT), [col][row]
  __shared__ T xs[kTB][kMaxRhs];       // x of the block being consumed
  __shared__ T part[4][kTB][kMaxRhs];  // partial sums of the four column quarters
  __shared__ T acc_s[kTB][kMaxRhs];
  __shared__ T drec[kTB];  // EXACT, upper: reciprocals of the diagonal (0: divide plainly)
  __shared__ int stop;
  const int nb = (n + kTB - 1) / kTB;
  const int r = threadIdx.x & (kTB - 1);  // row within the block
  const int qt = threadIdx.x >> 6;        // column quarter
  if (stuck_wait && blockIdx.x == 0) {
    if (threadIdx.x == 0) stop = !wait_ready(&flags[nb], abort_flag, status, wait_limit_ns);
    __syncthreads();
    if (stop) return;
  }
  for (int s = blockIdx.x; s < nb; s += gridDim.x) {
    // sweep position s -> block index (forward: ascending, backward: descending)
    const int bi = UPPER ? nb - 1 - s : s;
    const int i0 = bi * kTB;
    const int rows = min(kTB, n - i0);
    if (qt == 0 && r < rows)
      for (int k = 0; k < nrhs; ++k) acc_s[r][k] = x[(size_t)k * ldx + i0 + r];
    // the diagonal block and the first off-diagonal tile start loading now
    prefetch_tile<T>(dtile, lu, lda, i0, i0, rows, rows);
    cp_async_commit();
    if (s > 0) {
      const int bj = UPPER ? nb - 1 : 0;
      prefetch_tile<T>(tiles, lu, lda, i0, bj * kTB, rows, min(kTB, n - bj * kTB));
    }
    cp_async_commit();
    if constexpr (!EXACT) {
      // Invert the diagonal block now, while earlier blocks are still being
      // solved: the critical path then only pays a matrix-vector product.
      cp_async_wait<1>();  // the diagonal block (first group) has landed
      __syncthreads();
      if (threadIdx.x < rows) {
        const int c = threadIdx.x;
        T* xcol = dinv + c * kTB;
        if constexpr (!UPPER) {  // unit lower: x = L^{-1} e_c
          for (int rr = 0; rr < c; ++rr) xcol[rr] = T(0);
          xcol[c] = T(1);
          for (int rr = c + 1; rr < rows; ++rr) {
            T acc = T(0);
            for (int k = c; k < rr; ++k) acc = fma_rn(dtile[k * kTB + rr], xcol[k], acc);
            xcol[rr] = -acc;
          }
        } else {  // upper: x = U^{-1} e_c
          for (int rr = c + 1; rr < rows; ++rr) xcol[rr] = T(0);
          xcol[c] = div_rn(T(1), dtile[c * kTB + c]);
          for (int rr = c - 1; rr >= 0; --rr) {
            T acc = T(0);
            for (int k = rr + 1; k <= c; ++k) acc = fma_rn(dtile[k * kTB + rr], xcol[k], acc);
            xcol[rr] = -div_rn(acc, dtile[rr * kTB + rr]);
          }
        }
      }
    }
    if constexpr (EXACT && UPPER) {
      cp_async_wait<1>();
      __syncthreads();
      if (threadIdx.x < rows) {
        const T d = dtile[threadIdx.x * kTB + threadIdx.x];
        drec[threadIdx.x] = exp_fast_ok(d) ? rcp_rn(d) : T(0);
      }
    }
    __syncthreads();
    for (int t = 0; t < s; ++t) {
      const int bj = UPPER ? nb - 1 - t : t;
      const int j0 = bj * kTB;
      const int cols = min(kTB, n - j0);
      const T* tile = tiles + (size_t)(t & 1) * kTB * kTB;
      // next tile in flight while this one is consumed
      if (t + 1 < s) {
        const int bn = UPPER ? nb - 2 - t : t + 1;
        prefetch_tile<T>(tiles + (size_t)((t + 1) & 1) * kTB * kTB, lu, lda, i0, bn * kTB, rows,
                         min(kTB, n - bn * kTB));
      }
      cp_async_commit();
      // wait for block bj (bounded); a failure anywhere stops every CTA
      if (threadIdx.x == 0) stop = !wait_ready(&flags[bj], abort_flag, status, wait_limit_ns);
      __syncthreads();
      if (stop) {
        cp_async_wait<0>();
        return;
      }
      for (int idx = threadIdx.x; idx < cols * nrhs; idx += kTThreads) {
        const int c = idx % cols, k = idx / cols;
        xs[c][k] = __ldcg(&x[(size_t)k * ldx + j0 + c]);
      }
      cp_async_wait<1>();  // tile t has landed (tile t+1 may still be in flight)
      __syncthreads();
      if (r < rows) {
        if constexpr (EXACT) {
          if (qt == 0) {
            for (int k = 0; k < nrhs; ++k) {
              T a = acc_s[r][k];
#pragma unroll 8
              for (int c = 0; c < cols; ++c) a = msub<true>(a, tile[c * kTB + r], xs[c][k]);
              acc_s[r][k] = a;
            }
          }
        } else {
          const int c0 = qt * (kTB / 4), c1 = min(cols, c0 + kTB / 4);
          for (int k = 0; k < nrhs; ++k) {
            T p = T(0);
#pragma unroll 4
            for (int c = c0; c < c1; ++c) p = fma_rn(tile[c * kTB + r], xs[c][k], p);
            part[qt][r][k] = p;
          }
        }
      }
      __syncthreads();
      if constexpr (!EXACT) {
        if (qt == 0 && r < rows)
          for (int k = 0; k < nrhs; ++k)
            acc_s[r][k] = acc_s[r][k] - ((part[0][r][k] + part[1][r][k]) + (part[2][r][k] + part[3][r][k]));
        __syncthreads();
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    if constexpr (!EXACT) {
      // x_i = inv(D_ii) y_i: four column quarters per row, fixed-order combine
      if (r < rows) {
        const int c0 = qt * (kTB / 4), c1 = min(rows, c0 + kTB / 4);
        for (int k = 0; k < nrhs; ++k) {
          T p = T(0);
          for (int c = c0; c < c1; ++c) p = fma_rn(dinv[c * kTB + r], acc_s[c][k], p);
          part[qt][r][k] = p;
        }
      }
      __syncthreads();
      if (qt == 0 && r < rows)
        for (int k = 0; k < nrhs; ++k)
          acc_s[r][k] = (part[0][r][k] + part[1][r][k]) + (part[2][r][k] + part[3][r][k]);
    }
    if constexpr (EXACT) {
      if (threadIdx.x < 32) exact_diag<T, UPPER>(dtile, drec, acc_s, rows, nrhs);
    }
    __syncthreads();
    if (threadIdx.x < 64) {  // two warps store the block, one of them releases it
      if (r < rows)
        for (int k = 0; k < nrhs; ++k) x[(size_t)k * ldx + i0 + r] = acc_s[r][k];
      asm volatile("bar.sync 1, 64;" ::: "memory");
      if (threadIdx.x == 0) {
        __threadfence();  // cumulative: the block's stores, ordered by the barrier, before the flag
        st_release(&flags[bi], 1);
      }
    }
  }
}

template <typename T, bool EXACT, bool UPPER>
int launch_trsv(alg_ctx* ctx, const T* lu, int lda, int n, T* x, int ldx, int nrhs, int* flags, int* abort_flag) {
  const int nb = (n + kTB - 1) / kTB;
  static PerDevice resident;  // CTAs of the kernel that a device holds at once
  int device = 0, max_blocks = 0;
  ALG_CUDA_TRY(cudaGetDevice(&device));
  ALG_CUDA_TRY(static_cast<cudaError_t>(resident.get(device, max_blocks, [&](int& blocks) {
    int per_sm = 0;
    cudaError_t e = cudaFuncSetAttribute(trsv_dataflow_kernel<T, EXACT, UPPER>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem<T>);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trsv_dataflow_kernel<T, EXACT, UPPER>, kTThreads,
                                                        kTSmem<T>);
    blocks = std::max(1, per_sm) * ctx->sm_count;
    return static_cast<int>(e);
  })));
  int grid = std::min(nb, max_blocks);
  uint64_t limit = ctx->wait_limit_ns ? ctx->wait_limit_ns : kWaitLimitNs;
  int stuck = 0;
  if (ctx->stuck_waits > 0) {
    --ctx->stuck_waits;
    stuck = 1;
  }
  void* args[] = {(void*)&lu, (void*)&lda, (void*)&n, (void*)&x, (void*)&ldx, (void*)&nrhs,
                  (void*)&flags, (void*)&abort_flag, (void*)&ctx->d_status, (void*)&limit, (void*)&stuck};
  ALG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)trsv_dataflow_kernel<T, EXACT, UPPER>, dim3(grid),
                                           dim3(kTThreads), args, kTSmem<T>, ctx->stream));
  count_launches();
  return ALG_OK;
}

// x[:, k] = b[perm, k]; with `guard`, nothing when the factorization it reports
// on failed (a row order from a timed-out one is not used as an index).
template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ b, int ldb, const int* __restrict__ perm, int n, int nrhs,
                                   T* __restrict__ x, int ldx, const DevStatus* guard) {
  if (guard != nullptr && factor_failed(guard)) return;
  const size_t cnt = (size_t)n * nrhs;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += (size_t)gridDim.x * blockDim.x) {
    const size_t k = idx / n, i = idx % n;
    x[k * ldx + i] = b[k * ldb + perm[i]];
  }
}

template <typename T>
void gather_rows(alg_ctx* ctx, const T* b, int ldb, const int* perm, int n, int nrhs, T* x, int ldx,
                 const DevStatus* guard) {
  const size_t cnt = (size_t)n * nrhs;
  const int g = (int)std::max<size_t>(1, std::min<size_t>((cnt + 255) / 256, (size_t)ctx->sm_count * 8));
  gather_rows_kernel<T><<<g, 256, 0, ctx->stream>>>(b, ldb, perm, n, nrhs, x, ldx, guard);
  count_launches();
}

template <typename T>
__global__ void store_solution_kernel(const T* __restrict__ x, int n, int nrhs, T* __restrict__ b, int ldb,
                                      const DevStatus* guard) {
  if (factor_failed(guard)) return;
  const size_t cnt = (size_t)n * nrhs;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += (size_t)gridDim.x * blockDim.x)
    b[(idx / n) * ldb + idx % n] = x[idx];
}

}  // namespace

// b (n x nrhs, ldb) <- x (n x nrhs, ld n), with `guard` only when the
// factorization it reports on succeeded.
template <typename T>
int store_solution_dev(alg_ctx* ctx, const T* x, int n, int nrhs, T* b, int ldb, const DevStatus* guard) {
  if (guard == nullptr) {
    ALG_CUDA_TRY(cudaMemcpy2DAsync(b, sizeof(T) * (size_t)ldb, x, sizeof(T) * (size_t)n, sizeof(T) * (size_t)n, nrhs,
                                   cudaMemcpyDeviceToDevice, ctx->stream));
    return ALG_OK;
  }
  const size_t cnt = (size_t)n * nrhs;
  const int g = (int)std::max<size_t>(1, std::min<size_t>((cnt + 255) / 256, (size_t)ctx->sm_count * 8));
  store_solution_kernel<T><<<g, 256, 0, ctx->stream>>>(x, n, nrhs, b, ldb, guard);
  count_launches();
  ALG_CUDA_TRY(cudaGetLastError());
  return ALG_OK;
}
template int store_solution_dev<double>(alg_ctx*, const double*, int, int, double*, int, const DevStatus*);
template int store_solution_dev<float>(alg_ctx*, const float*, int, int, float*, int, const DevStatus*);

// b (n x nrhs, ldb) <- (LU)^{-1} P b, one gather + two dataflow launches per
// group of up to kMaxRhs right-hand sides.
template <typename T, bool EXACT>
int lu_solve_dataflow_dev(alg_ctx* ctx, const T* lu, int n, int lda, const int* perm, T* b, int nrhs, int ldb,
                          const DevStatus* guard) {
  if (n == 0 || nrhs == 0) return ALG_OK;
  const int nb = (n + kTB - 1) / kTB;
  T* x = nullptr;
  int* flags = nullptr;
  ALG_TRY(ws_get(ctx, WS_X, sizeof(T) * (size_t)n * nrhs, reinterpret_cast<void**>(&x)));
  ALG_TRY(ws_get(ctx, WS_LAB, sizeof(int) * (size_t)(2 * nb + 4) + sizeof(int) * n,
                 reinterpret_cast<void**>(&flags)));
  int* abort_flag = flags + 2 * nb + 2;
  const int tok = prof_begin(ctx, ALG_K_SOLVE);
  gather_rows<T>(ctx, b, ldb, perm, n, nrhs, x, n, guard);
  for (int k0 = 0; k0 < nrhs; k0 += kMaxRhs) {
    // both sweeps' flags, and before the first group the abort flag behind them
    ALG_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(int) * (size_t)(2 * nb + 2 + (k0 == 0 ? 1 : 0)), ctx->stream));
    const int kr = std::min(kMaxRhs, nrhs - k0);
    T* xk = x + (size_t)k0 * n;
    ALG_TRY((launch_trsv<T, EXACT, false>(ctx, lu, lda, n, xk, n, kr, flags, abort_flag)));
    ALG_TRY((launch_trsv<T, EXACT, true>(ctx, lu, lda, n, xk, n, kr, flags + nb + 1, abort_flag)));
  }
  ALG_TRY(store_solution_dev<T>(ctx, x, n, nrhs, b, ldb, guard));
  prof_end(ctx, tok, 2.0 * n * n * nrhs, sizeof(T) * (double(n) * n + 4.0 * n * nrhs));
  return ALG_OK;
}

// One triangular sweep (non-exact arithmetic) over the leading n x n block
// of column-major factors: unit-lower (upper = false) or upper. flags holds
// n / 64 + 1 ints (cleared here); abort_flag must be zero.
template <typename T>
int tri_solve_dev(alg_ctx* ctx, const T* lu, int lda, int n, T* x, bool upper, int* flags, int* abort_flag) {
  if (n <= 0) return ALG_OK;
  ALG_CUDA_TRY(cudaMemsetAsync(flags, 0, sizeof(int) * ((n + kTB - 1) / kTB + 1), ctx->stream));
  if (upper) return launch_trsv<T, false, true>(ctx, lu, lda, n, x, n, 1, flags, abort_flag);
  return launch_trsv<T, false, false>(ctx, lu, lda, n, x, n, 1, flags, abort_flag);
}

template int tri_solve_dev<double>(alg_ctx*, const double*, int, int, double*, bool, int*, int*);
template int tri_solve_dev<float>(alg_ctx*, const float*, int, int, float*, bool, int*, int*);
template int lu_solve_dataflow_dev<double, true>(alg_ctx*, const double*, int, int, const int*, double*, int, int,
    const DevStatus*);
template int lu_solve_dataflow_dev<double, false>(alg_ctx*, const double*, int, int, const int*, double*, int, int,
    const DevStatus*);
template int lu_solve_dataflow_dev<float, false>(alg_ctx*, const float*, int, int, const int*, float*, int, int,
    const DevStatus*);
template int lu_solve_dataflow_dev<float, true>(alg_ctx*, const float*, int, int, const int*, float*, int, int,
    const DevStatus*);

}  // namespace alg
