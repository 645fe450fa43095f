// Batched dgesv for many independent dense systems of uneven order, in one
// persistent launch per size bucket (capturable in a CUDA graph).
//
// Each system is the reference's dgesv (src/lapack/mod.rs:309-354): LU with
// partial pivoting (first index of max |a_ik|, NaN rule as the reference),
// multipliers by division, then the forward/back sweeps. A CTA pulls systems
// from a queue ordered by decreasing order n (largest first, for balance) and
// factorizes each one in place in its global buffer with a right-looking
// blocked schedule: a 16- or 32-column panel factored in shared memory with
// its rows in registers (cta_leaf), then the columns right of it in chunks:
// gathered in the panel's row order, U12 by a blocked unit-lower solve, and
// the trailing update on the FP64 tensor cores (FP32: register tiles). In the
// FP64 form the right-hand side is one more column of that sweep, so the
// forward substitution costs nothing of its own. The mixed form factorizes an
// FP32 copy and refines x in FP64 against the FP64 matrix until the system's
// normwise backward error is within tol.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>
#include <math_constants.h>

#include "batched.cuh"
#include "cta_lu.cuh"

namespace alg {
namespace {

constexpr int kMaxN = 512;    // largest order a CTA handles

// Columns of the trailing matrix taken at a time.
template <int NT>
__host__ __device__ constexpr int chunk_cols() {
  return NT / 4;
}

// Shared memory of cta_getrf for panels of up to `cap` rows: the leaf's
// records, the panel [col][row], two U12 chunks [k][col] and 2 pb + 4 ints.
template <typename T, int NT>
__host__ __device__ constexpr size_t getrf_smem(int cap, int pb) {
  return 2 * (NT / 32) * sizeof(PivotRec<T, kLeafW>) + sizeof(T) * (size_t)panel_ld(cap) * pb +
         2 * sizeof(T) * (size_t)chunk_ld<T>(chunk_cols<NT>()) * pb + (2 * pb + 4) * 4;
}

// LU with partial pivoting of the n x n matrix a (global, leading dim n) in
// place; ipiv (global, n ints): the sequential interchanges. rhs (may be null):
// one more column of n entries, left as L^{-1} P rhs. perm (shared, may be
// null): n ints, left as the row order. Returns 0 or 1 + the first column
// with a zero pivot. NT threads, RPT rows each (n <= NT * RPT), panel PB.
template <typename T, int NT, int RPT, int PB>
__device__ int cta_getrf(T* a, int n, T* rhs, int* ipiv, int* perm, unsigned char* smem, int cap) {
  using Rec = PivotRec<T, kLeafW>;
  constexpr int NW = NT / 32;
  constexpr int CH = chunk_cols<NT>();
  constexpr int ldu = chunk_ld<T>(chunk_cols<NT>());
  const int ldt = panel_ld(cap);
  Rec(*rec)[NW] = reinterpret_cast<Rec(*)[NW]>(smem);
  T* tile = reinterpret_cast<T*>(smem + 2 * NW * sizeof(Rec));  // [col][row]
  T* us = tile + (size_t)PB * ldt;                              // [k][col], two buffers (16-byte aligned)
  int* piv_slot = reinterpret_cast<int*>(us + 2 * PB * ldu);    // slot of each pivot row
  int* disp = piv_slot + PB;  // where a top row that is no pivot went (-1: it is one)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int zero = INT_MAX;
  if (perm != nullptr)
    for (int i = tid; i < n; i += NT) perm[i] = i;
  for (int k0 = 0; k0 < n; k0 += PB) {
    const int w = min(PB, n - k0);
    const int m = n - k0;  // panel rows
    // ---- panel into shared memory --------------------------------------
    int pos[RPT];
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int r = tid + k * NT;
      pos[k] = r < m ? r : -1;
      if (r < m) {
        const T* src = a + (size_t)(k0 + r) + (size_t)k0 * n;
#pragma unroll 8
        for (int c = 0; c < w; ++c) tile[c * ldt + r] = src[(size_t)c * n];
      }
    }
    if (tid < PB) disp[tid] = -1;
    // ---- its leaves (each thread reads its own rows: no barrier needed) ------
    for (int cl0 = 0; cl0 < w; cl0 += kLeafW) {
      const int wl = min(kLeafW, w - cl0), tc = w - cl0 - wl;
      const int z = cta_leaf<T, kLeafW, NT, RPT, false, false>(tile, ldt, m, cl0, wl, pos, rec, piv_slot, ipiv + k0);
      if (z != INT_MAX && zero == INT_MAX) zero = k0 + z;
      __syncthreads();
      if (tc > 0) {
        if (tid < tc) {  // U of the leaf's pivot rows in the panel's other columns
          T x[kLeafW];
          T* tcol = tile + (cl0 + kLeafW + tid) * ldt;
#pragma unroll
          for (int i = 0; i < kLeafW; ++i) x[i] = tcol[piv_slot[cl0 + i]];
#pragma unroll
          for (int i = 1; i < kLeafW; ++i) {
            const T* lrow = tile + cl0 * ldt + piv_slot[cl0 + i];
#pragma unroll
            for (int k = 0; k < i; ++k) x[i] = fma_t<T>(-lrow[k * ldt], x[k], x[i]);
          }
#pragma unroll
          for (int i = 0; i < kLeafW; ++i) {
            us[tid * kLeafW + i] = x[i];
            tcol[piv_slot[cl0 + i]] = x[i];
          }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RPT; ++k)
          if (pos[k] >= cl0 + kLeafW) {
            T* trow = tile + tid + k * NT;
            T l[kLeafW];
#pragma unroll
            for (int i = 0; i < kLeafW; ++i) l[i] = trow[(cl0 + i) * ldt];
#pragma unroll 4
            for (int c = 0; c < tc; ++c) {
              T acc = trow[(cl0 + kLeafW + c) * ldt];
              const T* uc = static_cast<const T*>(__builtin_assume_aligned(us + c * kLeafW, 16));
#pragma unroll
              for (int i = 0; i < kLeafW; ++i) acc = fma_t<T>(-l[i], uc[i], acc);
              trow[(cl0 + kLeafW + c) * ldt] = acc;
            }
          }
      }
    }
    // ---- rows into position order: pivots first, displaced top rows last ----
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (tid + k * NT < w && pos[k] >= w) disp[tid + k * NT] = pos[k];
    const bool moved = __syncthreads_or(tid < w && piv_slot[tid] != tid);
    if (moved) {
      constexpr int kIt = (PB * PB + NT - 1) / NT;
      T pv[kIt], dv[kIt];
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int e = tid + it * NT, i = e % PB, c = e / PB;
        if (i < w && c < w) {
          pv[it] = tile[c * ldt + piv_slot[i]];
          dv[it] = tile[c * ldt + i];
        }
      }
      __syncthreads();
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int e = tid + it * NT, i = e % PB, c = e / PB;
        if (i < w && c < w) {
          tile[c * ldt + i] = pv[it];
          if (disp[i] >= 0) tile[c * ldt + disp[i]] = dv[it];
        }
      }
      // the same interchanges on the columns left of the panel, a warp each
      for (int c = warp; c < k0 + (perm != nullptr ? 1 : 0); c += NW) {
        if (c < k0) {
          T* cp = a + (size_t)c * n + k0;
          T p0 = T(0), d0 = T(0);
          if (lane < w) {
            p0 = cp[piv_slot[lane]];
            d0 = cp[lane];
          }
          __syncwarp();
          if (lane < w) {
            cp[lane] = p0;
            if (disp[lane] >= 0) cp[disp[lane]] = d0;
          }
        } else {
          int p0 = 0, d0 = 0;
          if (lane < w) {
            p0 = perm[k0 + piv_slot[lane]];
            d0 = perm[k0 + lane];
          }
          __syncwarp();
          if (lane < w) {
            perm[k0 + lane] = p0;
            if (disp[lane] >= 0) perm[k0 + disp[lane]] = d0;
          }
        }
      }
      __syncthreads();
    }
    // sequential interchanges from positions within the panel to rows
    if (tid < w) ipiv[k0 + tid] += k0;
    for (int r = tid; r < m; r += NT) {
      T* dst = a + (size_t)(k0 + r) + (size_t)k0 * n;
#pragma unroll 8
      for (int c = 0; c < w; ++c) dst[(size_t)c * n] = tile[c * ldt + r];
    }
    // ---- the columns right of the panel (and the right-hand side) -----------
    const int kr = k0 + w, mt = n - kr;
    const int nright = mt + (rhs != nullptr ? 1 : 0);
    // (a chunk's rows of U12, in pivot order, are fetched while the chunk
    // before it is updated)
    auto fetch = [&](int cb, T* u) {
      const int cw = min(CH, nright - cb);
#pragma unroll
      for (int it = 0; it < PB * CH / NT; ++it) {
        const int e = tid + it * NT, i = e % PB, c = e / PB;
        if (i < w && c < cw)
          cp_async_entry(u + i * ldu + c, (cb + c < mt ? a + (size_t)(kr + cb + c) * n : rhs) + k0 + piv_slot[i]);
      }
      cp_async_commit();
    };
    if (nright > 0) fetch(0, us);
    for (int cb = 0, buf = 0; cb < nright; cb += CH, buf ^= 1) {
      T* u = us + buf * PB * ldu;
      const int cw = min(CH, nright - cb);
      auto col = [&](int c) { return cb + c < mt ? a + (size_t)(kr + cb + c) * n : rhs; };
      constexpr int kIt = PB * CH / NT;
      T dv[kIt];
      if (moved) {
#pragma unroll
        for (int it = 0; it < kIt; ++it) {
          const int e = tid + it * NT, i = e % PB, c = e / PB;
          if (i < w && c < cw) dv[it] = col(c)[k0 + i];
        }
      }
      cp_async_wait_all();
      __syncthreads();
      if (cb + CH < nright) fetch(cb + CH, us + (buf ^ 1) * PB * ldu);
      if (moved) {
#pragma unroll
        for (int it = 0; it < kIt; ++it) {
          const int e = tid + it * NT, i = e % PB, c = e / PB;
          if (i < w && c < cw && disp[i] >= 0) col(c)[k0 + disp[i]] = dv[it];
        }
      }
      if (tid < cw) solve16(tile, ldt, u + tid, ldu, min(w, kLeafW));
      __syncthreads();
      if (PB > kLeafW && w > kLeafW) {
        for (int e = tid; e < kLeafW * cw; e += NT) {
          const int i = kLeafW + e % kLeafW, c = e / kLeafW;
          if (i < w) {
            T acc = u[i * ldu + c];
#pragma unroll
            for (int k = 0; k < kLeafW; ++k) acc = fma_t<T>(-tile[k * ldt + i], u[k * ldu + c], acc);
            u[i * ldu + c] = acc;
          }
        }
        __syncthreads();
        if (tid < cw) solve16(tile + kLeafW * ldt + kLeafW, ldt, u + kLeafW * ldu + tid, ldu, w - kLeafW);
        __syncthreads();
      }
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int e = tid + it * NT, i = e % PB, c = e / PB;
        if (i < w && c < cw) col(c)[k0 + i] = u[i * ldu + c];
      }
      if (mt > 0) {  // (then w == PB)
        const int cm = min(cw, mt - cb);  // the chunk's matrix columns
        cta_update<PB, NW, true, sizeof(T) == 8 && (NT * RPT > 256)>(tile + PB, ldt, u, ldu, a + (size_t)(kr + cb) * n + kr, n, mt, cm);
        if (cm < cw)  // and the right-hand side
          for (int r = tid; r < mt; r += NT) {
            T acc = rhs[kr + r];
#pragma unroll
            for (int k = 0; k < PB; ++k) acc = fma_t<T>(-tile[k * ldt + PB + r], u[k * ldu + cm], acc);
            rhs[kr + r] = acc;
          }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  return zero == INT_MAX ? 0 : zero + 1;
}

constexpr int kSB = 32;  // rows of a block of the triangular sweeps

// xs (shared, n) <- U^{-1} xs, or with UNIT_LOWER L^{-1} xs, for the factors
// lu (global, n x n). By blocks of 32 rows: one warp solves the diagonal
// block (its rows in registers, one shuffle per step; quotients correctly
// rounded from reciprocals formed beforehand), then every thread subtracts
// the block's 32 terms from a row of the rest, its 32 loads in flight at once.
template <bool UNIT_LOWER, typename T, int NT>
__device__ __noinline__ void cta_sweep(const T* lu, int n, double* xs) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int nb = (n + kSB - 1) / kSB;
  for (int b = 0; b < nb; ++b) {
    const int k0 = (UNIT_LOWER ? b : nb - 1 - b) * kSB, w = min(kSB, n - k0);
    const T* blk = lu + (size_t)k0 * n;  // the block's columns
    if (tid < 32) {
      double u[kSB];
#pragma unroll
      for (int j = 0; j < kSB; ++j) u[j] = (lane < w && j < w) ? (double)blk[(size_t)(k0 + lane) + (size_t)j * n] : 0.0;
      double x = lane < w ? xs[k0 + lane] : 0.0;
      if (UNIT_LOWER) {
#pragma unroll
        for (int j = 0; j < kSB; ++j) {
          const double xj = __shfl_sync(0xffffffffu, x, j);
          if (lane > j) x = __fma_rn(-u[j], xj, x);
        }
      } else {
        double d = 1.0;
#pragma unroll
        for (int j = 0; j < kSB; ++j)
          if (lane == j && j < w) d = u[j];
        const bool fast = exp_fast_ok(d);
        const double y = fast ? rcp_rn(d) : 1.0;
#pragma unroll
        for (int j = kSB - 1; j >= 0; --j) {
          if (lane == j) x = quotient<double>(x, d, y, fast);
          const double xj = __shfl_sync(0xffffffffu, x, j);
          if (lane < j) x = __fma_rn(-u[j], xj, x);
        }
      }
      if (lane < w) xs[k0 + lane] = x;
    }
    __syncthreads();
    const int r0 = UNIT_LOWER ? k0 + w : 0, r1 = UNIT_LOWER ? n : k0;
    for (int i = r0 + tid; i < r1; i += NT) {
      const T* row = blk + i;
      double acc = xs[i];
      if (w == kSB) {
        T v[kSB];
#pragma unroll
        for (int j = 0; j < kSB; ++j) v[j] = row[(size_t)j * n];
#pragma unroll
        for (int j = 0; j < kSB; ++j) acc = __fma_rn(-(double)v[j], xs[k0 + j], acc);
      } else {
        for (int j = 0; j < w; ++j) acc = __fma_rn(-(double)row[(size_t)j * n], xs[k0 + j], acc);
      }
      xs[i] = acc;
    }
    __syncthreads();
  }
}

// xs (shared) <- (LU)^{-1} P x for one vector x (global).
template <typename T, int NT>
__device__ void cta_getrs(const T* lu, int n, const int* perm, const double* x, double* xs) {
  for (int i = threadIdx.x; i < n; i += NT) xs[i] = x[perm[i]];
  __syncthreads();
  cta_sweep<true, T, NT>(lu, n, xs);
  cta_sweep<false, T, NT>(lu, n, xs);
}

// Normwise backward error of x for A x = b (FP64, A n x n in global).
__device__ __noinline__ double cta_backward_error(const double* a, int n, const double* x, const double* b, double* rs,
                                     double* red) {
  double rmax = 0.0, amax = 0.0, xmax = 0.0, bmax = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double s = 0.0, ra = 0.0;
#pragma unroll 16
    for (int j = 0; j < n; ++j) {
      const double aij = a[(size_t)i + (size_t)j * n];
      s = __fma_rn(aij, x[j], s);
      ra += fabs(aij);
    }
    rs[i] = b[i] - s;
    rmax = fmax(rmax, fabs(rs[i]));
    amax = fmax(amax, ra);
    xmax = fmax(xmax, fabs(x[i]));
    bmax = fmax(bmax, fabs(b[i]));
  }
  for (int off = 16; off > 0; off >>= 1) {
    rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, off));
    amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, off));
    bmax = fmax(bmax, __shfl_xor_sync(0xffffffffu, bmax, off));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    red[4 * warp + 0] = rmax;
    red[4 * warp + 1] = amax;
    red[4 * warp + 2] = xmax;
    red[4 * warp + 3] = bmax;
  }
  __syncthreads();
  double R = 0, A = 0, X = 0, B = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    R = fmax(R, red[4 * w + 0]);
    A = fmax(A, red[4 * w + 1]);
    X = fmax(X, red[4 * w + 2]);
    B = fmax(B, red[4 * w + 3]);
  }
  __syncthreads();
  const double den = A * X + B;
  return den == 0.0 ? R : R / den;
}

struct BatchArgs {
  int count;
  const int* order;        // systems of this bucket, largest first
  const int* n;
  const long long* a_off;  // offsets (entries) of A in a
  const long long* b_off;  // offsets of b in b
  double* a;               // FP64 matrices (overwritten by the LU in the FP64 form)
  double* b;               // right-hand sides -> solutions
  float* a32;              // FP32 working copies (mixed form), same offsets as a
  int* ipiv;               // same offsets as b
  double* work;            // same offsets as b: residual / correction
  int* info;               // per system: 0, 1 + singular column, or -(iterations+1) without convergence
  double* eta;             // per system backward error (mixed form)
  int* queue;              // work counter
  int cap;                 // largest order in the bucket
  int mixed;               // 0: FP64 LU; 1: FP32 LU + FP64 refinement
  int max_ir;
  double tol_scale;        // tol = tol_scale * n * 2^-53
};

// RPT rows per thread: systems of up to NT * RPT rows. Bound by the column
// chain (latency) and, for the largest orders, by the trailing matrix's
// passes through L2 and HBM (8 n^3 / 3 PB bytes of it per system and direction);
// 20 000 systems of order 8..512, FP64: 81 ms before (panel columns with three
// barriers each in shared memory, the update on the CUDA cores, sweeps of two
// barriers a column), 27.4 ms now; 3 000 in the mixed form 11.1 and 5.1 ms.
template <int NT, int RPT, int PB>
__global__ void __launch_bounds__(NT, RPT == 4 ? 2 : 512 / NT) batched_gesv_kernel(BatchArgs p) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int next;
  __shared__ double red[4 * (NT / 32)];
  double* vs = reinterpret_cast<double*>(smem);  // cap doubles for vectors
  int* perm = reinterpret_cast<int*>(vs + p.cap);  // cap ints: the row order (mixed form)
  unsigned char* lus = reinterpret_cast<unsigned char*>(perm + ((p.cap + 3) & ~3));
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(p.queue, 1);
    __syncthreads();
    const int q = next;
    __syncthreads();
    if (q >= p.count) return;
    const int s = p.order[q];
    const int n = p.n[s];
    double* a = p.a + p.a_off[s];
    double* b = p.b + p.b_off[s];
    int* ipiv = p.ipiv + p.b_off[s];
    if (!p.mixed) {
      double* y = p.work + p.b_off[s];  // b stays as it is when the system is singular
      for (int i = threadIdx.x; i < n; i += NT) y[i] = b[i];
      __syncthreads();
      const int info = cta_getrf<double, NT, RPT, PB>(a, n, y, ipiv, nullptr, lus, p.cap);
      if (threadIdx.x == 0) p.info[s] = info;
      if (info == 0) {  // y = L^{-1} P b
        for (int i = threadIdx.x; i < n; i += NT) vs[i] = y[i];
        __syncthreads();
        cta_sweep<false, double, NT>(a, n, vs);
        for (int i = threadIdx.x; i < n; i += NT) b[i] = vs[i];
      }
      continue;
    }
    // ---- mixed: FP32 LU, FP64 refinement against the FP64 matrix ------------
    float* a32 = p.a32 + p.a_off[s];
    {
      const size_t nn = (size_t)n * n;
      size_t e = threadIdx.x;
      for (; e + 7 * NT < nn; e += 8 * NT) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = a[e + u * NT];
#pragma unroll
        for (int u = 0; u < 8; ++u) a32[e + u * NT] = __double2float_rn(v[u]);
      }
      for (; e < nn; e += NT) a32[e] = __double2float_rn(a[e]);
    }
    __syncthreads();
    const int info = cta_getrf<float, NT, RPT, PB>(a32, n, nullptr, ipiv, perm, lus, p.cap);
    if (info != 0) {
      if (threadIdx.x == 0) p.info[s] = info;
      continue;
    }
    double* res = p.work + p.b_off[s];             // residual (global)
    double* sol = vs;                              // solution (shared)
    double* r = reinterpret_cast<double*>(lus);    // solve staging (the panel area is free now)
    cta_getrs<float, NT>(a32, n, perm, b, r);
    for (int i = threadIdx.x; i < n; i += NT) sol[i] = r[i];
    __syncthreads();
    const double tol = p.tol_scale * n * 0x1p-53;
    int it = 0;
    double e = 0.0;
    for (;;) {
      e = cta_backward_error(a, n, sol, b, res, red);  // also res = b - A sol
      if (e <= tol || it >= p.max_ir || !(e == e)) break;
      cta_getrs<float, NT>(a32, n, perm, res, r);
      for (int i = threadIdx.x; i < n; i += NT) sol[i] += r[i];
      __syncthreads();
      ++it;
    }
    for (int i = threadIdx.x; i < n; i += NT) b[i] = sol[i];
    if (threadIdx.x == 0) {
      p.info[s] = (e <= tol) ? 0 : -(it + 1);
      p.eta[s] = e;
    }
    __syncthreads();
  }
}

// Every launch shape: NT threads, the rows per thread that cover the bucket's
// cap, the panel width.
using BatchKernel = void (*)(BatchArgs);
template <int NT, int PB>
BatchKernel batch_kernel_rpt(int cap) {
  if (cap <= NT) return batched_gesv_kernel<NT, 1, PB>;
  if constexpr (2 * NT <= kMaxN)
    if (cap <= 2 * NT) return batched_gesv_kernel<NT, 2, PB>;
  if constexpr (4 * NT <= kMaxN) return batched_gesv_kernel<NT, 4, PB>;
  return nullptr;
}
BatchKernel batch_kernel(int cap, int threads, int panel) {
  const bool narrow = panel == 16;
  switch (threads) {
    case 128: return narrow ? batch_kernel_rpt<128, 16>(cap) : batch_kernel_rpt<128, 32>(cap);
    case 512: return narrow ? batch_kernel_rpt<512, 16>(cap) : batch_kernel_rpt<512, 32>(cap);
    default: return narrow ? batch_kernel_rpt<256, 16>(cap) : batch_kernel_rpt<256, 32>(cap);
  }
}

// The launch shape of a bucket when no autotuner chose one. With more systems
// than SMs throughput counts: small CTAs, several to an SM, so that one
// system's column chain runs beside another's update (1 500 systems of order
// 257..512 in FP64: 128 x 16 10.8 ms, 256 x 16 11.3 ms, 512 x 32 11.8 ms; 3 000
// of 129..256: 128 x 16 3.36 ms, 256 x 16 3.45 ms, 256 x 32 4.0 ms; 4 000 of
// 65..128: 128 x 16 0.98 ms, 128 x 32 1.32 ms). The mixed form's longest systems
// prefer the wide panel (128 x 32 11.1 ms, 128 x 16 12.9 ms). A few systems
// run one to an SM: a thread per row and the wide panel's fewer sweeps.
void default_batch_shape(int cap, bool mixed, bool few, int* threads, int* panel) {
  if (few) {
    *threads = std::max(128, std::min(512, cap));
    *panel = 32;
  } else {
    *threads = 128;
    *panel = mixed && cap >= 512 ? 32 : 16;
  }
}

template <int NT>
size_t kernel_smem_nt(int cap, bool mixed, int pb) {
  const size_t g = mixed ? getrf_smem<float, NT>(cap, pb) : getrf_smem<double, NT>(cap, pb);
  return sizeof(double) * (size_t)cap + sizeof(int) * (size_t)((cap + 3) & ~3) +
         std::max(g, sizeof(double) * (size_t)cap) + 64;
}
size_t kernel_smem(int cap, bool mixed, int threads, int pb) {
  switch (threads) {
    case 128: return kernel_smem_nt<128>(cap, mixed, pb);
    case 512: return kernel_smem_nt<512>(cap, mixed, pb);
    default: return kernel_smem_nt<256>(cap, mixed, pb);
  }
}

// Lifts a kernel's shared-memory limit: one limit for every bucket sharing an
// instantiation, the largest any asks for.
cudaError_t allow_smem(BatchKernel k, int threads, int pb) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)std::max(kernel_smem(kMaxN, false, threads, pb), kernel_smem(kMaxN, true, threads, pb)));
}

}  // namespace

int batch_launch_bucket(alg_ctx* ctx, const BatchSpec& sp, const BucketLaunch& bl) {
  BatchArgs p;
  p.count = bl.count;
  p.order = bl.d_order;
  p.n = sp.d_n;
  p.a_off = sp.d_a_off;
  p.b_off = sp.d_b_off;
  p.a = sp.d_a;
  p.b = sp.d_b;
  p.a32 = sp.d_a32;
  p.ipiv = sp.d_ipiv;
  p.work = sp.d_work;
  p.info = sp.d_info;
  p.eta = sp.d_eta;
  p.queue = bl.d_queue;
  p.cap = bl.cap;
  p.mixed = sp.mixed;
  p.max_ir = sp.max_ir > 0 ? sp.max_ir : 10;
  p.tol_scale = sp.tol_scale > 0 ? sp.tol_scale : 10.0;
  ALG_CUDA_TRY(cudaMemsetAsync(bl.d_queue, 0, sizeof(int), ctx->stream));
  const BatchKernel k = batch_kernel(bl.cap, bl.threads, bl.panel);
  k<<<bl.grid, bl.threads, kernel_smem(bl.cap, sp.mixed != 0, bl.threads, bl.panel), ctx->stream>>>(p);
  count_launches();
  ALG_CUDA_TRY(cudaGetLastError());
  return ALG_OK;
}

// Host-side configuration (not stream work, so never inside a graph capture).
int batch_configure_bucket(alg_ctx* ctx, bool mixed, BucketLaunch* bl) {
  if (bl->panel != 16) bl->panel = 32;
  if (bl->threads != 128 && bl->threads != 512) bl->threads = 256;
  const BatchKernel k = batch_kernel(bl->cap, bl->threads, bl->panel);
  ALG_CUDA_TRY(allow_smem(k, bl->threads, bl->panel));
  int per_sm = 0;
  ALG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, bl->threads,
                                                             kernel_smem(bl->cap, mixed, bl->threads, bl->panel)));
  bl->grid = std::max(1, std::min(std::max(1, per_sm) * ctx->sm_count, bl->count));
  return ALG_OK;
}

int batch_max_order() { return kMaxN; }

}  // namespace alg

// ===========================================================================
// Plans and C entry points
// ===========================================================================
struct alg_batch {
  alg_ctx* ctx = nullptr;
  int count = 0;
  int mixed = 0;
  std::vector<int> n;
  std::vector<long long> a_off, b_off;
  long long a_total = 0, b_total = 0;
  double flops = 0.0;
  // device
  int* d_n = nullptr;
  long long* d_a_off = nullptr;
  long long* d_b_off = nullptr;
  int* d_order = nullptr;
  int* d_queues = nullptr;
  int* d_ipiv = nullptr;
  double* d_work = nullptr;
  double* d_eta = nullptr;
  float* d_a32 = nullptr;
  std::vector<alg::BucketLaunch> buckets;
  // captured graph of the launch sequence (for fixed buffers)
  cudaGraphExec_t graph = nullptr;
  cudaStream_t cap_stream = nullptr;  // capture stream (the context's may be the legacy stream)
  double* g_a = nullptr;
  double* g_b = nullptr;
  int* g_info = nullptr;
};

namespace {

// Size buckets (orders): the shared-memory panel of a CTA is sized for the
// largest order of its bucket, so small systems keep many CTAs per SM.
const int kBucketCaps[] = {32, 64, 128, 256, 512};

void free_batch(alg_batch* b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  if (b->cap_stream) cudaStreamDestroy(b->cap_stream);
  for (void* p : {(void*)b->d_n, (void*)b->d_a_off, (void*)b->d_b_off, (void*)b->d_order, (void*)b->d_queues,
                  (void*)b->d_ipiv, (void*)b->d_work, (void*)b->d_eta, (void*)b->d_a32})
    if (p) cudaFree(p);
}

int issue(alg_batch* b, double* d_a, double* d_b, int* d_info) {
  alg::BatchSpec sp;
  sp.count = b->count;
  sp.d_n = b->d_n;
  sp.d_a_off = b->d_a_off;
  sp.d_b_off = b->d_b_off;
  sp.d_a = d_a;
  sp.d_b = d_b;
  sp.d_a32 = b->d_a32;
  sp.d_ipiv = b->d_ipiv;
  sp.d_work = b->d_work;
  sp.d_info = d_info;
  sp.d_eta = b->d_eta;
  sp.mixed = b->mixed;
  sp.flops = b->flops;
  const int tok = alg::prof_begin(b->ctx, ALG_K_BATCH);
  for (const auto& bl : b->buckets) ALG_TRY(alg::batch_launch_bucket(b->ctx, sp, bl));
  alg::prof_end(b->ctx, tok, b->flops, 8.0 * (double)b->a_total);
  return ALG_OK;
}

}  // namespace

extern "C" {

int alg_batch_create(alg_ctx* ctx, int count, const int* n_host, int mixed, alg_batch** out) {
  if (ctx == nullptr || out == nullptr || count < 0 || (count > 0 && n_host == nullptr)) return ALG_INVALID_ARGUMENT;
  for (int i = 0; i < count; ++i)
    if (n_host[i] < 1 || n_host[i] > alg::batch_max_order()) return ALG_BAD_SHAPE;
  auto* b = new alg_batch();
  b->ctx = ctx;
  b->count = count;
  b->mixed = mixed ? 1 : 0;
  b->n.assign(n_host, n_host + count);
  b->a_off.resize(count);
  b->b_off.resize(count);
  for (int i = 0; i < count; ++i) {
    b->a_off[i] = b->a_total;
    b->b_off[i] = b->b_total;
    b->a_total += (long long)b->n[i] * b->n[i];
    b->b_total += b->n[i];
    const double nn = b->n[i];
    b->flops += 2.0 / 3.0 * nn * nn * nn + 2.0 * nn * nn;
  }
  // order: bucket by cap, largest orders first inside each bucket
  std::vector<int> idx(count);
  for (int i = 0; i < count; ++i) idx[i] = i;
  std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) { return b->n[x] > b->n[y]; });
  auto fail = [&](int rc) {
    free_batch(b);
    delete b;
    *out = nullptr;
    return rc;
  };
  auto dmalloc = [&](void** p, size_t bytes) { return cudaMalloc(p, std::max<size_t>(bytes, 16)); };
  if (dmalloc((void**)&b->d_n, sizeof(int) * count) || dmalloc((void**)&b->d_a_off, 8 * (size_t)count) ||
      dmalloc((void**)&b->d_b_off, 8 * (size_t)count) || dmalloc((void**)&b->d_order, sizeof(int) * count) ||
      dmalloc((void**)&b->d_queues, sizeof(int) * 16) || dmalloc((void**)&b->d_ipiv, sizeof(int) * b->b_total) ||
      dmalloc((void**)&b->d_work, sizeof(double) * b->b_total) || dmalloc((void**)&b->d_eta, sizeof(double) * count))
    return fail(ALG_OUT_OF_DEVICE_MEMORY);
  if (b->mixed && dmalloc((void**)&b->d_a32, sizeof(float) * b->a_total)) return fail(ALG_OUT_OF_DEVICE_MEMORY);
  cudaMemcpyAsync(b->d_n, b->n.data(), sizeof(int) * count, cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(b->d_a_off, b->a_off.data(), 8 * (size_t)count, cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(b->d_b_off, b->b_off.data(), 8 * (size_t)count, cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(b->d_order, idx.data(), sizeof(int) * count, cudaMemcpyHostToDevice, ctx->stream);
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return fail(ALG_CUDA_ERROR);
  int pos = 0, qi = 0;
  for (int bi = (int)(sizeof(kBucketCaps) / sizeof(int)) - 1; bi >= 0 && pos < count; --bi) {
    const int lo = bi > 0 ? kBucketCaps[bi - 1] : 0;
    int end = pos;
    while (end < count && b->n[idx[end]] > lo) ++end;
    if (end > pos) {
      alg::BucketLaunch bl;
      bl.count = end - pos;
      bl.cap = kBucketCaps[bi];
      alg::default_batch_shape(bl.cap, b->mixed != 0, bl.count <= ctx->sm_count, &bl.threads, &bl.panel);
      bl.d_order = b->d_order + pos;
      bl.d_queue = b->d_queues + qi++;
      const int rc = alg::batch_configure_bucket(ctx, b->mixed != 0, &bl);
      if (rc != ALG_OK) return fail(rc);
      b->buckets.push_back(bl);
    }
    pos = end;
  }
  *out = b;
  return ALG_OK;
}

int alg_batch_offsets(const alg_batch* b, int64_t* a_off, int64_t* b_off) {
  if (b == nullptr) return ALG_INVALID_ARGUMENT;
  for (int i = 0; i < b->count; ++i) {
    if (a_off) a_off[i] = b->a_off[i];
    if (b_off) b_off[i] = b->b_off[i];
  }
  return ALG_OK;
}

int alg_batch_solve(alg_batch* b, double* d_a, double* d_b, int* d_info) {
  if (b == nullptr || (b->count > 0 && (d_a == nullptr || d_b == nullptr || d_info == nullptr)))
    return ALG_INVALID_ARGUMENT;
  return issue(b, d_a, d_b, d_info);
}

int alg_batch_solve_graph(alg_batch* b, double* d_a, double* d_b, int* d_info) {
  if (b == nullptr || (b->count > 0 && (d_a == nullptr || d_b == nullptr || d_info == nullptr)))
    return ALG_INVALID_ARGUMENT;
  alg_ctx* ctx = b->ctx;
  if (b->graph == nullptr || b->g_a != d_a || b->g_b != d_b || b->g_info != d_info) {
    if (b->graph) {
      cudaGraphExecDestroy(b->graph);
      b->graph = nullptr;
    }
    // configure the kernels outside the capture (attributes are not stream work)
    ALG_TRY(issue(b, d_a, d_b, d_info));
    ALG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    if (b->cap_stream == nullptr) ALG_CUDA_TRY(cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    // capture on the plan's own stream, issuing through the context meanwhile
    cudaStream_t saved = ctx->stream;
    ctx->stream = b->cap_stream;
    const bool prof = ctx->prof_on;
    ctx->prof_on = false;
    cudaError_t e = cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeThreadLocal);
    int rc = e == cudaSuccess ? issue(b, d_a, d_b, d_info) : ALG_CUDA_ERROR;
    if (e == cudaSuccess) e = cudaStreamEndCapture(b->cap_stream, &g);
    ctx->prof_on = prof;
    ctx->stream = saved;
    if (rc != ALG_OK) return rc;
    ALG_CUDA_TRY(e);
    ALG_CUDA_TRY(cudaGraphInstantiate(&b->graph, g, 0));
    cudaGraphDestroy(g);
    b->g_a = d_a;
    b->g_b = d_b;
    b->g_info = d_info;
    return ALG_OK;  // the warm-up issue above already solved this batch
  }
  const int tok = alg::prof_begin(ctx, ALG_K_BATCH);
  ALG_CUDA_TRY(cudaGraphLaunch(b->graph, ctx->stream));
  alg::count_launches(b->buckets.size());
  alg::prof_end(ctx, tok, b->flops, 8.0 * (double)b->a_total);
  return ALG_OK;
}

// Tries every launch shape for each bucket on the given batch (which it
// solves several times: pass scratch copies) and keeps the fastest: 128 / 256
// / 512 threads per CTA times a 16- or 32-column panel (the split between the
// column-serial panel and the tiled update).
int alg_batch_autotune(alg_batch* b, double* d_a, double* d_b, int* d_info, const double* d_a_src,
                       const double* d_b_src, int* threads_out) {
  if (b == nullptr) return ALG_INVALID_ARGUMENT;
  alg_ctx* ctx = b->ctx;
  cudaEvent_t e0, e1;
  ALG_CUDA_TRY(cudaEventCreate(&e0));
  ALG_CUDA_TRY(cudaEventCreate(&e1));
  alg::BatchSpec sp;
  sp.count = b->count;
  sp.d_n = b->d_n;
  sp.d_a_off = b->d_a_off;
  sp.d_b_off = b->d_b_off;
  sp.d_a = d_a;
  sp.d_b = d_b;
  sp.d_a32 = b->d_a32;
  sp.d_ipiv = b->d_ipiv;
  sp.d_work = b->d_work;
  sp.d_info = d_info;
  sp.d_eta = b->d_eta;
  sp.mixed = b->mixed;
  for (size_t k = 0; k < b->buckets.size(); ++k) {
    auto& bl = b->buckets[k];
    float best = 1e30f;
    int best_t = bl.threads, best_p = bl.panel;
    for (int cfg = 0; cfg < 6; ++cfg) {
      const int t = 128 << (cfg >> 1), pb = (cfg & 1) ? 32 : 16;
      alg::BucketLaunch trial = bl;
      trial.threads = t;
      trial.panel = pb;
      ALG_TRY(alg::batch_configure_bucket(ctx, b->mixed != 0, &trial));
      for (int rep = 0; rep < 2; ++rep) {
        ALG_CUDA_TRY(cudaMemcpyAsync(d_a, d_a_src, 8 * (size_t)b->a_total, cudaMemcpyDeviceToDevice, ctx->stream));
        ALG_CUDA_TRY(cudaMemcpyAsync(d_b, d_b_src, 8 * (size_t)b->b_total, cudaMemcpyDeviceToDevice, ctx->stream));
        ALG_CUDA_TRY(cudaEventRecord(e0, ctx->stream));
        ALG_TRY(alg::batch_launch_bucket(ctx, sp, trial));
        ALG_CUDA_TRY(cudaEventRecord(e1, ctx->stream));
        ALG_CUDA_TRY(cudaEventSynchronize(e1));
        float ms = 0.f;
        ALG_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
        if (rep == 1 && ms < best) {
          best = ms;
          best_t = t;
          best_p = pb;
        }
      }
    }
    bl.threads = best_t;
    bl.panel = best_p;
    ALG_TRY(alg::batch_configure_bucket(ctx, b->mixed != 0, &bl));
    if (threads_out) threads_out[k] = best_t;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (b->graph) {
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
  }
  return ALG_OK;
}

int alg_batch_info(const alg_batch* b, int* n_buckets, int* caps, int* threads, int* counts, double* flops) {
  if (b == nullptr) return ALG_INVALID_ARGUMENT;
  if (n_buckets) *n_buckets = (int)b->buckets.size();
  for (size_t k = 0; k < b->buckets.size(); ++k) {
    if (caps) caps[k] = b->buckets[k].cap;
    if (threads) threads[k] = b->buckets[k].threads;
    if (counts) counts[k] = b->buckets[k].count;
  }
  if (flops) *flops = b->flops;
  return ALG_OK;
}

int alg_batch_panels(const alg_batch* b, int* panels) {
  if (b == nullptr || panels == nullptr) return ALG_INVALID_ARGUMENT;
  for (size_t k = 0; k < b->buckets.size(); ++k) panels[k] = b->buckets[k].panel;
  return ALG_OK;
}

int alg_batch_set_config(alg_batch* b, int bucket, int threads, int panel) {
  if (b == nullptr || bucket < 0 || bucket >= (int)b->buckets.size()) return ALG_INVALID_ARGUMENT;
  if ((threads != 128 && threads != 256 && threads != 512) || (panel != 16 && panel != 32))
    return ALG_INVALID_ARGUMENT;
  alg::BucketLaunch& bl = b->buckets[bucket];
  bl.threads = threads;
  bl.panel = panel;
  ALG_TRY(alg::batch_configure_bucket(b->ctx, b->mixed != 0, &bl));
  if (b->graph) {  // the captured launches used the old shape
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
  }
  return ALG_OK;
}

int alg_batch_eta(const alg_batch* b, double* eta_host) {
  if (b == nullptr || eta_host == nullptr) return ALG_INVALID_ARGUMENT;
  ALG_CUDA_TRY(cudaMemcpy(eta_host, b->d_eta, sizeof(double) * b->count, cudaMemcpyDeviceToHost));
  return ALG_OK;
}

int alg_batch_ipiv(const alg_batch* b, int* ipiv_host) {
  if (b == nullptr || ipiv_host == nullptr) return ALG_INVALID_ARGUMENT;
  if (b->b_total == 0) return ALG_OK;
  ALG_CUDA_TRY(cudaMemcpy(ipiv_host, b->d_ipiv, sizeof(int) * b->b_total, cudaMemcpyDeviceToHost));
  return ALG_OK;
}

// Frees the plan's device buffers (cudaFree waits for work that uses them).
// Does not touch the context, which the caller may already have destroyed.
void alg_batch_destroy(alg_batch* b) {
  if (b == nullptr) return;
  free_batch(b);
  delete b;
}

}  // extern "C"

// ===========================================================================
// Allocation-free solve of one small system (no counterpart in the reference)
// ===========================================================================
// Some callers cannot call cudaMalloc: code running inside another library's
// memory pool that owns the device's free memory, serving loops where the
// implicit device-wide synchronisation of cudaMalloc/cudaFree would stall
// unrelated streams, and callers that must never fail with out-of-memory after
// start-up. alg_dgesv_mixed_noalloc serves them: it runs the mixed form of the
// batched kernel above (FP32 LU with partial pivoting, FP64 refinement) on
// one system, and takes its working memory (the FP32 copy of A, the residual
// vector, the work counter) from the file-scope array below instead of from
// an allocation. Set-up per device (the array's address, the kernels' load
// and the shared-memory limit) is host-side work done by the first call in
// each CUDA context; a call with n = 0 does only the set-up. Every call on a
// device shares the one array, so calls that overlap on the GPU (different
// streams, or different host threads) race on it; calls on one stream are
// ordered and safe.
namespace alg {
namespace {

constexpr int kNoAllocMaxN = 512;
// Layout: FP32 copy of A (max order squared), residual (max order doubles),
// pivots (max order ints), then a 256-byte header of per-call fields.
constexpr size_t kNoAllocA32 = sizeof(float) * (size_t)kNoAllocMaxN * kNoAllocMaxN;
constexpr size_t kNoAllocWork = sizeof(double) * kNoAllocMaxN;
constexpr size_t kNoAllocIpiv = sizeof(int) * kNoAllocMaxN;
constexpr size_t kNoAllocHeader = 256;
constexpr size_t kNoAllocBytes = kNoAllocA32 + kNoAllocWork + kNoAllocIpiv + kNoAllocHeader;
static_assert(kNoAllocBytes == 1054976, "scratch size is part of the C interface");

struct NoAllocHeader {
  long long a_off;  // offset of the system in A, b, pivots and the FP32 copy (always 0)
  long long b_off;
  int queue;        // work counter of the persistent kernel: must be 0 when it starts
  int order;        // queue position -> system (always 0)
  int n;            // the system's order
  int info;         // spare slot (the caller's info pointer is required)
  double eta;       // used when the caller passes no backward-error pointer
};
static_assert(sizeof(NoAllocHeader) <= kNoAllocHeader, "header fits its slot");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Writes the per-call header, in stream order before the solve kernel; this
// is what resets the work counter to 0 for each call.
__global__ void noalloc_header_kernel(NoAllocHeader* h, int n) {
  h->a_off = 0;
  h->b_off = 0;
  h->queue = 0;
  h->order = 0;
  h->n = n;
  h->info = 0;
  h->eta = 0.0;
}

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
// Per device: the array's address and the unique id (cuCtxGetId) of the CUDA
// context it was looked up in. A __device__ symbol's address belongs to one
// context; after cudaDeviceReset, or when the caller makes another context
// current, the id differs and the set-up runs again.
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};
unsigned long long g_noalloc_ctx[kNoAllocMaxDevices] = {};

// The two driver calls are reached through the runtime's entry-point table,
// so the library does not link libcuda (it stays loadable on hosts without
// a driver, where every call reports ALG_NO_DEVICE).
int current_context_id(unsigned long long* id) {
  static PFN_cuCtxGetCurrent_v4000 get_current = nullptr;
  static PFN_cuCtxGetId_v12000 get_id = nullptr;
  if (get_current == nullptr || get_id == nullptr) {
    cudaDriverEntryPointQueryResult q1, q2;
    void* f1 = nullptr;
    void* f2 = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1) != cudaSuccess ||
        cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2) != cudaSuccess ||
        q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2) {
      cudaGetLastError();
      return ALG_CUDA_ERROR;
    }
    get_current = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(f1);
    get_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(f2);
  }
  CUcontext c = nullptr;
  if (get_current(&c) != CUDA_SUCCESS || c == nullptr) return ALG_CUDA_ERROR;
  if (get_id(c, id) != CUDA_SUCCESS) return ALG_CUDA_ERROR;
  return ALG_OK;
}

// Set-up (host side, not stream work), with `dev` current. cudaGetSymbolAddress
// loads this file's module if lazy loading (the CUDA 12 default) has not
// yet, which is when the static array comes into being on the device; the
// kernels are loaded here too (cudaFuncGetAttributes / cudaFuncSetAttribute),
// so no later call loads code or data.
int noalloc_setup(int dev, unsigned char** out) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  unsigned long long id = 0;
  if (g_noalloc_ptr[dev] == nullptr || current_context_id(&id) != ALG_OK || id != g_noalloc_ctx[dev]) {
    void* p = nullptr;
    ALG_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));  // also makes the primary context current
    ALG_TRY(current_context_id(&id));
    cudaFuncAttributes fa;
    ALG_CUDA_TRY(cudaFuncGetAttributes(&fa, noalloc_header_kernel));
    for (int cap = 32; cap <= kNoAllocMaxN; cap *= 2) {
      int threads, panel;
      default_batch_shape(cap, true, true, &threads, &panel);
      ALG_CUDA_TRY(allow_smem(batch_kernel(cap, threads, panel), threads, panel));
    }
    g_noalloc_ptr[dev] = p;
    g_noalloc_ctx[dev] = id;
  }
  *out = static_cast<unsigned char*>(g_noalloc_ptr[dev]);
  return ALG_OK;
}

}  // namespace
}  // namespace alg

extern "C" int alg_dgesv_mixed_noalloc(void* stream, const double* d_a, double* d_b, int n, int* d_ipiv,
                                       int* d_info, double* d_eta) {
  using namespace alg;
  if (n < 0 || n > kNoAllocMaxN) {
    if (std::getenv("ALG_VERBOSE"))
      std::fprintf(stderr, "alg_dgesv_mixed_noalloc: order %d outside 0..%d (the size of its static scratch)\n", n,
                   kNoAllocMaxN);
    return ALG_BAD_SHAPE;
  }
  if (n > 0 && (d_a == nullptr || d_b == nullptr || d_info == nullptr)) return ALG_INVALID_ARGUMENT;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return ALG_NO_DEVICE;
  }
  int dev = 0;
  ALG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return ALG_INVALID_ARGUMENT;
  unsigned char* base = nullptr;
  ALG_TRY(noalloc_setup(dev, &base));
  if (n == 0) return ALG_OK;  // the set-up call: nothing is queued
  auto* hdr = reinterpret_cast<NoAllocHeader*>(base + kNoAllocA32 + kNoAllocWork + kNoAllocIpiv);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the size bucket and CTA size a one-system plan of this order uses
  int cap = 32;
  while (cap < n) cap *= 2;
  int threads, panel;
  default_batch_shape(cap, true, true, &threads, &panel);
  BatchArgs p;
  p.count = 1;
  p.order = &hdr->order;
  p.n = &hdr->n;
  p.a_off = &hdr->a_off;
  p.b_off = &hdr->b_off;
  p.a = const_cast<double*>(d_a);  // the mixed form only reads A
  p.b = d_b;
  p.a32 = reinterpret_cast<float*>(base);
  p.ipiv = d_ipiv ? d_ipiv : reinterpret_cast<int*>(base + kNoAllocA32 + kNoAllocWork);
  p.work = reinterpret_cast<double*>(base + kNoAllocA32);
  p.info = d_info;
  p.eta = d_eta ? d_eta : &hdr->eta;
  p.queue = &hdr->queue;
  p.cap = cap;
  p.mixed = 1;
  p.max_ir = 10;
  p.tol_scale = 10.0;
  noalloc_header_kernel<<<1, 1, 0, s>>>(hdr, n);
  count_launches();
  ALG_CUDA_TRY(cudaGetLastError());
  batch_kernel(cap, threads, panel)<<<1, threads, kernel_smem(cap, true, threads, panel), s>>>(p);
  count_launches();
  ALG_CUDA_TRY(cudaGetLastError());
  return ALG_OK;
}
