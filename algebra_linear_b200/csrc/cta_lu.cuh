// Pieces of an LU by one CTA (batched systems, sparse small fronts): the panel's
// shared-memory layout, the chunks of columns right of it, their unit-lower
// solve and the tiled update.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "pivot.cuh"

namespace alg {

constexpr int kLeafW = 16;    // columns a leaf keeps in registers

template <typename T>
__device__ __forceinline__ T fma_t(T a, T b, T c);
template <>
__device__ __forceinline__ double fma_t<double>(double a, double b, double c) { return __fma_rn(a, b, c); }
template <>
__device__ __forceinline__ float fma_t<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Column strides in shared memory: 4 mod 16 entries, so that a half-warp's
// DMMA fragment loads (4 k x 4 rows or columns) fall in distinct banks.
__host__ __device__ constexpr int panel_ld(int cap) { return ((cap + 15) & ~15) + 4; }

// A chunk's row stride is odd in FP64: its columns arrive 32 k at a time
// (cp.async, a row of U each), and an even stride made those stores 8-way
// bank conflicts; the FP32 tiles need rows of whole 16 bytes.
template <typename T>
__host__ __device__ constexpr int chunk_ld(int cols) {
  return cols + (sizeof(T) == 8 ? 5 : 4);
}
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// An entry copied asynchronously from global to shared memory.
template <typename T>
__device__ __forceinline__ void cp_async_entry(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "n"(sizeof(T))
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// A 32 x 16 tile at (r0, c0) of C (mt x cw) -= L U held by one warp: L[k][row]
// (stride ldl) and U[k][col] (stride ldu) in shared memory, C global (leading
// dimension n). The K products are summed from zero, in increasing k, each one
// fused multiply-add, and the sum is subtracted from C once: accumulated into
// C, every product would be rounded at C's size (a front's contribution block
// under a dominant diagonal is much larger than its products): error of the
// sparse solution, geometric mean over 2-D and 3-D grids of 1 600 to 90 000
// unknowns, 1.27 times larger in FP64, 1.29 times in unrefined FP32, twice as
// large after refinement.
// Rows and columns past the edge read padding and are not stored.
struct TileF64 {  // FP64 tensor cores
  double c[4][2][2];
  __device__ __forceinline__ void load(const double* C, int n, int r0, int c0, int mt, int cw) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cc = c0 + 8 * j + 2 * t + e;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = r0 + 8 * i + g;
          c[i][j][e] = (cc < cw && r < mt) ? C[cc * n + r] : 0.0;
        }
      }
  }
  template <int K, bool ALIGNED>
  __device__ __forceinline__ void update(const double* L, int ldl, const double* U, int ldu, int r0, int c0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
    for (int k = 0; k < K; k += 4) {
      double av[4], bv[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = L[(k + t) * ldl + r0 + 8 * i + g];
#pragma unroll
      for (int j = 0; j < 2; ++j) bv[j] = U[(k + t) * ldu + c0 + 8 * j + g];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) dmma(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) c[i][j][e] -= acc[i][j][e];
  }
  __device__ __forceinline__ void store(double* C, int n, int r0, int c0, int mt, int cw) const {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cc = c0 + 8 * j + 2 * t + e;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = r0 + 8 * i + g;
          if (cc < cw && r < mt) C[cc * n + r] = c[i][j][e];
        }
      }
  }
};
struct TileF32 {  // CUDA cores; a lane has rows 4 rg .. 4 rg + 3 and columns 4 cg .. 4 cg + 3
  float c[4][4];
  __device__ __forceinline__ void load(const float* C, int n, int r0, int c0, int mt, int cw) {
    const int lane = threadIdx.x & 31, rg = lane & 7, cg = lane >> 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = c0 + 4 * cg + j;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + 4 * rg + i;
        c[i][j] = (cc < cw && r < mt) ? C[cc * n + r] : 0.f;
      }
    }
  }
  template <int K, bool ALIGNED>
  __device__ __forceinline__ void update(const float* L, int ldl, const float* U, int ldu, int r0, int c0) {
    const int lane = threadIdx.x & 31, rg = lane & 7, cg = lane >> 3;
    float acc[4][4] = {};
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
      const float* lp = L + k * ldl + r0 + 4 * rg;
      const float4 u = *reinterpret_cast<const float4*>(U + k * ldu + c0 + 4 * cg);
      const float uv[4] = {u.x, u.y, u.z, u.w};
      float lv[4];
      if constexpr (ALIGNED) {
        const float4 l = *reinterpret_cast<const float4*>(lp);
        lv[0] = l.x, lv[1] = l.y, lv[2] = l.z, lv[3] = l.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) lv[i] = lp[i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][j] = __fmaf_rn(lv[i], uv[j], acc[i][j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) c[i][j] -= acc[i][j];
  }
  __device__ __forceinline__ void store(float* C, int n, int r0, int c0, int mt, int cw) const {
    const int lane = threadIdx.x & 31, rg = lane & 7, cg = lane >> 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = c0 + 4 * cg + j;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + 4 * rg + i;
        if (cc < cw && r < mt) C[cc * n + r] = c[i][j];
      }
    }
  }
};

// All tiles of C (mt x cw) -= L U, dealt to the CTA's NW warps (ALIGNED: L
// starts on 16 bytes; U always does). A tile's C is asked for before its products
// are summed and needed after them, which hides the round trip to L2. AHEAD: a
// warp loads its next tile's C while it updates one, for matrices that come from
// HBM (1 500 FP64 systems of order 257..512: 10.8 ms with it, 11.3 without);
// elsewhere the second tile's registers cost more (3 000 of 129..256: 4.4 ms with
// it, 3.4 without; FP64 small fronts of the 300 x 300 grid 11.5 and 9.4 ms, FP32
// 8.4 and 8.0). Accumulated into C, with the next tile ahead: 11.2, 4.3, 11.2, 8.8.
template <int K, int NW, bool ALIGNED, bool AHEAD, typename T>
__device__ __noinline__ void cta_update(const T* L, int ldl, const T* U, int ldu, T* C, int n, int mt, int cw) {
  using Tile = std::conditional_t<sizeof(T) == 8, TileF64, TileF32>;
  const int tr = (mt + 31) / 32, tiles = tr * ((cw + 15) / 16);
  int cur = threadIdx.x >> 5;
  if constexpr (!AHEAD) {
    for (; cur < tiles; cur += NW) {
      Tile t;
      const int r0 = 32 * (cur % tr), c0 = 16 * (cur / tr);
      t.load(C, n, r0, c0, mt, cw);
      t.template update<K, ALIGNED>(L, ldl, U, ldu, r0, c0);
      t.store(C, n, r0, c0, mt, cw);
    }
    return;
  }
  if (cur >= tiles) return;
  Tile t0, t1;
  int r0 = 32 * (cur % tr), c0 = 16 * (cur / tr), r1 = 0, c1 = 0;
  t0.load(C, n, r0, c0, mt, cw);
  for (;;) {
    if ((cur += NW) < tiles) {
      r1 = 32 * (cur % tr), c1 = 16 * (cur / tr);
      t1.load(C, n, r1, c1, mt, cw);
    }
    t0.template update<K, ALIGNED>(L, ldl, U, ldu, r0, c0);
    t0.store(C, n, r0, c0, mt, cw);
    if (cur >= tiles) return;
    if ((cur += NW) < tiles) {
      r0 = 32 * (cur % tr), c0 = 16 * (cur / tr);
      t0.load(C, n, r0, c0, mt, cw);
    }
    t1.template update<K, ALIGNED>(L, ldl, U, ldu, r1, c1);
    t1.store(C, n, r1, c1, mt, cw);
    if (cur >= tiles) return;
  }
}

// x <- L^{-1} x for 16 entries x[i] = xs[i * lds]; L unit lower, entry (i, k)
// at l[k * ldl + i].
template <typename T>
__device__ __noinline__ void solve16(const T* l, int ldl, T* xs, int lds, int w) {
  T x[kLeafW];
#pragma unroll
  for (int i = 0; i < kLeafW; ++i) x[i] = i < w ? xs[i * lds] : T(0);
#pragma unroll
  for (int k = 0; k < kLeafW - 1; ++k)
#pragma unroll
    for (int i = k + 1; i < kLeafW; ++i) x[i] = fma_t<T>(-l[k * ldl + i], x[k], x[i]);
#pragma unroll
  for (int i = 0; i < kLeafW; ++i)
    if (i < w) xs[i * lds] = x[i];
}

}  // namespace alg
