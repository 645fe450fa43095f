// Pivot search and division shared by the panel LU kernels (dense blocks,
// batched systems, sparse small fronts).
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "common.cuh"

namespace alg {

template <typename T>
__device__ __forceinline__ bool div_fast_ok(T x) {
  const double ax = fabs(static_cast<double>(x));
  if constexpr (sizeof(T) == 8) {
    return ax >= 0x1p-500 && ax <= 0x1p500;
  } else {
    return ax >= 0x1p-60f && ax <= 0x1p60f;
  }
}
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// a / d correctly rounded; y = RN(1/d), fast = d passed div_fast_ok.
template <typename T>
__device__ __forceinline__ T quotient(T a, T d, T y, bool fast) {
  if (fast && div_fast_ok(a)) {
    const T q = mul_rn(a, y);
    const T r = fma_rn(-q, d, a);
    return fma_rn(r, y, q);
  }
  return div_rn(a, d);
}

// A pivot candidate: |v|'s bits as an ordered integer and the row's position;
// (0, INT_MAX) is no candidate (a zero entry is (0, its position), which wins
// over it). The reference's NaN rule (mod.rs:123-134): +inf on the diagonal,
// never chosen elsewhere.
template <bool DIAG_NAN = true>
__device__ __forceinline__ void pivot_candidate(double v, int pos, int J, unsigned long long& key, int& kpos) {
  key = pos >= J ? (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull : 0ull;
  kpos = pos >= J ? pos : INT_MAX;
  if (v != v) {
    key = DIAG_NAN && pos == J ? 0x7ff0000000000000ull : 0ull;
    kpos = DIAG_NAN && pos == J ? J : INT_MAX;
  }
}
template <bool DIAG_NAN = true>
__device__ __forceinline__ void pivot_candidate(float v, int pos, int J, unsigned& key, int& kpos) {
  key = pos >= J ? __float_as_uint(v) & 0x7fffffffu : 0u;
  kpos = pos >= J ? pos : INT_MAX;
  if (v != v) {
    key = DIAG_NAN && pos == J ? 0x7f800000u : 0u;
    kpos = DIAG_NAN && pos == J ? J : INT_MAX;
  }
}
// Warp-wide: the largest key, and among its lanes the smallest tag; true on
// the lanes that hold both.
__device__ __forceinline__ bool warp_pivot(unsigned long long key, int tag, unsigned long long& mk, int& mt) {
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)key : 0u);
  const bool eq = hi == mh && (unsigned)key == ml;
  mt = __reduce_min_sync(0xffffffffu, eq ? tag : INT_MAX);
  mk = ((unsigned long long)mh << 32) | ml;
  return eq && tag == mt;
}
__device__ __forceinline__ bool warp_pivot(unsigned key, int tag, unsigned& mk, int& mt) {
  mk = __reduce_max_sync(0xffffffffu, key);
  const bool eq = key == mk;
  mt = __reduce_min_sync(0xffffffffu, eq ? tag : INT_MAX);
  return eq && tag == mt;
}
// div_fast_ok on the exponent bits (also false for zero, infinity and NaN)
__device__ __forceinline__ bool exp_fast_ok(double v) {
  const unsigned e = ((unsigned)__double2hiint(v) >> 20) & 0x7ffu;
  return e - (1023u - 500u) < 1000u;  // [2^-500, 2^500)
}
__device__ __forceinline__ bool exp_fast_ok(float v) {
  const unsigned e = (__float_as_uint(v) >> 23) & 0xffu;
  return e - (127u - 60u) < 120u;  // [2^-60, 2^60)
}
// A pivot record, in 16-byte chunks: (key; position and the row's slot in its
// CTA), (reciprocal, unused), then the leaf's row, rotated as in registers.
template <typename T, int W>
struct alignas(16) PivotRec {
  using Key = std::conditional_t<sizeof(T) == 8, unsigned long long, unsigned>;
  unsigned long long key;
  unsigned pos, slot;
  T recip;
  alignas(16) T row[W];
  static constexpr int kChunks = 2 + W * (int)sizeof(T) / 16;
};

// The same over the records rec[0 .. count) (one lane each): the winner's
// index; its position in mp. Positions are below 2^20 (longer panels take
// another kernel), so position and index share one reduction.
template <typename Rec>
__device__ __forceinline__ int warp_pick(const Rec* rec, int count, int lane, int& mp) {
  typename Rec::Key k = 0, mk;
  int t = INT_MAX, mt;
  if (lane < count) {
    const ulonglong2 h = *reinterpret_cast<const ulonglong2*>(&rec[lane]);  // key; position and slot
    k = (typename Rec::Key)h.x;
    const unsigned pos = (unsigned)h.y;
    t = pos < (1u << 20) ? (int)(pos << 5 | (unsigned)lane) : INT_MAX - 31 + lane;
  }
  warp_pivot(k, t, mk, mt);
  mp = mt >> 5;
  return mt & 31;
}

// A barrier of the CTA's NT threads that its warps may reach at different places
// in the code (__syncthreads must be met at one place by all of them). Each warp
// comes to it whole; the form for warps that may not cost 1 % of a small front
// of 192 columns (649 us the call with this one, 656 with that).
template <int NT>
__device__ __forceinline__ void cta_barrier() {
  asm volatile("barrier.sync.aligned 1, %0;" ::"n"(NT) : "memory");
}

// One leaf of an LU by one CTA: columns [cl0, cl0 + w) (w <= W) of the m rows
// in tile[col][row] (column stride ldt), rows tid + k NT of it by this thread
// (m <= NT * RPT), pos[k] the row's position (-1: no row). The column chain
// of panel_reg_kernel without the exchange between CTAs: rows never move, the
// rank-1 update writes entry c into c - 1 so the pivot column is always entry
// 0, and finished entries go back to the tile, each row in its own slot.
// piv_slot[J] receives the slot of column J's pivot row and ipiv[J] its
// position at that step. RECIP: multipliers by the reciprocal (else the
// correctly rounded quotient, see panel_reg_kernel).
// With RECIP a NaN is never chosen, on the diagonal either (lu_front's rule).
// Warps without rows (late panels of a CTA sized for the first) only keep the
// barriers. Returns the first column of the leaf whose pivot is zero (INT_MAX:
// none); with RECIP the leaf stops there (a column without any number counts
// as zero). No barrier after the last column: the caller's follows.
// Not inlined: its registers are then allocated by themselves (inlined into
// a kernel with other phases, its loop spilled).
template <typename T, int W, int NT, int RPT, bool EXACT, bool RECIP>
__device__ __noinline__ int cta_leaf(T* tile, int ldt, int m, int cl0, int w, int* pos_io,
                                     PivotRec<T, W> (*rec)[NT / 32], int* piv_slot, int* ipiv) {
  using Key = typename PivotRec<T, W>::Key;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = min(NT / 32, (m + 31) / 32);  // warps with rows
  int zero = INT_MAX, mp;
  if (warp >= nw) {
#pragma unroll 1
    for (int j = 0; j < w; ++j) {
      cta_barrier<NT>();
      const int par = (cl0 + j) & 1;
      const T d = rec[par][warp_pick(&rec[par][0], nw, lane, mp)].row[0];
      if (RECIP) {
        if (!(fabs((double)d) > 0.0) || mp >= (1 << 20)) return cl0 + j;
      } else if (d == T(0) && zero == INT_MAX) {
        zero = cl0 + j;
      }
    }
    return zero;
  }
  int pos[RPT];
  T v[RPT][W];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int r = tid + k * NT;
    pos[k] = pos_io[k];
#pragma unroll
    for (int c = 0; c < W; ++c) v[k][c] = (c < w && r < m) ? tile[(cl0 + c) * ldt + r] : T(0);
  }
#pragma unroll 1
  for (int j = 0; j < w; ++j) {
    const int J = cl0 + j;
    const int par = J & 1;
    Key key, mk;
    int kpos, kslot = tid;
    T cand = v[0][0];
    pivot_candidate<!RECIP>(v[0][0], pos[0], J, key, kpos);
#pragma unroll
    for (int k = 1; k < RPT; ++k) {
      Key kk;
      int kp;
      pivot_candidate<!RECIP>(v[k][0], pos[k], J, kk, kp);
      if (kk > key || (kk == key && kp < kpos)) {
        key = kk;
        kpos = kp;
        kslot = tid + k * NT;
        cand = v[k][0];
      }
    }
    const T crecip = rcp_rn(RECIP || exp_fast_ok(cand) ? cand : T(1));
    if (warp_pivot(key, kpos, mk, mp)) {  // (no candidate at all: any lanes, an empty record)
      PivotRec<T, W>& s = rec[par][warp];
      s.key = mk;
      s.pos = (unsigned)mp;
      s.slot = kslot;
      s.recip = crecip;
#pragma unroll
      for (int k = 0; k < RPT; ++k)
        if (RPT == 1 || kslot == tid + k * NT) {
#pragma unroll
          for (int c = 0; c < W; ++c) s.row[c] = v[k][c];
        }
    }
    cta_barrier<NT>();
    const int win = warp_pick(&rec[par][0], nw, lane, mp);
    const PivotRec<T, W>& wr = rec[par][win];
    const T d = wr.row[0];
    const T y = wr.recip;
    if (RECIP) {
      if (!(fabs((double)d) > 0.0) || mp >= (1 << 20)) return J;  // uniform
    } else if (d == T(0) && zero == INT_MAX) {
      zero = J;
    }
    if (warp == (j % nw)) {  // one warp files the pivot row
      const int slot = (int)wr.slot;
      if (lane < w - j) tile[(J + lane) * ldt + slot] = wr.row[lane];
      if (lane == 0) {
        piv_slot[J] = slot;
        ipiv[J] = mp;
      }
    }
    const bool fast = exp_fast_ok(d);
    T l[RPT];
    bool odd = false;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      if (pos[k] == mp) pos[k] = J;
      else if (pos[k] == J) pos[k] = mp;
      const T av = v[k][0];
      if (RECIP) {
        l[k] = mul_rn(av, y);
      } else {
        const T qv = mul_rn(av, y);
        l[k] = fma_rn(fma_rn(-qv, d, av), y, qv);
        odd |= !(fast && exp_fast_ok(av)) && pos[k] > J;
      }
    }
    if (!RECIP && odd) {  // zeros; rarely the plain IEEE division
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const T av = v[k][0];
        if (!(fast && exp_fast_ok(av))) l[k] = (fast && av == T(0)) ? mul_rn(av, y) : div_rn(av, d);
      }
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (pos[k] > J) tile[J * ldt + tid + k * NT] = l[k];
    // (entries past the leaf's live columns, and rows that have left, hold
    // values that nothing reads)
#pragma unroll
    for (int c = 1; c < W; ++c) {
      const T u = wr.row[c];
#pragma unroll
      for (int k = 0; k < RPT; ++k) v[k][c - 1] = msub<EXACT>(v[k][c], l[k], u);
    }
  }
#pragma unroll
  for (int k = 0; k < RPT; ++k) pos_io[k] = pos[k];
  return zero;
}

}  // namespace alg
