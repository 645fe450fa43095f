// Kernels of the blocked right-looking LU with partial pivoting.
//
// Reference algorithm: lapack::dgetrf_with_pivots (src/lapack/mod.rs:112-163),
// an unblocked kij loop. The blocked schedule below gives every matrix entry
// exactly the same sequence of operations as that loop — the rank-1 terms
// `a_ij -= l_ik * u_kj` in increasing k, multipliers by true division, rows
// swapped before they are used — so with EXACT = true the factors are
// bit-identical to the reference; only the order in which *different* entries
// are processed changes.
//
// Layout: column-major, leading dimension lda, as the reference stores it.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "common.cuh"
#include "index_guard.h"
#include "pivot.cuh"

namespace alg {
namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------
// K1: leaf panel LU on one thread-block cluster.
//
// Factors the (m - c0) x w leaf panel whose top-left entry is (c0, c0). Its
// rows are split into C contiguous slabs, one per CTA of the cluster, held in
// shared memory for the whole panel (W = 16 or 32 columns, padded stride).
// Thread (g, c) of a CTA owns column c of the slab rows g, g+G, g+2G, ...
//
// Pivot exchange without cluster barriers: for column j every CTA sends a
// record — its candidate (first index of max |a_ij| with the reference's NaN
// rule, mod.rs:123-134), a copy of that row and its labels — into the
// mailbox of every CTA of the cluster with st.async DSMEM stores that count
// their bytes on the receiver's mbarrier; the owner of row j also sends a
// copy of row j. A CTA waits on its own mbarrier only, and every warp reduces
// the C records redundantly to the same winner. Mailboxes and mbarriers are
// double-buffered by column parity; a sender can only reach column j+2 after
// every CTA has consumed column j (it needs their column j+1 records), so a
// buffer is never overwritten while it is read.
//
// Per column j, after the exchange: swap rows j and p (mod.rs:141-146),
// divide the rows below by the pivot (true division, mod.rs:153-155), apply
// the rank-1 update (mod.rs:156-158) and scan column j+1 for the next
// candidate. Rows carry two labels through the swaps: the original row within
// the enclosing block-panel (for the deferred interchange of the matrix's
// other columns) and within this leaf (for the block-panel's other columns,
// which this kernel swaps itself before it exits).
// ---------------------------------------------------------------------------
template <typename T>
struct PanelArgs {
  T* a;
  int lda;
  int n;           // rows of the matrix
  int c0;          // first row and column of the leaf
  int w;           // leaf width (<= W)
  int kb0, kb1;    // columns of the enclosing block-panel
  int* ipiv;       // global interchanges (0-based global rows)
  int* lab;        // cumulative source labels of rows [kb0, n)
  int first_leaf;  // labels start as the identity
  DevStatus* status;
};

constexpr int kPanelThreads = 512;
constexpr int kPanelWarps = kPanelThreads / 32;
constexpr int kPanelMaxW = 32;
constexpr int kPanelMaxC = 16;
constexpr int kSideCols = 16;  // block-panel columns swapped per pass at exit

// One mailbox record, in 8-byte words: key, (row, cumulative label),
// (leaf label, unused), then the row's W entries.
template <typename T, int W>
struct PanelRec {
  static constexpr int kRowWords = (W * (int)sizeof(T)) / 8;
  static constexpr int kWords = (3 + kRowWords + 1) & ~1;     // padded to 16 bytes
  static constexpr int kBytes = 8 * kWords;
  static constexpr int kDiagWords = (1 + kRowWords + 1) & ~1;  // (cumulative, leaf label), row
  static constexpr int kDiagBytes = 8 * kDiagWords;
};

template <typename T, int W>
struct PanelSmem {
  unsigned long long mbar[2];
  alignas(16) unsigned long long rec[2][kPanelMaxC][PanelRec<T, W>::kWords];
  alignas(16) unsigned long long diag[2][PanelRec<T, W>::kDiagWords];
  alignas(16) unsigned long long outbox[2][PanelRec<T, W>::kWords];
  alignas(16) unsigned long long doutbox[2][PanelRec<T, W>::kDiagWords];
  double cand_key[kPanelWarps];
  int cand_idx[kPanelWarps];
  T side_vals[4 * kPanelMaxW][kSideCols];
  int side_rows[4 * kPanelMaxW];
  int side_cnt;
};

template <typename T, int W>
__host__ __device__ inline size_t panel_smem_bytes(int rows_per_cta) {
  size_t b = sizeof(PanelSmem<T, W>);
  b = (b + 15) & ~size_t(15);
  b += sizeof(T) * (size_t)rows_per_cta * (W + 1);  // slab
  b += sizeof(int) * 2 * (size_t)rows_per_cta;     // labels
  return (b + 127) & ~size_t(127);
}

__device__ __forceinline__ void keyidx_combine(double& k, int& i, double ok, int oi) {
  if (ok > k || (ok == k && oi < i)) {
    k = ok;
    i = oi;
  }
}

__device__ __forceinline__ double pivot_key(double v, bool is_diag) {
  const double a = fabs(v);
  if (isnan(a)) return is_diag ? CUDART_INF : -CUDART_INF;
  return a;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t a, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// One bulk copy (async proxy) of `bytes` from this CTA's shared memory into
// the shared memory of a CTA of the cluster, completing on that CTA's mbarrier.
// Addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_to_cta(uint32_t remote_dst, uint32_t local_src, int bytes, uint32_t remote_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :: "r"(remote_dst), "r"(local_src), "r"(bytes), "r"(remote_bar) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arm(uint32_t bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of the given parity; gives up after kWaitLimitNs and
// returns false. What completes the phase are other CTAs' st.async: acquire at
// cluster scope (their completion releases at that scope).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, int parity) {
  uint32_t done = 0;
  uint64_t t0 = 0;
  for (int it = 1;; ++it) {
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((it & 63) == 0) {  // the timer is read only once the wait is long
      const uint64_t t = global_timer_ns();
      if (t0 == 0) t0 = t;
      else if (t - t0 > kWaitLimitNs) return false;
    }
  }
}

template <typename T>
__device__ __forceinline__ unsigned long long pack2(T a, T b);
template <>
__device__ __forceinline__ unsigned long long pack2<float>(float a, float b) {
  return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}
__device__ __forceinline__ unsigned long long pack_ii(int a, int b) {
  return (unsigned long long)(unsigned)a | ((unsigned long long)(unsigned)b << 32);
}

// Word k of a slab row, as the record stores it.
template <typename T, int W>
__device__ __forceinline__ unsigned long long row_word(const T* row, int k) {
  if constexpr (sizeof(T) == 8) {
    return (unsigned long long)__double_as_longlong(static_cast<double>(row[k]));
  } else {
    return pack2<float>(static_cast<float>(row[2 * k]), static_cast<float>(row[2 * k + 1]));
  }
}
template <typename T>
__device__ __forceinline__ T rec_entry(const unsigned long long* words, int c) {
  if constexpr (sizeof(T) == 8) {
    return static_cast<T>(__longlong_as_double((long long)words[c]));
  } else {
    const unsigned long long wv = words[c >> 1];
    return static_cast<T>(__uint_as_float((unsigned)(c & 1 ? (wv >> 32) : wv)));
  }
}

template <typename T, int W, bool EXACT>
__global__ void __launch_bounds__(kPanelThreads, 1) panel_cluster_kernel(PanelArgs<T> p) {
  using Rec = PanelRec<T, W>;
  constexpr int G = kPanelThreads / W;  // row groups
  constexpr int LD = W + 1;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks();
  const int q = (int)cl.block_rank();
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int c = tid % W;   // column owned by this thread
  const int g = tid / W;   // row group
  const int m = p.n - p.c0;
  const int R = (m + C - 1) / C;
  const int rb = q * R;
  const int re = min(m, rb + R);
  const int nr = max(0, re - rb);
  const int w = p.w;
  const int step_bytes = C * Rec::kBytes + Rec::kDiagBytes;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  PanelSmem<T, W>& S = *reinterpret_cast<PanelSmem<T, W>*>(smem_raw);
  T* tile = reinterpret_cast<T*>(smem_raw + ((sizeof(PanelSmem<T, W>) + 15) & ~size_t(15)));
  int* lab_s = reinterpret_cast<int*>(tile + (size_t)R * LD);
  int* loc_s = lab_s + R;

  // ---- load the slab, set up the mailboxes ----------------------------------
  for (int cc = 0; cc < W; ++cc) {
    const T* col = p.a + (size_t)(p.c0 + cc) * p.lda + (p.c0 + rb);
    for (int r = tid; r < nr; r += kPanelThreads) tile[r * LD + cc] = cc < w ? col[r] : T(0);
  }
  for (int r = tid; r < nr; r += kPanelThreads) {
    const int gr = p.c0 + rb + r;
    lab_s[r] = p.first_leaf ? gr : p.lab[gr];
    loc_s[r] = gr;
  }
  if (tid == 0) {
    mbar_init(smem_u32(&S.mbar[0]), 1);
    mbar_init(smem_u32(&S.mbar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_arm(smem_u32(&S.mbar[0]), step_bytes);
    if (w > 1) mbar_arm(smem_u32(&S.mbar[1]), step_bytes);
  }
  cl.sync();  // mbarriers live in every CTA before anyone sends

  // first candidate (column 0)
  {
    double bk = -CUDART_INF;
    int bi = INT_MAX;
    if (c == 0) {
      for (int r = g; r < nr; r += G) {
        const double key = pivot_key((double)tile[r * LD], rb + r == 0);
        if (key > bk) { bk = key; bi = rb + r; }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double ok = __shfl_down_sync(0xffffffffu, bk, off);
      const int oi = __shfl_down_sync(0xffffffffu, bi, off);
      keyidx_combine(bk, bi, ok, oi);
    }
    if (lane == 0) { S.cand_key[warp] = bk; S.cand_idx[warp] = bi; }
  }
  __syncthreads();

  const uint32_t rec_base = smem_u32(&S.rec[0][0][0]);
  const uint32_t diag_base = smem_u32(&S.diag[0][0]);
  const uint32_t bar_base = smem_u32(&S.mbar[0]);
  bool ok_wait = true;

  for (int j = 0; j < w; ++j) {
    const int par = j & 1;
    // ---- send: CTA candidate record (+ row j) to every mailbox -------------
    if (warp == 0) {
      double bk = -CUDART_INF;
      int bi = INT_MAX;
      if (lane < kPanelWarps) { bk = S.cand_key[lane]; bi = S.cand_idx[lane]; }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double ok = __shfl_down_sync(0xffffffffu, bk, off);
        const int oi = __shfl_down_sync(0xffffffffu, bi, off);
        keyidx_combine(bk, bi, ok, oi);
      }
      bk = __shfl_sync(0xffffffffu, bk, 0);
      bi = __shfl_sync(0xffffffffu, bi, 0);
      const bool have = bi != INT_MAX;
      const T* crow = have ? tile + (size_t)(bi - rb) * LD : tile;
      const bool own_j = j >= rb && j < re;
      const T* drow = own_j ? tile + (size_t)(j - rb) * LD : tile;
      unsigned long long* ob = &S.outbox[par][0];
      unsigned long long* dob = &S.doutbox[par][0];
      for (int kw = lane; kw < Rec::kWords; kw += 32) {
        unsigned long long val = 0;
        if (kw == 0) val = (unsigned long long)__double_as_longlong(bk);
        else if (kw == 1) val = pack_ii(bi, have ? lab_s[bi - rb] : 0);
        else if (kw == 2) val = pack_ii(have ? loc_s[bi - rb] : 0, 0);
        else if (kw < 3 + Rec::kRowWords) val = row_word<T, W>(crow, kw - 3);
        ob[kw] = val;
      }
      if (own_j) {
        for (int kw = lane; kw < Rec::kDiagWords; kw += 32) {
          unsigned long long val = 0;
          if (kw == 0) val = pack_ii(lab_s[j - rb], loc_s[j - rb]);
          else if (kw < 1 + Rec::kRowWords) val = row_word<T, W>(drow, kw - 1);
          dob[kw] = val;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane < C) {
        const uint32_t rbar = mapa_u32(bar_base + 8u * par, lane);
        const uint32_t la = rec_base + 8u * (uint32_t)((par * kPanelMaxC + q) * Rec::kWords);
        bulk_to_cta(mapa_u32(la, lane), smem_u32(ob), Rec::kBytes, rbar);
        if (own_j) {
          const uint32_t ld2 = diag_base + 8u * (uint32_t)(par * Rec::kDiagWords);
          bulk_to_cta(mapa_u32(ld2, lane), smem_u32(dob), Rec::kDiagBytes, rbar);
        }
      }
    }
    // ---- receive: wait for this column's records ---------------------------
    // a wait that ran out stays failed: the rest of the leaf runs through
    // without waiting and the host reports ALG_TIMEOUT
    if (ok_wait && !mbar_wait(bar_base + 8u * par, (j >> 1) & 1)) {
      ok_wait = false;
      atomicExch(&p.status->timeout, 1);
    }
    __syncwarp();
    if (tid == 0 && j + 2 < w) mbar_arm(bar_base + 8u * par, step_bytes);
    // every warp reduces the C records to the same winner
    double wk = -CUDART_INF;
    int wi = INT_MAX, ws = 0;
    if (lane < C) {
      wk = __longlong_as_double((long long)S.rec[par][lane][0]);
      wi = (int)(unsigned)(S.rec[par][lane][1] & 0xffffffffu);
      ws = lane;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double ok = __shfl_down_sync(0xffffffffu, wk, off);
      const int oi = __shfl_down_sync(0xffffffffu, wi, off);
      const int os = __shfl_down_sync(0xffffffffu, ws, off);
      if (ok > wk || (ok == wk && oi < wi)) { wk = ok; wi = oi; ws = os; }
    }
    const int pr = __shfl_sync(0xffffffffu, wi, 0);  // winning panel row (>= j)
    const int ps = __shfl_sync(0xffffffffu, ws, 0);  // CTA that sent it
    const unsigned long long* wrow = &S.rec[par][ps][3];
    const T d = rec_entry<T>(wrow, j);
    const T u = rec_entry<T>(wrow, c);
    // swap rows j and pr where this thread owns them (same thread updates them later)
    if (j >= rb && j < re && (j - rb) % G == g) {
      tile[(j - rb) * LD + c] = u;
      if (c == 0) {
        lab_s[j - rb] = (int)(unsigned)(S.rec[par][ps][1] >> 32);
        loc_s[j - rb] = (int)(unsigned)(S.rec[par][ps][2] & 0xffffffffu);
      }
    }
    if (pr != j && pr >= rb && pr < re && (pr - rb) % G == g) {
      tile[(pr - rb) * LD + c] = rec_entry<T>(&S.diag[par][1], c);
      if (c == 0) {
        lab_s[pr - rb] = (int)(unsigned)(S.diag[par][0] & 0xffffffffu);
        loc_s[pr - rb] = (int)(unsigned)(S.diag[par][0] >> 32);
      }
    }
    if (tid == 0 && q == 0) {
      p.ipiv[p.c0 + j] = p.c0 + pr;
      if (fabs((double)d) <= 0.0) atomicMin(&p.status->singular_col, p.c0 + j);
    }
    __syncwarp();
    // multipliers (correctly rounded quotient, as K1r) for the group's rows
    // below j, spread over its lanes
    const int r_first = max(0, j + 1 - rb);
    const int r0 = r_first + ((g - r_first % G) + G) % G;  // first row >= r_first of group g
    {
      const bool fast = div_fast_ok(d);
      const T y = fast ? rcp_rn(d) : T(1);
      int k = 0;
      for (int r = r0 + c * G; r < nr; r += W * G, k += W) {
        const T av = tile[r * LD + j];
        tile[r * LD + j] = quotient<T>(av, d, y, fast);
      }
    }
    __syncwarp();
    // rank-1 update, 8 independent rows per batch; column j+1 yields the next candidate
    double bk = -CUDART_INF;
    int bi = INT_MAX;
    if (c > j && c < w) {
      constexpr int B = 8;
      for (int rs = r0; rs < nr; rs += B * G) {
        T av[B], lv[B];
#pragma unroll
        for (int t = 0; t < B; ++t) {
          const int r = rs + t * G;
          av[t] = r < nr ? tile[r * LD + c] : T(0);
          lv[t] = r < nr ? tile[r * LD + j] : T(0);
        }
#pragma unroll
        for (int t = 0; t < B; ++t) av[t] = msub<EXACT>(av[t], lv[t], u);
#pragma unroll
        for (int t = 0; t < B; ++t) {
          const int r = rs + t * G;
          if (r < nr) {
            tile[r * LD + c] = av[t];
            if (c == j + 1) {
              const double key = pivot_key((double)av[t], rb + r == j + 1);
              if (key > bk) { bk = key; bi = rb + r; }
            }
          }
        }
      }
    }
    if (j + 1 < w) {
      // collect the candidates of the warp's row groups (lanes with c == j+1)
      const int src0 = (lane / W) * W + (j + 1);  // own group's candidate lane
      double k0 = __shfl_sync(0xffffffffu, bk, src0 & 31);
      int i0 = __shfl_sync(0xffffffffu, bi, src0 & 31);
      if constexpr (W == 16) {
        const double k1 = __shfl_sync(0xffffffffu, bk, (j + 1 + 16 - (lane / W) * W) & 31);
        const int i1 = __shfl_sync(0xffffffffu, bi, (j + 1 + 16 - (lane / W) * W) & 31);
        keyidx_combine(k0, i0, k1, i1);
      }
      if (lane == 0) { S.cand_key[warp] = k0; S.cand_idx[warp] = i0; }
    }
    __syncthreads();
  }
  cl.sync();  // every record consumed; no DSMEM access outlives its owner

  // ---- swap the block-panel's other columns by this leaf's interchanges -----
  // Rows whose leaf label moved take the old content of the labelled row; all
  // reads of a pass precede the cluster barrier, all writes follow it.
  if (tid == 0) S.side_cnt = 0;
  __syncthreads();
  for (int r = tid; r < nr; r += kPanelThreads) {
    loc_s[r] = index_or(loc_s[r], p.c0, p.n, p.c0 + rb + r);
    if (loc_s[r] != p.c0 + rb + r) {
      const int s = atomicAdd(&S.side_cnt, 1);
      if (s < 4 * kPanelMaxW) S.side_rows[s] = r;
    }
  }
  __syncthreads();
  const int n_side = min(S.side_cnt, 4 * kPanelMaxW);
  const int side_w = (p.kb1 - p.kb0) - w;
  for (int cbase = 0; cbase < side_w; cbase += kSideCols) {
    const int ncol = min(kSideCols, side_w - cbase);
    for (int idx = tid; idx < n_side * kSideCols; idx += kPanelThreads) {
      const int s = idx / kSideCols, cc = idx % kSideCols;
      if (cc >= ncol) continue;
      int col = p.kb0 + cbase + cc;
      if (col >= p.c0) col += w;
      S.side_vals[s][cc] = p.a[(size_t)loc_s[S.side_rows[s]] + (size_t)col * p.lda];
    }
    cl.sync();
    for (int idx = tid; idx < n_side * kSideCols; idx += kPanelThreads) {
      const int s = idx / kSideCols, cc = idx % kSideCols;
      if (cc >= ncol) continue;
      int col = p.kb0 + cbase + cc;
      if (col >= p.c0) col += w;
      p.a[(size_t)(p.c0 + rb + S.side_rows[s]) + (size_t)col * p.lda] = S.side_vals[s][cc];
    }
    cl.sync();
  }

  // ---- write the slab back ------------------------------------------------
  for (int cc = 0; cc < w; ++cc) {
    T* col = p.a + (size_t)(p.c0 + cc) * p.lda + (p.c0 + rb);
    for (int r = tid; r < nr; r += kPanelThreads) col[r] = tile[r * LD + cc];
  }
  for (int r = tid; r < nr; r += kPanelThreads) p.lab[p.c0 + rb + r] = lab_s[r];
}

// ---------------------------------------------------------------------------
// K1r: LU of a block of columns by one thread-block cluster, rows resident on
// the chip (m <= 16 * NT * RPT).
//
// Factors columns [c0, c0 + bw) of rows [c0, n) in leaves of W columns. The
// kernel is bound by the latency of its column chain (search, exchange,
// divide, update), so each link is kept short and nothing else is launched
// between the leaves:
//  * A thread keeps RPT whole rows of the current leaf in registers. Rows
//    never move: a row carries its current position instead, an interchange
//    of rows j and p sets two positions, and the rows are written to their
//    final positions at the end.
//  * The rank-1 update writes entry c into entry c - 1, so the pivot column
//    is always entry 0 and one copy of the column's code (small enough for
//    the instruction cache: unrolled by four columns, fetching it was a third
//    of the time) serves the whole leaf with static register indices. What
//    leaves the register row is final and goes to the tile in shared memory:
//    a multiplier from its own thread, a pivot row from its record.
//  * Candidates are compared as integers by redux.sync over the high word,
//    the low word and the position.
//  * The reciprocal of a candidate is formed beside the search and travels
//    in its record, so no thread divides after the exchange.
//  * A pivot is filed (its U entries, the interchange) by one warp, another
//    each column.
// Per column: candidate -> redux -> the warp's best lane stages its row ->
// one CTA barrier -> the CTA's best record to every mailbox (16-byte st.async,
// the CTAs spread over the warps, completing on the receiver's mbarrier) ->
// wait on the own mbarrier -> redux over the C records -> divide and update.
// C == 1 skips the exchange. Mailboxes and mbarriers alternate by column
// parity as in K1.
//
// With more than one leaf (bw > W) the columns right of the leaf wait in the
// tile (tile[col][row]). At the leaf's end every CTA reads the pivot rows'
// entries there, and their multipliers, from their owners' tiles, solves
// U12 = L11^{-1} A12 for itself and updates its own rows, each entry's terms in
// increasing k. A cluster barrier comes before those reads: the tiles are
// written by ordinary stores, which a record's arrival does not order for
// another CTA. Nothing changes a pivot row afterwards, so none follows them.
//
// Division: the multiplier is the correctly rounded quotient a/d
// (mod.rs:154). With y = RN(1/d), q = RN(a*y) is within one ulp of a/d, the
// remainder a - q*d is exact under an FMA, and RN(q + (a - q*d)*y) is the
// correctly rounded quotient (Markstein's theorem), as long as nothing over-
// or underflows; a zero a keeps q, the zero with the quotient's sign; other
// entries and pivots outside [2^-500, 2^500] in magnitude and non-finite
// values take the plain IEEE division instead.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void st_async_v2(uint32_t remote, ulonglong2 v, uint32_t remote_bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];"
               :: "r"(remote), "l"(v.x), "l"(v.y), "r"(remote_bar) : "memory");
}
__device__ __forceinline__ void ld_cluster(double& v, uint32_t a) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_cluster(float& v, uint32_t a) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}

constexpr int kBlockMaxW = 64;  // columns of a block that one launch factors

// Dynamic shared memory: the tile and, with more than one leaf, the U12 rows
// of the current leaf ([col][k]) and its unit-lower block.
template <typename T, int W>
__host__ __device__ inline size_t block_panel_smem(int rows_per_cta, int bw) {
  return sizeof(T) * ((size_t)bw * ((rows_per_cta + 1) & ~1) + (bw > W ? (size_t)bw * W : 0));
}

template <typename T, int W, int NT, int RPT, bool EXACT>
__global__ void __launch_bounds__(NT, 1) panel_reg_kernel(PanelArgs<T> p) {
  using Rec = PivotRec<T, W>;
  using Key = typename Rec::Key;
  static_assert(sizeof(Rec) == 16 * Rec::kChunks && Rec::kChunks <= 16, "record layout");
  constexpr int NW = NT / 32;
  constexpr int kVec = 16 / (int)sizeof(T);
  struct alignas(16) Vec {
    T e[kVec];
  };
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks();
  const int q = (int)cl.block_rank();
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int m = p.n - p.c0;
  const int R = (m + C - 1) / C;
  const int rb = q * R;
  const int nr = max(0, min(m, rb + R) - rb);
  const int bw = p.w;  // columns of this launch
  const bool multi = bw > W;
  const int ldt = (R + 1) & ~1;  // tile column stride
  const int step_bytes = C * (int)sizeof(Rec);

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* l11 = reinterpret_cast<T*>(smem_raw);       // W x W: the leaf's unit-lower block, [row][col]
  T* ubuf = l11 + W * W;                         // (bw - W) x W: its U12, [col][k]
  T* tile = l11 + (multi ? (size_t)bw * W : 0);  // bw x ldt
  __shared__ unsigned long long mbar[2];
  // [par][0, C): the mailboxes; [par][kPanelMaxC + warp]: the warps' stages
  __shared__ Rec rec[2][kPanelMaxC + NW];
  __shared__ int side_src[2 * kBlockMaxW];
  __shared__ int side_dst[2 * kBlockMaxW];
  __shared__ int side_cnt;
  __shared__ int piv_src[W];  // the leaf's pivot rows: owner << 16 | slot there

  // ---- load --------------------------------------------------------------
  T v[RPT][W];
  int pos[RPT];  // the row's position in the panel (-1: no row)
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int r = tid + k * NT;  // local row
    const bool in = r < nr;
    const T* row = p.a + (size_t)(p.c0 + rb + r) + (size_t)p.c0 * p.lda;
    pos[k] = in ? rb + r : -1;
#pragma unroll
    for (int c = 0; c < W; ++c) v[k][c] = (in && c < bw) ? row[(size_t)c * p.lda] : T(0);
    if (multi && r < ldt) {
#pragma unroll 8
      for (int c = W; c < bw; ++c) tile[c * ldt + r] = in ? row[(size_t)c * p.lda] : T(0);
    }
  }
  if (tid == 0) {
    side_cnt = 0;
    if (C > 1) {
      mbar_init(smem_u32(&mbar[0]), 1);
      mbar_init(smem_u32(&mbar[1]), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_arm(smem_u32(&mbar[0]), step_bytes);
      if (bw > 1) mbar_arm(smem_u32(&mbar[1]), step_bytes);
    }
  }
  cl.sync();

  const uint32_t bar_base = smem_u32(&mbar[0]);
  const uint32_t tile_base = smem_u32(tile);
  bool ok_wait = true;
  // the mailboxes (slot q, this lane's chunk) and mbarriers this lane sends to
  constexpr int kSends = (kPanelMaxC + 2 * NW - 1) / (2 * NW);
  const int chunk = lane & 15;
  uint32_t rem_rec[kSends], rem_bar[kSends];
#pragma unroll
  for (int i = 0; i < kSends; ++i) {
    const int t = min(warp + NW * (2 * i + (lane >> 4)), C - 1);
    rem_rec[i] = mapa_u32(smem_u32(&rec[0][q]) + 16u * chunk, t);
    rem_bar[i] = mapa_u32(bar_base, t);
  }

#pragma unroll 1
  for (int cl0 = 0; cl0 < bw; cl0 += W) {
    const int w = min(W, bw - cl0);
    const int tc = bw - cl0 - w;  // columns of the block right of the leaf
#pragma unroll 1
    for (int j = 0; j < w; ++j) {
      const int J = cl0 + j;  // column of the launch = row position of its pivot
      const int par = J & 1;
      int mp;
      // ---- 1. the thread's, then the warp's candidate ------------------------
      Key key, mk;
      int kpos, kslot = tid;
      T cand = v[0][0];
      pivot_candidate(v[0][0], pos[0], J, key, kpos);
#pragma unroll
      for (int k = 1; k < RPT; ++k) {
        Key kk;
        int kp;
        pivot_candidate(v[k][0], pos[k], J, kk, kp);
        if (kk > key || (kk == key && kp < kpos)) {
          key = kk;
          kpos = kp;
          kslot = tid + k * NT;
          cand = v[k][0];
        }
      }
      const T crecip = rcp_rn(exp_fast_ok(cand) ? cand : T(1));
      if (warp_pivot(key, kpos, mk, mp)) {  // (no candidate at all: any lanes, an empty record)
        Rec& s = rec[par][kPanelMaxC + warp];
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
      __syncthreads();
      // ---- 2. the CTA's candidate ----------------------------------------
      int win = kPanelMaxC + warp_pick(&rec[par][kPanelMaxC], NW, lane, mp), owner = q;
      if (C > 1) {
        // the record to every mailbox: half-warps of 16-byte chunks, CTAs
        // t = warp, warp + NW, ... (slot q of the mailboxes)
        if (chunk < Rec::kChunks) {
          const ulonglong2 val = reinterpret_cast<const ulonglong2*>(&rec[par][win])[chunk];
          const uint32_t off = (uint32_t)(par * (kPanelMaxC + NW) * (int)sizeof(Rec));
#pragma unroll
          for (int i = 0; i < kSends; ++i)
            if (warp + NW * (2 * i + (lane >> 4)) < C) st_async_v2(rem_rec[i] + off, val, rem_bar[i] + 8u * par);
        }
        // ---- 3. wait for this column's records; every warp picks the winner
        // (a wait that ran out stays failed: the rest of the launch runs
        // through without waiting and the host reports ALG_TIMEOUT)
        if (ok_wait && !mbar_wait(bar_base + 8u * par, (J >> 1) & 1)) {
          ok_wait = false;
          atomicExch(&p.status->timeout, 1);
        }
        if (tid == 0 && J + 2 < bw) mbar_arm(bar_base + 8u * par, step_bytes);
        __syncwarp();
        win = owner = warp_pick(&rec[par][0], C, lane, mp);
      }
      const Rec& wr = rec[par][win];
      const int pr = ok_wait ? mp : J;  // winning row's position (>= J)
      const T d = wr.row[0];
      const T y = wr.recip;
      // one warp files the pivot row ------------------------------------
      if (warp == (j % NW)) {
        const int slot = ok_wait ? index_or((int)wr.slot, 0, ldt, 0) : 0;
        if (owner == q && lane < w - j) tile[(J + lane) * ldt + slot] = wr.row[lane];
        if (lane == 0 && q == 0) {
          p.ipiv[p.c0 + J] = p.c0 + pr;
          if (d == T(0)) atomicMin(&p.status->singular_col, p.c0 + J);
        }
        if (lane == 0) piv_src[j] = owner << 16 | slot;
      }
      // ---- 4. rows J and pr change places; divide and update below J -------
      const bool fast = exp_fast_ok(d);
      T l[RPT];
      bool odd = false;
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        if (pos[k] == pr) pos[k] = J;
        else if (pos[k] == J) pos[k] = pr;
        const T av = v[k][0];
        const T qv = mul_rn(av, y);
        l[k] = fma_rn(fma_rn(-qv, d, av), y, qv);
        odd |= !(fast && exp_fast_ok(av)) && pos[k] > J;
      }
      if (odd) {  // zeros; rarely the plain IEEE division
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
    if (tc > 0) {  // (then w == W)
      if (C > 1) cl.sync();
      else __syncthreads();
      // entry e: pivot row j = e % W, column c = e / W of the leaf and those right of it
      constexpr int kPull = 8;  // in flight per thread
      const int pulls = W * (W + tc);
      for (int e0 = tid; e0 < pulls; e0 += kPull * NT) {
        T pv[kPull];
#pragma unroll
        for (int i = 0; i < kPull; ++i) {
          const int e = e0 + i * NT, j = e % W, c = e / W;
          if (e < pulls && (c < j || c >= W)) {
            const int src = piv_src[j];
            ld_cluster(pv[i], mapa_u32(tile_base + (uint32_t)sizeof(T) * ((cl0 + c) * ldt + (src & 0xffff)), src >> 16));
          }
        }
#pragma unroll
        for (int i = 0; i < kPull; ++i) {
          const int e = e0 + i * NT, j = e % W, c = e / W;
          if (e < pulls && c < j) l11[j * W + c] = pv[i];
          if (e < pulls && c >= W) ubuf[(c - W) * W + j] = pv[i];
        }
      }
      __syncthreads();
      if (tid < tc) {
        T* x = ubuf + tid * W;
        T xr[W];
#pragma unroll
        for (int i = 0; i < W; ++i) xr[i] = x[i];
#pragma unroll
        for (int k = 0; k < W; ++k)
#pragma unroll
          for (int i = k + 1; i < W; ++i) xr[i] = msub<EXACT>(xr[i], l11[i * W + k], xr[k]);
#pragma unroll
        for (int i = 0; i < W; ++i) x[i] = xr[i];
        if (q == 0) {
          T* out = p.a + (size_t)(p.c0 + cl0) + (size_t)(p.c0 + cl0 + w + tid) * p.lda;
#pragma unroll
          for (int i = 0; i < W; ++i) out[i] = xr[i];
        }
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const int r = tid + k * NT;
        if (pos[k] >= cl0 + w) {
#pragma unroll
          for (int i = 0; i < W; ++i) v[k][i] = tile[(cl0 + i) * ldt + r];
          T* trow = tile + (size_t)(cl0 + w) * ldt + r;
#pragma unroll 1
          for (int c = 0; c < tc; c += 4) {  // tc: a multiple of 4 unless the block is ragged
            T acc[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] = c + e < tc ? trow[(c + e) * ldt] : T(0);
#pragma unroll
            for (int i = 0; i < W; i += kVec)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const Vec u = *reinterpret_cast<const Vec*>(ubuf + min(c + e, tc - 1) * W + i);
#pragma unroll
                for (int t = 0; t < kVec; ++t) acc[e] = msub<EXACT>(acc[e], v[k][i + t], u.e[t]);
              }
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (c + e < tc) trow[(c + e) * ldt] = acc[e];
          }
        }
      }
      // the next leaf's rows
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const int r = tid + k * NT;
#pragma unroll
        for (int c = 0; c < W; ++c) v[k][c] = (c < tc && r < ldt) ? tile[(cl0 + w + c) * ldt + r] : T(0);
      }
    }
  }
  __syncthreads();

  // ---- rows to their final positions; swap the block-panel's other columns --
  // The row loaded from c0 + rb + r moved to position pos: its content in the
  // other columns goes the same way. All reads of a pass precede the cluster
  // barrier, all writes follow it; the first barrier also ends the DSMEM
  // exchange (every record and pull done before a CTA may exit).
  int lab[RPT];  // the rows' source labels, read before any CTA writes one
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int r = tid + k * NT;
    if (pos[k] >= 0) pos[k] = index_or(pos[k], 0, m, rb + r);
    lab[k] = p.c0 + rb + r;
    if (pos[k] >= 0 && !p.first_leaf) lab[k] = p.lab[p.c0 + rb + r];
    if (pos[k] >= 0 && pos[k] != rb + r) {
      const int s = atomicAdd(&side_cnt, 1);
      if (s < 2 * kBlockMaxW) {
        side_src[s] = p.c0 + rb + r;
        side_dst[s] = p.c0 + pos[k];
      }
    }
  }
  __syncthreads();
  const int side_w = (p.kb1 - p.kb0) - bw;
  const int n_side = min(side_cnt, 2 * kBlockMaxW);
  // A pass takes the same columns in every CTA (a CTA moves at most 2 bw rows).
  constexpr int kSidePer = 16;  // values in flight per thread and pass
  const int pass_w = kSidePer * NT / (2 * bw);
  const int passes = (side_w + pass_w - 1) / pass_w;
  for (int ps = 0; ps < passes; ++ps) {
    const int s0 = ps * pass_w;
    const int n_move = n_side * min(pass_w, side_w - s0);
    T sv[kSidePer];
#pragma unroll
    for (int i = 0; i < kSidePer; ++i) {
      const int e = i * NT + tid;
      if (e < n_move) {
        int col = p.kb0 + s0 + e / n_side;
        if (col >= p.c0) col += bw;
        sv[i] = p.a[(size_t)side_src[e % n_side] + (size_t)col * p.lda];
      }
    }
    cl.sync();
#pragma unroll
    for (int i = 0; i < kSidePer; ++i) {
      const int e = i * NT + tid;
      if (e < n_move) {
        int col = p.kb0 + s0 + e / n_side;
        if (col >= p.c0) col += bw;
        p.a[(size_t)side_dst[e % n_side] + (size_t)col * p.lda] = sv[i];
      }
    }
  }
  if (passes == 0) cl.sync();

  // ---- back to the matrix -----------------------------------------------
  // (a pivot row's U entries right of its leaf are already there)
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    if (pos[k] >= 0) {
      T* row = p.a + (size_t)(p.c0 + pos[k]) + (size_t)p.c0 * p.lda;
      const int ce = pos[k] < bw ? min(bw, (pos[k] / W + 1) * W) : bw;
      const T* trow = tile + tid + k * NT;
#pragma unroll 8
      for (int c = 0; c < ce; ++c) row[(size_t)c * p.lda] = trow[c * ldt];
      p.lab[p.c0 + pos[k]] = lab[k];
    }
  }
}

// ---------------------------------------------------------------------------
// K2: deferred row interchange of the columns outside a block-panel.
// Row r (r in [k0, n)) of every such column takes the old content of row
// lab[r]; the rows that move are compacted once per CTA, and one warp owns a
// column (all loads of a column precede its stores).
// The net permutation `perm` is carried the same way (CTA 0, one extra pass).
// ---------------------------------------------------------------------------
constexpr int kSwapThreads = 256;
constexpr int kSwapMaxMoves = 512;
constexpr int kSwapScan = 16;  // labels a thread reads per round trip of the scan

template <typename T>
__global__ void __launch_bounds__(kSwapThreads) laswp_outside_kernel(
    T* a, int lda, int n, int cb, int ce, int k0, int kb, const int* lab, int* perm, int* perm_tmp) {
  __shared__ int mv_dst[kSwapMaxMoves];
  __shared__ int mv_src[kSwapMaxMoves];
  __shared__ int mv_cnt;
  if (threadIdx.x == 0) mv_cnt = 0;
  __syncthreads();
  for (int r0 = k0 + threadIdx.x; r0 < n; r0 += kSwapScan * kSwapThreads) {
    int src[kSwapScan];
#pragma unroll
    for (int i = 0; i < kSwapScan; ++i) {
      const int r = r0 + i * kSwapThreads;
      src[i] = r < n ? index_or(lab[r], k0, n, r) : r;
    }
#pragma unroll
    for (int i = 0; i < kSwapScan; ++i) {
      const int r = r0 + i * kSwapThreads;
      if (src[i] != r) {
        const int slot = atomicAdd(&mv_cnt, 1);
        if (slot < kSwapMaxMoves) { mv_dst[slot] = r; mv_src[slot] = src[i]; }
      }
    }
  }
  __syncthreads();
  const int moves = min(mv_cnt, kSwapMaxMoves);
  const int lane = threadIdx.x & 31;
  const int warps_total = gridDim.x * (kSwapThreads / 32);
  const int gwarp = blockIdx.x * (kSwapThreads / 32) + (threadIdx.x >> 5);
  // columns of the window [cb, ce) outside the block [k0, k0 + kb)
  const int n_before = max(0, min(ce, k0) - cb);
  const int after0 = max(cb, k0 + kb);
  const int n_out = n_before + max(0, ce - after0);
  constexpr int kPer = kSwapMaxMoves / 32;
  for (int cidx = gwarp; cidx < n_out; cidx += warps_total) {
    const int col = cidx < n_before ? cb + cidx : after0 + (cidx - n_before);
    T* colp = a + (size_t)col * lda;
    T vals[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int s = lane + 32 * t;
      if (s < moves) vals[t] = colp[mv_src[s]];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int s = lane + 32 * t;
      if (s < moves) colp[mv_dst[s]] = vals[t];
    }
  }
  if (perm != nullptr && blockIdx.x == 0) {
    // perm_new[r] = perm_old[lab[r]] over the moved rows
    for (int s = threadIdx.x; s < moves; s += kSwapThreads) perm_tmp[s] = perm[mv_src[s]];
    __syncthreads();
    for (int s = threadIdx.x; s < moves; s += kSwapThreads) perm[mv_dst[s]] = perm_tmp[s];
  }
}

// ---------------------------------------------------------------------------
// K2c / K2p: the interchanges of the columns left of each block, all at once
// after the last block. Block b's labels lie at lab + b * n; the columns of
// block b take the interchanges of the blocks b + 1, ..., nblk - 1 one after
// the other: their row r takes the old content of row
//   comp_b[r] = lab_{b+1}[... lab_{nblk-1}[r]],
// which one thread per row follows backwards through the blocks (a block
// moves rows from its own first one on, so row r starts at block r / nb).
// comp_b lies at comp + b * n; the chain's last element is the net
// permutation.
// A move within a column costs 32 to 64 bytes of DRAM traffic for 4 or 8
// bytes of data, and one block's interchanges move up to 2 nb rows of every
// column. Here a column is read and written once, consecutively, with the
// exchange in shared memory (bound by HBM).
// ---------------------------------------------------------------------------
__global__ void compose_swaps_kernel(const int* lab, int n, int nb, int nblk, int* comp, int* perm) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  int s = r;
  for (int b = min(nblk - 1, r / nb); b >= 0; --b) {
    s = index_or(lab[(size_t)b * n + s], b * nb, n, s);
    if (b > 0) comp[(size_t)(b - 1) * n + r] = s;
  }
  if (perm != nullptr) perm[r] = s;
}

constexpr int kPermThreads = 1024;

// One CTA per column; dynamic shared memory: the longest column's moving rows.
template <typename T>
__global__ void __launch_bounds__(kPermThreads) permute_left_kernel(T* a, int lda, int n, int nb, const int* comp) {
  extern __shared__ __align__(16) unsigned char perm_smem[];
  T* old = reinterpret_cast<T*>(perm_smem);
  const int c = blockIdx.x, b = c / nb;
  const int base = (b + 1) * nb, cnt = n - base;
  T* col = a + (size_t)c * lda + base;
  const int* src = comp + (size_t)b * n + base;
#pragma unroll 8
  for (int i = threadIdx.x; i < cnt; i += kPermThreads) old[i] = col[i];
  __syncthreads();
#pragma unroll 8
  for (int i = threadIdx.x; i < cnt; i += kPermThreads) {
    const int s = src[i] - base;
    col[i] = old[(unsigned)s < (unsigned)cnt ? s : i];
  }
}

__global__ void iota_kernel(int* v, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

// ---------------------------------------------------------------------------
// K3: U12 = L11^{-1} A12 for rows [r0, r0+kb) of columns [cb, ce), unit lower
// L11 = a[r0:r0+kb, r0:r0+kb]. Entry (i, c) receives `-= l_ik * u_kc` for
// k = r0 .. i-1 in that order (one rounded multiply-subtract each in the
// exact form), the reference's order for those entries. No block barrier
// inside: L11 (kb <= 128) staged in shared memory, each warp owns
// CPW whole columns with lane l holding rows l, l + 32, ... in
// registers; step k broadcasts x_k from its owner lane by a shuffle.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr int kTrsmThreads = 256;

// CPW columns per warp, RPT rows per lane (kb <= 32 RPT; L's columns are
// 32 RPT apart). Bound by the issue of the shuffles and multiply-subtracts
// with 8 columns, by the chain shuffle -> multiply-subtract with 2.
// The row group rk of the broadcast is unrolled, so that x_k needs no selection
// among a lane's rows, and L arrives by asynchronous copies of its lower half.
// Inside an LU of n = 16384, us per launch of 128 rows, many columns / a
// block's columns (before: selection by k, L through registers): FP64
// 66 / 35 -> 30 / 16, FP32 41 / 23 -> 24 / 12; 64 rows of a block's
// columns, n = 5001 exact: 8.4 -> 5.2.
template <typename T, bool EXACT, int RPT, int CPW>
__global__ void __launch_bounds__(kTrsmThreads, 1) trsm_lower_unit_reg_kernel(T* a, int lda, int r0, int kb, int cb,
                                                                           int ce) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* L = reinterpret_cast<T*>(smem_raw);
  constexpr int kLd = 32 * RPT;
  constexpr int kCtaCols = CPW * (kTrsmThreads / 32);
  const int c_first = cb + blockIdx.x * kCtaCols;
  const int ncol = min(kCtaCols, ce - c_first);
  if (ncol <= 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // L's strictly lower part (the rest is not read, rows beyond kb to no effect)
  {
    const int i = threadIdx.x % kLd;
    const T* src = a + (size_t)(r0 + i) + (size_t)r0 * lda;
    if (i < kb)
      for (int k = threadIdx.x / kLd; k < i; k += kTrsmThreads / kLd) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(L + k * kLd + i);
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src + (size_t)k * lda),
                     "n"(sizeof(T)) : "memory");
      }
    cp_async_commit_group();
  }
  T x[CPW][RPT];
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int cc = warp * CPW + c;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int i = lane + 32 * r;
      x[c][r] = (cc < ncol && i < kb) ? a[(size_t)(r0 + i) + (size_t)(c_first + cc) * lda] : T(0);
    }
  }
  cp_async_wait_group<0>();
  __syncthreads();
#pragma unroll
  for (int rk = 0; rk < RPT; ++rk) {
    const T* lk = L + (size_t)(32 * rk) * kLd + lane;
    const int steps = min(32, kb - 1 - 32 * rk);
#pragma unroll 4
    for (int kk = 0; kk < steps; ++kk, lk += kLd) {
      T l[RPT], u[CPW];
#pragma unroll
      for (int r = rk; r < RPT; ++r) l[r] = lk[32 * r];
#pragma unroll
      for (int c = 0; c < CPW; ++c) u[c] = __shfl_sync(0xffffffffu, x[c][rk], kk);
      if (lane > kk) {
#pragma unroll
        for (int c = 0; c < CPW; ++c) x[c][rk] = msub<EXACT>(x[c][rk], l[rk], u[c]);
      }
#pragma unroll
      for (int r = rk + 1; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < CPW; ++c) x[c][r] = msub<EXACT>(x[c][r], l[r], u[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int cc = warp * CPW + c;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int i = lane + 32 * r;
      if (cc < ncol && i < kb) a[(size_t)(r0 + i) + (size_t)(c_first + cc) * lda] = x[c][r];
    }
  }
}

// ---------------------------------------------------------------------------
// K3i: the inverses of the diagonal blocks of packed LU factors, for the
// blocked many-right-hand-side solve (fused arithmetic). Block b = rows and
// columns [b kb, b kb + kb) (the last one may be short; its inverse is
// zero-padded to kb x kb): inv + b kb^2 <- T_bb^{-1}, column-major with
// leading dimension kb, T_bb unit lower (UPPER false) or upper. Grid: column
// groups x blocks. The K3 layout: T_bb (kb <= 128) in shared memory, each
// warp owns CPW columns of the identity with lane l holding rows l, l + 32,
// ... in registers; step k broadcasts row k from its owner lane (upper:
// x_k / u_kk, from the last row up).
// ---------------------------------------------------------------------------
template <typename T, bool UPPER, int RPT, int CPW>
__global__ void __launch_bounds__(kTrsmThreads, 1) tri_block_inverse_kernel(const T* lu, int lda, int n, int kb,
                                                                         T* inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* M = reinterpret_cast<T*>(smem_raw);  // kb x kb, column-major
  constexpr int kCtaCols = CPW * (kTrsmThreads / 32);
  const int r0 = blockIdx.y * kb;
  const int bk = min(kb, n - r0);
  const int c_first = blockIdx.x * kCtaCols;
  if (c_first >= kb) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T v[CPW][RPT];
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int col = c_first + warp * CPW + c;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int i = lane + 32 * r;
      v[c][r] = (i == col && col < bk) ? T(1) : T(0);
    }
  }
  for (int idx = threadIdx.x; idx < kb * kb; idx += kTrsmThreads) {
    const int i = idx % kb, k = idx / kb;
    const bool keep = (i < bk && k < bk) && (UPPER ? i <= k : i > k);
    M[idx] = keep ? lu[(size_t)(r0 + i) + (size_t)(r0 + k) * lda] : T(0);
  }
  __syncthreads();
  if constexpr (!UPPER) {
    for (int k = 0; k + 1 < bk; ++k) {
      const int owner = k & 31, rk = k >> 5;
      T u[CPW];
#pragma unroll
      for (int c = 0; c < CPW; ++c) {
        T xv = v[c][0];
#pragma unroll
        for (int r = 1; r < RPT; ++r)
          if (r == rk) xv = v[c][r];
        u[c] = __shfl_sync(0xffffffffu, xv, owner);
      }
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int i = lane + 32 * r;
        if (i > k && i < bk) {
          const T l = M[i + (size_t)k * kb];
#pragma unroll
          for (int c = 0; c < CPW; ++c) v[c][r] = msub<false>(v[c][r], l, u[c]);
        }
      }
    }
  } else {
    for (int k = bk - 1; k >= 0; --k) {
      const int owner = k & 31, rk = k >> 5;
      const T d = M[k + (size_t)k * kb];
      T u[CPW];
#pragma unroll
      for (int c = 0; c < CPW; ++c) {
        T xv = v[c][0];
#pragma unroll
        for (int r = 1; r < RPT; ++r)
          if (r == rk) xv = v[c][r];
        if (lane == owner) {
          xv = xv / d;
#pragma unroll
          for (int r = 0; r < RPT; ++r)
            if (r == rk) v[c][r] = xv;
        }
        u[c] = __shfl_sync(0xffffffffu, xv, owner);
      }
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int i = lane + 32 * r;
        if (i < k) {
          const T m = M[i + (size_t)k * kb];
#pragma unroll
          for (int c = 0; c < CPW; ++c) v[c][r] = msub<false>(v[c][r], m, u[c]);
        }
      }
    }
  }
  T* out = inv + (size_t)blockIdx.y * kb * kb;
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int col = c_first + warp * CPW + c;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int i = lane + 32 * r;
      if (col < kb && i < kb) out[i + (size_t)col * kb] = v[c][r];
    }
  }
}


// ---------------------------------------------------------------------------
// K3b: one step of the blocked many-right-hand-side solve. Y[k0:k0+kbe] holds
// the solved rows of a block; every CTA updates its 128 rows of the rows not
// yet solved, X[rows, tile] -= T[rows, k0:k0+kbe] Y[k0:k0+kbe, tile] (lower:
// the rows below the block; upper: the rows above), and the CTA whose rows
// are the next block goes on to Y[rows, tile] = T_bb^{-1} X[rows, tile] (the
// block's inverse from K3i). `first`: no update, the block [k0, k0 + kbe)
// itself is formed. A tile of 128 rows x 32 right-hand sides per CTA, 4 x 4
// entries per thread; both products read their 128-row operand in chunks of
// K through one cp.async ring, so the inverse arrives during the update. (Every
// CTA forming the block's solution for itself, operands whole in shared
// memory: 33 us a step, FP32, 64 right-hand sides, n = 5 000; 16 us now.)
// ---------------------------------------------------------------------------
constexpr int kSolveKb = 128;
constexpr int kSolveCols = 32;  // right-hand sides per CTA

template <typename T>
struct StepCfg {
  static constexpr int kV = 16 / (int)sizeof(T);
  static constexpr int kKC = 8 * kV, kStages = 3;  // K per chunk
  static constexpr int kBS = kKC + kV;             // row stride of the Y chunk, [c][k]
  static constexpr int kXS = kSolveKb + kV;        // row stride of the block's X, [c][k]
  static constexpr int kStage = kKC * kSolveKb + kSolveCols * kBS;
  static constexpr size_t kSmem = sizeof(T) * (kStages * kStage + kSolveCols * kXS);
};

template <typename T, bool UPPER, bool VEC>
__global__ void __launch_bounds__(256) block_solve_step_kernel(const T* __restrict__ lu, int lda, int n, int k0,
                                                               int kbe, const T* __restrict__ inv, T* __restrict__ x,
                                                               T* __restrict__ y, int nrhs, int first) {
  using Cfg = StepCfg<T>;
  constexpr int kV = Cfg::kV, kKC = Cfg::kKC, kStages = Cfg::kStages, kBS = Cfg::kBS, kXS = Cfg::kXS;
  struct alignas(16) Vec {
    T e[kV];
  };
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  T* Xs = ring + kStages * Cfg::kStage;
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int c0 = blockIdx.y * kSolveCols;
  const int nc = min(kSolveCols, nrhs - c0);
  // this CTA's rows; CTA x = 0 has the next block's
  int r0, r1;
  if (first) {
    r0 = k0, r1 = k0 + kbe;
  } else if (UPPER) {
    r1 = k0 - blockIdx.x * kSolveKb, r0 = r1 - kSolveKb;
  } else {
    r0 = k0 + kbe + blockIdx.x * kSolveKb, r1 = min(n, r0 + kSolveKb);
  }
  const int nr = r1 - r0;
  const int nch1 = first ? 0 : (kbe + kKC - 1) / kKC;
  const int nch = nch1 + (blockIdx.x == 0 ? (nr + kKC - 1) / kKC : 0);

  auto copy = [&](T* dst, const T* src, int count) {  // kV entries (VEC) or one; count of them valid
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (VEC)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src),
                   "r"(max(0, min(kV, count)) * (int)sizeof(T)) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(sizeof(T)),
                   "r"(count > 0 ? (int)sizeof(T) : 0) : "memory");
  };
  constexpr int P = VEC ? kV : 1;
  auto load_chunk = [&](int ch) {
    T* As = ring + (ch % kStages) * Cfg::kStage;  // [k][i]
    T* Bs = As + kKC * kSolveKb;                  // [c][k]
    const bool upd = ch < nch1;
    const int kc = (upd ? ch : ch - nch1) * kKC;
#pragma unroll 4
    for (int e = tid; e < kKC * kSolveKb / P; e += 256) {
      const int i = P * (e % (kSolveKb / P)), k = e / (kSolveKb / P);
      if (upd) {
        const int cnt = kc + k < kbe ? nr - i : 0;
        copy(As + k * kSolveKb + i, cnt > 0 ? lu + (size_t)(r0 + i) + (size_t)(k0 + kc + k) * lda : lu, cnt);
      } else {  // the inverse is padded with zeros to kSolveKb x kSolveKb
        copy(As + k * kSolveKb + i, inv + i + (size_t)(kc + k) * kSolveKb, kV);
      }
    }
    if (upd)
      for (int e = tid; e < kSolveCols * kKC / P; e += 256) {
        const int k = P * (e % (kKC / P)), c = e / (kKC / P);
        const int cnt = c < nc ? kbe - (kc + k) : 0;
        copy(Bs + c * kBS + k, cnt > 0 ? y + (size_t)(k0 + kc + k) + (size_t)(c0 + c) * n : y, cnt);
      }
  };
#pragma unroll
  for (int st = 0; st < kStages - 1; ++st) {
    if (st < nch) load_chunk(st);
    cp_async_commit_group();
  }
  T acc[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = tx + 32 * r, cc = ty * 4 + c;
      acc[r][c] = (i < nr && cc < nc) ? x[(size_t)(r0 + i) + (size_t)(c0 + cc) * n] : T(0);
    }
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait_group<kStages - 2>();
    if (ch == nch1) {  // the block's rows are final: on to its inverse
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          Xs[(ty * 4 + c) * kXS + tx + 32 * r] = acc[r][c];
          acc[r][c] = T(0);
        }
    }
    __syncthreads();  // chunk ch is here for every thread, and chunk ch - 1's stage is free
    if (ch + kStages - 1 < nch) load_chunk(ch + kStages - 1);
    cp_async_commit_group();
    const bool upd = ch < nch1;
    const T* As = ring + (ch % kStages) * Cfg::kStage;
    const T* Bs = upd ? As + kKC * kSolveKb : Xs + (ch - nch1) * kKC;
    const int bs = upd ? kBS : kXS;
#pragma unroll 2
    for (int k = 0; k < kKC; k += kV) {
      Vec bv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) bv[c] = *reinterpret_cast<const Vec*>(Bs + (ty * 4 + c) * bs + k);
#pragma unroll
      for (int q = 0; q < kV; ++q) {
        T av[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const T v = As[(k + q) * kSolveKb + tx + 32 * r];
          av[r] = upd ? -v : v;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fma_rn(av[r], bv[c].e[q], acc[r][c]);
      }
    }
  }
  cp_async_wait_group<0>();
  T* out = blockIdx.x == 0 ? y : x;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = tx + 32 * r, cc = ty * 4 + c;
      if (i < nr && cc < nc) out[(size_t)(r0 + i) + (size_t)(c0 + cc) * n] = acc[r][c];
    }
}

// x[i, c] = b[perm[i], c] (the row interchanges of P, n x ncols); with a guard,
// nothing when its factorization failed
template <typename T>
__global__ void gather_perm_rows_kernel(const T* __restrict__ b, int ldb, const int* __restrict__ perm, int n,
                                        int ncols, T* __restrict__ x, int ldx, const DevStatus* guard) {
  if (guard != nullptr && factor_failed(guard)) return;
  const size_t cnt = (size_t)n * ncols;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < cnt; e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), c = (int)(e / n);
    x[(size_t)i + (size_t)c * ldx] = b[(size_t)perm[i] + (size_t)c * ldb];
  }
}

// ---------------------------------------------------------------------------
// K4: C -= A B on the CUDA cores (the exact FP64 update and the FP32 one).
// Every entry takes its terms in increasing k, each a rounded multiply-
// subtract (EXACT: rounded product, then rounded difference), so it equals
// the rank-1 order of the reference's loop bit for bit.
//
// 128 threads per 64 x (8 NJ) tile: thread (tx, ty) has rows tx + 16 r and
// columns ty + 8 c, so a warp's C accesses are whole 128-byte lines and its
// shared-memory reads are free of bank conflicts; A [k][m] and B [n][k] in
// chunks of 16 k through a three-stage cp.async ring (16-byte copies when the
// operands allow, else element by element; out-of-range elements are
// zero-filled, which leaves every in-range entry unchanged bit for bit). A CTA
// also asks L2 for the C tile its slot takes next. Bound by the FP64 (FP32)
// pipe. Measured: see the table at gemm_sub_dev.
// ---------------------------------------------------------------------------
template <typename T, int NJ>
struct SubCfg {
  static constexpr int kBM = 64, kBN = 8 * NJ, kBK = 16, kThreads = 128, kStages = 3;
  static constexpr int kV = 16 / (int)sizeof(T);
  static constexpr int kBS = kBK + kV;  // B's row stride
  static constexpr int kStage = kBK * kBM + kBN * kBS;
  static constexpr size_t kSmem = sizeof(T) * kStages * kStage;
  static constexpr int kCtas = sizeof(T) == 8 && NJ == 8 ? 4 : 5;  // per SM
};

template <typename T, bool EXACT, int NJ, bool VEC>
__global__ void __launch_bounds__(128, SubCfg<T, NJ>::kCtas)
    gemm_sub_kernel(int M, int N, int K, const T* __restrict__ A, int lda, const T* __restrict__ B, int ldb,
                    T* __restrict__ Cm, int ldc, int ahead) {
  using Cfg = SubCfg<T, NJ>;
  constexpr int kBM = Cfg::kBM, kBN = Cfg::kBN, kBK = Cfg::kBK, kThreads = Cfg::kThreads, kStages = Cfg::kStages;
  constexpr int kV = Cfg::kV, kBS = Cfg::kBS, kStage = Cfg::kStage;
  struct alignas(16) Vec {
    T e[kV];
  };
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* smem = reinterpret_cast<T*>(smem_raw);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;

  auto load_stage = [&](int stage, int k0) {
    T* As = smem + stage * kStage;  // [k][m]
    T* Bs = As + kBK * kBM;         // [n][k]
    constexpr int P = VEC ? kV : 1;  // entries per copy
    auto copy = [&](T* dst, const T* src, int count) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
      if constexpr (VEC)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src),
                     "r"(max(0, min(kV, count)) * (int)sizeof(T)) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(sizeof(T)),
                     "r"(count > 0 ? (int)sizeof(T) : 0) : "memory");
    };
#pragma unroll
    for (int r = 0; r < kBK * kBM / (P * kThreads); ++r) {
      const int e = tid + r * kThreads;
      const int mm = P * (e % (kBM / P)), kk = e / (kBM / P);
      const int gm = m0 + mm, gk = k0 + kk;
      const int cnt = gk < K ? M - gm : 0;
      copy(As + kk * kBM + mm, cnt > 0 ? A + (size_t)gm + (size_t)gk * lda : A, cnt);
    }
#pragma unroll
    for (int r = 0; r < kBK * kBN / (P * kThreads); ++r) {
      const int e = tid + r * kThreads;
      const int kk = P * (e % (kBK / P)), nn = e / (kBK / P);
      const int gn = n0 + nn, gk = k0 + kk;
      const int cnt = gn < N ? K - gk : 0;
      copy(Bs + nn * kBS + kk, cnt > 0 ? B + (size_t)gk + (size_t)gn * ldb : B, cnt);
    }
  };

  const int nch = (K + kBK - 1) / kBK;
#pragma unroll
  for (int st = 0; st < kStages - 1; ++st) {
    if (st < nch) load_stage(st, st * kBK);
    cp_async_commit_group();
  }
  T acc[4][NJ];
#pragma unroll
  for (int c = 0; c < NJ; ++c) {
    const int nj = n0 + ty + 8 * c;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int mi = m0 + tx + 16 * r;
      acc[r][c] = (mi < M && nj < N) ? Cm[(size_t)mi + (size_t)nj * ldc] : T(0);
    }
  }
  {
    constexpr int kLine = 128 / (int)sizeof(T);
    const int nxt = (int)(blockIdx.x + blockIdx.y * gridDim.x) + ahead;
    if (nxt < (int)(gridDim.x * gridDim.y)) {
      const int pm = (nxt % (int)gridDim.x) * kBM, pn = (nxt / (int)gridDim.x) * kBN;
      for (int e = tid; e < kBN * (kBM / kLine); e += kThreads) {
        const int r = pm + kLine * (e % (kBM / kLine)), c = pn + e / (kBM / kLine);
        if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(Cm + (size_t)r + (size_t)c * ldc));
      }
    }
  }
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait_group<kStages - 2>();  // chunk ch has landed
    __syncthreads();                     // ... for every thread, and chunk ch - 1's stage is free
    if (ch + kStages - 1 < nch) load_stage((ch + kStages - 1) % kStages, (ch + kStages - 1) * kBK);
    cp_async_commit_group();
    const T* As = smem + (ch % kStages) * kStage;
    const T* Bs = As + kBK * kBM;
#pragma unroll
    for (int k0 = 0; k0 < kBK; k0 += kV) {
      Vec bv[NJ];
#pragma unroll
      for (int c = 0; c < NJ; ++c) bv[c] = *reinterpret_cast<const Vec*>(Bs + (ty + 8 * c) * kBS + k0);
#pragma unroll
      for (int q = 0; q < kV; ++q) {
        T av[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) av[r] = As[(k0 + q) * kBM + tx + 16 * r];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < NJ; ++c) acc[r][c] = msub<EXACT>(acc[r][c], av[r], bv[c].e[q]);
      }
    }
  }
  cp_async_wait_group<0>();
#pragma unroll
  for (int c = 0; c < NJ; ++c) {
    const int nj = n0 + ty + 8 * c;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int mi = m0 + tx + 16 * r;
      if (mi < M && nj < N) Cm[(size_t)mi + (size_t)nj * ldc] = acc[r][c];
    }
  }
}

}  // namespace alg
