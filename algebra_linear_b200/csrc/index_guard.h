// Row numbers that kernels exchange (labels, positions, slots) are unset or
// stale once a bounded wait has run out; the launch then runs to its end and
// the host reports ALG_TIMEOUT. They are checked where they become an index.
// Plain C++.
#pragma once

#if defined(__CUDACC__)
#define ALG_HD __host__ __device__ __forceinline__
#else
#define ALG_HD inline
#endif

namespace alg {

// index if first <= index < end, else the fallback.
ALG_HD int index_or(int index, int first, int end, int fallback) {
  return index >= first && index < end ? index : fallback;
}

}  // namespace alg
