// Loops of a thread over every STEP-th row of a channel, and the types that number the
// rows.  Plain C++ beside the kernels' use.
#pragma once
#include <type_traits>

#ifdef __CUDACC__
#define VFRB_WALK_HD __host__ __device__ __forceinline__
#else
#define VFRB_WALK_HD inline
#endif

namespace vfrb {

// Whole-block bandpass: 64 bits for channels in memory, which may hold more rows than
// 32 bits count past the last step; 32 bits for those that a CTA keeps.
template <bool MEMORY>
using BpFullRow = std::conditional_t<MEMORY, long long, unsigned>;
constexpr int kBpFullThreads = 256;  // threads of a channel

// Channel statistics: the rows of a block are an int, whose largest a last step passes.
using StatsRow = unsigned;

// f(t) for t = first, first + STEP, ... < nrows; UNROLL 0: unrolled as the compiler likes
template <int STEP, int UNROLL, typename Row, typename F>
VFRB_WALK_HD void walk_rows(Row first, Row nrows, F f) {
  if constexpr (UNROLL == 0) {
    for (Row t = first; t < nrows; t += STEP) f(t);
  } else {
#ifdef __CUDA_ARCH__
#pragma unroll UNROLL
#endif
    for (Row t = first; t < nrows; t += STEP) f(t);
  }
}

}  // namespace vfrb
