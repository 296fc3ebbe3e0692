// The rows that a thread of the whole-block bandpass takes of a long channel.  Plain
// C++ beside the kernel's use.
#pragma once
#include <type_traits>

#ifdef __CUDACC__
#define VFRB_ROWS_HD __host__ __device__ __forceinline__
#else
#define VFRB_ROWS_HD inline
#endif

namespace vfrb {

constexpr int kBpFullThreads = 256;  // threads of a channel

// A row's number: 64 bits for channels in memory, which may hold more rows than 32
// bits count past the last step; 32 bits for those that a CTA keeps.
template <bool MEMORY>
using BpFullRow = std::conditional_t<MEMORY, long long, unsigned>;

// f(t) for t = first, first + kBpFullThreads, ... < nrows
template <int UNROLL, typename Row, typename F>
VFRB_ROWS_HD void bp_full_rows(Row first, Row nrows, F f) {
#ifdef __CUDA_ARCH__
#pragma unroll UNROLL
#endif
  for (Row t = first; t < nrows; t += kBpFullThreads) f(t);
}

}  // namespace vfrb
