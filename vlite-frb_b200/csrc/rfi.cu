// Optional bandpass / zero-DM modes that the reference keeps as dead code
// (its calls are commented out), offered here for RFI-heavy data.  Both work
// in place on the channel-major FP32 filterbank fb[c * chan_stride + row].
//
//  * k_subtract_bp_full -- subtractbp (PIPE:1372-1424): one clipped mean per
//    channel over the whole block instead of per 128-row cal window.  Kept as
//    the reference computes it: the first mean divides the channel's sum by
//    NCHANOUT (the number of channels) rather than by the number of rows, the
//    variance ("sig") is taken about that value, the clip is the open interval
//    ave +- 3 sig, and an empty clip window divides by zero.
//  * k_subtract_zero -- subtractZERO (PIPE:1478-1515): per time row, the
//    clipped mean across channels (count floored at 1) is subtracted from
//    every channel, removing the zero-DM (undispersed) signal.
//
// Sums are FP64 (the reference sums sequentially in FP32).  The statistics need
// three passes over the same values (mean, variance, clipped mean) and a fourth
// to subtract.  Both kernels keep the values in shared memory meanwhile, so
// memory is read once and written once; lengths that do not fit there go
// through memory four times.
#include "vfrb_common.cuh"

#include <algorithm>

namespace vfrb {

__device__ __forceinline__ double rfi_wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// x < hi (x > lo) of a float against a double threshold, decided in FP32: the
// threshold rounded away from the interval's inside orders every float alike
// (NaN stays NaN, and compares false)
__device__ __forceinline__ float clip_hi(double hi) { return __double2float_ru(hi); }
__device__ __forceinline__ float clip_lo(double lo) { return __double2float_rd(lo); }

// ---- whole-block clipped channel mean ------------------------------------------
// one CTA (256 threads) per channel.  CACHED: the channel's rows in shared memory
// (30 kB at 7680 rows: several CTAs per SM hide each other's passes).  7680 rows x
// 6250 channels: 144 us with four passes over memory, 102 us.
template <bool CACHED>
__global__ void __launch_bounds__(256) k_subtract_bp_full(float* __restrict__ fb, long long chan_stride, long long row0,
                                                          unsigned row_mask, int nchan, long long nrows) {
  extern __shared__ float bp_smem[];
  __shared__ double red[2][8];
  const int c = blockIdx.x;
  float* x = fb + (long long)c * chan_stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // 32-bit row arithmetic is enough: the ring's (or linear run's) rows are below 2^32
  const unsigned r0 = (unsigned)row0;
  auto mem = [&](unsigned t) -> float& { return x[(r0 + t) & row_mask]; };
  const unsigned n32 = (unsigned)nrows;
  auto block_sum2 = [&](double a, double b, double& sa, double& sb) {
    a = rfi_wsum(a);
    b = rfi_wsum(b);
    __syncthreads();
    if (lane == 0) {
      red[0][warp] = a;
      red[1][warp] = b;
    }
    __syncthreads();
    sa = sb = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      sa += red[0][w];
      sb += red[1][w];
    }
  };
  auto at = [&](unsigned t) -> float { return CACHED ? bp_smem[t] : mem(t); };
  double s = 0.0, dummy;
  if (CACHED) {
    unsigned t = threadIdx.x;
    for (; t + 7 * 256 < n32; t += 8 * 256) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = mem(t + 256 * u);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        bp_smem[t + 256 * u] = v[u];
        s += (double)v[u];
      }
    }
    for (; t < n32; t += 256) {
      const float v = mem(t);
      bp_smem[t] = v;
      s += (double)v;
    }
  } else {
    for (unsigned t = threadIdx.x; t < n32; t += 256) s += (double)mem(t);
  }
  double tot;
  block_sum2(s, 0.0, tot, dummy);
  const double ave = tot / (double)nchan;  // the reference divides by NCHANOUT
  double d1 = 0.0, d2 = 0.0;
#pragma unroll 4
  for (unsigned t = threadIdx.x; t < n32; t += 256) {
    const double d = (double)at(t) - ave;
    d1 += d;
    d2 += d * d;
  }
  double sum, sum2;
  block_sum2(d1, d2, sum, sum2);
  const double n = (double)nrows;
  const double sig = (sum2 - sum * sum / n) / (n - 1.0);
  const float hi = clip_hi(ave + 3.0 * sig), lo = clip_lo(ave - 3.0 * sig);
  double cs = 0.0;
  int cn = 0;
#pragma unroll 4
  for (unsigned t = threadIdx.x; t < n32; t += 256) {
    const float v = at(t);
    if (v < hi && v > lo) {
      cs += (double)v;
      ++cn;
    }
  }
  double csum, cnt;
  block_sum2(cs, (double)cn, csum, cnt);
  const float m = (float)(csum / cnt);  // cnt == 0 gives NaN, as the reference's ave/=i
#pragma unroll 4
  for (unsigned t = threadIdx.x; t < n32; t += 256) mem(t) = at(t) - m;
}

// ---- zero-DM ----------------------------------------------------------------------
// A CTA takes 8 consecutive rows of every channel: 32-byte runs, a whole sector of
// memory each, into shared memory (200 kB at 6250 channels) with asynchronous
// copies.  Thread t has row t % 8 and every 64th channel, so a warp's shared
// accesses are 32 consecutive words.  The clipped mean of a row that loses nothing
// to the clip is its sum, so the third pass only compares, in FP32.  7680 rows x
// 6250 channels: 4.99 ms with a thread per row and four passes over memory (30
// CTAs), 0.21 ms.  Clusters of eight CTAs with 32-row tiles (full 128-byte lines,
// two CTAs per SM) took 0.23 ms.
constexpr int kZeroRows = 8;
constexpr int kZeroThreads = 512;
constexpr int kZeroLanes = kZeroThreads / kZeroRows;  // threads per row

__global__ void __launch_bounds__(kZeroThreads) k_subtract_zero(float* __restrict__ fb, long long chan_stride,
                                                                long long row0, unsigned row_mask, int nchan,
                                                                long long nrows) {
  extern __shared__ float z_smem[];  // [nchan][8]
  __shared__ double red[2][kZeroThreads / 32][kZeroRows];
  const int rl = threadIdx.x % kZeroRows, cl = threadIdx.x / kZeroRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long t = (long long)blockIdx.x * kZeroRows + rl;
  const bool live = t < nrows;
  float* x = fb + ((unsigned long long)(row0 + (live ? t : 0)) & (unsigned long long)row_mask);
  for (int c = cl; c < nchan; c += kZeroLanes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(z_smem + c * kZeroRows + rl);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(x + (long long)c * chan_stride),
                 "r"(live ? 4 : 0));
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  // (a thread reads back only what it copied: no barrier needed)
  auto row_sum2 = [&](double a, double b, double& sa, double& sb) {
    a += __shfl_xor_sync(0xffffffffu, a, 8);
    b += __shfl_xor_sync(0xffffffffu, b, 8);
    a += __shfl_xor_sync(0xffffffffu, a, 16);
    b += __shfl_xor_sync(0xffffffffu, b, 16);
    __syncthreads();
    if (lane < kZeroRows) {
      red[0][warp][lane] = a;
      red[1][warp][lane] = b;
    }
    __syncthreads();
    sa = sb = 0.0;
#pragma unroll
    for (int w = 0; w < kZeroThreads / 32; ++w) {
      sa += red[0][w][rl];
      sb += red[1][w][rl];
    }
  };
  double s = 0.0, dummy;
#pragma unroll 4
  for (int c = cl; c < nchan; c += kZeroLanes) s += (double)z_smem[c * kZeroRows + rl];
  double tot;
  row_sum2(s, 0.0, tot, dummy);
  const double ave = tot / (double)nchan;
  double d1 = 0.0, d2 = 0.0;
#pragma unroll 4
  for (int c = cl; c < nchan; c += kZeroLanes) {
    const double d = (double)z_smem[c * kZeroRows + rl] - ave;
    d1 += d;
    d2 += d * d;
  }
  double s1, s2;
  row_sum2(d1, d2, s1, s2);
  const double n = (double)nchan;
  const double sig = (s2 - s1 * s1 / n) / (n - 1.0);
  const float hi = clip_hi(ave + 3.0 * sig), lo = clip_lo(ave - 3.0 * sig);
  int out = 0;  // values that the clip rejects
#pragma unroll 4
  for (int c = cl; c < nchan; c += kZeroLanes) {
    const float v = z_smem[c * kZeroRows + rl];
    out += (v < hi && v > lo) ? 0 : 1;
  }
  double cs = 0.0, cnt = n;
  if (__syncthreads_or(out)) {  // some row loses values: sum what is kept
    int kept = 0;
    for (int c = cl; c < nchan; c += kZeroLanes) {
      const float v = z_smem[c * kZeroRows + rl];
      if (v < hi && v > lo) {
        cs += (double)v;
        ++kept;
      }
    }
    double csum;
    row_sum2(cs, (double)kept, csum, cnt);
    cs = csum;
  } else {
    cs = tot;
  }
  const float m = (float)(cs / (cnt > 0.0 ? cnt : 1.0));
  if (live) {
#pragma unroll 4
    for (int c = cl; c < nchan; c += kZeroLanes) x[(long long)c * chan_stride] = z_smem[c * kZeroRows + rl] - m;
  }
}

// More channels than fit in shared memory: one thread per row; a warp covers 32
// consecutive rows, so every channel's load is one 128-byte segment
__global__ void __launch_bounds__(256) k_subtract_zero_wide(float* __restrict__ fb, long long chan_stride, long long row0,
                                                            unsigned row_mask, int nchan, long long nrows) {
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
  if (t >= nrows) return;
  float* x = fb + ((unsigned long long)(row0 + t) & (unsigned long long)row_mask);
  double s = 0.0;
  for (int c = 0; c < nchan; ++c) s += (double)x[(long long)c * chan_stride];
  const double ave = s / (double)nchan;
  double d1 = 0.0, d2 = 0.0;
  for (int c = 0; c < nchan; ++c) {
    const double d = (double)x[(long long)c * chan_stride] - ave;
    d1 += d;
    d2 += d * d;
  }
  const double n = (double)nchan;
  const double sig = (d2 - d1 * d1 / n) / (n - 1.0);
  const double hi = ave + 3.0 * sig, lo = ave - 3.0 * sig;
  double cs = 0.0;
  int cnt = 0;
  for (int c = 0; c < nchan; ++c) {
    const double v = (double)x[(long long)c * chan_stride];
    if (v < hi && v > lo) {
      cs += v;
      ++cnt;
    }
  }
  const float m = (float)(cs / (double)(cnt > 0 ? cnt : 1));
  for (int c = 0; c < nchan; ++c) x[(long long)c * chan_stride] -= m;
}

// rows [row0, row0 + nrows) of every channel must lie in its chan_stride
// elements: a power-of-two ring (row_mask + 1 <= chan_stride) or a linear run
static bool rfi_args_ok(const float* fb, long long chan_stride, long long row0, unsigned row_mask, int nchan,
                        long long nrows) {
  if (!fb || nchan < 2 || nrows < 2 || chan_stride < 1) return false;
  if (row_mask != 0xffffffffu) {
    const unsigned long long r = (unsigned long long)row_mask + 1ULL;
    if ((r & (r - 1)) != 0 || (long long)r < nrows || chan_stride < (long long)r) return false;
  } else if (row0 < 0 || row0 + nrows > chan_stride) {
    return false;
  }
  return true;
}

constexpr int kRfiSmem = 220 * 1024;  // of the dynamic kind, beside the sums

template <typename K>
static int rfi_smem(K kern) {  // one limit, whoever launches
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRfiSmem) != cudaSuccess) {
    cudaGetLastError();
    return VFRB_ERR_CUDA;
  }
  return VFRB_OK;
}

int launch_subtract_bp_full(float* fb, long long chan_stride, long long row0, unsigned row_mask, int nchan,
                            long long nrows, cudaStream_t s) {
  if (!rfi_args_ok(fb, chan_stride, row0, row_mask, nchan, nrows)) return VFRB_ERR_ARG;
  if (nrows * 4 <= kRfiSmem) {
    if (const int st = rfi_smem(k_subtract_bp_full<true>)) return st;
    k_subtract_bp_full<true><<<nchan, 256, (size_t)nrows * 4, s>>>(fb, chan_stride, row0, row_mask, nchan, nrows);
  } else {
    k_subtract_bp_full<false><<<nchan, 256, 0, s>>>(fb, chan_stride, row0, row_mask, nchan, nrows);
  }
  return cuda_status(cudaGetLastError());
}

int launch_subtract_zero(float* fb, long long chan_stride, long long row0, unsigned row_mask, int nchan,
                         long long nrows, cudaStream_t s) {
  if (!rfi_args_ok(fb, chan_stride, row0, row_mask, nchan, nrows)) return VFRB_ERR_ARG;
  const long long smem = (long long)nchan * kZeroRows * 4;
  if (smem <= kRfiSmem) {
    const long long nb = (nrows + kZeroRows - 1) / kZeroRows;
    if (nb > 0x7fffffffLL) return VFRB_ERR_UNSUPPORTED;
    if (const int st = rfi_smem(k_subtract_zero)) return st;
    k_subtract_zero<<<(unsigned)nb, kZeroThreads, (size_t)smem, s>>>(fb, chan_stride, row0, row_mask, nchan, nrows);
  } else {
    const long long nb = (nrows + 255) / 256;
    if (nb > 0x7fffffffLL) return VFRB_ERR_UNSUPPORTED;
    k_subtract_zero_wide<<<(unsigned)nb, 256, 0, s>>>(fb, chan_stride, row0, row_mask, nchan, nrows);
  }
  return cuda_status(cudaGetLastError());
}

}  // namespace vfrb

extern "C" int vfrb_subtract_bp_full(float* fb_cm, int64_t chan_stride, int64_t row0, uint32_t row_mask, int nchan,
                                     int64_t nrows, void* stream) {
  return vfrb::launch_subtract_bp_full(fb_cm, chan_stride, row0, row_mask, nchan, nrows, (cudaStream_t)stream);
}

extern "C" int vfrb_subtract_zero(float* fb_cm, int64_t chan_stride, int64_t row0, uint32_t row_mask, int nchan,
                                  int64_t nrows, void* stream) {
  return vfrb::launch_subtract_zero(fb_cm, chan_stride, row0, row_mask, nchan, nrows, (cudaStream_t)stream);
}
