// K2: bandpass + noise-cal subtraction, K4: per-channel statistics, and the
// channel-major -> time-major copy.  HBM-bound kernels for sm_100a.
//
// K2 replaces subtractbpCAL (PIPE:1427-1474; STATS:869-908; TS:1365-1407).
// A CTA takes one window of <=128 rows x 32 channels of the raw time-major
// filterbank (coalesced 128-byte row segments), transposes it in shared memory,
// and computes in FP64: mean, the variance the reference calls "sig", the
// open-interval clip ave +- 3 sig and the clipped mean (count floored at 1).  Eight
// lanes share a channel, 16 rows each, so a sum takes three shuffles and four
// channels reduce at once, and a row is converted to FP64 once.  (A warp per
// channel, four rows per lane, spent more on its five-step reductions than on the
// rows.)  The subtracted rows are written channel-major (512-byte runs per
// channel), the layout the dedisperser streams, in FP32, FP16 (z = x/s_c) or int8
// (round(z*q)) form.  subtract_mode 1 skips the statistics and writes the rows
// unchanged (the input of the whole-block subtractbp in rfi.cu).  The FP16 form
// can also write a copy shifted by one row, out1[c][r - 1] = out[c][r] (absolute
// rows, the same ring geometry): with both copies the four-trial pattern kernel
// reads any window of halves with aligned 4-byte loads.
//
// Bound by instruction issue: it was 50 instructions per value, most of them row
// addresses through the rings' masks; where a window does not wrap a ring (all but
// one in a ring's length) rows are pointer steps.  7680 rows x 6250 channels: 201 ->
// 92 us; FP16 with the shifted copy, 1024 rows: 37 -> 22 us.
#include "row_walk.h"
#include "vfrb_common.cuh"

#include <algorithm>

namespace vfrb {

constexpr int kBpThreads = 256;  // 8 warps
constexpr int kBpChan = 32;      // channels per CTA
constexpr int kBpMaxWin = 128;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// over each eight neighbouring lanes
__device__ __forceinline__ double sum8(double v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int STORAGE>
struct BpOut;
template <>
struct BpOut<VFRB_F32> {
  using T = float;
  __device__ static T of(float y, float, float) { return y; }
};
template <>
struct BpOut<VFRB_F16> {
  using T = __half;
  __device__ static T of(float y, float inv, float) { return __float2half_rn(y * inv); }
};
template <>
struct BpOut<VFRB_I8> {
  using T = int8_t;
  __device__ static T of(float y, float inv, float q) {
    return (int8_t)fminf(fmaxf(rintf(y * inv * q), -127.f), 127.f);
  }
};

// FULL: the window has kBpMaxWin rows and every channel of the tile exists
template <int STORAGE, bool FULL>
__device__ __forceinline__ void bp_window(const vfrb_bp_args& a, __half* __restrict__ out1,
                                          float (&tile)[kBpChan][kBpMaxWin + 1]) {
  using T = typename BpOut<STORAGE>::T;
  constexpr int kWarps = kBpThreads / 32;
  constexpr int kRows = kBpMaxWin / kWarps;  // rows a warp loads, and rows a lane sums
  const int win = blockIdx.y;
  const int c0 = blockIdx.x * kBpChan;
  const long long r0 = (long long)win * a.window;
  const int npts = FULL ? kBpMaxWin : (int)min((long long)a.window, (long long)a.nrows - r0);
  const int nc = FULL ? kBpChan : min(kBpChan, a.nchan - c0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  // rows (time-major) -> tile[ch][row]: a warp's 16 rows are loaded into registers
  // first, so all 16 row segments are in flight together
  {
    float v[kRows];
    const unsigned long long first = (unsigned long long)(a.in_row0 + r0) & (unsigned long long)a.in_row_mask;
    if (FULL && first + kBpMaxWin <= (unsigned long long)a.in_row_mask + 1ULL) {
      const float* src = a.in + (long long)(first + warp) * a.in_row_stride + c0 + lane;
      const long long step = kWarps * a.in_row_stride;
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        v[k] = *src;
        src += step;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        const int r = warp + kWarps * k;
        const unsigned long long rr = (unsigned long long)(a.in_row0 + r0 + r) & (unsigned long long)a.in_row_mask;
        v[k] = (r < npts && lane < nc) ? a.in[(long long)rr * a.in_row_stride + c0 + lane] : 0.f;
      }
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) tile[lane][warp + kWarps * k] = v[k];
  }
  __syncthreads();

  if (a.subtract_mode == 0 || a.win_mean || a.win_var) {
    // lanes g, g + 8, ... of channel cl = warp + 8 (lane / 8): with the tile's odd
    // pitch the 32 lanes of a load touch 32 banks
    const int g = lane & 7, cl = warp + kWarps * (lane >> 3);
    float* row = tile[cl] + g;
    double cave = 0.0, sig = 0.0;  // subtract_mode 1: copy only (cave = 0)
    if (a.subtract_mode == 0) {
      double xd[kRows];
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        xd[k] = (double)row[8 * k];  // rows past the window hold zeros
        s += xd[k];
      }
      const double n = (double)npts;
      s = sum8(s);
      const double ave = s / n;
      double sd = 0.0, sd2 = 0.0;
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        if (FULL || g + 8 * k < npts) {
          const double d = xd[k] - ave;
          sd += d;
          sd2 += d * d;
        }
      }
      sd = sum8(sd);
      sd2 = sum8(sd2);
      sig = (sd2 - (sd * sd) / n) / (n - 1.0);  // variance, NaN when npts == 1
      const double hi = ave + 3.0 * sig, lo = ave - 3.0 * sig;
      bool all = true;
#pragma unroll
      for (int k = 0; k < kRows; ++k)
        if (FULL || g + 8 * k < npts) all = all && xd[k] < hi && xd[k] > lo;
      double cnt = n, cs = s;
      if (!__all_sync(0xffffffffu, all)) {  // some channel of the warp loses rows
        int kept = 0;
        cs = 0.0;
#pragma unroll
        for (int k = 0; k < kRows; ++k)
          if ((FULL || g + 8 * k < npts) && xd[k] < hi && xd[k] > lo) {
            cs += xd[k];
            ++kept;
          }
        cs = sum8(cs);
        cnt = sum8((double)kept);
        if (cnt == 0.0) cnt = 1.0;
      }
      cave = cs / cnt;
#pragma unroll
      for (int k = 0; k < kRows; ++k) row[8 * k] = (float)(xd[k] - cave);
    }
    if (g == 0 && cl < nc) {
      if (a.win_mean) a.win_mean[(long long)win * a.nchan + c0 + cl] = (float)cave;
      if (a.win_var) a.win_var[(long long)win * a.nchan + c0 + cl] = (float)sig;
    }
    __syncthreads();
  }

  // tile -> channel-major rows, a warp per channel
  const unsigned long long omask = (unsigned long long)a.out_row_mask;
  const unsigned long long first = (unsigned long long)(a.out_row0 + r0) & omask;
  const bool straight = FULL && first + kBpMaxWin <= omask + 1ULL;
  T* const out = reinterpret_cast<T*>(a.out);
#pragma unroll 1
  for (int cl = warp; cl < nc; cl += kWarps) {
    const float inv = (STORAGE == VFRB_F32) ? 1.f : a.inv_scale[c0 + cl];
    T* dst = out + (long long)(c0 + cl) * a.out_chan_stride;
    const float* row = tile[cl];
    if (straight && STORAGE == VFRB_F16 && ((uintptr_t)(dst + first) & 3) == 0) {
      // two rows per store; the shifted copy's pairs (rows 2i + 1, 2i + 2) start where
      // this one's do, and its row before the window and the window's last row alone
      __half2* d2 = reinterpret_cast<__half2*>(dst + first);
      __half* d1 = out1 ? out1 + (long long)(c0 + cl) * a.out_chan_stride : nullptr;
#pragma unroll
      for (int k = 0; k < kBpMaxWin / 64; ++k) {
        const int i = lane + 32 * k;
        const __half lo = __float2half_rn(row[2 * i] * inv), hi = __float2half_rn(row[2 * i + 1] * inv);
        d2[i] = __halves2half2(lo, hi);
        if (d1) {
          const __half up = __shfl_down_sync(0xffffffffu, lo, 1);  // row 2i + 2 of the next lane
          if (lane < 31) {
            if (((uintptr_t)(d1 + first) & 3) == 0) {
              reinterpret_cast<__half2*>(d1 + first)[i] = __halves2half2(hi, up);
            } else {
              d1[first + 2 * i] = hi;
              d1[first + 2 * i + 1] = up;
            }
          } else {
            d1[first + 2 * i] = hi;
            if (2 * i + 2 < kBpMaxWin) d1[first + 2 * i + 1] = __float2half_rn(row[2 * i + 2] * inv);
          }
          if (i == 0 && a.out_row0 + r0 >= 1)
            d1[(unsigned long long)(a.out_row0 + r0 - 1) & omask] = lo;
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < kBpMaxWin / 32; ++k) {
        const int r = lane + 32 * k;
        if (FULL || r < npts) {
          const T v = BpOut<STORAGE>::of(row[r], inv, a.q_scale);
          const long long ra = a.out_row0 + r0 + r;  // absolute row; row ra - 1 of the shifted copy
          if (straight) dst[first + r] = v;
          else dst[(unsigned long long)ra & omask] = v;
          if constexpr (STORAGE == VFRB_F16) {
            if (out1 && ra >= 1)
              out1[(long long)(c0 + cl) * a.out_chan_stride + (long long)((unsigned long long)(ra - 1) & omask)] = v;
          }
        }
      }
    }
  }
  if (a.tm_out) {
    for (int r = warp; r < npts; r += kWarps)
      if (lane < nc) a.tm_out[(r0 + r) * a.tm_row_stride + c0 + lane] = tile[lane][r];
  }
}

// (four CTAs per SM: 64 registers; 92 us at 7680 x 6250, with three 100, with five,
// which spills, 102)
template <int STORAGE>
__global__ void __launch_bounds__(kBpThreads, 4) k_bandpass(const __grid_constant__ vfrb_bp_args a,
                                                         __half* __restrict__ out1) {
  __shared__ float tile[kBpChan][kBpMaxWin + 1];
  const bool full = a.window == kBpMaxWin && (long long)(blockIdx.y + 1) * kBpMaxWin <= a.nrows &&
                    ((int)blockIdx.x + 1) * kBpChan <= a.nchan;
  if (full) bp_window<STORAGE, true>(a, out1, tile);
  else bp_window<STORAGE, false>(a, out1, tile);
}

int launch_bandpass(const vfrb_bp_args& a, cudaStream_t s) {
  if (a.nrows <= 0) return a.nrows == 0 ? VFRB_OK : VFRB_ERR_ARG;
  if (a.out_shift1 && (a.storage != VFRB_F16 || a.out_row0 < 0 || ((uintptr_t)a.out_shift1 & 1))) return VFRB_ERR_ARG;
  if (!a.in || !a.out || a.nchan <= 0 || a.window <= 0 || a.window > kBpMaxWin) return VFRB_ERR_ARG;
  if (a.storage != VFRB_F32 && !a.inv_scale) return VFRB_ERR_ARG;
  if (a.subtract_mode != 0 && a.subtract_mode != 1) return VFRB_ERR_ARG;
  const int nwin = (a.nrows + a.window - 1) / a.window;
  dim3 grid((a.nchan + kBpChan - 1) / kBpChan, nwin);
  switch (a.storage) {
    case VFRB_F32: k_bandpass<VFRB_F32><<<grid, kBpThreads, 0, s>>>(a, nullptr); break;
    case VFRB_F16: k_bandpass<VFRB_F16><<<grid, kBpThreads, 0, s>>>(a, static_cast<__half*>(a.out_shift1)); break;
    case VFRB_I8: k_bandpass<VFRB_I8><<<grid, kBpThreads, 0, s>>>(a, nullptr); break;
    default: return VFRB_ERR_ARG;
  }
  return cuda_status(cudaGetLastError());
}

// ---- K4: per-channel statistics (STATS:910-946) ---------------------------
// One warp per (channel, statistics block); the block's rows are contiguous in the
// channel-major layout.  FP64 mean and variance; the outlier count uses the
// reference's float comparison x > ave + 5*sig (decided in FP32 against the threshold
// rounded down, which orders every float alike) and stores the integer quotient
// count/npts.
//
// REGS: every block has exactly kStatsRows rows, which stay in registers (32 per lane,
// all loads in flight at once) over the three passes: 6250 channels x 7 blocks 85 -> 55
// us, 3908 x 8 64 -> 42 us.  Other blocks are read three times, mostly from the caches;
// registers with a test for every row, of one to eight warps a block, were slower: 6250
// x 7680, blocks of 1025 rows 91 against 342 us, 4096 86 against 105; 3908 x 7680,
// blocks of 300 88 against 182 us, of 16 0.86 against 3.2 ms.
constexpr int kStatsRows = 1024;
template <bool REGS>
__global__ void __launch_bounds__(256) k_chan_stats(const __grid_constant__ vfrb_cs_args a) {
  constexpr int R = kStatsRows / 32;
  const int lane = threadIdx.x & 31;
  const long long gw = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (gw >= (long long)a.nchan * a.nstatblks) return;
  const int c = (int)(gw % a.nchan);
  const int k = (int)(gw / a.nchan);
  const long long colmin = (long long)a.ncolstatblk * k;
  long long colmax = colmin + a.ncolstatblk;
  if (colmax > a.nrows) colmax = a.nrows;
  const int npts = (int)(colmax - colmin);
  const float* base = a.fb + (long long)c * a.chan_stride;
  const unsigned r0 = (unsigned)(a.row0 + colmin);  // ring rows are 32-bit
  auto at = [&](unsigned i) { return base[(r0 + i) & a.row_mask]; };
  float x[REGS ? R : 1];
  if constexpr (REGS) {
    const unsigned long long first = r0 & a.row_mask;
    if (first + kStatsRows <= (unsigned long long)a.row_mask + 1ULL) {  // the rows do not wrap the ring
      const float* src = base + first + lane;
#pragma unroll
      for (int i = 0; i < R; ++i) x[i] = src[32 * i];
    } else {
#pragma unroll
      for (int i = 0; i < R; ++i) x[i] = at(lane + 32 * i);
    }
  }
  auto each = [&](auto&& f) {
    if constexpr (REGS) {
#pragma unroll
      for (int i = 0; i < R; ++i) f(x[i]);
    } else {
      walk_rows<32, 0, StatsRow>(lane, npts, [&](StatsRow i) { f(at(i)); });
    }
  };
  double s = 0.0;
  each([&](float v) { s += (double)v; });
  const double n = (double)npts;
  const double ave = warp_sum(s) / n;
  double sd = 0.0, sd2 = 0.0;
  each([&](float v) {
    const double d = (double)v - ave;
    sd += d;
    sd2 += d * d;
  });
  sd = warp_sum(sd);
  sd2 = warp_sum(sd2);
  const double sig = (sd2 - sd * sd / n) / (n - 1.0);
  const float hi = __double2float_rd(ave + 5.0 * sig);  // x > hi of a float: x > the threshold rounded down
  int out = 0;
  each([&](float v) { out += v > hi ? 1 : 0; });
  out = __reduce_add_sync(0xffffffffu, out);
  if (lane == 0) {
    const long long o = (long long)k * a.nchan + c;
    a.ave[o] = (float)ave;
    a.sig[o] = (float)sig;
    a.outlier[o] = (float)(npts > 0 ? out / npts : 0);
  }
}

int launch_chan_stats(const vfrb_cs_args& a, cudaStream_t s) {
  if (!a.fb || !a.ave || !a.sig || !a.outlier || a.nchan <= 0 || a.nstatblks <= 0 || a.ncolstatblk <= 1)
    return VFRB_ERR_ARG;
  if ((long long)a.ncolstatblk * (a.nstatblks - 1) >= a.nrows) return VFRB_ERR_ARG;
  const unsigned blocks = (unsigned)(((long long)a.nchan * a.nstatblks + 7) / 8);
  const int rows = std::min(a.ncolstatblk, a.nrows);  // of the longest block
  if (rows == kStatsRows && (long long)rows * a.nstatblks <= a.nrows)
    k_chan_stats<true><<<blocks, 256, 0, s>>>(a);
  else
    k_chan_stats<false><<<blocks, 256, 0, s>>>(a);
  return cuda_status(cudaGetLastError());
}

// ---- spectral kurtosis per (channel, statistics block) ----------------------
// Generalised SK estimator (Nita & Gary 2010) of the raw (not bandpass-
// subtracted) power: with M rows in the block, S1 = sum x, S2 = sum x^2 and
// nsum = N*d raw power values per FB sample (2 pols x NAVE spectra, each an
// exponential variable for Gaussian noise),
//   SK = (M*nsum + 1)/(M - 1) * (M*S2/S1^2 - 1),
// whose expectation is 1 for Gaussian noise; narrowband RFI drives it below 1
// (steady tones) or far above it (bursts); a one-row block gives inf/NaN as
// M - 1 = 0.  FP64 sums.  The FB is time-major, so a warp reads 32 consecutive
// channels of a row: 128-byte segments.
// A CTA takes CH channels of one block: SETS sets of threads share its rows out (set g
// rows g, g + SETS, ..., eight loads in flight per thread), and the sets' sums are added
// in order.  64 x 16 for blocks of kSkLong rows or more: a thread per channel alone gives
// 175 CTAs of 1024 serial loads at 6250 channels x 7 blocks (93 -> 39 us).  256 x 1 for
// shorter ones, which leave most of the sets without a row (3908 channels x 7680 rows,
// blocks of 64 55 -> 29 us, of 16 172 -> 29 us; at 192 35 against 31, at 256 31 against 35).
constexpr int kSkLong = 224;
template <int CH, int SETS>
__global__ void __launch_bounds__(CH * SETS) k_chan_sk(const float* __restrict__ fb, long long row_stride,
                                                       long long row0, unsigned long long row_mask, int nchan,
                                                       int nrows, int ncolstatblk, int nstatblks, double nsum,
                                                       float* __restrict__ sk) {
  __shared__ double red[2][SETS][SETS > 1 ? CH : 1];
  const int cl = threadIdx.x % CH, g = threadIdx.x / CH;
  const int c = blockIdx.x * CH + cl;
  const int k = blockIdx.y;
  const long long r0 = (long long)ncolstatblk * k;
  const long long r1 = min(r0 + ncolstatblk, (long long)nrows);
  const float* x = fb + min(c, nchan - 1);
  auto at = [&](long long r) { return x[(long long)((unsigned long long)(row0 + r) & row_mask) * row_stride]; };
  double s1 = 0.0, s2 = 0.0;
  long long r = r0 + g;
  constexpr int U = 8;
  for (; r + (U - 1) * SETS < r1; r += U * SETS) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = at(r + u * SETS);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double d = (double)v[u];
      s1 += d;
      s2 += d * d;
    }
  }
  for (; r < r1; r += SETS) {
    const double d = (double)at(r);
    s1 += d;
    s2 += d * d;
  }
  if constexpr (SETS > 1) {
    red[0][g][cl] = s1;
    red[1][g][cl] = s2;
    __syncthreads();
  }
  if (g != 0 || c >= nchan) return;
  for (int q = 1; q < SETS; ++q) {
    s1 += red[0][q][cl];
    s2 += red[1][q][cl];
  }
  const double m = (double)(r1 - r0);
  const double v = (m * nsum + 1.0) / (m - 1.0) * (m * s2 / (s1 * s1) - 1.0);
  sk[(long long)k * nchan + c] = (float)v;
}

// rows r < nrows of the block start at ring row (row0 + r) & row_mask
// (row_mask ~0: a linear array)
int launch_chan_sk_ring(const float* fb_tm, long long row_stride, long long row0, unsigned long long row_mask,
                        int nchan, int nrows, int ncolstatblk, int nstatblks, int nsum, float* sk, cudaStream_t s) {
  if (!fb_tm || !sk || nchan <= 0 || nstatblks <= 0 || ncolstatblk <= 1 || nsum < 1 || row_stride < nchan ||
      (long long)nrows - (long long)ncolstatblk * (nstatblks - 1) < 1 || nstatblks > 65535 || row0 < 0)
    return VFRB_ERR_ARG;
  auto run = [&](auto kern, int ch, int threads) {
    kern<<<dim3((unsigned)((nchan + ch - 1) / ch), (unsigned)nstatblks), threads, 0, s>>>(
        fb_tm, row_stride, row0, row_mask, nchan, nrows, ncolstatblk, nstatblks, (double)nsum, sk);
  };
  if (std::min(ncolstatblk, nrows) >= kSkLong) run(k_chan_sk<64, 16>, 64, 1024);
  else run(k_chan_sk<256, 1>, 256, 256);
  return cuda_status(cudaGetLastError());
}

int launch_chan_sk(const float* fb_tm, long long row_stride, int nchan, int nrows, int ncolstatblk, int nstatblks,
                   int nsum, float* sk, cudaStream_t s) {
  return launch_chan_sk_ring(fb_tm, row_stride, 0, ~0ULL, nchan, nrows, ncolstatblk, nstatblks, nsum, sk, s);
}

// ---- channel-major -> time-major copy ---------------------------------------
// Tiles of 64 x 64: each warp has eight 256-byte runs' loads in flight before it
// stores the first to the tile (a 32 x 32 tile with four loads per thread ran at
// 45% of the copy rate).  32 x 32 for up to twelve channels, most of whose tile is
// empty: 8 channels x 2^20 rows 55 -> 39 us.
template <int T>
__global__ void __launch_bounds__(256) k_transpose(const float* __restrict__ src, long long chan_stride,
                                                   unsigned row_mask, long long row0, int nchan, int nrows,
                                                   float* __restrict__ dst, long long dst_row_stride) {
  __shared__ float t[T][T + 1];
  constexpr int H = T / 32;
  const int cb = blockIdx.x * T, rb = blockIdx.y * T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned r = (unsigned)(row0 + rb + lane);
  float v[T / 8][H];
#pragma unroll
  for (int i = 0; i < T / 8; ++i)
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int c = cb + warp + 8 * i;
      v[i][h] = (c < nchan && rb + lane + 32 * h < nrows) ? src[(long long)c * chan_stride + ((r + 32u * h) & row_mask)]
                                                          : 0.f;
    }
#pragma unroll
  for (int i = 0; i < T / 8; ++i)
#pragma unroll
    for (int h = 0; h < H; ++h) t[warp + 8 * i][lane + 32 * h] = v[i][h];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < T / 8; ++i)
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int row = rb + warp + 8 * i, c = cb + lane + 32 * h;
      if (row < nrows && c < nchan) dst[(long long)row * dst_row_stride + c] = t[lane + 32 * h][warp + 8 * i];
    }
}

int launch_fb_transpose(const float* src_cm, long long chan_stride, unsigned row_mask, long long row0, int nchan,
                        int nrows, float* dst_tm, long long dst_row_stride, cudaStream_t s) {
  if (!src_cm || !dst_tm || nchan <= 0 || nrows < 0) return VFRB_ERR_ARG;
  if (nrows == 0) return VFRB_OK;
  auto run = [&](auto kern, int T) {
    kern<<<dim3((nchan + T - 1) / T, (nrows + T - 1) / T), 256, 0, s>>>(src_cm, chan_stride, row_mask, row0, nchan,
                                                                        nrows, dst_tm, dst_row_stride);
  };
  // (up to the rows that a grid of the small tiles has)
  if (nchan <= 12 && nrows <= 65535 * 32) run(k_transpose<32>, 32);
  else run(k_transpose<64>, 64);
  return cuda_status(cudaGetLastError());
}

}  // namespace vfrb
