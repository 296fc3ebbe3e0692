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
// to subtract.  Both kernels keep the values in registers or shared memory
// meanwhile, so memory is read once and written once; lengths that do not fit
// there go through memory four times.
#include "row_walk.h"
#include "vfrb_common.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace cg = cooperative_groups;

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
// One CTA (256 threads) per channel.  NV > 0: a thread keeps NV rows of the channel
// in registers, all of their loads in flight at once, in quads of neighbouring rows
// where these are aligned (VEC).  NV = 0: in shared memory (CACHED), or, for channels
// too long for it, read in every pass.
//
// NV = 32 leaves 64 registers a thread, four CTAs per SM; 8192 rows are its limit.
// Bound by the FP64 sums and conversions (three per value) and the three reductions.
// 7680 rows x 6250 channels: 144 us with four passes over memory, 117 us through shared
// memory, 100 us in registers and quads; 3071 x 3908 49 -> 39 us, 60 x 3908 20 -> 19 us.
template <int NV, bool VEC, bool CACHED>
__global__ void __launch_bounds__(256, NV ? 4 : 1) k_subtract_bp_full(float* __restrict__ fb, long long chan_stride, long long row0,
                                                          unsigned row_mask, int nchan, long long nrows) {
  extern __shared__ float bp_smem[];
  __shared__ double red[3][2][8];
  __shared__ double s_ave;
  __shared__ float s_hi, s_lo, s_m;
  const int c = blockIdx.x;
  float* x = fb + (long long)c * chan_stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // rows are taken modulo 2^32, the widest mask; their count may be larger (NV = 0)
  const unsigned r0 = (unsigned)row0;
  auto mem = [&](unsigned t) -> float& { return x[(r0 + t) & row_mask]; };
  using Row = BpFullRow<NV == 0 && !CACHED>;
  const Row n = (Row)nrows;
  // done(A, B), by thread 0 (FP64 divisions are dozens of instructions), with the
  // CTA's sums of a and b
  auto block_sum2 = [&](int phase, double a, double b, auto done) {
    a = rfi_wsum(a);
    b = rfi_wsum(b);
    if (lane == 0) {
      red[phase][0][warp] = a;
      red[phase][1][warp] = b;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
      double v = red[phase][threadIdx.x >> 3][threadIdx.x & 7];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffu, v, o);
      const double w = __shfl_down_sync(0xffffu, v, 8);
      if (threadIdx.x == 0) done(v, w);
    }
    __syncthreads();
  };
  // row of register k; a pass over all rows
  auto row = [&](int k) { return VEC ? 4 * (threadIdx.x + 256 * (k / 4)) + k % 4 : threadIdx.x + 256 * k; };
  float v[NV ? NV : 1];
  if constexpr (NV > 0 && VEC) {
#pragma unroll
    for (int k = 0; k < NV; k += 4)
      if (row(k) < n) {
        const float4 q = *reinterpret_cast<const float4*>(&mem(row(k)));
        v[k] = q.x, v[k + 1] = q.y, v[k + 2] = q.z, v[k + 3] = q.w;
      }
  } else if constexpr (NV > 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (row(k) < n) v[k] = mem(row(k));
  } else if constexpr (CACHED) {  // (a thread reads back only its own rows)
    walk_rows<kBpFullThreads, 8, Row>(threadIdx.x, n, [&](Row t) { bp_smem[t] = mem(t); });
  }
  auto each = [&](auto f) {
    if constexpr (NV > 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (row(k) < n) f(v[k]);
    } else {
      walk_rows<kBpFullThreads, 4, Row>(threadIdx.x, n, [&](Row t) { f(CACHED ? bp_smem[t] : mem((unsigned)t)); });
    }
  };
  const double nd = (double)nrows;
  double s = 0.0;
  each([&](float u) { s += (double)u; });
  block_sum2(0, s, 0.0, [&](double a, double) { s_ave = a / (double)nchan; });  // the reference divides by NCHANOUT
  const double ave = s_ave;
  double d1 = 0.0, d2 = 0.0;
  each([&](float u) {
    const double d = (double)u - ave;
    d1 += d;
    d2 += d * d;
  });
  block_sum2(1, d1, d2, [&](double sum, double sum2) {
    const double sig = (sum2 - sum * sum / nd) / (nd - 1.0);
    s_hi = clip_hi(ave + 3.0 * sig);
    s_lo = clip_lo(ave - 3.0 * sig);
  });
  const float hi = s_hi, lo = s_lo;
  double cs = 0.0;
  int cn = 0;
  each([&](float u) {
    if (u < hi && u > lo) {
      cs += (double)u;
      ++cn;
    }
  });
  block_sum2(2, cs, (double)cn, [&](double a, double b) { s_m = (float)(a / b); });  // no rows kept: NaN, as the reference's ave/=i
  const float m = s_m;
  if constexpr (NV > 0 && VEC) {
#pragma unroll
    for (int k = 0; k < NV; k += 4)
      if (row(k) < n)
        *reinterpret_cast<float4*>(&mem(row(k))) = make_float4(v[k] - m, v[k + 1] - m, v[k + 2] - m, v[k + 3] - m);
  } else if constexpr (NV > 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (row(k) < n) mem(row(k)) = v[k] - m;
  } else {
    walk_rows<kBpFullThreads, 4, Row>(threadIdx.x, n, [&](Row t) {
      float& at = mem((unsigned)t);
      at = (CACHED ? bp_smem[t] : at) - m;
    });
  }
}

// ---- zero-DM ----------------------------------------------------------------------
// A cluster of CTAs takes 8 consecutive rows of every channel, 32-byte runs (a whole
// sector of memory each), a slice of the channels per CTA, into shared memory with
// asynchronous copies.  A thread has four rows of every (kZeroThreads / 2)-th channel:
// 16-byte copies and accesses where the rows are aligned.  The slices' row sums are
// added in rank order through distributed shared memory.
//
// Slices of up to 52 kB let four CTAs share an SM, so that one's copies run beside
// another's sums.  Bound by the latency of the three reductions and of the FP64
// sums; 384 MB at 2.9 TB/s.  7680 rows x 6250 channels: 4.99 ms with a thread per row
// and four passes over memory (30 CTAs); 0.209 ms with one CTA of 200 kB for all
// channels and 4-byte accesses; 0.147 ms with four slices; 0.134 ms with the
// divisions in one thread per row and reductions that halve the values at each step.
// Two slices of 512 threads 0.146 ms; eight of 128 threads 0.131 ms, not worth the
// larger clusters.
constexpr int kZeroRows = 8;
constexpr int kZeroThreads = 256;
constexpr int kZeroSlice = 52 * 1024;

template <bool VEC>
__global__ void __launch_bounds__(kZeroThreads, 1024 / kZeroThreads)
    k_subtract_zero(float* __restrict__ fb, long long chan_stride, long long row0, unsigned row_mask, int nchan,
                    long long nrows, int per) {
  extern __shared__ float4 z_smem[];  // [per][2]: rows 0..3 and 4..7 of a channel
  constexpr int kWarps = kZeroThreads / 32;
  __shared__ double red[kWarps][2][kZeroRows];
  __shared__ double part[3][2][kZeroRows];  // this slice's sums: read by the whole cluster
  __shared__ double row_ave[kZeroRows];
  __shared__ float row_hi[kZeroRows], row_lo[kZeroRows], row_m[kZeroRows];
  cg::cluster_group cluster = cg::this_cluster();
  const int nslice = (int)cluster.num_blocks();
  const int c0 = (int)cluster.block_rank() * per;
  const int nq = 2 * max(0, min(per, nchan - c0));  // quads of this slice
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = tid & 1;
  const long long t0 = (long long)(blockIdx.x / nslice) * kZeroRows + 4 * h;
  const int live = (int)max(0LL, min(4LL, nrows - t0));
  auto row_at = [&](int i) {
    return (unsigned long long)(row0 + (i < live ? t0 + i : 0)) & (unsigned long long)row_mask;
  };
  float* x[VEC ? 1 : 4];
#pragma unroll
  for (int i = 0; i < (VEC ? 1 : 4); ++i) x[i] = fb + (c0 + tid / 2) * chan_stride + row_at(i);
  const long long step = (kZeroThreads / 2) * chan_stride;
  {
    long long o = 0;
    for (int q = tid; q < nq; q += kZeroThreads, o += step) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(z_smem + q);
      if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(x[0] + o), "r"(4 * live));
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d + 4 * i), "l"(x[i] + o),
                       "r"(i < live ? 4 : 0));
      }
    }
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  // (a thread reads back only what it copied: no barrier needed)
  // done(row, A, B) with the cluster's sums of a and b over the channels: by one
  // thread per row (FP64 divisions are dozens of instructions)
  auto row_sums = [&](int phase, double (&a)[4], double (&b)[4], auto done) {
    // half of the values are handed over in each step, so a lane ends with one
    auto fold = [&](bool up, double keep, double other, int o) {
      return (up ? other : keep) + __shfl_xor_sync(0xffffffffu, up ? keep : other, o);
    };
    const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
    double v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = fold(u16, a[i], b[i], 16);
    v[0] = fold(u8, v[0], v[2], 8);
    v[1] = fold(u8, v[1], v[3], 8);
    v[0] = fold(u4, v[0], v[1], 4);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    if (!(lane & 2)) red[warp][u16][4 * h + 2 * u8 + u4] = v[0];
    __syncthreads();
    if (tid < 2 * kZeroRows) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += red[w][tid / kZeroRows][tid % kZeroRows];
      part[phase][tid / kZeroRows][tid % kZeroRows] = v;
    }
    cluster.sync();
    if (tid < 2 * kZeroRows) {
      double v = 0.0;
      for (int r = 0; r < nslice; ++r)
        v += cluster.map_shared_rank(&part[phase][tid / kZeroRows][tid % kZeroRows], r)[0];
      const double w = __shfl_down_sync((1u << 2 * kZeroRows) - 1, v, kZeroRows);
      if (tid < kZeroRows) done(tid, v, w);
    }
    __syncthreads();
  };
  const double n = (double)nchan;
  double a[4] = {}, b[4] = {};
#pragma unroll 2
  for (int q = tid; q < nq; q += kZeroThreads) {
    const float4 v = z_smem[q];
    a[0] += (double)v.x;
    a[1] += (double)v.y;
    a[2] += (double)v.z;
    a[3] += (double)v.w;
  }
  row_sums(0, a, b, [&](int r, double s, double) { row_ave[r] = s / n; });
  double ave[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ave[i] = row_ave[4 * h + i];
    a[i] = b[i] = 0.0;
  }
#pragma unroll 2
  for (int q = tid; q < nq; q += kZeroThreads) {
    const float4 v = z_smem[q];
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double d = (double)f[i] - ave[i];
      a[i] += d;
      b[i] = fma(d, d, b[i]);
    }
  }
  row_sums(1, a, b, [&](int r, double s1, double s2) {
    const double sig = (s2 - s1 * s1 / n) / (n - 1.0);
    row_hi[r] = clip_hi(row_ave[r] + 3.0 * sig);
    row_lo[r] = clip_lo(row_ave[r] - 3.0 * sig);
  });
  float hi[4], lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    hi[i] = row_hi[4 * h + i];
    lo[i] = row_lo[4 * h + i];
  }
  bool out = false;  // the clip rejects values of a row
#pragma unroll 2
  for (int q = tid; q < nq; q += kZeroThreads) {
    const float4 v = z_smem[q];
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) out |= i < live && !(f[i] < hi[i] && f[i] > lo[i]);
  }
  if (__syncthreads_or(out)) {
    int kept[4] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = 0.0;
    for (int q = tid; q < nq; q += kZeroThreads) {
      const float4 v = z_smem[q];
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (f[i] < hi[i] && f[i] > lo[i]) {
          a[i] += (double)f[i];
          ++kept[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = (double)kept[i];
  } else {  // the slice loses nothing: its sum is the first pass's
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = tid < 2 ? part[0][0][4 * h + i] : 0.0;
      b[i] = tid < 2 ? (double)(nq / 2) : 0.0;
    }
  }
  row_sums(2, a, b, [&](int r, double s, double cnt) { row_m[r] = (float)(s / (cnt > 0.0 ? cnt : 1.0)); });
  cluster.barrier_arrive();  // this CTA has read the others' sums
  float m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = row_m[4 * h + i];
  {
    long long o = 0;
#pragma unroll 2
    for (int q = tid; q < nq; q += kZeroThreads, o += step) {
      const float4 v = z_smem[q];
      const float4 y = make_float4(v.x - m[0], v.y - m[1], v.z - m[2], v.w - m[3]);
      if (VEC && live == 4) {
        *reinterpret_cast<float4*>(x[0] + o) = y;
      } else {
        const float f[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < live) (VEC ? x[0] + i : x[VEC ? 0 : i])[o] = f[i];
      }
    }
  }
  cluster.barrier_wait();  // no CTA leaves while another may read its sums
}

// More channels than fit in shared memory, or many rows for them (launch_subtract_zero):
// one thread per row; a warp covers 32 consecutive rows, so every channel's load is one
// 128-byte segment
__global__ void __launch_bounds__(256) k_subtract_zero_rows(float* __restrict__ fb, long long chan_stride, long long row0,
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

// rows row0 + 4 i .. + 3 are 16 aligned bytes of memory
static bool rfi_quads(const float* fb, long long chan_stride, long long row0, unsigned row_mask) {
  return ((uintptr_t)fb & 15) == 0 && (chan_stride & 3) == 0 && (row0 & 3) == 0 && (row_mask & 3) == 3;
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
  const bool vec = rfi_quads(fb, chan_stride, row0, row_mask) && (nrows & 3) == 0;
  auto run = [&](auto kern, size_t smem) {
    kern<<<nchan, kBpFullThreads, smem, s>>>(fb, chan_stride, row0, row_mask, nchan, nrows);
  };
  // Registers where their number is nearly the rows', and by quads for the larger one;
  // else shared memory, which has no test for each row in its loops.  3908 channels, us,
  // registers against shared memory: 60 rows 25 / 19, 1024 25 / 25, 2000 33 (27 in quads)
  // / 35, 3071 70 / 39, 5000 (quads) 55 / 49, 7680 88 (66) / 78.
  if (nrows > 4 * 256 && nrows <= 8 * 256) {
    vec ? run(k_subtract_bp_full<8, true, false>, 0) : run(k_subtract_bp_full<8, false, false>, 0);
  } else if (vec && nrows > 24 * 256 && nrows <= 32 * 256) {
    run(k_subtract_bp_full<32, true, false>, 0);
  } else if (nrows * 4 <= kRfiSmem) {
    if (const int st = rfi_smem(k_subtract_bp_full<0, false, true>)) return st;
    run(k_subtract_bp_full<0, false, true>, (size_t)nrows * 4);
  } else {
    run(k_subtract_bp_full<0, false, false>, 0);
  }
  return cuda_status(cudaGetLastError());
}

int launch_subtract_zero(float* fb, long long chan_stride, long long row0, unsigned row_mask, int nchan,
                         long long nrows, cudaStream_t s) {
  if (!rfi_args_ok(fb, chan_stride, row0, row_mask, nchan, nrows)) return VFRB_ERR_ARG;
  auto slice = [&](int k) { return (long long)((nchan + k - 1) / k) * kZeroRows * 4; };
  int k = 1;
  while (k < 8 && slice(k) > kZeroSlice) k *= 2;
  const long long smem = slice(k);
  // A thread per row reads its channels four times: from the caches where 256 rows of
  // all channels fit there, and with enough rows for every SM; with very many rows its
  // plain loads keep more in flight than the clusters' short lives.  us, thread per row
  // against clusters: 64 channels x 1024 rows 10.3 / 8.8, 7680 10.3 / 14.4, 2^17 29 / 153;
  // 192 x 7680 45 / 16, 2^14 23 / 29, 2^17 102 / 195; 256 x 2^15 64 / 53, 2^17 245 / 207,
  // 2^19 581 / 865; 1024 x 2^17 969 / 386, 2^19 2312 / 2327, 2^20 4632 / 5744.
  const bool rows = (nchan <= 192 && nrows >= 84LL * nchan) || (nchan <= 1024 && nrows >= 1LL << 19);
  if (smem <= kRfiSmem && !rows) {
    const long long nb = (nrows + kZeroRows - 1) / kZeroRows * k;
    if (nb > 0x7fffffffLL) return VFRB_ERR_UNSUPPORTED;
    const bool vec = rfi_quads(fb, chan_stride, row0, row_mask);
    auto* kern = vec ? k_subtract_zero<true> : k_subtract_zero<false>;
    if (const int st = rfi_smem(kern)) return st;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nb);
    cfg.blockDim = dim3(kZeroThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)k;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, fb, chan_stride, row0, row_mask, nchan, nrows,
                                             (nchan + k - 1) / k);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return cuda_status(e);
    }
  } else {
    const long long nb = (nrows + 255) / 256;
    if (nb > 0x7fffffffLL) return VFRB_ERR_UNSUPPORTED;
    k_subtract_zero_rows<<<(unsigned)nb, 256, 0, s>>>(fb, chan_stride, row0, row_mask, nchan, nrows);
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
