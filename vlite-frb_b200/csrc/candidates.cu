// Boxcar width search over dedispersed series (new-build extension of the
// reference's calcstats peak, PIPE:1337-1370, which has no width).
//
// Per DM trial: for widths w = 1, 2, 4, ..., max_width the window sums
// S_w(t) = sum_{i<w} x[t+i] (FP64 sliding sums, t = 0 .. nt-w) and
// snr_w(t) = (S_w(t) - w*ave) / (sigma*sqrt(w)) with the trial's calcstats
// ave and sigma, so width 1 is calcstats' peak.  The best (snr, start,
// width) is kept; ties go to the smaller width, then the earlier start.
//
// One CTA per trial.  Widths up to kBoxTree: tiles of the series in shared memory,
// where a width's sums are two of the half width's, S_2w(t) = S_w(t) + S_w(t + w):
// one FP64 add per sample and width, and the series is read once, coalesced.  Wider
// searches, and those of series too short for a tile, slide a window per thread over a
// contiguous stretch of the series, which otherwise costs more in the windows' first
// sums (w adds for a few samples per thread) than in the sliding.
#include "vfrb_common.cuh"

#include <cmath>

namespace vfrb {

constexpr int kBoxThreads = 256;

struct BoxBest {
  double snr;
  int t, w;
};

__device__ __forceinline__ bool box_better(const BoxBest& a, const BoxBest& b) {
  if (a.snr != b.snr) return a.snr > b.snr;
  if (a.w != b.w) return a.w < b.w;
  return a.t < b.t;
}

__global__ void __launch_bounds__(kBoxThreads) k_boxcar_slide(const float* __restrict__ dd, long long nt, long long stride,
                                                         const float* __restrict__ ave, const float* __restrict__ sigma,
                                                         int max_width, float* __restrict__ snr_out,
                                                         int* __restrict__ t_out, int* __restrict__ w_out) {
  const int d = blockIdx.x;
  const float* x = dd + (long long)d * stride;
  const double a = (double)ave[d];
  const double s = (double)sigma[d];
  const long long per = (nt + kBoxThreads - 1) / kBoxThreads;
  const long long t_lo = (long long)threadIdx.x * per;
  BoxBest best{-INFINITY, 0x7fffffff, 0x7fffffff};
  for (int w = 1; w <= max_width && w <= nt; w *= 2) {
    const long long t_hi = min(t_lo + per, nt - w + 1);  // starts t in [t_lo, t_hi)
    if (t_lo >= t_hi) continue;
    const double inv = 1.0 / (s * sqrt((double)w));
    double S = 0.0;
    for (int i = 0; i < w; ++i) S += (double)x[t_lo + i];
    for (long long t = t_lo;; ++t) {
      const double v = (S - (double)w * a) * inv;
      if (v > best.snr) best = BoxBest{v, (int)t, w};
      if (t + 1 >= t_hi) break;
      S += (double)x[t + w] - (double)x[t];
    }
  }
  // CTA reduction with the tie rule
  __shared__ BoxBest red[kBoxThreads];
  red[threadIdx.x] = best;
  __syncthreads();
  for (int o = kBoxThreads / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o && box_better(red[threadIdx.x + o], red[threadIdx.x])) red[threadIdx.x] = red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    snr_out[d] = (float)red[0].snr;
    t_out[d] = red[0].t;
    w_out[d] = red[0].w;
  }
}

constexpr int kBoxTree = 256;  // widest boxcar of the tree kernel
constexpr int kBoxTile = 1024;  // starts per tile
constexpr int kBoxPer = kBoxTile / kBoxThreads;

// WMAX: the widest boxcar, a power of two; the tile holds WMAX - 1 more samples
__global__ void __launch_bounds__(kBoxThreads) k_boxcar_tree(const float* __restrict__ dd, long long nt,
                                                             long long stride, const float* __restrict__ ave,
                                                             const float* __restrict__ sigma, int wmax,
                                                             float* __restrict__ snr_out, int* __restrict__ t_out,
                                                             int* __restrict__ w_out) {
  __shared__ double S[kBoxTile + kBoxTree];
  __shared__ BoxBest red[kBoxThreads / 32];
  const int d = blockIdx.x, tid = threadIdx.x;
  const float* x = dd + (long long)d * stride;
  const double a = (double)ave[d];
  const double s = (double)sigma[d];
  BoxBest best{-INFINITY, 0x7fffffff, 0x7fffffff};
  // (64-bit tile starts: nt may be the largest int, past which the last step goes)
  for (long long t0 = 0; t0 < nt; t0 += kBoxTile) {
    const float* xt = x + t0;
    const int have = (int)min(nt - t0, (long long)(kBoxTile + kBoxTree));  // samples of the tile that there are
    // this thread's samples: tid + 256 i, the last of them in the halo
    double v[kBoxPer + 1];
#pragma unroll
    for (int i = 0; i <= kBoxPer; ++i) {
      const int p = tid + kBoxThreads * i;
      v[i] = p < kBoxTile + wmax - 1 && p < have ? (double)xt[p] : 0.0;
    }
    for (int w = 1;; w *= 2) {
      const double wa = (double)w * a, inv = 1.0 / (s * sqrt((double)w));
      const int last = have - w;  // starts t0 + p <= nt - w
#pragma unroll
      for (int i = 0; i < kBoxPer; ++i) {
        const int p = tid + kBoxThreads * i;
        const double q = (v[i] - wa) * inv;
        // ties: the smaller width (tiles are walked in time, so the earlier start of a width comes first)
        if (p <= last && (q > best.snr || (q == best.snr && w < best.w))) best = BoxBest{q, (int)t0 + p, w};
      }
      if (2 * w > wmax) break;
      __syncthreads();  // the half width's (or the last tile's) sums have been read
#pragma unroll
      for (int i = 0; i <= kBoxPer; ++i) {
        const int p = tid + kBoxThreads * i;
        if (p < kBoxTile + kBoxTree) S[p] = v[i];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i <= kBoxPer; ++i) {
        const int p = tid + kBoxThreads * i;  // (what lies past the halo is not used)
        v[i] += p + w < kBoxTile + kBoxTree ? S[p + w] : 0.0;
      }
    }
  }
  // CTA reduction with the tie rule
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    BoxBest b;
    b.snr = __shfl_xor_sync(0xffffffffu, best.snr, o);
    b.t = __shfl_xor_sync(0xffffffffu, best.t, o);
    b.w = __shfl_xor_sync(0xffffffffu, best.w, o);
    if (box_better(b, best)) best = b;
  }
  if ((tid & 31) == 0) red[tid >> 5] = best;
  __syncthreads();
  if (tid == 0) {
    for (int q = 1; q < kBoxThreads / 32; ++q)
      if (box_better(red[q], best)) best = red[q];
    snr_out[d] = (float)best.snr;
    t_out[d] = best.t;
    w_out[d] = best.w;
  }
}

int launch_boxcar(const float* dd, int ndm, long long nt, long long stride, const float* ave, const float* sigma,
                  int max_width, float* snr, int* t, int* w, cudaStream_t s) {
  if (!dd || !ave || !sigma || !snr || !t || !w || ndm < 1 || nt < 1 || stride < nt || max_width < 1)
    return VFRB_ERR_ARG;
  if (nt > 0x7fffffffLL) return VFRB_ERR_UNSUPPORTED;
  int wmax = 1;  // the widest width tried: powers of two up to max_width and nt
  while (2LL * wmax <= max_width && 2LL * wmax <= nt) wmax *= 2;
  // (a short series leaves most of a tile's threads idle: 8192 trials x 100 samples, widths
  // to 8, 45 us with tiles, 41 sliding; x 200 45 / 45; with one width 23 / 26)
  if (wmax <= kBoxTree && (nt >= 192 || wmax == 1))
    k_boxcar_tree<<<ndm, kBoxThreads, 0, s>>>(dd, nt, stride, ave, sigma, wmax, snr, t, w);
  else
    k_boxcar_slide<<<ndm, kBoxThreads, 0, s>>>(dd, nt, stride, ave, sigma, max_width, snr, t, w);
  return cuda_status(cudaGetLastError());
}

}  // namespace vfrb

extern "C" int vfrb_boxcar(const float* dd, int ndm, int64_t nt, int64_t stride, const float* ave,
                           const float* sigma, int max_width, float* snr, int32_t* start, int32_t* width,
                           void* stream) {
  return vfrb::launch_boxcar(dd, ndm, nt, stride, ave, sigma, max_width, snr, start, width, (cudaStream_t)stream);
}
