// Band-wise dedispersion: the exact brute-force sums with shared partial sums.
//
//   out[d][t] = (1/nchan) sum_c w_c fb[c][t + off[d][c]]
//
// Eight adjacent trials (a group) of an equally spaced DM list have, in channel
// c, delays that grow by y_c rows per trial.  The kernel works on one band of
// channels at a time, a band being the channels whose y_c rounds to the same
// whole number m.  Within it trial j of a group is accumulated m*j rows
// earlier, so the eight delays differ by a digital straight line of slope
// y_c - m, at most 1/2 row per trial: they span at most 4 rows, and there are
// only 67 such patterns, 8 or 9 of which occur among 60 neighbouring channels.
// Channels with the same pattern are summed FIRST, one add per window element, and
// their sum is then added to the eight trials at the pattern's eight shifts.  Every series is the sum of exactly the
// samples that the brute-force sum takes; only the order of the FP32 additions
// differs, and it is shorter (runs of a few channels, then chunks, then bands),
// which lowers the rounding error.
//
// What bounds it: a lane owns TT consecutive samples (a warp 32 TT) and loads TT +
// 1.75 elements per channel on average for 8 TT sums, 0.15 shared loads per sum
// at TT = 9, against 0.38 for the four-trial windows of the pattern kernel and 1
// for a plain sum.  At 2048 trials x 6250 channels x 16384 samples the loads keep
// the shared-memory pipe 57% busy; the rest is latency (dependent branches of the
// staircases and load latency, four warps per scheduler).  13.5 ms (pattern
// kernel) -> 6.53 ms; 2048 x 1024 in FP16 1.50 -> 0.74 ms; 201 trials x 5145
// samples 1.65 -> 0.59 ms, in int8 2.37 (staged kernel) -> 0.83 ms.  Longer runs
// per lane with fewer warps have fewer loads and instructions per sum but were no
// faster: TT 11 with 12 warps 7.0 ms, TT 17 with 8 warps 8.5 ms; nor were more
// warps with shorter runs, TT 7 x 20 warps 7.3 ms.  Two 8-warp CTAs per SM hold
// half as many channels per chunk, so runs are shorter: 8.1 ms.
//
// Each band is a launch of its own: trial d's accumulators cover the samples
// t = t' - skew(d, band) of a tile [t0, t0 + NT) of t', skew being the delay of
// the group's first trial at the band's middle channel plus m*j, so a CTA's
// trials need nearly the same rows of a channel (the tile is NT plus a few tens
// of rows) although their delays differ by hundreds.  The first band stores the
// sums into `out`, the later ones add (each element belongs to one thread per
// launch, so the order of the sums is fixed), the last one scales.  The launches
// overlap (programmatic dependent launch), which took 7.2 to 6.6 ms, and 1.15 to
// 0.78 ms at 1024 samples, where a band has fewer CTAs than the device SMs.
//
// A chunk of channels is staged by bulk asynchronous copies into one of two
// shared-memory buffers while the other is summed (zeros outside the valid rows and
// the last few of them are written by the warps), with the chunk's sorted
// channel lists (one record per group, made when the plan is created: slots by
// pattern, and the runs).
#include "dedisp_band.h"

#include "bulk_copy.cuh"
#include "dedisp_band_tables.h"

#include <memory>

namespace vfrb {

struct BandTables {
  BandHost h;
  unsigned char* d_all = nullptr;  // one allocation, of which the rest are parts
  int* d_bmin = nullptr;
  int* d_skew = nullptr;
  unsigned char* d_rec = nullptr;
  unsigned* d_shift = nullptr;
};

struct BandParams {
  int njobs;
  DdJob jobs[kDdMaxJobs];
  const void* fb;
  const float* chan_scale;
  float out_scale;
  long long chan_stride, row0, nrows_valid, nt_out, out_stride;
  unsigned row_mask;
  int nchan, ndm, ngroups, gper;
  float* out;
  const int* bmin;
  const int* skew;      // this band's
  const unsigned char* rec;  // this band's records
  const unsigned* shift;
  int rec_bytes, ch_cap;
  int c_lo, nch, m, ch, lm;
  int first, last;
  int* err;
};

// ---- window sums ---------------------------------------------------------------
// S[k] (+)= w * window[k], k < NW, the window starting at element `off` of the
// staged rows.  FP32: packed adds of pairs.  FP16: aligned 4-byte loads and a
// byte permute for an odd start, mixed-precision adds.  int8: the same with a
// start anywhere in the word; bytes become floats exactly.
template <typename T, bool WT, int NW, bool FIRST, int NS>
__device__ __forceinline__ void band_window(float (&S)[NS], const T* tile, int off, float wc) {
  if constexpr (sizeof(T) == 4) {
    const float* src = reinterpret_cast<const float*>(tile) + off;
    if constexpr (FIRST) {
#pragma unroll
      for (int k = 0; k < NW; ++k) S[k] = src[k];
    } else {
      float w[NW];
#pragma unroll
      for (int k = 0; k < NW; ++k) w[k] = src[k];
#pragma unroll
      for (int k = 0; k + 1 < NW; k += 2) {
        const float2 r = __fadd2_rn(make_float2(S[k], S[k + 1]), make_float2(w[k], w[k + 1]));
        S[k] = r.x;
        S[k + 1] = r.y;
      }
      if constexpr ((NW & 1) != 0) S[NW - 1] += w[NW - 1];
    }
  } else if constexpr (sizeof(T) == 2) {
    constexpr int N2 = (NW + 1) / 2;
    const unsigned* src = reinterpret_cast<const unsigned*>(tile + (off & ~1));
    const unsigned sel = (off & 1) ? 0x5432u : 0x3210u;
    unsigned w[N2 + 1];
#pragma unroll
    for (int k = 0; k <= N2; ++k) w[k] = src[k];
#pragma unroll
    for (int k = 0; k < N2; ++k) {
      const unsigned v = __byte_perm(w[k], w[k + 1], sel);
      unsigned short lo, hi;
      asm("mov.b32 {%0, %1}, %2;" : "=h"(lo), "=h"(hi) : "r"(v));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (2 * k + e < NW) {
          const unsigned short h = e ? hi : lo;
          float& s = S[2 * k + e];
          if constexpr (WT) {
            const float x = __half2float(__ushort_as_half(h));
            s = FIRST ? wc * x : fmaf(wc, x, s);
          } else if constexpr (FIRST) {
            s = __half2float(__ushort_as_half(h));
          } else {
            asm("add.rn.f32.f16 %0, %1, %0;" : "+f"(s) : "h"(h));
          }
        }
      }
    }
  } else {
    constexpr int N4 = (NW + 3) / 4;
    const unsigned* src = reinterpret_cast<const unsigned*>(tile + (off & ~3));
    const unsigned sel = 0x3210u + 0x1111u * (unsigned)(off & 3);
    unsigned w[N4 + 1];
#pragma unroll
    for (int k = 0; k <= N4; ++k) w[k] = src[k];
#pragma unroll
    for (int k = 0; k < N4; ++k) {
      // byte b + 128 in the low bits of 2^23: minus (2^23 + 128) leaves b exactly
      const unsigned v = __byte_perm(w[k], w[k + 1], sel) ^ 0x80808080u;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (4 * k + e < NW) {
          const float x = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u + (unsigned)e)) - 8388736.0f;
          float& s = S[4 * k + e];
          if constexpr (WT) {
            s = FIRST ? wc * x : fmaf(wc, x, s);
          } else {
            s = FIRST ? x : s + x;
          }
        }
      }
    }
  }
}

// a slot: tile offset (18 bits) and channel of the chunk
__device__ __forceinline__ int slot_off(unsigned e) { return (int)(e & 0x3ffffu); }
__device__ __forceinline__ int slot_chan(unsigned e) { return (int)(e >> 18); }

// S = the sum of n channels' windows of NW elements.  `off` is the first one's
// start in the tile, and the start after the last one's on return: each start is
// worked out while the window before it is on its way (past the last run of a
// chunk it comes from the record's padding and is not used).
template <typename T, bool WT, int NW, int NS>
__device__ __forceinline__ void band_run(float (&S)[NS], const T* tile, const unsigned*& slot, int n, int lane_off,
                                         const float* wts, int& off) {
  unsigned e = slot[1];
  band_window<T, WT, NW, true>(S, tile, off, WT ? wts[slot_chan(slot[0])] : 1.f);
#pragma unroll 1
  for (int i = 1; i < n; ++i) {
    ++slot;
    const int at = slot_off(e) + lane_off;
    const float wc = WT ? wts[slot_chan(e)] : 1.f;
    e = slot[1];
    band_window<T, WT, NW, false>(S, tile, at, wc);
  }
  ++slot;
  off = slot_off(e) + lane_off;
}

// acc[J][t] += S[t + SH] (an even shift adds register pairs)
template <int J, int SH, int TT, int NS>
__device__ __forceinline__ void band_add(float (&acc)[kBandD][TT], const float (&S)[NS]) {
  if constexpr (SH <= kBandSmax && SH + TT <= NS) {
    if constexpr ((SH & 1) == 0) {
#pragma unroll
      for (int t = 0; t + 1 < TT; t += 2) {
        const float2 r = __fadd2_rn(make_float2(acc[J][t], acc[J][t + 1]), make_float2(S[t + SH], S[t + SH + 1]));
        acc[J][t] = r.x;
        acc[J][t + 1] = r.y;
      }
      if constexpr ((TT & 1) != 0) acc[J][TT - 1] += S[TT - 1 + SH];
    } else {
#pragma unroll
      for (int t = 0; t < TT; ++t) acc[J][t] += S[t + SH];
    }
  }
}

// acc[j][t] += S[t + shift_j] for shifts that are a staircase of unit steps:
// a walk over the nodes (trial, shift), from each to the next trial at the same
// or the next shift, so that every add has static registers and the code is 40
// short blocks per direction.  (Straight-line code for each of the 67 patterns
// is 100 kB that the warps run out of step: it stalled on instruction fetches,
// 10.0 ms.  Moving the window down a register at each step becomes more moves
// than adds, 13.1 ms.)
template <int TT, int NS, bool DOWN>
__device__ __forceinline__ void band_stairs(float (&acc)[kBandD][TT], const float (&S)[NS], unsigned code) {
#define VFRB_NODE(Q, SH)                                            \
  n##Q##_##SH : band_add<DOWN ? kBandD - 1 - Q : Q, SH>(acc, S);
#define VFRB_STEP(Q, R, SH, SN)         \
  if (code & (1u << Q)) goto n##R##_##SN; \
  goto n##R##_##SH;
#define VFRB_ROW(Q, R)                                          \
  VFRB_NODE(Q, 0) VFRB_STEP(Q, R, 0, 1) VFRB_NODE(Q, 1) VFRB_STEP(Q, R, 1, 2) \
  VFRB_NODE(Q, 2) VFRB_STEP(Q, R, 2, 3) VFRB_NODE(Q, 3) VFRB_STEP(Q, R, 3, 4) \
  VFRB_NODE(Q, 4) goto n##R##_4;
  band_add<DOWN ? kBandD - 1 : 0, 0>(acc, S);
  VFRB_STEP(0, 1, 0, 1)
  VFRB_NODE(1, 0) VFRB_STEP(1, 2, 0, 1) VFRB_NODE(1, 1) VFRB_STEP(1, 2, 1, 2)
  VFRB_NODE(2, 0) VFRB_STEP(2, 3, 0, 1) VFRB_NODE(2, 1) VFRB_STEP(2, 3, 1, 2) VFRB_NODE(2, 2) VFRB_STEP(2, 3, 2, 3)
  VFRB_NODE(3, 0) VFRB_STEP(3, 4, 0, 1) VFRB_NODE(3, 1) VFRB_STEP(3, 4, 1, 2) VFRB_NODE(3, 2) VFRB_STEP(3, 4, 2, 3)
  VFRB_NODE(3, 3) VFRB_STEP(3, 4, 3, 4)
  VFRB_ROW(4, 5)
  VFRB_ROW(5, 6)
  VFRB_ROW(6, 7)
  VFRB_NODE(7, 0) return;
  VFRB_NODE(7, 1) return;
  VFRB_NODE(7, 2) return;
  VFRB_NODE(7, 3) return;
  VFRB_NODE(7, 4) return;
#undef VFRB_ROW
#undef VFRB_STEP
#undef VFRB_NODE
}

// shifts that are no staircase (rounding of the trials' values): selects
template <int TT, int NS>
__device__ __forceinline__ void band_any(float (&acc)[kBandD][TT], const float (&S)[NS], unsigned shifts) {
#pragma unroll
  for (int j = 0; j < kBandD; ++j) {
    const int sh = (int)(shifts >> (4 * j)) & 15;
    float v[TT];
#pragma unroll
    for (int t = 0; t < TT; ++t) {
      v[t] = S[t];
#pragma unroll
      for (int q = 1; q <= kBandSmax; ++q) v[t] = sh == q ? S[t + q] : v[t];
    }
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[j][t] += v[t];
  }
}

// TT samples per lane.  The lane stride in bytes is an odd number of words, so
// that a load touches 32 banks (int8 loads few words: two ways of conflict cost
// less there than the registers of a longer run)
template <typename T>
struct BandTT;
template <>
struct BandTT<float> {
  static constexpr int v = 9;
};
template <>
struct BandTT<__half> {
  static constexpr int v = 10;
};
template <>
struct BandTT<int8_t> {
  static constexpr int v = 8;
};

// Waits until the band launched before has ended and its sums are visible (the
// first band's launch is an ordinary one: nothing to wait for).
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// GIVE_UP: waits for staged rows give up at once (a test's form; as a launch parameter it
// cost 1% of the 201-trial case)
template <typename T, bool WT, bool GIVE_UP>
__global__ void __launch_bounds__(kBandW * 32, 1) k_dedisp_band(const __grid_constant__ BandParams p) {
  constexpr int TT = BandTT<T>::v;
  constexpr int NT = 32 * TT;
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int W = kBandW;
  static_assert(NT % kBandAlign == 0 && NT <= kBandNtMax, "tile starts stay aligned");
  // Once every CTA of this band runs, the next band's may start on free SMs; they
  // touch `out` only after this band has ended (grid_wait below).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const bool batch = p.njobs > 0;
  const DdJob& job = p.jobs[batch ? blockIdx.z : 0];
  const long long nt_out = batch ? job.nt_out : p.nt_out;
  const int blk = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = p.gper;
  const int gl = warp % G, set = warp / G;  // the CTA's group, and the set of warps
  const int gw = blk * G + gl;
  const int* skew = p.skew + blk * G;
  const long long t0 = (skew[0] / NT + (long long)blockIdx.y) * NT;  // first t' of the tile
  {  // the block's smallest and largest skew: its first and last trial's
    const int nd = min(G, p.ngroups - blk * G);
    const long long lo = skew[0], hi = (long long)skew[nd - 1] + (kBandD - 1) * p.m;
    if (t0 >= hi + nt_out || t0 + NT <= lo) {
      grid_wait();
      return;
    }
  }
  const long long row0 = batch ? job.row0 : p.row0;
  const long long vend = row0 + (batch ? job.nrows_valid : p.nrows_valid);
  const T* fb = reinterpret_cast<const T*>(batch ? job.fb : p.fb);
  const unsigned long long rmask = (unsigned long long)p.row_mask;
  const int CH = p.ch, LM = p.lm;

  // shared: full[2] mbarriers | rec[2][W][rec_bytes] | wts[2][CH] (WT) | tile[2][CH][LM]
  extern __shared__ __align__(128) unsigned char band_smem[];
  unsigned long long* s_full = reinterpret_cast<unsigned long long*>(band_smem);
  unsigned char* s_rec = band_smem + 16;
  float* s_w = reinterpret_cast<float*>(s_rec + 2 * W * p.rec_bytes);
  const int wpad = WT ? (CH + 3) / 4 * 4 : 0;
  T* s_tile = reinterpret_cast<T*>(s_w + 2 * wpad);
  if (tid == 0) {
    mbar_init(&s_full[0], W);
    mbar_init(&s_full[1], W);
    mbar_fence_init();
  }
  __syncthreads();

  const long long ta = (row0 + t0) & ~(long long)(kBandAlign - 1);  // tile rows start at ta + bmin
  const int phase = (int)(row0 + t0 - ta);
  const int nchunks = (p.nch + CH - 1) / CH;
  const int per = (CH + W - 1) / W;
  const int* bminp = p.bmin + (long long)blk * p.nchan + p.c_lo;
  // warp w stages channels [w*per, ...) of a chunk; their first rows are loaded a chunk ahead
  auto first_rows = [&](int k) -> int {
    const int cl = warp * per + lane;
    return k < nchunks && lane < per && cl < min(CH, p.nch - k * CH) ? __ldg(bminp + k * CH + cl) : 0;
  };
  auto stage = [&](int k, int b, int bm) {
    const int nc = min(CH, p.nch - k * CH);
    const int cb = warp * per;
    const int cn = max(0, min(per, nc - cb));
    const T* src0 = fb + (long long)(p.c_lo + k * CH + cb) * p.chan_stride;
    T* dst0 = s_tile + ((long long)b * CH + cb) * LM;
    // This lane's channel: the whole 16-byte groups among the valid rows of its tile
    // row [a, a + LM) come in one bulk copy (two where they wrap the ring), the warp
    // writes zeros and the last few rows beside them.
    const long long a = ta + bm;
    const BandRows rows_of = band_rows(a, LM, row0, vend, VEC);
    const long long lo = rows_of.lo, hi = rows_of.hi;
    const int nrow = lane < cn ? rows_of.n : 0;
    const bool part = lane < cn && nrow < LM;
    unsigned todo = __ballot_sync(0xffffffffu, part);
    while (todo) {
      const int cl = __ffs(todo) - 1;
      todo &= todo - 1;
      const long long ac = __shfl_sync(0xffffffffu, a, cl), hc = __shfl_sync(0xffffffffu, hi, cl);
      const int before = (int)(__shfl_sync(0xffffffffu, lo, cl) - ac);
      const int have = before + max(0, __shfl_sync(0xffffffffu, nrow, cl));
      const T* src = src0 + (long long)cl * p.chan_stride;
      T* dst = dst0 + (long long)cl * LM;
      for (int v = lane * VEC; v < min(before, LM); v += 32 * VEC) *reinterpret_cast<int4*>(dst + v) = make_int4(0, 0, 0, 0);
      for (int v = have + lane * VEC; v < LM; v += 32 * VEC) {
        union {
          int4 u;
          T t[VEC];
        } val;
        val.u = make_int4(0, 0, 0, 0);
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          if (ac + v + e < hc) val.t[e] = src[(unsigned long long)(ac + v + e) & rmask];
        *reinterpret_cast<int4*>(dst + v) = val.u;
      }
    }
    if (WT && lane < cn) s_w[b * wpad + cb + lane] = __ldg(p.chan_scale + p.c_lo + k * CH + cb + lane);
    __syncwarp();
    const unsigned rows = __reduce_add_sync(0xffffffffu, (unsigned)max(0, nrow));
    const unsigned rb = warp == 0 ? (unsigned)(W * p.rec_bytes) : 0u;
    fence_proxy_async_smem();  // earlier generic accesses of this buffer before the async writes
    if (lane == 0) mbar_arrive_expect_tx(&s_full[b], rows * (unsigned)sizeof(T) + rb);
    __syncwarp();
    if (nrow > 0) {
      T* dst = dst0 + (long long)lane * LM + (lo - a);
      const T* src = src0 + (long long)lane * p.chan_stride;
      const unsigned long long r = (unsigned long long)lo & rmask;
      const int n1 = (int)min((unsigned long long)nrow, rmask + 1ULL - r);  // rows before the ring's end
      bulk_g2s(dst, src + r, (unsigned)(n1 * (int)sizeof(T)), &s_full[b]);
      if (n1 < nrow) bulk_g2s(dst + n1, src, (unsigned)((nrow - n1) * (int)sizeof(T)), &s_full[b]);
    }
    if (rb && lane == 0)
      bulk_g2s(s_rec + (long long)b * W * p.rec_bytes,
               p.rec + ((long long)k * gridDim.x + blk) * W * p.rec_bytes, rb, &s_full[b]);
  };

  float acc[kBandD][TT];
#pragma unroll
  for (int j = 0; j < kBandD; ++j)
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[j][i] = 0.f;

  stage(0, 0, first_rows(0));
  int bm_next = first_rows(1);
  const int lane_off = lane * TT + phase;
  int k = 0;  // nchunks at the end; one more where this warp's wait gave up
  for (; k < nchunks; ++k) {
    __syncthreads();  // every warp is done with chunk k - 1: its buffer can be refilled
    const int b = k & 1;
    if (k + 1 < nchunks) stage(k + 1, b ^ 1, bm_next);
    bm_next = first_rows(k + 2);
    if (__any_sync(0xffffffffu, GIVE_UP || !mbar_wait(&s_full[b], (unsigned)(k >> 1) & 1u))) {
      drain_copies(s_full, k, nchunks);
      while (++k < nchunks) __syncthreads();  // the other warps' barriers
      k = nchunks + 1;
      break;
    }
    const unsigned char* rec = s_rec + ((long long)b * W + warp) * p.rec_bytes;
    const unsigned* slot = reinterpret_cast<const unsigned*>(rec);
    const unsigned short* run = reinterpret_cast<const unsigned short*>(rec + 4 * p.ch_cap);
    const int nrun = run[p.ch_cap];
    const T* tile = s_tile + (long long)b * CH * LM;
    const float* wts = s_w + b * wpad;
    unsigned rd = run[0];
    int off = slot_off(slot[0]) + lane_off;
#pragma unroll 1
    for (int r = 0; r < nrun; ++r) {
      const int n = (int)(rd >> 8);
      const unsigned code = rd & 0xffu;
      rd = run[r + 1];  // the last one reads nrun itself, unused
      float sum[TT + kBandSmax];
      if (n) {
        switch (__popc(code & 0x7fu)) {  // the rows that the shifts span
          case 0: band_run<T, WT, TT>(sum, tile, slot, n, lane_off, wts, off); break;
          case 1: band_run<T, WT, TT + 1>(sum, tile, slot, n, lane_off, wts, off); break;
          case 2: band_run<T, WT, TT + 2>(sum, tile, slot, n, lane_off, wts, off); break;
          case 3: band_run<T, WT, TT + 3>(sum, tile, slot, n, lane_off, wts, off); break;
          default: band_run<T, WT, TT + 4>(sum, tile, slot, n, lane_off, wts, off); break;
        }
        if (code & 0x80u)
          band_stairs<TT, TT + kBandSmax, true>(acc, sum, code);
        else
          band_stairs<TT, TT + kBandSmax, false>(acc, sum, code);
      } else {
        const unsigned e = slot[0];
        band_window<T, WT, TT + kBandSmax, true>(sum, tile, slot_off(e) + lane_off, WT ? wts[slot_chan(e)] : 1.f);
        const int c = p.c_lo + k * CH + slot_chan(e);
        band_any<TT, TT + kBandSmax>(acc, sum, __ldg(p.shift + (long long)min(gw, p.ngroups - 1) * p.nchan + c));
        ++slot;
        off = slot_off(slot[0]) + lane_off;
      }
    }
  }

  // out (+)= sums, through shared memory so that the global accesses run along time;
  // the sets' sums of a group are added in order
  float* sw = reinterpret_cast<float*>(s_tile) + warp * NT;
  const int gs = min(gw * kBandD, p.ndm - kBandD);  // the last group starts early enough to be whole
  const float fn = (float)p.nchan;
  const float scale = batch ? job.out_scale : p.out_scale;
  const float fs = scale / fn;
  float* out = batch ? job.out : p.out;
  const long long ostride = batch ? job.out_stride : p.out_stride;
  const int sk0 = gw < p.ngroups ? skew[gl] : 0;
  __syncthreads();  // the tiles have been read
  grid_wait();
#pragma unroll
  for (int j = 0; j < kBandD; ++j) {
    // (skipped: the other sets, padding, and the trials of an overlapping last group that the one before has)
    const bool mine = set == 0 && gw < p.ngroups && gs + j >= gw * kBandD;
    float* orow = out + (long long)(gs + j) * ostride;
    const long long tb = t0 - sk0 - j * p.m + lane;
    float old[TT];
    if (p.last && !p.first) {
#pragma unroll
      for (int i = 0; i < TT; ++i) {
        const long long t = tb + 32 * i;
        old[i] = mine && t >= 0 && t < nt_out ? orow[t] : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < TT; ++i) sw[lane * TT + i] = acc[j][i];
    if (G == W) __syncwarp();
    else __syncthreads();
    if (mine) {
#pragma unroll
      for (int i = 0; i < TT; ++i) {
        const long long t = tb + 32 * i;
        float v = sw[lane + 32 * i];
        for (int q = G; q < W; q += G) v += sw[q * NT + lane + 32 * i];
        if (t < 0 || t >= nt_out) continue;
        if (p.last) {
          if (!p.first) v += old[i];
          orow[t] = scale == 1.f ? v / fn : v * fs;
        } else if (p.first) {
          orow[t] = v;
        } else {
          atomicAdd(orow + t, v);  // nobody else touches it in this launch: an add that nothing waits for
        }
      }
    }
    if (G == W) __syncwarp();
    else __syncthreads();
  }
  int* derr = batch ? job.err : p.err;
  if (k > nchunks && lane == 0 && derr) atomicOr(derr, kErrTimeout);  // the sums are not whole
}

// ---- host side ------------------------------------------------------------------
void band_destroy(BandTables* t) {
  if (!t) return;
  cudaFree(t->d_all);
  delete t;
}

int band_launches(const BandTables* t) { return (int)t->h.bands.size(); }

int band_create(BandTables** out, const int32_t* off, int ndm, int nchan) {
  *out = nullptr;
  std::unique_ptr<BandTables> t(new BandTables());
  BandHost& h = t->h;
  if (!band_build(h, off, ndm, nchan)) return VFRB_OK;
  size_t used = 0;
  auto place = [&](const auto& v) {
    const size_t at = used;
    used = (used + v.size() * sizeof(v[0]) + 255) / 256 * 256;
    return at;
  };
  const size_t at_bmin = place(h.bmin), at_skew = place(h.skew), at_rec = place(h.rec), at_shift = place(h.shift);
  auto put = [&](size_t at, const auto& v) {
    return v.empty() ||
           cudaMemcpy(t->d_all + at, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice) == cudaSuccess;
  };
  if (cudaMalloc((void**)&t->d_all, used) != cudaSuccess || !put(at_bmin, h.bmin) || !put(at_skew, h.skew) ||
      !put(at_rec, h.rec) || !put(at_shift, h.shift)) {
    cudaGetLastError();
    band_destroy(t.release());
    return VFRB_ERR_NOMEM;
  }
  t->d_bmin = reinterpret_cast<int*>(t->d_all + at_bmin);
  t->d_skew = reinterpret_cast<int*>(t->d_all + at_skew);
  t->d_rec = t->d_all + at_rec;
  t->d_shift = h.shift.empty() ? nullptr : reinterpret_cast<unsigned*>(t->d_all + at_shift);
  // the device has them; the launches need the bands and the skew ranges only
  h.bmin = {};
  h.skew = {};
  h.rec = {};
  h.shift = {};
  *out = t.release();
  return VFRB_OK;
}

template <typename T, bool WT, bool GIVE_UP = false>
static int band_launch_t(const BandTables* t, BandParams& k, long long nt_max, cudaStream_t s, int* launched) {
  constexpr int NT = 32 * BandTT<T>::v;
  const int nb = t->h.nblocks;
  const int nbands = (int)t->h.bands.size();
  // grid y: the most tiles a block has
  auto tiles = [&](int bi) {
    long long most = 1;
    for (int q = 0; q < nb; ++q) {
      const long long lo = floor_div(t->h.skmin[(size_t)bi * nb + q], NT);
      const long long hi = floor_div(t->h.skmax[(size_t)bi * nb + q] + nt_max - 1, NT);
      most = std::max(most, hi - lo + 1);
    }
    return most;
  };
  for (int bi = 0; bi < nbands; ++bi)
    if (tiles(bi) > 65535) return VFRB_OK;
  // one limit for every band and plan: launches of other threads set the same
  if (cudaFuncSetAttribute(k_dedisp_band<T, WT, GIVE_UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBandSmemMax) !=
      cudaSuccess) {
    cudaGetLastError();
    return VFRB_ERR_CUDA;
  }
  for (int bi = 0; bi < nbands; ++bi) {
    const BandDesc& b = t->h.bands[bi];
    k.c_lo = b.c_lo;
    k.nch = b.nch;
    k.m = b.m;
    k.ch = b.ch;
    k.lm = b.lm;
    k.skew = t->d_skew + (size_t)bi * nb * t->h.gper;
    k.rec = t->d_rec + (size_t)b.chunk0 * nb * kBandW * t->h.rec_bytes;
    k.first = bi == 0;
    k.last = bi == nbands - 1;
    const size_t smem = band_smem(b.ch, b.lm, t->h.rec_bytes, sizeof(T), WT);
    const dim3 grid((unsigned)nb, (unsigned)tiles(bi), (unsigned)std::max(1, k.njobs));
    // A band overlaps the one before it (programmatic dependent launch): its
    // CTAs fill the SMs that the last wave leaves free, and stage and sum their
    // first chunks, before they wait for it to end.  (All CTAs of the band before
    // are resident by then, so none waits for an SM.)
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kBandW * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = bi > 0 ? 1 : 0;
    const int st = cuda_status(cudaLaunchKernelEx(&cfg, k_dedisp_band<T, WT, GIVE_UP>, k));
    if (st) {
      cudaGetLastError();
      return st;
    }
  }
  *launched = 1;
  return VFRB_OK;
}

int band_launch(const BandTables* t, const vfrb_dd_args& a, const DdJob* jobs, int njobs, bool give_up,
                cudaStream_t s, int* launched) {
  *launched = 0;
  if (!t) return VFRB_OK;
  const int vec = a.storage == VFRB_F32 ? 4 : a.storage == VFRB_F16 ? 8 : 16;
  if (a.chan_stride % vec || ((unsigned long long)a.row_mask + 1ULL) % vec || ((uintptr_t)a.fb & 15)) return VFRB_OK;
  BandParams k{};
  k.njobs = njobs;
  for (int i = 0; i < njobs; ++i) {
    if ((uintptr_t)jobs[i].fb & 15) return VFRB_OK;
    k.jobs[i] = jobs[i];
  }
  long long nt = a.nt_out;
  for (int i = 0; i < njobs; ++i) nt = std::max(nt, jobs[i].nt_out);
  const bool weighted = a.storage != VFRB_F32 && a.chan_scale;
  k.fb = a.fb;
  k.chan_scale = a.chan_scale;
  k.out_scale = a.storage == VFRB_F32 || weighted ? 1.f : a.uniform_scale;
  k.chan_stride = a.chan_stride;
  k.row0 = a.row0;
  k.row_mask = a.row_mask;
  k.nrows_valid = a.nrows_valid;
  k.nt_out = a.nt_out;
  k.out = a.out;
  k.out_stride = a.out_stride;
  k.nchan = t->h.nchan;
  k.ndm = t->h.ndm;
  k.ngroups = t->h.ngroups;
  k.gper = t->h.gper;
  k.bmin = t->d_bmin;
  k.shift = t->d_shift;
  k.rec_bytes = t->h.rec_bytes;
  k.ch_cap = t->h.ch_cap;
  k.err = a.d_err;
  switch (a.storage) {
    case VFRB_F32:
      return give_up ? band_launch_t<float, false, true>(t, k, nt, s, launched)
                     : band_launch_t<float, false>(t, k, nt, s, launched);
    case VFRB_F16:
      return weighted ? band_launch_t<__half, true>(t, k, nt, s, launched)
                      : band_launch_t<__half, false>(t, k, nt, s, launched);
    case VFRB_I8:
      return weighted ? band_launch_t<int8_t, true>(t, k, nt, s, launched)
                      : band_launch_t<int8_t, false>(t, k, nt, s, launched);
    default: return VFRB_ERR_ARG;
  }
}

}  // namespace vfrb
