// K1: fused channeliser for sm_100a.
//
// Replaces convertarray, cufftExecR2C (x2), sumpower, avepower and the
// per-row D2D channel-select copies of PIPE:574-632 (STATS:377-405,
// TS:603-636): raw 8-bit VDIF payload bytes of both polarisations in, one
// NAVE-averaged, NFREQ-normalised, pol-summed power spectrum row out.
//
// The two polarisations' real windows are transformed as ONE complex sequence of
// N = 12500 points, z[n] = (x0[n] - 128) + i (x1[n] - 128).  With Z = FFT(z) the
// spectra are X0 = (Z[k] + conj Z[N-k]) / 2 and X1 = (Z[k] - conj Z[N-k]) / 2i, so
// the pol-summed power needs no split at all:
//   |X0[k]|^2 + |X1[k]|^2 = (|Z[k]|^2 + |Z[N-k]|^2) / 2.
// The -128 offset only changes bin 0, which no output channel uses (NSKIP >= 1),
// and keeps the FP32 transform well conditioned.
//
// Passes of radix 20, 25 and 25 in 100 kB of shared memory.  A thread runs the same
// butterfly j of the last pass, bins j + 500 k, in every window, so the NAVE
// average of its 25 bins' powers stays in registers; only when a row is complete do
// the bins meet their mirrors (through shared memory) and go out.
//
// One persistent 512-thread CTA per SM: a radix-25 butterfly is 50 floats and the
// powers 25, which fits 128 registers, so 16 warps run.  (Before, each pol was a
// 6250-point transform of its even/odd samples and a thread ran both pols' radix-25
// butterflies in packed instructions: 100 floats, 255 registers, 8 warps, and the
// schedulers idle 60% of the time on dependent instructions.)  The raw bytes of the
// next window are copied from the frame ring into the other of two shared-memory
// byte buffers with cp.async while the current window is transformed, by
// warps 4..15: pass 1 has 625 butterflies for 512 threads, and the 113 second-round
// ones of warps 0 to 3 run meanwhile.  (Payloads are 8 mod 16 apart, so no shift of
// the window makes all its pieces legal 16-byte or bulk copies.)
//
// What bounds it: instruction issue (62% of the slots; FMA pipe 54%, shared memory 50%
// of the wavefronts), with the slots that stay empty at the start of each pass, where
// loads come faster than they are served.  8192 rows x 10 windows: 4.33 ms -> 3.46 ms.
// On the way: the transform alone 4.26, its passes in place 4.05, threads mapped so
// that half warps touch different banks 3.75, 8-byte staging copies 3.64, loads
// interleaved with the inner DFTs 3.53, packed adds and FMAs for (re, im) in the DFT-4
// and DFT-5 (14% fewer instructions) 3.46.  A second Z, which saves a barrier per
// window but leaves room for one staging buffer only: 3.70.
//
// Few rows: a row's NAVE windows are one after another in a CTA, so a 32-row bundle
// would use 32 SMs.  Where all windows of a call fit the device at once, a cluster of
// NAVE CTAs takes a row, one window each, and adds the powers in window order
// through distributed shared memory: the same sums bit for bit.  A 32-row bundle of 4
// windows: 36.9 -> 14.4 us.
#include "vfrb_common.cuh"
#include "dft_codelets.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>

namespace cg = cooperative_groups;

namespace vfrb {

constexpr int kN = kFftN;              // 12500
constexpr int kThreads = 512;          // one CTA per SM, 16 warps (up to 128 registers)
constexpr int kB1 = kN / 20;           // 625 butterflies in pass 1 (radix 20)
constexpr int kB = kN / 25;            // 500 in passes 2 and 3 (radix 25)
constexpr int kStage = 12512;          // one pol's window bytes, shifted by up to 7, padded to 16
constexpr int kStageT0 = 128;          // the staging copies are issued by threads 128..511
constexpr int kStageThreads = kThreads - kStageT0;
constexpr int kMaxCluster = 8;

// Twiddle tables, computed on the host in double precision:
//   g_tw2[(r-1)*20 + m] = W_500^(m r)                (pass 2, Ns = 20)
//   g_tw3[i*500 + j] = W_12500^(j e_i), e = 1 2 3 4 5 10 15 20: pass 3's twiddle of
//                      input r = 5a + b is the product of two of these
constexpr int kTw2 = 24 * 20;
constexpr int kTw3 = 8 * kB;
__device__ float2 g_tw2[kTw2];
__device__ float2 g_tw3[kTw3];

// Every pass works in place: output k of pass 1's butterfly j goes to j + 625 k, and
// passes 2 and 3 leave outputs where their inputs were, so no barrier parts a pass's
// reads and writes.  Butterfly (m, g), m < 20, g < 25, of pass 2 has its points at
// g + 25 r + 625 m, that of pass 3 (number m + 20 g) at r + 25 g + 625 m.  In both,
// and in the twiddle tables, the 16 lanes of a half warp touch different banks when
// they share g and have 16 neighbouring m, or have the last four m and every fourth
// g; threads are given butterflies that way.
__device__ __forceinline__ void butterfly_of(int tid, int& m, int& g) {
  if (tid < 400) {
    m = tid % 16;
    g = tid / 16;
  } else {
    const int i = tid - 400;
    m = 16 + i % 4;
    g = i < 64 ? i / 16 + 4 * (i % 16 / 4) : i / 4;
  }
}

// shared memory: Z | tw2 | tw3 | staged bytes [2 buffers][2 pols][kStage] | shifts | a zero
constexpr size_t kSmZ = sizeof(float2) * kN;
constexpr size_t kSmTab = sizeof(float2) * (kTw2 + kTw3);
constexpr size_t kSmem = kSmZ + kSmTab + 4 * kStage + 32;  // ... | shifts [2][2] | a zero
static_assert(kSmem <= 227 * 1024, "channeliser shared memory");
static_assert(kB1 - kThreads <= kStageT0 && kB <= kThreads, "pass 1 in two rounds, the second beside the staging");
static_assert((kSmZ + kSmTab) % 16 == 0 && kStage % 16 == 0, "16-byte aligned staging");

static std::mutex g_tw_mu;
static bool g_tw_ready[64];

static int ensure_twiddles() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return VFRB_ERR_CUDA;
  std::lock_guard<std::mutex> lk(g_tw_mu);
  if (g_tw_ready[dev]) return VFRB_OK;
  static float2 p2[kTw2], p3[kTw3];
  auto unit = [](double num, double den) {
    const double a = -2.0 * M_PI * num / den;
    return make_float2((float)cos(a), (float)sin(a));
  };
  for (int r = 1; r < 25; ++r)
    for (int m = 0; m < 20; ++m) p2[(r - 1) * 20 + m] = unit((double)((m * r) % 500), 500.0);
  static const int e[8] = {1, 2, 3, 4, 5, 10, 15, 20};
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j < kB; ++j) p3[i * kB + j] = unit((double)((j * e[i]) % kN), (double)kN);
  if (cudaMemcpyToSymbol(g_tw2, p2, sizeof(p2)) != cudaSuccess) return VFRB_ERR_CUDA;
  if (cudaMemcpyToSymbol(g_tw3, p3, sizeof(p3)) != cudaSuccess) return VFRB_ERR_CUDA;
  g_tw_ready[dev] = true;
  return VFRB_OK;
}

__device__ __forceinline__ void cp_async_commit_k1() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_k1() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// f(0), ..., f(4) with compile-time arguments.  A butterfly's inner DFTs take every
// fifth input: each group of loads is followed by its arithmetic and kept there (the
// empty asm), so that a warp computes while the others' loads are served, where all
// loads first would leave the arithmetic idle until the last one.
template <typename F>
__device__ __forceinline__ void each5(F&& f) {
  f(std::integral_constant<int, 0>{});
  asm volatile("" ::: "memory");
  f(std::integral_constant<int, 1>{});
  asm volatile("" ::: "memory");
  f(std::integral_constant<int, 2>{});
  asm volatile("" ::: "memory");
  f(std::integral_constant<int, 3>{});
  asm volatile("" ::: "memory");
  f(std::integral_constant<int, 4>{});
}

// byte b as the float b - 128, exactly: 0x4B0000bb is the float 2^23 + b
__device__ __forceinline__ float centred(unsigned b) { return __uint_as_float(0x4B000000u | b) - 8388736.0f; }

// Stage the raw bytes of one 12500-sample window of both pols (stream positions
// pos0 ..) into st[pol]; the window's first byte lands at st[pol] + sh[pol].
// ALIGNED (pos0 % 4 == 0, payloads at 4-byte offsets): asynchronous copies, each
// inside one payload, zero-filled for fill frames (slot -1).  Payloads are 5000
// bytes, so where a pol's pieces have one alignment mod 8 (frames back to back:
// 5032 bytes apart) the copies are 8 bytes, the window shifted to that alignment;
// 8-byte units then never straddle payloads, and the bytes beside the window that
// the first and last unit bring are payload bytes too.  Otherwise 4-byte copies,
// or, not ALIGNED, synchronous byte loads.  Positions outside the slot table and
// misaligned payloads set kErrSlotRange and read as zero bytes.
template <int B>
__device__ __forceinline__ void cp_async_k1(void* smem_dst, const void* gsrc, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(gsrc), "n"(B), "r"(src_bytes));
}

// window bytes [0, kN) of one pol in units of B bytes: piece q covers payload-linear
// bytes [5000 q, 5000 (q + 1)), which start at src0 = frames + slot - 5000 q
template <int B>
__device__ __forceinline__ void stage_pieces(unsigned char* st, int sh, const unsigned char* frames,
                                             const long long (&sv)[4], int off0, int t) {
  const int v0 = off0 - sh, v1 = off0 + kN;  // payload-linear bytes that the units cover
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int lo = max(v0, q * kDataLen), hi = min(v1, (q + 1) * kDataLen);
    if (lo >= hi) continue;
    const bool fill = sv[q] < 0;
    const unsigned char* src = frames + (fill ? 0 : sv[q] - (long long)q * kDataLen + lo);
    unsigned char* dst = st + (lo - v0);
    for (int v = B * t; v < hi - lo; v += B * kStageThreads) cp_async_k1<B>(dst + v, fill ? frames : src + v, fill ? 0 : B);
  }
}

template <bool ALIGNED>
__device__ __forceinline__ void stage_window(unsigned char* __restrict__ st, int* __restrict__ sh,
                                             const vfrb_chan_args& a, long long pos0, int& err) {
  const int t = (int)threadIdx.x - kStageT0;  // staging thread index
  if (t < 0) return;
  if (ALIGNED) {
    // the window's bytes start at payload offset off0 of slot slot0 and cover up to 4 payload pieces
    const long long slot0 = pos0 >= 0 ? pos0 / kDataLen : -1;
    const int off0 = pos0 >= 0 ? (int)(pos0 - slot0 * kDataLen) : 0;
    long long sv[2][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long slot = slot0 + q;
      const bool used = q * kDataLen - off0 < kN;
      const bool in = slot0 >= 0 && slot < a.nslots && used;
      sv[0][q] = in ? __ldg(a.slots0 + slot) : -1;
      sv[1][q] = in ? __ldg(a.slots1 + slot) : -1;
      if (!in && used) err |= kErrSlotRange;
    }
#pragma unroll
    for (int pol = 0; pol < 2; ++pol) {
      // 8-byte units: every payload at the same offset mod 8 as payload-linear bytes
      unsigned bad4 = 0, bad8 = (unsigned)(uintptr_t)a.frames & 7u;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (sv[pol][q] < 0) continue;
        if (sv[pol][q] & 3) {  // payloads must start on a 4-byte boundary
          bad4 = 1;
          sv[pol][q] = -1;
        } else {
          bad8 |= (unsigned)sv[pol][q] & 7u;
        }
      }
      if (bad4) err |= kErrSlotRange;
      unsigned char* const dst = st + pol * kStage;
      if (bad8 == 0) {
        stage_pieces<8>(dst, off0 & 7, a.frames, sv[pol], off0, t);
        if (t == 0) sh[pol] = off0 & 7;
      } else {
        stage_pieces<4>(dst, 0, a.frames, sv[pol], off0, t);
        if (t == 0) sh[pol] = 0;
      }
    }
  } else {
    for (int n = t; n < kN; n += kStageThreads) {
      const long long pos = pos0 + n;
      const long long slot = pos >= 0 ? pos / kDataLen : -1;
      unsigned char v0 = 0, v1 = 0;
      if (slot < 0 || slot >= a.nslots) {
        err |= kErrSlotRange;
      } else {
        const int off = (int)(pos - slot * kDataLen);
        const long long s0 = __ldg(a.slots0 + slot), s1 = __ldg(a.slots1 + slot);
        if (s0 >= 0) v0 = __ldg(a.frames + s0 + off);
        if (s1 >= 0) v1 = __ldg(a.frames + s1 + off);
      }
      st[n] = v0;
      st[kStage + n] = v1;
    }
    if (t < 2) sh[t] = 0;
  }
}

// CLUSTER: a cluster's CTAs take one row, a window each; else a CTA takes rows
// blockIdx.x, blockIdx.x + gridDim.x, ..., all windows of a row.
template <bool ALIGNED, bool CLUSTER>
__global__ void __launch_bounds__(kThreads, 1) k_channelise(const __grid_constant__ vfrb_chan_args a) {
  extern __shared__ float2 smem_f2[];
  float2* const Z = smem_f2;
  float2* const tw2 = smem_f2 + kN;
  float2* const tw3 = tw2 + kTw2;
  unsigned char* const stage = reinterpret_cast<unsigned char*>(tw3 + kTw3);  // [2 buffers][2 pols][kStage]
  int* const shifts = reinterpret_cast<int*>(stage + 4 * kStage);  // [2 buffers][2 pols]
  volatile int* const zero = shifts + 4;
  const int tid = threadIdx.x;
  int err = 0;
  const int nct = CLUSTER ? a.nave : 1;
  const int rank = CLUSTER ? (int)blockIdx.x % nct : 0;
  const int row0 = CLUSTER ? (int)blockIdx.x / nct : (int)blockIdx.x;
  // this CTA's windows are (row, w), rows row0 + k * gridDim.x, w < NAVE, in that order
  // (32-bit bookkeeping: a launch has fewer than 2^31 rows)
  const int nrows_cta = CLUSTER ? 1 : (a.nrows - row0 + (int)gridDim.x - 1) / (int)gridDim.x;
  const int nwin = CLUSTER ? 1 : a.nave;
  const long long win0 = a.sample0 + ((long long)row0 * a.nave + rank) * kN;  // the first one
  const long long row_step = (long long)gridDim.x * a.nave * kN;              // to the CTA's next row
  if (nrows_cta > 0) stage_window<ALIGNED>(stage, shifts, a, win0, err);
  cp_async_commit_k1();
  for (int i = tid; i < kTw2; i += kThreads) tw2[i] = g_tw2[i];
  for (int i = tid; i < kTw3; i += kThreads) tw3[i] = g_tw3[i];
  if (tid == 0) *zero = 0;
  // NFREQ-normalised pol-summed power, averaged over NAVE (PIPE:1296, 1310)
  const float scale = 0.5f / ((float)a.nfreq * (float)a.nave);
  int m, g;  // this thread's butterfly of passes 2 and 3
  butterfly_of(tid, m, g);
  const int j3 = m + 20 * g;
  float acc[25];
  int w = 0, rk = 0, buf = 0;  // window within the row, row of this CTA, staging buffer
  cp_async_wait_k1();
  __syncthreads();
#pragma unroll 1
  while (rk < nrows_cta) {
    const int wn = w + 1 < nwin ? w + 1 : 0, rn = w + 1 < nwin ? rk : rk + 1;
    const unsigned char* x0 = stage + (size_t)buf * 2 * kStage + shifts[2 * buf];
    const unsigned char* x1 = stage + (size_t)buf * 2 * kStage + kStage + shifts[2 * buf + 1];
    // the next window's buffer was last read by pass 1 of the window before, which every thread has left
    if (rn < nrows_cta)
      stage_window<ALIGNED>(stage + (size_t)(buf ^ 1) * 2 * kStage, shifts + 2 * (buf ^ 1), a,
                            win0 + rn * row_step + (long long)wn * kN, err);
    cp_async_commit_k1();
    // The tables' addresses, offset by a zero the compiler cannot see through: their
    // entries are then read where used instead of being kept in registers across the
    // whole loop, which would not fit.
    const int z = *zero;
    if (w == 0) {
#pragma unroll
      for (int k = 0; k < 25; ++k) acc[k] = 0.f;
    }
    // pass 1: R = 20, Ns = 1, from the staged bytes
    for (int j = tid; j < kB1; j += kThreads) {
      Cx v[20];
      each5([&](auto q) {
        constexpr int Q = decltype(q)::value;
#pragma unroll
        for (int r = Q; r < 20; r += 5) v[r] = Cx{centred(x0[j + kB1 * r]), centred(x1[j + kB1 * r])};
        dft20_inner<Q>(v);
      });
      dft20_outer(v);
#pragma unroll
      for (int k = 0; k < 20; ++k) Z[j + kB1 * k] = make_float2(v[dft20_pos(k)].re, v[dft20_pos(k)].im);
    }
    __syncthreads();
    // pass 2: R = 25, Ns = 20
    Cx v[25];
    if (tid < kB) {
      float2* io = Z + g + kB1 * m;
      const float2* tw = tw2 + m + z;
      each5([&](auto q) {
        constexpr int Q = decltype(q)::value;
#pragma unroll
        for (int r = Q; r < 25; r += 5) {
          const float2 x = io[25 * r];
          v[r] = Cx{x.x, x.y};
          if (r) {
            const float2 t = tw[(r - 1) * 20];
            cx_mul(v[r], t.x, t.y);
          }
        }
        dft25_inner<Q>(v);
      });
      dft25_outer(v);
#pragma unroll
      for (int k = 0; k < 25; ++k) io[25 * k] = make_float2(v[dft25_pos(k)].re, v[dft25_pos(k)].im);
    }
    __syncthreads();
    // pass 3: R = 25, Ns = 500
    if (tid < kB) {
      const float2* src = Z + 25 * g + kB1 * m;
#pragma unroll
      for (int r = 0; r < 25; ++r) {
        const float2 q = src[r];
        v[r] = Cx{q.x, q.y};
      }
    }
    cp_async_wait_k1();  // this thread's copies of the next window have landed
    __syncthreads();     // ... and everybody else's, and Z has been read
    if (tid < kB) {
      const float2* tw = tw3 + j3 + z;
      Cx lo[5], hi;
#pragma unroll
      for (int i = 1; i < 5; ++i) {
        const float2 t = tw[(i - 1) * kB];
        lo[i] = Cx{t.x, t.y};
        cx_mul(v[i], t.x, t.y);
      }
#pragma unroll
      for (int q = 1; q < 5; ++q) {
        const float2 t = tw[(3 + q) * kB];
        hi = Cx{t.x, t.y};
        cx_mul(v[5 * q], t.x, t.y);
#pragma unroll
        for (int i = 1; i < 5; ++i) {
          const Cx p = cx_prod(hi, lo[i]);
          cx_mul(v[5 * q + i], p.re, p.im);
        }
      }
      each5([&](auto q) { dft25_inner<decltype(q)::value>(v); });
      dft25_outer(v);
#pragma unroll
      for (int k = 0; k < 25; ++k) {
        const Cx x = v[dft25_pos(k)];
        acc[k] += fmaf(x.im, x.im, x.re * x.re);
      }
    }
    if (w + 1 == nwin) {  // the row is complete: |Z[k]|^2 + |Z[N-k]|^2
      float* P = reinterpret_cast<float*>(Z);
      const int row = row0 + rk * (int)gridDim.x;
      const unsigned long long orow = (unsigned long long)(a.out_row0 + row) & (unsigned long long)a.out_row_mask;
      float* dst = a.out + (long long)orow * a.out_row_stride;
      if (tid < kB) {
#pragma unroll
        for (int k = 0; k < 25; ++k) P[j3 + kB * k] = acc[k];
      }
      if constexpr (CLUSTER) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        for (int c = rank * kThreads + tid; c < a.nchanout; c += nct * kThreads) {
          const int bin = c + a.nskip;
          float p = 0.f, q = 0.f;
          for (int r = 0; r < nct; ++r) {
            const float* R = cluster.map_shared_rank(P, r);
            p = r ? p + R[bin] : R[bin];
            q = r ? q + R[kN - bin] : R[kN - bin];
          }
          dst[c] = (p + q) * scale;
        }
        cluster.sync();  // no CTA leaves while another may read its powers
      } else {
        __syncthreads();
        for (int c = tid; c < a.nchanout; c += kThreads) dst[c] = (P[c + a.nskip] + P[kN - c - a.nskip]) * scale;
        __syncthreads();
      }
    }
    w = wn;
    rk = rn;
    buf ^= 1;
  }
  if (err && a.d_err) atomicOr(a.d_err, err);
}

template <bool ALIGNED>
static int chan_launch(const vfrb_chan_args& a, int nsm, cudaStream_t s) {
  for (const void* kern : {(const void*)k_channelise<ALIGNED, false>, (const void*)k_channelise<ALIGNED, true>})
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess) {
      cudaGetLastError();
      return VFRB_ERR_CUDA;
    }
  // few rows: a cluster per row where every window can have an SM of its own
  // (clusters of NAVE leave some SMs of a GPC free: 7/8 of them)
  if (a.nave >= 2 && a.nave <= kMaxCluster && (long long)a.nrows * a.nave <= nsm * 7LL / 8) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(a.nrows * a.nave));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)a.nave;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const int st = cuda_status(cudaLaunchKernelEx(&cfg, k_channelise<ALIGNED, true>, a));
    if (st) cudaGetLastError();
    return st;
  }
  // persistent: one CTA per SM, rows dealt round robin
  const int grid = (int)std::min<long long>(a.nrows, (long long)nsm);
  k_channelise<ALIGNED, false><<<grid, kThreads, kSmem, s>>>(a);
  return cuda_status(cudaGetLastError());
}

int launch_channelise(const vfrb_chan_args& a, cudaStream_t s) {
  if (a.nrows <= 0) return a.nrows == 0 ? VFRB_OK : VFRB_ERR_ARG;
  if (!a.frames || !a.slots0 || !a.slots1 || !a.out || a.nave <= 0) return VFRB_ERR_ARG;
  if (a.twonchan != kFftN || a.nfreq != kFftN / 2 + 1) return VFRB_ERR_UNSUPPORTED;
  if (a.nskip < 1 || a.nchanout < 1 || a.nskip + a.nchanout > kFftN / 2 + 1) return VFRB_ERR_ARG;
  int st = ensure_twiddles();
  if (st) return st;
  int dev = 0, nsm = 148;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm < 1) {
    cudaGetLastError();
    nsm = 148;
  }
  return (a.sample0 % 4) == 0 ? chan_launch<true>(a, nsm, s) : chan_launch<false>(a, nsm, s);
}

}  // namespace vfrb
