// Tables of the band-wise dedispersion kernel (dedisperse_band.cu), built on the
// host from a delay table when a plan is created.  Plain C++.
#pragma once
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define VFRB_HD __host__ __device__ __forceinline__
#else
#define VFRB_HD inline
#endif

namespace vfrb {

constexpr int kBandD = 8;                 // trials per group
constexpr int kBandW = 16;                // warps per CTA, one CTA per SM
constexpr int kBandSmax = 4;              // most rows that a group's shifts span
constexpr int kBandAlign = 16;            // rows: tile starts of every storage form are 16-byte aligned
constexpr int kBandNtMax = 320;           // longest tile (FP16): the row length in shared memory is common to all forms
constexpr int kBandSmem = 220 * 1024;     // that the tables plan for
constexpr int kBandSmemMax = 227 * 1024;  // a CTA's limit
constexpr int kBandMaxCh = 96;
constexpr int kBandMax = 64;              // bands
// Code of eight shifts that go up (or down) by 0 or 1 from trial to trial: bit q =
// the step after the q-th trial, counted from the trial with shift 0; bit 7 = the
// shifts fall (the count starts at the last trial).
constexpr int kBandGeneric = 256;         // shifts that are no such staircase

struct BandDesc {
  int c_lo, nch;    // channels [c_lo, c_lo + nch)
  int m;            // rows per trial taken off
  int ch, nchunks;  // channels per chunk
  int lm;           // tile row length in elements
  int chunk0;       // index of its first chunk among the plan's records
};

// a group's record of a chunk: slot[ch_cap] (tile offset | channel << 18), run[ch_cap] (code | count << 8), nrun
constexpr int band_rec_bytes(int ch_cap) { return (ch_cap * 6 + 2 + 15) / 16 * 16; }

// Shared memory of a launch: two mbarriers, two buffers of records, of weights and of
// tile rows; the rows' place also takes the sums of the longest tile at the end.
inline size_t band_smem(int ch, int lm, int rec_bytes, int elem, bool weighted) {
  const size_t fixed = 16 + (size_t)2 * kBandW * rec_bytes + (weighted ? (size_t)2 * ((ch + 3) / 4 * 4) * 4 : 0);
  return fixed + std::max((size_t)2 * ch * lm * elem, (size_t)kBandW * kBandNtMax * 4);
}

struct BandHost {
  int ndm = 0, nchan = 0, ngroups = 0, nblocks = 0;
  // Groups per CTA.  Its kBandW warps are `split` sets of them: with fewer
  // groups each chunk's channels are divided among the sets, whose sums are
  // added at the end, so a plan of few trials still has CTAs for every SM.  It
  // depends on the trials alone: the order of the sums must not change with the
  // number of samples.  (201 trials x 5145 samples: 16 groups per CTA give 44 CTAs
  // and 1.49 ms, 4 groups 154 CTAs and 0.94 ms.)
  int gper = kBandW, split = 1;
  std::vector<BandDesc> bands;
  std::vector<int> skmin, skmax;   // [band][block] skews of the block's first and last trial
  int rec_bytes = 0, ch_cap = 0;
  std::vector<int> bmin;           // [block][nchan] first staged row of the channel, relative to row0 + t'
  std::vector<int> skew;           // [band][nblocks * gper] skew of each group's first trial
  std::vector<unsigned char> rec;  // [chunk][nblocks][split][gper][rec_bytes]
  std::vector<unsigned> shift;     // [group][nchan] eight shifts, 4 bits each; empty when all are staircases
};

// Rows [lo, lo + n) of a tile row that starts at row a (a multiple of kBandAlign):
// the valid rows among its lm in whole groups of vec (16 bytes; the first group may
// begin before row0), and hi, the end of all its valid rows.  Only valid rows are
// read: a ring need be no longer than these, so a run of more would meet itself, or
// pass the ring's end twice.  n <= ring rows: the run is one copy, or two where it
// passes the end once.
struct BandRows {
  long long lo, hi;
  int n;
};
VFRB_HD BandRows band_rows(long long a, int lm, long long row0, long long vend, int vec) {
  const long long first = (row0 > 0 ? row0 : 0) & ~(long long)(vec - 1);
  const long long lo = a > first ? a : first, end = a + lm < vend ? a + lm : vend;
  const long long hi = end > lo ? end : lo;
  return BandRows{lo, hi, (int)((hi & ~(long long)(vec - 1)) - lo)};
}

inline long long floor_div(long long a, long long b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }
inline int floor_to(int a, int b) { return (int)floor_div(a, b) * b; }

// False when the kernel does not apply to the delay table: fewer than eight
// trials, or trials that are not close to equally spaced.
inline bool band_build(BandHost& h, const int32_t* off, int ndm, int nchan) {
  if (ndm < kBandD) return false;
  BandHost* t = &h;
  const int D = kBandD;
  t->ndm = ndm;
  t->nchan = nchan;
  const int ng = t->ngroups = (ndm + D - 1) / D;
  const int G = t->gper = ng <= 40 ? 4 : ng <= 80 ? 8 : 16;
  const int SP = t->split = kBandW / G;
  const int nb = t->nblocks = (ng + G - 1) / G;
  auto start = [&](int g) { return std::min(g * D, ndm - D); };
  auto row = [&](int d) { return off + (long long)d * nchan; };
  // bands: runs of channels whose mean delay step per trial rounds to one number
  std::vector<long long> step(nchan, 0);
  for (int g = 0; g < ng; ++g) {
    const int32_t *a = row(start(g)), *z = row(start(g) + D - 1);
    for (int c = 0; c < nchan; ++c) step[c] += z[c] - a[c];
  }
  // (the mean over a few dozen neighbouring channels: whole-number delays make a single channel's noisy)
  const double per = 1.0 / ((double)ng * (D - 1));
  std::vector<long long> cum(nchan + 1, 0);
  for (int c = 0; c < nchan; ++c) cum[c + 1] = cum[c] + step[c];
  int m = 0;
  for (int c = 0; c < nchan; ++c) {
    const int w = std::min(std::min(c, nchan - 1 - c), nchan / 256);
    const double y = (double)(cum[c + w + 1] - cum[c - w]) * per / (2 * w + 1);
    if (c == 0 || y > m + 0.51 || y < m - 0.51) {
      const int mn = (int)std::lrint(y);
      if (c == 0 || mn != m) {
        if ((int)t->bands.size() == kBandMax || mn > 4096 || mn < -4096) return false;
        m = mn;
        BandDesc b{};
        b.c_lo = c;
        b.m = m;
        t->bands.push_back(b);
      }
    }
    ++t->bands.back().nch;
  }
  const int nbands = (int)t->bands.size();
  // per (group, channel): window start relative to row0 + t', pattern, shifts
  std::vector<int> base((size_t)ng * nchan);
  std::vector<unsigned short> pat((size_t)ng * nchan);
  std::vector<unsigned>& shift = t->shift;
  std::vector<int>& skew = t->skew;
  skew.assign((size_t)nbands * nb * G, 0);
  for (int bi = 0; bi < nbands; ++bi) {
    const BandDesc& b = t->bands[bi];
    const int mid = b.c_lo + b.nch / 2;
    for (int g = 0; g < ng; ++g) {
      const int gs = start(g);
      const int sk = row(gs)[mid];
      skew[(size_t)bi * nb * G + g] = sk;
      const int32_t* r[D];
      for (int j = 0; j < D; ++j) r[j] = row(gs + j);
      const size_t i0 = (size_t)g * nchan;
      int worst = 0;
      unsigned odd = 0;
      for (int c = b.c_lo; c < b.c_lo + b.nch; ++c) {  // straight-line: the compiler vectorises it
        int v = r[0][c], mn = v, mx = v;
        unsigned up = 0, down = 0, no_up = 0, no_down = 0;
#pragma GCC unroll 8
        for (int j = 1; j < D; ++j) {
          const int n = r[j][c] - j * b.m, d = n - v;
          v = n;
          mn = std::min(mn, n);
          mx = std::max(mx, n);
          up |= (unsigned)(d & 1) << (j - 1);
          down |= (unsigned)(d & 1) << (D - 1 - j);
          no_up |= (unsigned)d & ~1u;
          no_down |= (unsigned)-d & ~1u;
        }
        worst = std::max(worst, mx - mn);
        const unsigned code = no_up == 0 ? up : no_down == 0 ? 128u | down : (unsigned)kBandGeneric;
        odd |= code;
        base[i0 + c] = mn - sk;
        pat[i0 + c] = (unsigned short)code;
      }
      if (worst > kBandSmax) return false;  // not (nearly) equally spaced
      if (odd & (unsigned)kBandGeneric) {
        if (shift.empty()) shift.assign((size_t)ng * nchan, 0u);
        for (int c = b.c_lo; c < b.c_lo + b.nch; ++c) {
          if (pat[i0 + c] != kBandGeneric) continue;
          unsigned sh = 0;
          for (int j = 0; j < D; ++j) sh |= (unsigned)(r[j][c] - j * b.m - sk - base[i0 + c]) << (4 * j);
          shift[i0 + c] = sh;
        }
      }
    }
  }
  size_t ngen = 0;
  if (!shift.empty())
    for (unsigned short q : pat) ngen += q == kBandGeneric;
  if (ngen * 20 > pat.size()) return false;  // more than 5% off the staircases: the other kernels are faster
  // per block: first staged row of each channel, and the tile row length of each band
  std::vector<int>& bmin = t->bmin;
  bmin.assign((size_t)nb * nchan, 0);
  std::vector<int> span(nbands, 0);
  for (int bi = 0; bi < nbands; ++bi)
    for (int c = t->bands[bi].c_lo; c < t->bands[bi].c_lo + t->bands[bi].nch; ++c)
      for (int k = 0; k < nb; ++k) {
        int mn = 0x7fffffff, mx = -0x7fffffff;
        for (int g = k * G; g < std::min(ng, (k + 1) * G); ++g) {
          mn = std::min(mn, base[(size_t)g * nchan + c]);
          mx = std::max(mx, base[(size_t)g * nchan + c]);
        }
        mn = floor_to(mn, kBandAlign);
        bmin[(size_t)k * nchan + c] = mn;
        span[bi] = std::max(span[bi], mx - mn);
      }
  int cap = 1;
  auto chunks = [&](BandDesc& b, int most) {
    b.nchunks = (b.nch + most - 1) / most;
    b.ch = (b.nch + b.nchunks - 1) / b.nchunks;  // even chunks
  };
  for (int bi = 0; bi < nbands; ++bi) {
    BandDesc& b = t->bands[bi];
    b.lm = (kBandAlign - 1 + span[bi] + kBandNtMax + kBandSmax + 1 + kBandAlign - 1) / kBandAlign * kBandAlign;
    // two buffers of FP32 rows and records
    int ch = (kBandSmem - 64) / (2 * (b.lm * 4 + 6 * kBandW + 4) + 64);
    ch = std::min(ch, kBandMaxCh);
    ch = std::min(ch, 32 * kBandW);
    if (ch < 8) return false;  // the block's trials spread too far to share staged rows
    chunks(b, ch);
    cap = std::max(cap, (b.ch + SP - 1) / SP);
  }
  cap = (cap + 2) & ~1;  // and a slot of padding, read ahead
  // Every band's records have the room of the largest chunk's: a band of long rows,
  // whose own chunks are short, may have to take still fewer channels beside them.
  int chunk0 = 0;
  for (BandDesc& b : t->bands) {
    while (band_smem(b.ch, b.lm, band_rec_bytes(cap), 4, false) > (size_t)kBandSmemMax) {
      if (b.ch <= 4) return false;
      chunks(b, b.ch - 1);
    }
    b.chunk0 = chunk0;
    chunk0 += b.nchunks;
  }
  t->ch_cap = cap;
  t->rec_bytes = band_rec_bytes(cap);
  const size_t ngp = (size_t)nb * G;
  std::vector<unsigned char>& rec = t->rec;
  rec.assign((size_t)chunk0 * nb * kBandW * t->rec_bytes, 0);
  for (int bi = 0; bi < nbands; ++bi) {
    const BandDesc& b = t->bands[bi];
    for (int k = 0; k < b.nchunks; ++k)
      for (int g = 0; g < ng; ++g) {
        const int c0 = b.c_lo + k * b.ch, nc = std::min(b.ch, b.nch - k * b.ch);
        const unsigned short* pp = &pat[(size_t)g * nchan + c0];
        int cnt[257] = {0}, pos[257], n = 0;
        unsigned char ord[kBandMaxCh];
        for (int i = 0; i < nc; ++i) ++cnt[pp[i]];
        for (int i = 0; i < 257; ++i) {
          pos[i] = n;
          n += cnt[i];
        }
        for (int i = 0; i < nc; ++i) ord[pos[pp[i]]++] = (unsigned char)i;
        for (int sp = 0; sp < SP; ++sp) {  // this set's share of the sorted channels
          unsigned char* q =
              rec.data() + (((size_t)(b.chunk0 + k) * nb + g / G) * kBandW + sp * G + g % G) * t->rec_bytes;
          unsigned* slot = reinterpret_cast<unsigned*>(q);
          unsigned short* run = reinterpret_cast<unsigned short*>(q + 4 * cap);
          int nrun = 0, last = -1;
          const int lo = nc * sp / SP, hi = nc * (sp + 1) / SP;
          for (int i = lo; i < hi; ++i) {
            const int cl = ord[i], code = pp[cl];
            const int rel = base[(size_t)g * nchan + c0 + cl] - bmin[(size_t)(g / G) * nchan + c0 + cl];
            slot[i - lo] = (unsigned)(cl * b.lm + rel) | ((unsigned)cl << 18);
            if (code == kBandGeneric) run[nrun++] = 0;  // no count: one channel with its own shifts
            else if (code == last) run[nrun - 1] += 1 << 8;
            else run[nrun++] = (unsigned short)(code | (1 << 8));
            last = code;
          }
          run[cap] = (unsigned short)nrun;
        }
      }
  }
  // skews of a block's first and last trial, per band (launch geometry)
  t->skmin.resize((size_t)nbands * nb);
  t->skmax.resize((size_t)nbands * nb);
  for (int bi = 0; bi < nbands; ++bi)
    for (int k = 0; k < nb; ++k) {
      int mn = 0x7fffffff, mx = -0x7fffffff;
      for (int g = k * G; g < std::min(ng, (k + 1) * G); ++g)
        for (int j = 0; j < D; j += D - 1) {
          mn = std::min(mn, skew[(size_t)bi * ngp + g] + j * t->bands[bi].m);
          mx = std::max(mx, skew[(size_t)bi * ngp + g] + j * t->bands[bi].m);
        }
      t->skmin[(size_t)bi * nb + k] = mn;
      t->skmax[(size_t)bi * nb + k] = mx;
      // the kernel takes them from the first and the last group (delays grow with the trial)
      const int g0 = k * G, g1 = std::min(ng, (k + 1) * G) - 1;
      if (mn != skew[(size_t)bi * ngp + g0] || mx != skew[(size_t)bi * ngp + g1] + (D - 1) * t->bands[bi].m)
        return false;
    }
  return true;
}

}  // namespace vfrb
