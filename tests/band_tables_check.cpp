// Walks the band-wise dedispersion kernel's tables on the host as the kernel
// does: stages tile rows, sums windows by pattern, adds them to the trials'
// skewed accumulators and writes every output once per band, with every tile
// access checked against the row length.  Reads a delay table and a case from
// stdin, sums whole numbers (exact in any order) and compares with the plain
// sum.  Exit code 0: equal, 3: the kernel does not apply, 1: a mismatch.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "dedisp_band_tables.h"

using namespace vfrb;

#define CHECK(x)                                       \
  do {                                                 \
    if (!(x)) {                                        \
      std::printf("line %d: %s\n", __LINE__, #x);      \
      return 1;                                        \
    }                                                  \
  } while (0)

int main() {
  int ndm, nchan, tt, over;
  long long row0, mask, nvalid, nt;
  if (std::scanf("%d %d %lld %lld %lld %lld %d %d", &ndm, &nchan, &row0, &mask, &nvalid, &nt, &tt, &over) != 8) return 2;
  std::vector<int32_t> off((size_t)ndm * nchan);
  for (auto& v : off)
    if (std::scanf("%d", &v) != 1) return 2;
  BandHost h;
  if (!band_build(h, off.data(), ndm, nchan)) return 3;
  // a value per (channel, absolute row); rows outside the valid ones hold a poison value
  auto value = [&](int c, long long r) -> long long {
    if (r < 0 || r >= row0 + nvalid) return 0;  // staged as zeros
    if (r < row0) return 1000003;               // another part of the ring: must never count
    return (long long)((unsigned)(c * 2654435761u + (unsigned)r * 40503u) >> 16) - 32768;
  };
  const int NT = 32 * tt;
  const int W = kBandW, G = h.gper, nb = h.nblocks;
  CHECK(G * h.split == W);
  std::vector<long long> out((size_t)ndm * nt, 0);
  std::vector<int> written((size_t)ndm * nt, 0);
  int channels = 0;
  for (size_t bi = 0; bi < h.bands.size(); ++bi) {
    const BandDesc& b = h.bands[bi];
    CHECK(b.c_lo == channels);
    channels += b.nch;
    CHECK((b.ch + h.split - 1) / h.split < h.ch_cap && b.ch <= kBandMaxCh && b.ch <= 32 * W);
    CHECK((size_t)2 * b.ch * b.lm * 4 + 2 * W * h.rec_bytes + 16 + 2 * 4 * (b.ch + 3) <= (size_t)kBandSmem);
    long long gy = 1;
    for (int k = 0; k < nb; ++k)
      gy = std::max(gy, floor_div(h.skmax[bi * nb + k] + nt - 1, NT) - floor_div(h.skmin[bi * nb + k], NT) + 1);
    for (int k = 0; k < nb; ++k)
      for (long long y = 0; y < gy; ++y) {
        const int* skew = &h.skew[(bi * nb + k) * G];
        CHECK(skew[0] >= 0);
        const long long t0 = (skew[0] / NT + y) * NT;
        const int nd = std::min(G, h.ngroups - k * G);
        if (t0 >= (long long)skew[nd - 1] + (kBandD - 1) * b.m + nt || t0 + NT <= skew[0]) continue;
        const long long ta = (row0 + t0) & ~(long long)(kBandAlign - 1);
        const int phase = (int)(row0 + t0 - ta);
        for (int w = 0; w < G; ++w) {
          const int g = k * G + w;
          std::vector<long long> acc((size_t)kBandD * NT, 0);
          for (int q = 0; q < b.nchunks; ++q) {
            int total = 0;
            std::vector<int> seen(b.ch, 0);
            for (int set = 0; set < h.split; ++set) {
            const unsigned char* rec = &h.rec[(((size_t)(b.chunk0 + q) * nb + k) * W + set * G + w) * h.rec_bytes];
            const unsigned* slot = reinterpret_cast<const unsigned*>(rec);
            const unsigned short* run = reinterpret_cast<const unsigned short*>(rec + 4 * h.ch_cap);
            const int nrun = run[h.ch_cap];
            int at = 0;
            for (int r = 0; r < nrun; ++r) {
              const int n = run[r] >> 8, code = run[r] & 255;
              for (int i = 0; i < std::max(n, 1); ++i, ++at) {
                const int cl = (int)(slot[at] >> 18), rel = (int)(slot[at] & 0x3ffff) - cl * b.lm;
                const int c = b.c_lo + q * b.ch + cl;
                CHECK(cl < std::min(b.ch, b.nch - q * b.ch) && rel >= 0 && !seen[cl]++);
                int sh[8], most = 0;
                for (int j = 0; j < 8; ++j) {
                  const int q = code & 128 ? 7 - j : j;  // trials before it in the staircase
                  sh[j] = n ? __builtin_popcount(code & ((1 << q) - 1)) : (int)(h.shift[(size_t)g * nchan + c] >> (4 * j)) & 15;
                  most = std::max(most, sh[j]);
                }
                CHECK(most <= kBandSmax);
                CHECK(rel + phase + NT + kBandSmax + over <= b.lm);
                const long long a = ta + h.bmin[(size_t)k * nchan + c];
                CHECK(a % kBandAlign == 0);
                for (int j = 0; j < 8; ++j)
                  for (int i2 = 0; i2 < NT; ++i2) acc[j * NT + i2] += value(c, a + rel + phase + i2 + sh[j]);
              }
            }
            total += at;
            }
            CHECK(total == (g < h.ngroups ? std::min(b.ch, b.nch - q * b.ch) : 0));
          }
          if (g >= h.ngroups) continue;
          const int gs = std::min(g * kBandD, ndm - kBandD);
          for (int j = 0; j < kBandD; ++j) {
            if (gs + j < g * kBandD) continue;
            for (int i = 0; i < NT; ++i) {
              const long long t = t0 - skew[w] - j * b.m + i;
              if (t < 0 || t >= nt) continue;
              out[(size_t)(gs + j) * nt + t] += acc[j * NT + i];
              ++written[(size_t)(gs + j) * nt + t];
            }
          }
        }
      }
  }
  CHECK(channels == nchan);
  for (int d = 0; d < ndm; ++d)
    for (long long t = 0; t < nt; ++t) {
      CHECK(written[(size_t)d * nt + t] == (int)h.bands.size());
      long long s = 0;
      for (int c = 0; c < nchan; ++c) s += value(c, row0 + t + off[(size_t)d * nchan + c]);
      CHECK(s == out[(size_t)d * nt + t]);
    }
  std::printf("bands %zu generic %d\n", h.bands.size(), (int)!h.shift.empty());
  return 0;
}
