// Walks the staging of the band-wise dedispersion kernel on the host for rings that
// are hardly longer than the valid rows: every copy must lie inside its channel's
// ring, every staged row must be a valid one (or share a 16-byte group with one), and
// every row that an output sums must be staged from its own place.  Reads a delay
// table and a case from stdin.  Exit code 0: so, 3: the kernel does not apply, 1: not.
#include <cstdio>
#include <vector>

#include "dedisp_band_tables.h"

using namespace vfrb;

#define CHECK(x)                                  \
  do {                                            \
    if (!(x)) {                                   \
      std::printf("line %d: %s\n", __LINE__, #x); \
      return 1;                                   \
    }                                             \
  } while (0)

int main() {
  int ndm, nchan, tt, vec;
  long long row0, ring, nvalid, nt;
  if (std::scanf("%d %d %lld %lld %lld %lld %d %d", &ndm, &nchan, &row0, &ring, &nvalid, &nt, &tt, &vec) != 8) return 2;
  std::vector<int32_t> off((size_t)ndm * nchan);
  for (auto& v : off)
    if (std::scanf("%d", &v) != 1) return 2;
  BandHost h;
  if (!band_build(h, off.data(), ndm, nchan)) return 3;
  const int NT = 32 * tt, nb = h.nblocks, G = h.gper;
  const long long vend = row0 + nvalid, mask = ring - 1;
  long long copies = 0, twice = 0;
  for (size_t bi = 0; bi < h.bands.size(); ++bi) {
    const BandDesc& b = h.bands[bi];
    for (int k = 0; k < nb; ++k) {
      const int* skew = &h.skew[(bi * nb + k) * G];
      const int g0 = k * G, g1 = std::min(h.ngroups, g0 + G);
      for (long long y = 0;; ++y) {
        const long long t0 = (skew[0] / NT + y) * NT;
        if (t0 >= (long long)skew[g1 - g0 - 1] + (kBandD - 1) * b.m + nt) break;
        const long long ta = (row0 + t0) & ~(long long)(kBandAlign - 1);
        for (int c = b.c_lo; c < b.c_lo + b.nch; ++c) {
          const long long a = ta + h.bmin[(size_t)k * nchan + c];
          const BandRows q = band_rows(a, b.lm, row0, vend, vec);
          CHECK(q.lo >= a && q.lo % vec == 0 && q.n % vec == 0 && q.n <= ring && q.lo + q.n <= vend);
          std::vector<long long> from(b.lm, -1);  // ring row each tile element was copied from
          if (q.n > 0) {
            const long long r = q.lo & mask, n1 = std::min<long long>(q.n, ring - r);
            ++copies;
            twice += n1 < q.n;
            CHECK(r % vec == 0 && n1 % vec == 0);
            CHECK(r + n1 <= ring && q.n - n1 <= ring);
            CHECK(q.lo - a + q.n <= b.lm);
            for (int i = 0; i < q.n; ++i) from[q.lo - a + i] = i < n1 ? r + i : i - n1;
          }
          // the last rows, one by one
          for (long long x = q.lo + std::max(q.n, 0); x < q.hi; ++x) {
            CHECK(x > row0 - vec && x < vend && x - a < b.lm);
            from[x - a] = x & mask;
          }
          for (int i = 0; i < b.lm; ++i)
            if (from[i] >= 0) CHECK(a + i > row0 - vec && a + i < vend && from[i] == ((a + i) & mask));
          for (int g = g0; g < g1; ++g) {
            const int gs = std::min(g * kBandD, ndm - kBandD);
            for (int j = 0; j < kBandD; ++j) {
              const long long tb = t0 - skew[g - g0] - j * b.m;  // the trial's sample at t' = t0
              for (long long t = std::max(0LL, tb); t < std::min(nt, tb + NT); ++t) {
                const long long x = row0 + t + off[(size_t)(gs + j) * nchan + c];
                CHECK(x >= a && x - a < b.lm && from[x - a] == (x & mask));
              }
            }
          }
        }
      }
    }
  }
  std::printf("copies %lld, in two parts %lld\n", copies, twice);
  return 0;
}
