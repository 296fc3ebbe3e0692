"""Shared memory of the band-wise dedispersion launches, for lists equally spaced in
two parts: beside a gap a group block's rows spread, and the band's chunks shrink with
them, down to lists that the kernel refuses.  No launch may ask for more than a CTA's
limit: the plan was accepted, so its calls have no other kernel."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include "dedisp_band_tables.h"
using namespace vfrb;
int main() {
  // 146 channels without delay (the longest chunks), then 80 of one row per trial, every
  // other one with a gap of x rows between the eighth and ninth group of a CTA's sixteen
  const int ndm = 768, na = 146, nb = 80, nchan = na + nb;
  int built = 0, refused = 0;
  size_t most = 0;
  for (int x = 0; x < 4000; x += 16) {
    std::vector<int32_t> off((size_t)ndm * nchan, 0);
    for (int d = 0; d < ndm; ++d)
      for (int c = na; c < nchan; ++c) off[(size_t)d * nchan + c] = d + (c & 1 && d % 128 >= 64 ? x : 0) * (d < 128);
    for (int d = 128; d < ndm; ++d)
      for (int c = na; c < nchan; ++c) off[(size_t)d * nchan + c] += x;
    BandHost h;
    if (!band_build(h, off.data(), ndm, nchan)) {
      ++refused;
      continue;
    }
    ++built;
    int chunk = 0, chan = 0;
    for (const BandDesc& b : h.bands) {
      // as the launch has it: two mbarriers, two buffers of 16 records and of rows
      const size_t smem = 16 + (size_t)2 * kBandW * h.rec_bytes + (size_t)2 * b.ch * b.lm * 4;
      most = std::max(most, smem);
      if (b.chunk0 != chunk || b.c_lo != chan || b.ch * b.nchunks < b.nch || b.ch * (b.nchunks - 1) >= b.nch) return 1;
      chunk += b.nchunks;
      chan += b.nch;
    }
    if (h.rec.size() != (size_t)chunk * h.nblocks * kBandW * h.rec_bytes || chan != nchan) return 2;
  }
  std::printf("%d %d %zu\n", built, refused, most);
  return 0;
}
"""


def test_launches_fit_a_cta(tmp_path):
    src, exe = tmp_path / "smem.cpp", tmp_path / "smem"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "vlite-frb_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0
    built, refused, most = map(int, r.stdout.split())
    assert built > 100 and refused > 0
    assert most <= 227 * 1024, most
