"""The row walk of the whole-block bandpass at counts that 32 bits do not hold: a
thread's last rows near 2^32 are its own, in order, and the walk ends."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "rfi_rows.h"
int main(int, char** v) {
  const long long nrows = std::atoll(v[1]), tid = std::atoll(v[2]);
  // the thread's rows from shortly before the end
  const long long first = tid + (nrows - tid - 2000) / vfrb::kBpFullThreads * vfrb::kBpFullThreads;
  long long want = first, n = 0;
  vfrb::bp_full_rows<4, vfrb::BpFullRow<true>>(first, nrows, [&](auto t) {
    if (t != want || ++n > 100) std::exit(1);
    want += vfrb::kBpFullThreads;
  });
  return want >= nrows && want < nrows + vfrb::kBpFullThreads ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    (d / "w.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "vlite-frb_b200", "csrc"), str(d / "w.cpp"),
                    "-o", str(d / "w")], check=True)
    return lambda n, t: subprocess.run([str(d / "w"), str(n), str(t)]).returncode


@pytest.mark.parametrize("nrows", [60000, 2**31 + 7, 2**32 - 257, 2**32 - 255, 2**32, 2**32 + 1, 2**33 + 12345])
def test_walk_ends_at_the_last_row(walk, nrows):
    assert [walk(nrows, t) for t in (0, 1, 100, 255)] == [0, 0, 0, 0]

