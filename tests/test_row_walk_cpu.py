"""The row walks of the whole-block bandpass and the channel statistics at counts near
the largest that they take: a thread's last rows are its own, in order, and the walk
ends."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdlib>
#include "row_walk.h"
template <int STEP, typename Row>
int walk(long long nrows, long long tid) {
  // the thread's rows from shortly before the end
  const long long first = tid + (nrows - tid - 2000) / STEP * STEP;
  long long want = first, n = 0;
  vfrb::walk_rows<STEP, STEP == 32 ? 0 : 4, Row>((Row)first, (Row)nrows, [&](auto t) {
    if (t != want || ++n > 200) std::exit(1);
    want += STEP;
  });
  return want >= nrows && want < nrows + STEP ? 0 : 2;
}
int main(int, char** v) {
  const long long nrows = std::atoll(v[2]), tid = std::atoll(v[3]);
  if (v[1][0] == 'b') return walk<vfrb::kBpFullThreads, vfrb::BpFullRow<true>>(nrows, tid);
  return walk<32, vfrb::StatsRow>(nrows, tid);
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    (d / "w.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "vlite-frb_b200", "csrc"), str(d / "w.cpp"),
                    "-o", str(d / "w")], check=True)
    return lambda kind, n, t: subprocess.run([str(d / "w"), kind, str(n), str(t)]).returncode


@pytest.mark.parametrize("nrows", [60000, 2**31 + 7, 2**32 - 257, 2**32 - 255, 2**32, 2**32 + 1, 2**33 + 12345])
def test_bandpass_walk_ends_at_the_last_row(walk, nrows):
    assert [walk("b", nrows, t) for t in (0, 1, 100, 255)] == [0, 0, 0, 0]


@pytest.mark.parametrize("nrows", [9000, 2**31 - 33, 2**31 - 31, 2**31 - 1])
def test_statistics_walk_ends_at_the_last_row(walk, nrows):
    assert [walk("s", nrows, t) for t in (0, 1, 17, 31)] == [0, 0, 0, 0]
