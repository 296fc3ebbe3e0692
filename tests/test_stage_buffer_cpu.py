"""Growth of the staging buffers for pageable input, with an allocator that fails: a push
is never left without a buffer, nor with one smaller than it is told."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "stage_buffer.h"
using vfrb::StageBuffer;
using vfrb::stage_room;
#define CHECK(x) if (!(x)) return __LINE__
int main() {
  uint8_t few[16], large[1];  // addresses only
  int calls = 0;
  auto fails = [&](size_t) { ++calls; return (uint8_t*)nullptr; };
  auto works = [&](size_t n) { ++calls; return n == 8192 ? large : nullptr; };
  StageBuffer a{few, 16, false};
  CHECK(stage_room(a, 3, 8192, fails) == 3 && calls == 0);      // fits: nothing is asked for
  CHECK(stage_room(a, 500, 8192, fails) == 16 && a.p == few && a.frames == 16 && calls == 1);
  CHECK(stage_room(a, 10, 8192, fails) == 10 && a.p == few);    // the next small push
  CHECK(stage_room(a, 9000, 8192, fails) == 16 && calls == 1);  // and the next long one
  StageBuffer b{few, 16, false};
  calls = 0;
  CHECK(stage_room(b, 17, 8192, works) == 17 && b.p == large && b.frames == 8192 && calls == 1);
  CHECK(stage_room(b, 8192, 8192, works) == 8192 && stage_room(b, 1, 8192, works) == 1 && calls == 1);
  return 0;
}
"""


def test_a_failed_growth_leaves_the_small_buffer(tmp_path):
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + os.path.join(ROOT, "vlite-frb_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
