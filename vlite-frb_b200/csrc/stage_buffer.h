// A staging buffer for pageable input: a few frames when its stream opens, grown when a
// push first brings more.  Plain C++.
#pragma once
#include <cstddef>
#include <cstdint>

namespace vfrb {

struct StageBuffer {
  uint8_t* p = nullptr;
  size_t frames = 0;   // that it holds
  bool whole = false;  // grown, or growing failed: it stays as it is
};

// Frames that the next push of `want` frames may copy through b.  alloc(frames) returns a
// page-locked buffer, or NULL: the old one then serves in smaller pieces.  The buffer
// that is replaced stays with its owner (copies from it may be in flight).
template <typename Alloc>
size_t stage_room(StageBuffer& b, size_t want, size_t full, Alloc alloc) {
  if (want > b.frames && !b.whole) {
    b.whole = true;
    if (uint8_t* q = alloc(full)) {
      b.p = q;
      b.frames = full;
    }
  }
  return want < b.frames ? want : b.frames;
}

}  // namespace vfrb
