// pinned.h -- page-locked host memory that a handle can do without.
#pragma once

#include <cstddef>

namespace nl {

// `base` bytes that the handle needs and `extra` more that only save it a staged copy:
// where the host does not grant both, `base` alone.  alloc(void**, bytes): true where
// it could allocate.  False where not even `base` could be had; *got: bytes past
// `base`.
template <typename Alloc>
bool alloc_pinned(Alloc alloc, void** p, size_t base, size_t extra, size_t* got) {
  *got = 0;
  if (extra > 0 && alloc(p, base + extra)) {
    *got = extra;
    return true;
  }
  return alloc(p, base);
}

}  // namespace nl
