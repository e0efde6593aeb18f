// alloc_pinned on an allocator that refuses large requests, and one that refuses all.
#include <cstdlib>

#include "../../nelson_b200/csrc/pinned.h"

int main() {
  size_t limit = 0, got = 9;
  int calls = 0;
  auto alloc = [&](void** p, size_t n) {
    calls++;
    if (n > limit) return false;
    *p = std::malloc(n);
    return true;
  };
  auto once = [&](size_t lim, size_t base, size_t extra, bool want, size_t want_got, int want_calls) {
    void* p = nullptr;
    limit = lim;
    calls = 0;
    const bool ok = nl::alloc_pinned(alloc, &p, base, extra, &got);
    std::free(p);
    return ok == want && (p != nullptr) == want && got == want_got && calls == want_calls;
  };
  if (!once(1 << 20, 4096, 1000, true, 1000, 1)) return 1;  // granted in full
  if (!once(8192, 4096, 1 << 20, true, 0, 2)) return 2;     // only the base
  if (!once(8192, 4096, 0, true, 0, 1)) return 3;           // none wanted
  if (!once(1000, 4096, 1000, false, 0, 2)) return 4;       // nothing granted
  return 0;
}
