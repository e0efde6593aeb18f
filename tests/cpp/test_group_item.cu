// group_item over whole grids: every item once per lane, none below zero, for numbers of
// items where items x lanes passes 2^31.  Runs on the host.
#include <cstdio>

#include "../../nelson_b200/csrc/nl_common.cuh"

int main() {
  const int nt = 128;
  for (int lanes : {4, 8, 16})
    for (long long items : {1LL, 31LL, 33LL, 1000LL, (1LL << 31) / lanes - 1, (1LL << 31) / lanes + 1, 200000000LL, 700000001LL}) {
      const long long ctas = (lanes * items + nt - 1) / nt;
      long long next = 0;  // item of the CTA's first thread
      for (long long b = 0; b < ctas; b += (b < 4 || b + 5 > ctas || ctas < 3000000) ? 1 : ctas / 1000003 + 1) {
        next = b * (nt / lanes);
        for (int t = 0; t < nt; t++)
          if (nl::group_item((unsigned)b, nt, t, lanes) != next + t / lanes) {
            std::printf("lanes %d items %lld CTA %lld thread %d\n", lanes, items, b, t);
            return 1;
          }
      }
      if (nl::group_item((unsigned)(ctas - 1), nt, nt - 1, lanes) + 1 < items) return 2;  // the grid covers the items
    }
  return 0;
}
