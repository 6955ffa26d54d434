// Checks resident_rule.hpp on the CPU (tests/test_resident_rule.py): LPs without long rows, LPs on both sides of
// the lines, and that a longer row never turns the choice back to the resident form.
#include <cstdio>

#include "resident_rule.hpp"

using namespace b200;

static int failures = 0;
static void check(bool ok, const char* what) {
  if (!ok) std::printf("failed: %s\n", what), ++failures;
}

// An LP of m rows of `per` entries and 1.5·m columns, with `count` more rows of `length` entries.
static bool pays(int m, int per, int count, int length, bool fp32, bool columns = false) {
  const int n = m * 3 / 2, blocks = 148;
  const double nnz = static_cast<double>(m) * per + static_cast<double>(count) * length;
  const int warps = (n / blocks + 32) / 32 + (m / blocks + 32) / 32 + 1, threads = 32 * std::min(32, warps);
  const int a_warp = std::min(count, 32) * length, narrow = 4 * per;
  RowLengths longs{256 * per, per, per > 32 ? 32 * per : 0}, others{256 * narrow / 6, narrow / 4, 0};
  if (count > 0) {
    longs.slab = std::max(longs.slab, (256 - std::min(count, 256)) * per + std::min(count, 256) * length);
    longs.longest = std::max(per, length);
    longs.together = length > 32 ? a_warp : longs.together;
  }
  return resident_pays(columns ? others : longs, columns ? longs : others, nnz, blocks, threads,
                       (static_cast<double>(m) + n) / blocks, fp32);
}

int main() {
  for (const int m : {1000, 10000, 30000, 60000, 100000}) {
    for (const bool fp32 : {false, true}) {
      check(pays(m, 6, 0, 0, fp32), "no long rows");
      check(pays(m, 6, 1, 16, fp32), "one of 16");
      for (const bool columns : {false, true})
        for (const int count : {1, 4, 32})
          for (int length = 32, was = 1; length <= 8192; length += 32) {
            const int now = pays(m, 6, count, length, fp32, columns) ? 1 : 0;
            // past the line between the two ways of summing it (32 or 64), one row never gets cheaper
            if (count == 1 && length > 64) check(now <= was, "a longer row turns the choice back");
            was = now;
          }
    }
  }
  check(pays(1000, 6, 1, 512, false) && pays(10000, 6, 1, 512, false), "512 beside 10k rows");
  check(pays(60000, 6, 1, 256, false), "256 beside 60k rows");
  check(!pays(60000, 6, 1, 1024, false), "1,024 beside 60k rows");
  check(!pays(10000, 6, 1, 4096, false) && !pays(10000, 6, 1, 4096, false, true), "4,096 beside 10k rows");
  check(!pays(60000, 6, 32, 256, false), "32 of 256 beside 60k rows");
  check(pays(1000, 50, 0, 0, false) && pays(1000, 200, 0, 0, true) && pays(300, 400, 0, 0, false), "long rows everywhere");
  if (failures == 0) std::puts("ok");
  return failures != 0;
}
