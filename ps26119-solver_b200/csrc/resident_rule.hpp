// resident_rule.hpp — whether the epochs of an LP that fits the SMs' shared memory are resident
// (resident.cuh) or run by the step kernels (spmv.cuh): what the long rows and columns cost in either form.
//
// Without long rows the resident form is faster wherever it fits. A long row makes every iteration wait: in the
// resident form for the thread that walks it (a trip to L2 for every 16, 8 or 4 entries, by the launch's
// block size) or for the warp that sums it (resident_long); in the step kernels, in the launch variant that does
// best there (tune.hpp measures it), for one addition per entry, and for a tile of 2,048 entries after another
// where a slab of 256 rows has more. The costs below are fits to 407 LPs of 1k to 100k rows with 1 to 128 more
// rows or columns of 16 to 4,096 entries, and with 12 to 600 entries in every row, fp64 and mixed: the form
// chosen was nowhere slower than the other's best variant by more than 25% (14 of 407, the step kernels chosen), and
// the resident form, where chosen, nowhere slower by more than 3%. On both sides of the line, us per iteration,
// resident / step kernels, one more row: 10k rows, 512 entries 7.4 / 10.0, 1,024 11.7 / 12.4, 4,096 36.9 / 29.7; 60k
// rows, 256 9.7 / 13.6, 1,024 20.5 / 15.5. Rows of 400 entries everywhere (300 x 500): 30 / 268.
#pragma once

#include <algorithm>

namespace b200 {

// The rows of a matrix (or its columns), in nonzeros.
struct RowLengths {
  int slab = 0;      // the most of 256 consecutive rows
  int longest = 0;   // the most of a row
  int together = 0;  // the most of the rows of more than 32, of 32 consecutive rows
};

// A launch's form, by its threads a block: 0 up to 256, 1 up to 512, 2 up to 1,024 (16, 8 or 4 entries in flight
// for a thread).
constexpr int resident_form(int threads) { return threads <= 256 ? 0 : threads <= 512 ? 1 : 2; }
// Rows of more entries are long: the warp sums those it has together, one after the other, if they have fewer
// than kResidentShare times the entries of the longest (more of them do better with a thread each).
constexpr int resident_long_row(int form) { return form == 0 ? 64 : 32; }
constexpr int kResidentShare = 6;

// What one side adds to an iteration of the resident form, us. share: the entries of a block's even share.
inline double resident_long_us(const RowLengths& r, double share, int threads, bool fp32) {
  const int form = resident_form(threads);
  const double walk[3] = {0.031, 0.069, 0.108}, warp[3] = {0.0086, 0.009, 0.014};  // an entry
  const double together = std::min<double>(r.together, r.longest + share);
  if (r.longest > resident_long_row(form) && together < static_cast<double>(kResidentShare) * r.longest)
    return warp[form] * (fp32 ? 0.6 : 1.0) * together;
  const double beside = std::min(32.0, static_cast<double>(r.slab) / std::max(1, r.longest));  // long rows in a warp
  return walk[form] * std::max(0, r.longest - 16) * (1.0 + beside / 64.0);
}
// What it adds to an iteration of the step kernels, us.
inline double step_long_us(const RowLengths& r) {
  const double added = std::max<double>(r.longest, r.together / 2048.0 * std::min(r.longest, 2048));
  return 0.0056 * added + 2.0 * std::max(0, r.slab - 2048) / 2048.0;
}
// The choice, for a launch of `blocks` blocks of `threads` threads, `elements` rows and columns each. What the
// resident form is ahead by without long rows: 1k rows 2.7 / 6.9 us, 10k 3.0 / 6.8, 60k 6.1 / 11.5, but
// 100k (1,689 a block) 10.0 / 11.5.
inline bool resident_pays(const RowLengths& rows, const RowLengths& cols, double nnz, int blocks, int threads,
                          double elements, bool fp32) {
  const double share = nnz / blocks, ahead = elements < 1300 ? 5.0 : 2.0;
  return resident_long_us(rows, share, threads, fp32) + resident_long_us(cols, share, threads, fp32) <=
         ahead + step_long_us(rows) + step_long_us(cols);
}

}  // namespace b200
