// How the threads of a CTA are laid over rows of `units` columns (or groups of columns) when every thread keeps its column and
// walks over rows: a CTA takes as many whole rows as fit; rows wider than the CTA are cut into equal parts (grid.y).
#pragma once
#include "common.cuh"

namespace f2c {

struct Lanes { int parts, part, rows_per_cta, threads; };

// Of the CTA sizes between half of `most` and `most` (multiples of 32 that hold a part) the one with the fewest idle threads:
// 101 columns fill 505 of 512 threads, 357 columns 357 of 384.  Work that does not fill the chip is spread over all its
// multiprocessors in CTAs of 128 threads.
static inline Lanes lanes_of_rows(int64_t units, int64_t rows, int sms, int most) {
  Lanes l;
  if (rows * units < (int64_t)sms * 3 * 512) most = 128;
  if (units > most && most < 512) most = units >= 512 ? 512 : (int)ceil_div(units, 32) * 32;
  l.parts = (int)ceil_div(units, most);
  l.part = (int)ceil_div(units, l.parts);
  l.threads = most;
  double best = 0.0;
  for (int t = most; t >= most / 2; t -= 32) {
    if (t < l.part) break;
    const double used = (double)(t / l.part * l.part) / t;
    if (used > best + 0.02) { best = used; l.threads = t; }
  }
  l.rows_per_cta = l.threads / l.part;
  return l;
}

}  // namespace f2c
