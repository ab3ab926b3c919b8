// row_batches (csrc/csr_rows.hpp) over all lanes of a row: the positions that
// the batches cover, counted per position from `begin`.
#include "csr_rows.hpp"

extern "C" long walk(int begin, int end, unsigned char *seen) {
  constexpr int COUNT = 9, LANES = 4;
  long batches = 0;
  for (int lane = 0; lane < LANES; ++lane)
    pda::row_batches<COUNT, LANES>(begin, end, lane, [&](unsigned q) {
      if (++batches > 1000) throw "runs away";
      for (unsigned u = 0; u < COUNT; ++u)
        if (q + u * LANES < (unsigned)end) ++seen[q + u * LANES - (unsigned)begin];
    });
  return batches;
}
