// Walk over the CSR positions [begin, end) of a row by one of several lanes,
// in batches of COUNT positions STRIDE apart.  Positions are unsigned: a matrix
// may have up to 2^31 - 2 entries, and the position after a lane's last batch
// (up to COUNT * STRIDE - 1 beyond the row's end) does not fit an int then.
#pragma once

#ifdef __CUDACC__
#define PDA_ROW_FN __host__ __device__ __forceinline__
#else
#define PDA_ROW_FN inline
#endif

namespace pda {

// f(q): the lane's batch q, q + STRIDE, ..., of which those below `end` belong to the row
template <int COUNT, int STRIDE, class F>
PDA_ROW_FN void row_batches(int begin, int end, int lane, F f) {
  for (unsigned q = (unsigned)begin + lane; q < (unsigned)end; q += COUNT * STRIDE) f(q);
}

}  // namespace pda
