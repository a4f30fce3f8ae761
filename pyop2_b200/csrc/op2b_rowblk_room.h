// Size of the packet array of row blocks (op2b_rowblk.cu), on the host.
#pragma once

#include <cstdint>

namespace op2b {

// 16-byte units for elements shared by 1.7 blocks and targets by 2; what the
// blocks really take is known after the first pass over them.  All products in 64
// bits: nelem * ra * ca goes up to 2^31 and each part is a multiple of it.
inline int64_t row_block_room(int64_t nelem, int64_t ra, int64_t ca, int64_t nrows, int64_t nentries,
                              int64_t nblocks, bool ids, int nstage, const int32_t *stage_arity) {
  int64_t bytes = ((ids ? 4 : 0) + 2 * ra) * nelem * 17 / 10 + 8 * nentries + nelem * ra * ca / 2;
  for (int q = 0; q < nstage; ++q) bytes += 8 * nrows + 2 * stage_arity[q] * nelem * 17 / 10;
  return bytes / 16 + nblocks * (7 + 2 * nstage);
}

}  // namespace op2b
