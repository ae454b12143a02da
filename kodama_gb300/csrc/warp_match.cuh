// Lanes of a warp that hold the same code.
#pragma once

#include <cuda_runtime.h>

namespace kgb {

// Those of `act` whose code (of `bits` bits) equals this lane's, by a ballot a bit.
// __match_any_sync takes two cycles of the whole SM per distinct code, which suits a
// vote's few (by ballots 20000 x 50 rows took 13.1 ms in place of 12.1) but not a sort's.
__device__ __forceinline__ unsigned same_code(int code, unsigned act, int bits) {
  unsigned m = act;
  for (int b = 0; b < bits; ++b) {
    const unsigned v = __ballot_sync(0xffffffffu, (code >> b) & 1);
    m &= (code >> b) & 1 ? v : ~v;
  }
  return m;
}

}  // namespace kgb
