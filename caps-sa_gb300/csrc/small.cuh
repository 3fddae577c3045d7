// small.cuh — suffix arrays of small plain texts in one launch (small.cu).
#pragma once

#include "common.cuh"

namespace capssa {

// Longest text one block sorts (13-bit bins, 16-bit positions, 100 KB of
// shared memory).
constexpr uint32_t kSmallText = 8192;

// Suffix array of a whole plain text of 1 .. kSmallText symbols under an
// unbounded context into the device buffer out_sa (4 or 8 bytes an entry).
// Waits for the device.  *done false: the text's ties ran too deep for one
// block (nothing useful was written) and the caller takes the general path.
capssa_status small_build(Ctx &c, const void *text, int sym_bytes, uint32_t n, int longer_first,
                          void *out_sa, int out_bytes, bool *done);

}  // namespace capssa
