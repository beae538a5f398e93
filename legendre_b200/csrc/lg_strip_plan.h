// Unit heights of the strip kernel that are fixed (the others: lg_modelc_tile.cuh).
// Host code only.
#pragma once

#include <algorithm>
#include <cstdint>

namespace lg {

// Rows per unit of the FP32 batched step on a device of `sms` SMs.  The first
// row of a unit may be contracted otherwise than the rows inside it, so other
// heights move the states by their last bits and the gradients through them by
// 1e-7 of their size, which their FP64 outputs show.  At least 8 rows, more
// where 96 units an SM have work, at most 32 and whole fours.  By the cost of
// the other forms 4 instances of 48^2 would take 5.9 instead of 8.7 us a step,
// 32 of 128^2 the same time.
inline int strip_batch_rows_f32(int64_t nblocks, int strips, int n1, int sms) {
    const int64_t want = (int64_t)sms * 96, per_chunk = nblocks * strips;
    const int chunks = (int)std::max<int64_t>(1, std::min<int64_t>(n1, (want + per_chunk - 1) / per_chunk));
    const int rows = std::max(1, std::min({std::max(8, (n1 + chunks - 1) / chunks), 32, n1}));
    return n1 >= 4 ? std::max(4, rows / 4 * 4) : rows;
}

}  // namespace lg
