// delta.cuh -- carries of delta_f columns.
//
// A delta_f column's value i is the running sum of lane i mod 8
// (delta.h:229-262).  The column is cut into segments of blocks, one per warp;
// a pass over the packed deltas sums every segment lane by lane, one CTA scans
// those sums, and a warp that decodes a whole segment then keeps its carry in
// registers from block to block.  Operators that take blocks in any order get
// the carry of every block.
#pragma once

#include "fastpath.cuh"
#include "internal.h"

namespace ms {

struct DeltaSegs {
    uint64_t nseg;
    unsigned blocks;         // per segment
    const uint64_t *prefix;  // 8 lane values before each segment
};

// A column's view without the carries of delta_f (prepare_view adds them).
int prepare_view_plain(const ms_col *c, ms_arena *a, cudaStream_t st, ColView *v);

// Segments of view `w`'s compressed part; carry_in: the 8 lane values before
// its first row (device, nullptr: zeros).  carry (optional): nb x 8 words that
// receive every block's lane values.  total (optional, device): the 8 lane
// sums over the column.
int delta_segments(const ColView &w, const uint64_t *carry_in, uint64_t *carry, uint64_t *total, DeltaSegs *out,
                   ms_arena *a, cudaStream_t st);

}  // namespace ms
