// Which heads of a block-sparse call belong to which of the two persistent kernels.
#pragma once
#include "attn_kernels.h"

namespace h3b {

// The pair kernel (attn_sparse_pair.cu) multiplies both tiles of a pair by every KV tile of the UNION of their
// lists, the single kernel (attn_sparse_t.cu) multiplies each tile by its own list only. A head goes to the pair
// kernel when joining the lists leaves less than SPARSE_PAIR_PERCENT of their entries. Whole calls, single against
// pair kernel for every head: 287 tiles x 56 heads, 67 % left: 2766 / 2439 us; 905 tiles x 24 heads, 87.5 %
// left: 9368 / 10330 us. A union tile costs 1.25 to 1.3 list entries, so the line lies near 77 %.
// The decision is the head's own, so that a head's result does not depend on which other heads are in the call,
// and a kernel takes its heads whole and in order: what runs at one time shares the K and V of few heads in L2
// (handed out pair by pair in the order in which a pre-pass happened to list them, the single kernel took 8.4 ms
// instead of 7.0 for the same 24 heads of 905 tiles).
constexpr unsigned SPARSE_PAIR_PERCENT = 75;

__device__ __forceinline__ bool head_joins(const SparseWork &w, int head) {
    if (w.assign >= 0) return w.assign != 0;
    return 100ull * w.head_sums[2 * head + 1] < (unsigned long long)SPARSE_PAIR_PERCENT * w.head_sums[2 * head];
}
// The head number k (from 0) of those that join (or do not); -1: there are fewer. For a whole warp.
__device__ __forceinline__ int nth_head(const SparseWork &w, int heads, bool joins, unsigned k) {
    const int lane = threadIdx.x & 31;
    for (int h0 = 0; h0 < heads; h0 += 32) {
        const unsigned mine = __ballot_sync(0xffffffffu, h0 + lane < heads && head_joins(w, h0 + lane) == joins);
        const unsigned n = __popc(mine);
        if (k < n) return h0 + (int)__fns(mine, 0, (int)k + 1);
        k -= n;
    }
    return -1;
}

}  // namespace h3b
