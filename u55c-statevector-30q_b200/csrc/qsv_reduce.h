// qsv_reduce.h -- sizes of the FP64 reductions (host).
#pragma once
#include <stdint.h>

namespace qsv {

constexpr int kRedChunkBits = 13;            // a block of reduce_chunks_kernel takes chunks of 2^13 amplitudes

constexpr int reduce_bits_of(int n) {
    int B = n - 10;
    if (B < 13) B = 13;
    if (B > n) B = n;
    if (B > 25) B = 25;
    return B;
}
// doubles of block partials that the declared scratch of an n-qubit reduction holds
constexpr long long reduce_room(int n) { return (1ll << (n - reduce_bits_of(n))) * (reduce_bits_of(n) + 1); }

// The block partials of a reduction: `blocks` blocks of nout doubles. Up to 2^9 chunks (n = 22) every chunk is a
// block of its own with the sums of its 13 bits; above, a fixed grid takes chunks in turn and keeps the sums of all n
// bits, as many blocks as fit the scratch. The grid, and so the order of the sums and their last bits, depends on n
// alone: 592 blocks are four on each of a B200's 148 SMs, and on a part of one (fewer SMs) the results stay the same.
constexpr int kReduceBlocks = 592;
struct ReduceGrid {
    int64_t blocks;
    int nout;
};
constexpr ReduceGrid reduce_grid(int n) {
    if (n <= kRedChunkBits) return {1, n + 1};
    if (n <= 22) return {1ll << (n - kRedChunkBits), kRedChunkBits + 1};
    int64_t g = kReduceBlocks;
    if (g > reduce_room(n) / (n + 1)) g = reduce_room(n) / (n + 1);
    if (g > 1ll << (n - kRedChunkBits)) g = 1ll << (n - kRedChunkBits);
    return {g, n + 1};
}

}  // namespace qsv
