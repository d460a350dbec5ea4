// Grid size of single-source BFS over lists (plain C++: no CUDA needed).
#pragma once

#include <algorithm>
#include <cstdint>

namespace blest {

// Blocks of `threads` threads for a graph of n vertices and nnz edges, at most
// max_blocks of them resident per SM. blocks_per_sm > 0 is the caller's choice
// and is taken as it is (up to what is resident).
//
// Otherwise a small graph takes no more than it has work for, since every
// block costs every barrier of every level: a thread per vertex or per four
// edges, and below 2^20 vertices one 512-thread block's threads per SM.
// Density does not move that line (a block more per SM helps the passes over
// vertices, not those over edges). One and two blocks per SM, device us of a
// BFS: RMAT 2^16 x 16 40.1 / 41.9, 2^18 x 16 47.0 / 49.6, 2^19 x 64 (56 M
// edges) 51.3 / 52.6; uniform 2^14 x 16 32.9 / 34.3, 2^19 x 16 72.1 / 68.2,
// 2^19 x 64 (67 M edges) 63.8 / 65.6, 2^20 x 32 97.7 / 90.6, 2^21 x 16 109 /
// 96; RMAT 2^21 x 16 83 / 74; grids 2^16 370 / 386, 2^20 588 / 636.
inline int bfs_lists_blocks(uint32_t n, uint64_t nnz, int sms, int max_blocks, int blocks_per_sm, int threads) {
    if (blocks_per_sm > 0) return std::min(blocks_per_sm, max_blocks) * sms;
    uint64_t want = std::max<uint64_t>(n, nnz / 4) + 512;
    if (n < (1u << 20)) want = std::min<uint64_t>(want, 512ull * sms);
    const uint64_t blocks = (want + threads - 1) / threads;
    return (int)std::min<uint64_t>(blocks, (uint64_t)max_blocks * sms);
}

}  // namespace blest
