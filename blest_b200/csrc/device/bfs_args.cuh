// Arguments and pull-phase constants shared by the single-source BFS kernels:
// over adjacency lists (bfs_lists.cu) and over BVSS tiles (bfs.cu).
#pragma once

#include "common.cuh"

namespace blest {
namespace dev {

struct BfsArgs {
    DevGraph g;
    uint32_t* levels;
    uint32_t* parents;
    uint32_t* visited;
    uint32_t* frontier0;
    uint32_t* frontier1;
    uint32_t* frontier2;
    uint32_t* q_rset;
    uint32_t* q_off;
    RunCounters* ctr;
    uint32_t words;
    uint32_t src;
    int direction;
    float alpha;
    float beta;
    blest_level_trace* trace;  // optional per-level records
    // Frontier summary per level (1 bit per 2^sum_shift frontier words),
    // staged in shared memory by the pull phase to skip empty words.
    uint32_t* summary0;
    uint32_t* summary1;
    uint32_t* summary2;
    uint32_t sum_shift;
    uint32_t sum_words;
    // Pull: unvisited vertices whose remaining list is longer than
    // heavy_min are scanned by all warps in kHeavyChunk pieces after a
    // mid-level barrier. heavy: {vertex, first, end, chunk offset} records.
    uint4* heavy;
    uint32_t heavy_cap;
    uint32_t heavy_min;
    // Push over lists: the queues of reached vertices with out-edges, {first
    // edge, edges, vertex, first piece}: short lists from 0, long ones from n.
    uint4* pieces;
    // Where the run's outcome goes (null: nowhere) and the call number it
    // carries.
    RunRecord* record;
    uint64_t seq;
};

// Neighbours a lane scans alone in the pull phase before the warp takes over,
// and how many of them it has in flight at once (a warp waits for its
// slowest lane, so fewer, wider rounds finish sooner).
constexpr uint32_t kPullLaneScan = 32;
constexpr uint32_t kPullUnroll = 4;
// Neighbours per piece of a heavy (very long) in-neighbour list.
constexpr uint32_t kHeavyChunk = 256;

// The run's record but its seq, which the host polls and which must become
// visible after the rest.
__device__ __forceinline__ void fill_record(RunRecord* r, const BfsArgs& a, uint64_t start_ns) {
    const RunCounters* c = a.ctr;
    r->start_ns = start_ns;
    r->end_ns = global_ns();
    r->error = ld_relaxed(&c->error);
    r->discovered = c->discovered;
    r->degree = c->degree;
    r->levels = c->levels;
    r->push_levels = c->push_levels;
    r->pull_levels = c->pull_levels;
    r->source = a.src;
}

__device__ __forceinline__ void publish_record(RunRecord* r, uint64_t seq) {
    __threadfence_system();
    *(volatile unsigned long long*)&r->seq = seq;
}

}  // namespace dev
}  // namespace blest
