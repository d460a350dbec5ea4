// Single-source direction-optimising BFS over adjacency lists, as ONE
// persistent cooperative kernel per BFS: the default kernel behind blest_bfs
// and blest_bfs_ws (bfs.cu keeps the kernel over BVSS tiles for the b1-MMA
// slice test and for blest_bfs_noalloc, whose callers hand over tiles only).
//
// Same levels as the six BFS kernels of BFS/BVSSBFSKernel.cuh (:33-1261). A
// push level over tiles reads every slice of every set that holds one
// frontier vertex (a uniform graph's level of 41 k vertices: 49 MB of tiles
// for 1.3 M edges, 62 us); here it reads the frontier's own out-lists.
//
// The frontier has two forms, and each level uses the one its direction
// reads:
//  - two queues of {first edge, edges, vertex} (push): lists of at most 128
//    edges, of which a warp takes 32 and walks their edges as one flat range,
//    and longer ones, whose 128-edge pieces are numbered through (each entry
//    holds its first piece's number) and split evenly over the warps. One
//    entry per vertex: writing out the pieces themselves took 24 us for the
//    317 k pieces of RMAT-22's second level, its edges 7 us;
//  - a bitmap with a summary of its non-empty words (pull, and the result of
//    a lazy push).
// A change of form costs one more grid barrier, once or twice in a run; in
// return push levels keep no bitmap and pull levels queue nothing.
//
// What bounds it: levels are short, so chains of dependent L2 round trips
// (~0.7 us each) and words that every warp updates (about one access a
// nanosecond per word). A block therefore gathers its level's discoveries in
// shared memory and appends them with one atomic, and while the frontier is
// small ("solo" levels) block 0 runs the levels alone out of shared memory,
// with block barriers only, while the others wait in one grid barrier.
// Against the kernel over tiles (a whole call): RMAT 2^10 63 -> 42 us, RMAT-16
// 72 -> 53, RMAT-22 215 -> 129 a BFS, grid 2901 x 2801 3080 -> 1090 (widest
// level, 306 k vertices: 71 -> 20; smallest levels 8 -> 3), uniform 2 M
// vertices x degree 32 211 -> 103 (41 k-vertex level 62 -> 26).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "../host/common.hpp"
#include "../host/errors.hpp"
#include "bfs_args.cuh"
#include "bfs_grid.hpp"
#include "common.cuh"
#include "runtime.hpp"

namespace blest {
namespace dev {
namespace {

constexpr uint32_t kPiece = kBfsPieceEdges;
constexpr uint32_t kPullWords = 16;     // words a warp takes at a time in a pull level
constexpr uint32_t kPullItems = 2;      // vertices a lane tries at a time
constexpr uint32_t kPullWarpScan = 128; // list remainders above this are scanned by the whole warp
constexpr uint32_t kMaxWarps = 16;      // per block (512 threads)
constexpr uint32_t kWinners = 2048;     // discoveries a block gathers before it appends one warp at a time
// A level is run by block 0 alone when its pieces and edges fit these: one
// flat step of its warps (16 warps x 128 edges).
constexpr uint32_t kSoloPieces = 512;
constexpr uint32_t kSoloEdges = 2048;
// Solo levels in a row, after which the waiting blocks' barrier is renewed
// (its wait is bounded, a solo level takes a few microseconds).
constexpr uint32_t kSoloLevels = 512;

// A queue position or size: short lists, long lists, pieces of the long lists.
struct Span {
    uint32_t a, b, u;
};

static_assert(4 * kSoloPieces >= kWinners, "BlockState::pulled holds as many as the other buffer");
struct BlockState {
    union {
        struct {  // push: the level's discoveries (vertex, first out-edge, out-degree)
            uint32_t win_v[kWinners], win_b[kWinners], win_d[kWinners];
        };
        struct {  // pull, per warp: the chunk's vertices, those set aside, found bits
            uint16_t items[kMaxWarps][32 * kPullWords];
            uint16_t later[kMaxWarps][32 + 32 * kPullItems];
            uint32_t found[kMaxWarps][kPullWords];
        };
    };
    union {
        uint4 solo[kSoloPieces];  // one-block levels: the frontier's pieces
        uint32_t pulled[4 * kSoloPieces];  // pull: vertices to queue
    };
    uint32_t win_cnt, win_end;       // appended; where the first append that did not fit starts
    uint32_t tot_ab[kMaxWarps], tot_u[kMaxWarps], tot_d[kMaxWarps], tot_disc[kMaxWarps], tot_deg[kMaxWarps];
    Span base;
    uint32_t ok;
    unsigned long long val[kSlotWords];  // the step's counters after its barrier
};

// The run's state, the same in every block.
struct Run {
    uint32_t level;
    uint32_t step;        // rounds of the main loop: counter slot (step % 3), record of the solo levels (step % 2)
    Span from, size;      // the frontier's entries in the two queues (from.u is unused)
    uint32_t D2, D1;      // vertices discovered up to the last level but one / the last level
    uint32_t nf_prev;
    uint32_t push, pull;  // levels run (kept here: a counter in memory costs its warp a round trip a level)
    unsigned long long G2, G1;  // their degree sums
};

__device__ __forceinline__ uint32_t* bitmap_of(const BfsArgs& a, uint32_t gen) {
    const uint32_t m = gen % 3;
    return m == 0 ? a.frontier0 : (m == 1 ? a.frontier1 : a.frontier2);
}

__device__ __forceinline__ uint32_t* summary_of(const BfsArgs& a, uint32_t gen) {
    const uint32_t m = gen % 3;
    return m == 0 ? a.summary0 : (m == 1 ? a.summary1 : a.summary2);
}

__device__ __forceinline__ void mark_summary(const BfsArgs& a, uint32_t* sum, uint32_t word) {
    const uint32_t sb = word >> a.sum_shift;
    atomicOr(&sum[sb >> 5], 1u << (sb & 31));
}

__device__ __forceinline__ uint32_t pieces_of(uint32_t degree) { return (degree + kPiece - 1) / kPiece; }

// Where a step appends: entries from `from` on, counted by *ca (short lists)
// and *cb (long lists, packed entries << kQShift | pieces), which start at 0.
struct Tail {
    Span from;
    unsigned long long* ca;
    unsigned long long* cb;
};

__device__ __forceinline__ Span span_of(unsigned long long ca, unsigned long long cb) {
    return Span{(uint32_t)ca, (uint32_t)(cb >> kQShift), (uint32_t)(cb & kQUnitMask)};
}

// Reserve room for `need` entries (one thread); returns where they go.
__device__ __forceinline__ Span reserve(const Tail& t, const Span& need) {
    Span at{0u, 0u, 0u};
    if (need.a) at.a = t.from.a + (uint32_t)atomicAdd(t.ca, (unsigned long long)need.a);
    if (need.b) {
        const unsigned long long o = atomicAdd(t.cb, ((unsigned long long)need.b << kQShift) | need.u);
        at.b = t.from.b + (uint32_t)(o >> kQShift);
        at.u = (uint32_t)(o & kQUnitMask);
    }
    return at;
}

// Write vertex v's entry and advance `at` past it. Every vertex is queued at
// most once, so the queues cannot overflow.
__device__ __forceinline__ void put_entry(const BfsArgs& a, Span& at, uint32_t v, uint32_t b, uint32_t d) {
    if (d == 0) return;
    const bool is_long = d > kPiece;
    const uint32_t e = is_long ? a.g.n + at.b : at.a;
    if (is_long ? e < a.g.piece_cap : e < a.g.n) a.pieces[e] = make_uint4(b, d, v, is_long ? at.u : 0u);
    else set_error(a.ctr, BLEST_ERR_DEVICE_INDEX);
    if (is_long) {
        ++at.b;
        at.u += pieces_of(d);
    } else {
        ++at.a;
    }
}

__device__ __forceinline__ uint32_t warp_incl(uint32_t x) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, x, s);
        if (lane >= s) x += o;
    }
    return x;
}

// A warp's discoveries (bit k of `won`: vertex v[k], out-list at b[k] of length
// d[k]) straight to the global queues, with one reservation.
__device__ __forceinline__ void append(const BfsArgs& a, const uint32_t (&v)[4], const uint32_t (&b)[4],
                                       const uint32_t (&d)[4], uint32_t won, const Tail& tail) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t ab = 0, u = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!((won >> k) & 1u) || !d[k]) continue;
        ab += d[k] > kPiece ? 0x10000u : 1u;
        u += d[k] > kPiece ? pieces_of(d[k]) : 0u;
    }
    const uint32_t iab = warp_incl(ab), iu = warp_incl(u);
    Span at{0u, 0u, 0u};
    if (lane == 31) at = reserve(tail, Span{iab & 0xFFFFu, iab >> 16, iu});
    at.a = __shfl_sync(0xFFFFFFFFu, at.a, 31) + ((iab - ab) & 0xFFFFu);
    at.b = __shfl_sync(0xFFFFFFFFu, at.b, 31) + ((iab - ab) >> 16);
    at.u = __shfl_sync(0xFFFFFFFFu, at.u, 31) + iu - u;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if ((won >> k) & 1u) put_entry(a, at, v[k], b[k], d[k]);
}

// Hand a warp's discoveries to the block's buffer; when it is full, to the global queues.
__device__ __forceinline__ void emit(const BfsArgs& a, BlockState& B, const uint32_t (&v)[4], const uint32_t (&b)[4],
                                     const uint32_t (&d)[4], uint32_t won, const Tail& tail) {
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    uint32_t off[4], total = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, (won >> k) & 1u);
        off[k] = total + __popc(m & below);
        total += __popc(m);
    }
    if (!total) return;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&B.win_cnt, total);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (base + total <= kWinners) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (!((won >> k) & 1u)) continue;
            B.win_v[base + off[k]] = v[k];
            B.win_b[base + off[k]] = b[k];
            B.win_d[base + off[k]] = d[k];
        }
        return;
    }
    // the counter only grows, so every later append fails too and the entries
    // before the first failed one are exactly those written
    if (lane == 0) atomicMin(&B.win_end, base);
    append(a, v, b, d, won, tail);
}

// The block's buffered discoveries as queue entries: into the global queues
// (one reservation per block), or, when `solo` and they fit, as pieces into
// B.solo. Adds the block's discovery count and degree sum to lvl[1], lvl[2]
// (when lvl). The buffer's counters stay as they are: every warp reads them
// here, so they are reset behind a barrier that follows (reset_buffer).
struct Flushed {
    uint32_t pieces, disc, deg;
    bool in_solo;
};
__device__ __forceinline__ void reset_buffer(BlockState& B) {  // one thread, between two block barriers
    B.win_cnt = 0;
    B.win_end = kWinners;
}
__device__ __forceinline__ Flushed flush(const BfsArgs& a, BlockState& B, const Tail& tail, unsigned long long* lvl,
                                         uint32_t disc, uint32_t deg, bool solo) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    const uint32_t m = min(B.win_cnt, B.win_end);
    const bool spilled = B.win_end != kWinners;
    // Few discoveries (m is the same in every thread), as in most levels: one
    // warp does it all, and the discoveries' own degrees are the counts (a
    // block-wide scan costs two more barriers, a microsecond of a 6 us level).
    if (m <= 32 && !spilled && a.g.out_ptrs == a.g.csr_ptrs) {
        Flushed F{0, m, 0, false};
        if (w == 0) {
            const uint32_t d = lane < m ? B.win_d[lane] : 0u, b = lane < m ? B.win_b[lane] : 0u;
            const uint32_t v = lane < m ? B.win_v[lane] : 0u;
            const uint32_t ab = d > kPiece ? 0x10000u : (d ? 1u : 0u), u = d > kPiece ? pieces_of(d) : 0u;
            const uint32_t iab = warp_incl(ab), iu = warp_incl(u), sum = __reduce_add_sync(0xFFFFFFFFu, d);
            const uint32_t all_ab = __shfl_sync(0xFFFFFFFFu, iab, 31), all_u = __shfl_sync(0xFFFFFFFFu, iu, 31);
            const uint32_t pieces = (all_ab & 0xFFFFu) + all_u;
            const bool fits = solo && pieces <= kSoloPieces && sum <= kSoloEdges;
            const uint32_t pab = iab - ab, pu = iu - u;
            if (fits) {
                uint32_t at = (pab & 0xFFFFu) + pu;
                for (uint32_t k = 0; k < d; k += kPiece) B.solo[at++] = make_uint4(b + k, min(kPiece, d - k), v, 0u);
            } else if (pieces) {
                Span at{0u, 0u, 0u};
                if (lane == 0) at = reserve(tail, Span{all_ab & 0xFFFFu, all_ab >> 16, all_u});
                at.a = __shfl_sync(0xFFFFFFFFu, at.a, 0) + (pab & 0xFFFFu);
                at.b = __shfl_sync(0xFFFFFFFFu, at.b, 0) + (pab >> 16);
                at.u = __shfl_sync(0xFFFFFFFFu, at.u, 0) + pu;
                put_entry(a, at, v, b, d);
            }
            if (lane == 0) {
                if (lvl && m) {
                    atomicAdd(&lvl[1], (unsigned long long)m);
                    atomicAdd(&lvl[2], (unsigned long long)sum);
                }
                B.tot_u[0] = pieces;
                B.tot_deg[0] = sum;
                B.ok = fits;
            }
        }
        if (lvl) return F;  // (the caller reads nothing of it, and its barrier follows)
        __syncthreads();
        F.pieces = B.tot_u[0];
        F.deg = B.tot_deg[0];
        F.in_solo = B.ok;
        return F;
    }
    uint32_t ab = 0, u = 0, ed = 0;  // short | long << 16 entries, pieces of the long ones, edges
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
        const uint32_t d = B.win_d[i];
        ab += d > kPiece ? 0x10000u : (d ? 1u : 0u);
        u += d > kPiece ? pieces_of(d) : 0u;
        ed += d;
    }
    const uint32_t iab = warp_incl(ab), iu = warp_incl(u);
    ed = __reduce_add_sync(0xFFFFFFFFu, ed);
    disc = __reduce_add_sync(0xFFFFFFFFu, disc);
    deg = __reduce_add_sync(0xFFFFFFFFu, deg);
    if (lane == 31) {
        B.tot_ab[w] = iab;
        B.tot_u[w] = iu;
        B.tot_d[w] = ed;
        B.tot_disc[w] = disc;
        B.tot_deg[w] = deg;
    }
    __syncthreads();
    Flushed F{0, 0, 0, false};
    uint32_t before_ab = 0, before_u = 0, all_ab = 0, all_u = 0, edges = 0;
    for (uint32_t i = 0; i < nw; ++i) {
        if (i == w) {
            before_ab = all_ab;
            before_u = all_u;
        }
        all_ab += B.tot_ab[i];
        all_u += B.tot_u[i];
        edges += B.tot_d[i];
        F.disc += B.tot_disc[i];
        F.deg += B.tot_deg[i];
    }
    F.pieces = (all_ab & 0xFFFFu) + all_u;
    F.in_solo = solo && !spilled && F.pieces <= kSoloPieces && edges <= kSoloEdges;
    if (threadIdx.x == 0) {
        if (lvl && F.disc) {
            atomicAdd(&lvl[1], (unsigned long long)F.disc);
            atomicAdd(&lvl[2], (unsigned long long)F.deg);
        }
        if (!F.in_solo) B.base = reserve(tail, Span{all_ab & 0xFFFFu, all_ab >> 16, all_u});
    }
    __syncthreads();
    const uint32_t pab = before_ab + iab - ab, pu = before_u + iu - u;
    if (F.in_solo) {
        uint32_t at = (pab & 0xFFFFu) + pu;
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
            const uint32_t b = B.win_b[i], d = B.win_d[i], v = B.win_v[i];
            for (uint32_t k = 0; k < d; k += kPiece) B.solo[at++] = make_uint4(b + k, min(kPiece, d - k), v, 0u);
        }
    } else {
        Span at{B.base.a + (pab & 0xFFFFu), B.base.b + (pab >> 16), B.base.u + pu};
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) put_entry(a, at, B.win_v[i], B.win_b[i], B.win_d[i]);
    }
    return F;
}

// The out-edges of the pieces that a warp's lanes hold (p.y = 0: none): each
// unvisited end is claimed by its bit in `visited` and recorded, or, in a lazy
// level, only marked in fcur (the sweep drops what was visited).
template <bool PARENTS, bool LAZY>
__device__ __forceinline__ void push_batch(const BfsArgs& a, BlockState& B, const uint4& p, uint32_t level,
                                           bool precheck, uint32_t* fcur, const Tail& tail, uint32_t& disc,
                                           uint32_t& deg) {
    const uint32_t lane = threadIdx.x & 31;
    const DevGraph& g = a.g;
    const bool own_lists = g.out_ptrs != g.csr_ptrs;  // directed: degrees are counted over the in-lists
    const uint32_t incl = warp_incl(p.y);
    const uint32_t off = incl - p.y;
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    const uint32_t from = p.x - off;  // edge of flat index i in this piece: from + i
    for (uint32_t base = 0; base < total; base += 128) {
        uint32_t row[4], src[4], live = 0;
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t i = base + u * 32 + lane;
            uint32_t lo = 0;
#pragma unroll
            for (uint32_t st = 16; st > 0; st >>= 1) {
                const uint32_t o = __shfl_sync(0xFFFFFFFFu, off, lo + st);  // lo + st <= 31
                if (o <= i) lo += st;
            }
            const uint32_t f = __shfl_sync(0xFFFFFFFFu, from, lo);
            src[u] = PARENTS ? __shfl_sync(0xFFFFFFFFu, p.z, lo) : 0u;
            row[u] = i < total ? __ldg(&g.out_ids[f + i]) : kUnreached;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) live |= (row[u] < g.n ? 1u : 0u) << u;
        if (precheck) {
            uint32_t vis[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) vis[u] = (live >> u) & 1u ? __ldcg(&a.visited[row[u] >> 5]) : 0u;
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                if ((vis[u] >> (row[u] & 31)) & 1u) live &= ~(1u << u);
        }
        if (LAZY) {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                if ((live >> u) & 1u) atomicOr(&fcur[row[u] >> 5], 1u << (row[u] & 31));
            continue;
        }
        // the claims and the winners' list bounds in flight together
        uint32_t old[4], b[4], d[4], won = 0;
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            old[u] = (live >> u) & 1u ? atomicOr(&a.visited[row[u] >> 5], 1u << (row[u] & 31)) : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            b[u] = (live >> u) & 1u ? __ldg(&g.out_ptrs[row[u]]) : 0u;
            d[u] = (live >> u) & 1u ? __ldg(&g.out_ptrs[row[u] + 1]) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            if ((old[u] >> (row[u] & 31)) & 1u) continue;
            won |= 1u << u;
            d[u] -= b[u];
            a.levels[row[u]] = level;
            if (PARENTS) a.parents[row[u]] = src[u];
            ++disc;
            deg += own_lists ? __ldg(&g.csr_ptrs[row[u] + 1]) - __ldg(&g.csr_ptrs[row[u]]) : d[u];
        }
        emit(a, B, row, b, d, won, tail);
    }
}

// A push level over the frontier's entries in the global queues: batches of
// short lists, spread over the warps, then each warp's share of the long
// lists' pieces (its first piece's entry by a 32-way search).
template <bool PARENTS, bool LAZY>
__device__ __forceinline__ void push_level(const BfsArgs& a, BlockState& B, const Run& s, uint32_t warp,
                                           uint32_t nwarps, bool precheck, uint32_t* fcur, const Tail& tail,
                                           uint32_t& disc, uint32_t& deg) {
    const uint32_t lane = threadIdx.x & 31;
    {
        const uint4* q = a.pieces + s.from.a;
        const uint32_t T = s.size.a, per = min(32u, (T + nwarps - 1) / nwarps);
        for (uint64_t e0 = (uint64_t)warp * per; e0 < T; e0 += (uint64_t)nwarps * per) {
            uint4 p = make_uint4(0u, 0u, 0u, 0u);
            if (lane < per && e0 + lane < T) p = __ldcg(&q[e0 + lane]);
            push_batch<PARENTS, LAZY>(a, B, p, s.level, precheck, fcur, tail, disc, deg);
        }
    }
    const uint4* q = a.pieces + a.g.n + s.from.b;
    const uint32_t T = s.size.b, U = s.size.u;
    // with few pieces a warp takes one; shares start at the other end of the
    // warps, which have no short lists
    const uint32_t share = (U + nwarps - 1) / nwarps;
    uint32_t x = (nwarps - 1 - warp) * share;
    const uint32_t end = min(U, x + share);
    if (x >= end) return;
    uint32_t lo = 0, hi = T;
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32, idx = lo + lane * step;
        const bool ok = idx < hi && __ldcg(&q[idx].w) <= x;
        const uint32_t nlo = lo + (__popc(__ballot_sync(0xFFFFFFFFu, ok)) - 1) * step;
        hi = min(hi, nlo + step);
        lo = nlo;
    }
    {
        const bool ok = lo + lane < hi && __ldcg(&q[lo + lane].w) <= x;
        lo += __popc(__ballot_sync(0xFFFFFFFFu, ok)) - 1;
    }
    while (x < end) {
        // lane j takes piece x + j, while it lies in the share
        const uint32_t take = min(32u, end - x);
        // entries lo .. lo + 31 cover at least 32 pieces from x on
        const uint4 e = lo + lane < T ? __ldcg(&q[lo + lane]) : make_uint4(0u, 0u, 0u, 0xFFFFFFFFu);
        uint32_t own = 0;
#pragma unroll
        for (uint32_t st = 16; st > 0; st >>= 1) {
            const uint32_t o = __shfl_sync(0xFFFFFFFFu, e.w, own + st);
            if (o <= x + lane) own += st;
        }
        const uint32_t eb = __shfl_sync(0xFFFFFFFFu, e.x, own), ed = __shfl_sync(0xFFFFFFFFu, e.y, own);
        const uint32_t ev = __shfl_sync(0xFFFFFFFFu, e.z, own), ew = __shfl_sync(0xFFFFFFFFu, e.w, own);
        uint4 p = make_uint4(0u, 0u, 0u, 0u);
        if (lane < take) {
            const uint32_t k = (x + lane - ew) * kPiece;
            if (k < ed) p = make_uint4(eb + k, min(kPiece, ed - k), ev, 0u);
            else set_error(a.ctr, BLEST_ERR_DEVICE_INDEX);  // offsets and lengths disagree: cannot happen
        }
        push_batch<PARENTS, LAZY>(a, B, p, s.level, precheck, fcur, tail, disc, deg);
        x += take;
        lo += __shfl_sync(0xFFFFFFFFu, own, take - 1);
    }
}

// End of a level (or of a part of it): the grid barrier, then thread 0 reads
// the level's counters; the block's buffer is empty again. Adds the block's
// disc/deg first when `add`. Returns false when the run has an error recorded.
__device__ __forceinline__ bool level_end(const BfsArgs& a, BlockState& B, unsigned long long* lvl, bool add,
                                          uint32_t disc, uint32_t deg) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (add) {
        disc = __reduce_add_sync(0xFFFFFFFFu, disc);
        deg = __reduce_add_sync(0xFFFFFFFFu, deg);
        if (lane == 0) {
            B.tot_disc[w] = disc;
            B.tot_deg[w] = deg;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        reset_buffer(B);
        if (add) {
            uint32_t sd = 0, sg = 0;
            for (uint32_t i = 0; i < nw; ++i) {
                sd += B.tot_disc[i];
                sg += B.tot_deg[i];
            }
            if (sd) {
                atomicAdd(&lvl[1], (unsigned long long)sd);
                atomicAdd(&lvl[2], (unsigned long long)sg);
            }
        }
        const uint64_t v = barrier_arrive_wait(a.ctr);
#pragma unroll
        for (uint32_t i = 0; i < kSlotWords; ++i) B.val[i] = ld_relaxed64(&lvl[i]);
        B.ok = (v & kArriveError) == 0;
    }
    __syncthreads();
    return B.ok;
}

__device__ __forceinline__ void trace_level(const BfsArgs& a, uint32_t level, int dir, uint32_t nf, uint32_t units) {
    if (!a.trace || level > BLEST_TRACE_CAPACITY) return;
    blest_level_trace& t = a.trace[level - 1];
    t.start_ns = global_ns();
    t.level = level;
    t.direction = (uint32_t)dir;
    t.frontier = nf;
    t.work_units = units;
    t.sweep_ns = 0;
    t.longest_scan = 0;
}

// Take up to four of a lane's set bits (vertices first + bit) with their list
// bounds, for emit or append.
__device__ __forceinline__ uint32_t take_bits(const DevGraph& g, uint32_t first, uint32_t& bits, uint32_t (&v)[4],
                                              uint32_t (&b)[4], uint32_t (&d)[4]) {
    uint32_t won = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        v[k] = b[k] = d[k] = 0u;
        if (bits) {
            v[k] = first + __ffs(bits) - 1;
            bits &= bits - 1;
            won |= 1u << k;
            b[k] = __ldg(&g.out_ptrs[v[k]]);
            d[k] = __ldg(&g.out_ptrs[v[k] + 1]) - b[k];
        }
    }
    return won;
}

// The frontier's out-edges, from its entries in the global queues (all threads;
// every block gets the same).
__device__ __forceinline__ uint32_t frontier_edges(const BfsArgs& a, BlockState& B, const Run& s) {
    uint32_t sum = 0;
    for (uint32_t i = threadIdx.x; i < s.size.a + s.size.b; i += blockDim.x)
        sum += __ldcg(&a.pieces[i < s.size.a ? s.from.a + i : a.g.n + s.from.b + (i - s.size.a)].y);
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if ((threadIdx.x & 31) == 0) B.tot_d[threadIdx.x >> 5] = sum;
    __syncthreads();
    sum = 0;
    for (uint32_t i = 0; i < blockDim.x >> 5; ++i) sum += B.tot_d[i];
    return sum;
}

// Levels run by block 0 alone, from the queues on, until the frontier outgrows
// a block (its entries are then in the global queues again), is empty, or
// kSoloLevels are done.
template <bool PARENTS>
__device__ __forceinline__ void solo_levels(const BfsArgs& a, BlockState& B, Run& s, const Tail& tail) {
    RunCounters* c = a.ctr;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t T = s.size.a + s.size.u, done = 0;
    for (uint32_t i = threadIdx.x; i < s.size.a; i += blockDim.x) B.solo[i] = __ldcg(&a.pieces[s.from.a + i]);
    for (uint32_t i = threadIdx.x; i < s.size.b; i += blockDim.x) {
        const uint4 e = __ldcg(&a.pieces[a.g.n + s.from.b + i]);
        for (uint32_t k = 0; k < e.y; k += kPiece)
            B.solo[s.size.a + e.w + k / kPiece] = make_uint4(e.x + k, min(kPiece, e.y - k), e.z, 0u);
    }
    __syncthreads();
    for (bool inside = true; inside;) {
        const uint32_t nf = s.D1 - s.D2;
        if (threadIdx.x == 0 && done) trace_level(a, s.level, BLEST_DIR_PUSH, nf, T);
        ++s.push;
        s.nf_prev = nf;
        uint32_t disc = 0, deg = 0;
        const uint32_t per = min(32u, (T + nw - 1) / nw);
        for (uint32_t e0 = w * per; e0 < T; e0 += nw * per) {
            uint4 p = make_uint4(0u, 0u, 0u, 0u);
            if (lane < per && e0 + lane < T) p = B.solo[e0 + lane];
            push_batch<PARENTS, false>(a, B, p, s.level, false, nullptr, tail, disc, deg);
        }
        ++done;
        const Flushed F = flush(a, B, tail, nullptr, disc, deg, done < kSoloLevels);
        // flush's last barrier follows every read of the counters
        if (threadIdx.x == 0) reset_buffer(B);
        s.D2 = s.D1;
        s.G2 = s.G1;
        s.D1 += F.disc;
        s.G1 += F.deg;
        ++s.level;
        T = F.pieces;
        inside = F.in_solo && F.disc && s.level <= a.g.n + 1;
        __syncthreads();  // B.solo and the buffer's reset are visible
    }
    if (threadIdx.x == 0) {
        // what the last level left in the global queues; two records in turn:
        // a block may still be reading the last one (degree sums are below
        // 2^32, as nnz is)
        s.from.a += s.size.a;
        s.from.b += s.size.b;
        s.size = span_of(ld_relaxed64(tail.ca), ld_relaxed64(tail.cb));
        unsigned long long* r = c->solo[s.step % 2];
        r[0] = ((unsigned long long)s.nf_prev << 32) | s.level;
        r[1] = ((unsigned long long)s.from.a << 32) | s.size.a;
        r[2] = ((unsigned long long)s.from.b << 32) | s.size.b;
        r[3] = ((unsigned long long)s.push << 32) | s.size.u;
        r[4] = ((unsigned long long)s.D2 << 32) | s.D1;
        r[5] = (s.G2 << 32) | s.G1;
    }
}

// The frontier of a pull level: its bitmap, read through L1 (nobody writes it
// in this level), behind its summary in shared memory, which keeps most
// probes of a small frontier off L2.
struct Frontier {
    const uint32_t* bits;
    const uint32_t* summary;
    uint32_t shift;
    // Which of v[0..N) are in the frontier (entries may be kUnreached, which is
    // not). All N bitmap loads are in flight together.
    template <int N>
    __device__ __forceinline__ void test(const uint32_t (&v)[N], bool (&hit)[N]) const {
        bool may[N];
        uint32_t word[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const uint32_t sb = (v[j] >> 5) >> shift;
            may[j] = v[j] != kUnreached && (summary[v[j] != kUnreached ? sb >> 5 : 0u] >> (sb & 31)) & 1u;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) word[j] = may[j] ? bits[v[j] >> 5] : 0u;
#pragma unroll
        for (int j = 0; j < N; ++j) hit[j] = (word[j] >> (v[j] & 31)) & 1u;
    }
    // First of v[0..N) in the frontier, kUnreached if none.
    template <int N>
    __device__ __forceinline__ uint32_t first(const uint32_t (&v)[N]) const {
        bool hit[N];
        test(v, hit);
        uint32_t x = kUnreached;
#pragma unroll
        for (int j = N - 1; j >= 0; --j)
            if (hit[j]) x = v[j];
        return x;
    }
};

// Bottom-up level: a warp owns the words wi = warp + t * nwarps and takes them
// 16 at a time, two lanes per word (a half each): the unvisited vertices with
// in-neighbours go into one list in shared memory that the lanes take 32 at a
// time, so no lane idles on a visited vertex. (Finding a lane's vertex in the
// words by shuffles and __fns instead cost more issue slots than the scan.)
//
// First every vertex tries its first four in-neighbours (those of highest
// degree, DevGraph::heads: one aligned 16-byte load with the degree in its
// spare bits, so no list bound is read; two vertices a lane, the next two's
// loads in flight meanwhile). Most are settled by that: found, or their list
// is done. The others are set aside, and lanes then take
// them one by one, eight neighbours at a time, a lane that finishes taking the
// next, so that no lane waits for the warp's longest scan in every round.
// Lists with more than kPullWarpScan edges left are scanned by the whole warp,
// very long ones by all warps after the level (heavy queue).
//
// Found vertices set their bit in the warp's word slots in shared memory;
// after the chunk lane 2j writes word j's visited and frontier words, and with
// `queue_too` they are also gathered in B.pulled for the queue `tail` (straight
// to it once that is full).
template <bool PARENTS>
__device__ __forceinline__ void pull_level(const BfsArgs& a, BlockState& B, uint32_t level, uint32_t warp,
                                           uint32_t nwarps, uint32_t* fcur, uint32_t* fsum, unsigned long long* lvl,
                                           const Frontier& front, bool queue_too, const Tail& tail, uint32_t& disc,
                                           uint32_t& deg) {
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    const DevGraph& g = a.g;
    const uint32_t W = (g.n + 31) / 32;
    const uint32_t tailMask = (g.n & 31) ? ((1u << (g.n & 31)) - 1) : 0xFFFFFFFFu;
    uint32_t longest = 0;
    const uint32_t w = threadIdx.x >> 5;
    uint32_t* const found_slots = B.found[w];
    uint16_t* const items = B.items[w];  // word slot << 5 | bit
    uint16_t* const later = B.later[w];
    // word `lane / 2` of the chunk at t0: visited word and the vertices to try
    auto words = [&](uint32_t t0, uint32_t& vis) -> uint32_t {
        const uint32_t wj = warp + (t0 + (lane >> 1)) * nwarps;
        vis = 0xFFFFFFFFu;
        if (wj >= W) return 0u;
        vis = __ldcg(&a.visited[wj]);
        const uint32_t hj = g.has_in ? __ldg(&g.has_in[wj]) : 0xFFFFFFFFu;
        return ~vis & hj & (wj == W - 1 ? tailMask : 0xFFFFFFFFu);
    };
    uint32_t nvis, nunv = words(0, nvis);
    for (uint32_t t0 = 0; warp + t0 * nwarps < W; t0 += kPullWords) {
        const uint32_t vis = nvis, unv = nunv;
        if (warp + (t0 + kPullWords) * nwarps < W) nunv = words(t0 + kPullWords, nvis);
        uint32_t half = unv & (lane & 1 ? 0xFFFF0000u : 0xFFFFu);
        uint32_t at = warp_incl(__popc(half));
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, at, 31);
        if (total == 0) continue;
        at -= __popc(half);
        if (lane < kPullWords) found_slots[lane] = 0u;
        for (; half; half &= half - 1) items[at++] = (uint16_t)((lane >> 1) << 5 | (__ffs(half) - 1));
        __syncwarp();
        auto vertex = [&](uint32_t code) { return (warp + (t0 + (code >> 5)) * nwarps) * 32 + (code & 31u); };
        auto record = [&](uint32_t code, uint32_t u, uint32_t parent, uint32_t d) {
            a.levels[u] = level;
            if (PARENTS) a.parents[u] = parent;
            atomicOr(&found_slots[code >> 5], 1u << (code & 31u));
            ++disc;
            deg += d;
        };
        // the set-aside items later[0..cnt): lanes take them until none is left
        auto drain = [&](uint32_t cnt) {
            __syncwarp();
            uint32_t code = 0, u = 0, p = 0, pe = 0, d = 0, next = 0;
            bool busy = false;
            for (;;) {
                const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy);
                if (idle && next < cnt) {
                    const uint32_t k = next + __popc(idle & below);
                    if (!busy && k < cnt) {
                        code = later[k];
                        u = vertex(code);
                        p = __ldg(&g.csr_ptrs[u]);
                        pe = __ldg(&g.csr_ptrs[u + 1]);
                        d = pe - p;
                        p += 4;
                        busy = true;
                    }
                    next = min(cnt, next + __popc(idle));
                }
                if (!__any_sync(0xFFFFFFFFu, busy)) break;
                if (busy) {
                    // two aligned quads (the lists are padded to whole quads)
                    const uint32_t q = p & ~3u;
                    const uint4 x = __ldg(reinterpret_cast<const uint4*>(g.csr_ids + q));
                    const uint4 y = q + 4 < pe ? __ldg(reinterpret_cast<const uint4*>(g.csr_ids + q + 4))
                                               : make_uint4(0u, 0u, 0u, 0u);
                    uint32_t v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        if (q + j < p || q + j >= pe) v[j] = kUnreached;
                    const uint32_t parent = front.first(v);
                    p = q + 8;
                    if (parent != kUnreached) record(code, u, parent, d);
                    busy = parent == kUnreached && p < pe;
                }
            }
            __syncwarp();
        };
        uint32_t ncode[kPullItems], waiting = 0;
        uint4 nhead[kPullItems];
        auto fetch = [&](uint32_t base) {
#pragma unroll
            for (uint32_t k = 0; k < kPullItems; ++k) {
                const uint32_t idx = base + 32 * k + lane;
                ncode[k] = 0;
                nhead[k] = make_uint4(0u, 0u, 0u, 0u);  // an empty list
                if (idx < total) {
                    ncode[k] = items[idx];
                    nhead[k] = __ldg(&g.heads[vertex(ncode[k])]);
                }
            }
        };
        fetch(0);
        for (uint32_t base = 0; base < total; base += 32 * kPullItems) {
            uint32_t code[kPullItems], d[kPullItems], parent[kPullItems], v[kPullItems][4];
#pragma unroll
            for (uint32_t k = 0; k < kPullItems; ++k) {
                code[k] = ncode[k];
                const uint4 h = nhead[k];
                d[k] = head_degree(h);
                const uint32_t x[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) v[k][j] = d[k] > j ? x[j] & kHeadId : kUnreached;
            }
            if (base + 32 * kPullItems < total) fetch(base + 32 * kPullItems);
            // Two neighbours, then two more: 32 lanes' probes are 32 L1 lines
            // (one a clock), so probes past the first hit cost more than the
            // round trip that testing all four at once would save.
            {
                uint32_t x[2 * kPullItems];
                bool hit[2 * kPullItems];
#pragma unroll
                for (uint32_t k = 0; k < kPullItems; ++k) {
                    x[2 * k] = v[k][0];
                    x[2 * k + 1] = v[k][1];
                }
                front.test(x, hit);
                bool more = false;
#pragma unroll
                for (uint32_t k = 0; k < kPullItems; ++k) {
                    parent[k] = hit[2 * k] ? x[2 * k] : (hit[2 * k + 1] ? x[2 * k + 1] : kUnreached);
                    const bool on = parent[k] == kUnreached && d[k] > 2;
                    more |= on;
                    x[2 * k] = on ? v[k][2] : kUnreached;
                    x[2 * k + 1] = on ? v[k][3] : kUnreached;
                }
                if (more) {
                    front.test(x, hit);
#pragma unroll
                    for (uint32_t k = 0; k < kPullItems; ++k) {
                        if (hit[2 * k + 1]) parent[k] = x[2 * k + 1];
                        if (hit[2 * k]) parent[k] = x[2 * k];
                    }
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kPullItems; ++k) {
                const uint32_t u = vertex(code[k]);
                uint32_t p = 0, pe = 0;
                const bool is_long = d[k] > kPullWarpScan + 4;
                if (d[k] >= kHeadDegreeMax || (is_long && parent[k] == kUnreached)) {
                    p = __ldg(&g.csr_ptrs[u]);
                    pe = __ldg(&g.csr_ptrs[u + 1]);
                    d[k] = pe - p;
                    p += 4;
                    if (parent[k] != kUnreached) p = pe;  // settled
                }
                // Very long lists go to the heavy queue (all warps split them
                // after the level barrier).
                if (p < pe && pe - p > a.heavy_min) {
                    const uint32_t chunks = (pe - p + kHeavyChunk - 1) / kHeavyChunk;
                    const uint64_t hs = atomicAdd(&lvl[3], (unsigned long long)((1ull << kQShift) | chunks));
                    const uint32_t idx = (uint32_t)(hs >> kQShift);
                    if (idx < a.heavy_cap) {
                        a.heavy[idx] = make_uint4(u, p, pe, (uint32_t)(hs & kQUnitMask));
                        p = pe;  // handed over
                    } else {
                        set_error(a.ctr, BLEST_ERR_DEVICE_INDEX);  // capacity is sized so this cannot happen
                    }
                }
                // Long lists: the whole warp scans them, one vertex at a time.
                for (uint32_t rest = __ballot_sync(0xFFFFFFFFu, p < pe); rest; rest &= rest - 1) {
                    const uint32_t ln = __ffs(rest) - 1;
                    const uint32_t q0 = __shfl_sync(0xFFFFFFFFu, p, ln);
                    const uint32_t q1 = __shfl_sync(0xFFFFFFFFu, pe, ln);
                    longest = max(longest, q1 - q0);
                    uint32_t hitv = kUnreached;
                    for (uint32_t qb = q0; qb < q1 && hitv == kUnreached; qb += 128) {
                        uint32_t x[4];
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j) {
                            const uint32_t idx = qb + 32 * j + lane;
                            x[j] = idx < q1 ? __ldg(&g.csr_ids[idx]) : kUnreached;
                        }
                        const uint32_t mine = front.first(x);
                        const uint32_t hb = __ballot_sync(0xFFFFFFFFu, mine != kUnreached);
                        if (hb) hitv = __shfl_sync(0xFFFFFFFFu, mine, __ffs(hb) - 1);
                    }
                    if (lane == ln) parent[k] = hitv;
                }
                if (parent[k] != kUnreached) record(code[k], u, parent[k], d[k]);
                const bool aside = parent[k] == kUnreached && d[k] > 4 && !is_long;
                const uint32_t am = __ballot_sync(0xFFFFFFFFu, aside);
                if (aside) later[waiting + __popc(am & below)] = (uint16_t)code[k];
                waiting += __popc(am);
            }
            if (waiting >= 32) {
                drain(waiting);
                waiting = 0;
            }
        }
        drain(waiting);
        // write back the chunk's words (lanes 2j: word j)
        const uint32_t nb = lane & 1 ? 0u : found_slots[lane >> 1];
        __syncwarp();
        if (nb) {
            const uint32_t wj = warp + (t0 + (lane >> 1)) * nwarps;
            fcur[wj] = nb;
            a.visited[wj] = vis | nb;
            mark_summary(a, fsum, wj);
        }
        if (queue_too && __any_sync(0xFFFFFFFFu, nb)) {
            const uint32_t first = (warp + (t0 + (lane >> 1)) * nwarps) * 32;
            const uint32_t end = warp_incl(__popc(nb));
            uint32_t at = 0, bits = nb;
            if (lane == 31) at = atomicAdd(&B.win_cnt, end);
            at = __shfl_sync(0xFFFFFFFFu, at, 31);
            if (at + __shfl_sync(0xFFFFFFFFu, end, 31) <= kWinners) {
                for (at += end - __popc(nb); bits; bits &= bits - 1) B.pulled[at++] = first + __ffs(bits) - 1;
            } else {
                if (lane == 0) atomicMin(&B.win_end, at);
                while (__any_sync(0xFFFFFFFFu, bits)) {
                    uint32_t v[4], b[4], d[4];
                    const uint32_t won = take_bits(g, first, bits, v, b, d);
                    append(a, v, b, d, won, tail);
                }
            }
        }
    }
    if (a.trace && lane == 0 && longest && level <= BLEST_TRACE_CAPACITY)
        atomicMax((unsigned long long*)&a.trace[level - 1].longest_scan, (unsigned long long)longest);
}

// The heavy lists of a pull level: every warp takes an equal share of their
// pieces.
template <bool PARENTS>
__device__ __forceinline__ void heavy_level(const BfsArgs& a, uint64_t hq, uint32_t level, uint32_t warp,
                                            uint32_t nwarps, uint32_t* fcur, uint32_t* fsum, const Frontier& front,
                                            uint32_t& disc, uint32_t& deg) {
    const uint32_t lane = threadIdx.x & 31;
    const DevGraph& g = a.g;
    const uint32_t hitems = min((uint32_t)(hq >> kQShift), a.heavy_cap);
    const uint32_t hchunks = (uint32_t)(hq & kQUnitMask);
    const uint32_t hk = (hchunks + nwarps - 1) / nwarps;
    for (uint32_t ch = warp * hk; hitems && ch < min(hchunks, warp * hk + hk); ++ch) {
        // owner: largest item with chunk offset <= ch
        uint32_t lo = 0, hi = hitems;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (__ldcg(&a.heavy[mid].w) <= ch) lo = mid;
            else hi = mid;
        }
        const uint4 it = __ldcg(&a.heavy[lo]);
        const uint32_t hu = it.x, w = hu >> 5, b = 1u << (hu & 31);
        const uint32_t q0 = it.y + (ch - it.w) * kHeavyChunk;
        const uint32_t q1 = min(it.z, q0 + kHeavyChunk);
        uint32_t hitv = kUnreached;
        for (uint32_t base = q0; base < q1 && hitv == kUnreached; base += 32) {
            // another piece found it (lanes need not read the same while
            // that happens: the warp leaves as one)
            if (__any_sync(0xFFFFFFFFu, __ldcg(&a.visited[w]) & b)) break;
            const uint32_t idx = base + lane;
            const uint32_t v[1] = {idx < q1 ? __ldg(&g.csr_ids[idx]) : kUnreached};
            const uint32_t hb = __ballot_sync(0xFFFFFFFFu, front.first(v) != kUnreached);
            if (hb) hitv = __shfl_sync(0xFFFFFFFFu, v[0], __ffs(hb) - 1);
        }
        if (hitv != kUnreached && lane == 0 && !(atomicOr(&a.visited[w], b) & b)) {
            a.levels[hu] = level;
            if (PARENTS) a.parents[hu] = hitv;
            ++disc;
            deg += __ldg(&g.csr_ptrs[hu + 1]) - __ldg(&g.csr_ptrs[hu]);
            atomicOr(&fcur[w], b);
            mark_summary(a, fsum, w);
        }
    }
}

template <bool PARENTS>
__device__ __forceinline__ void lists_run(const BfsArgs& a) {
    extern __shared__ uint32_t s_sum[];
    __shared__ BlockState B;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nth = gridDim.x * blockDim.x;
    // warps are numbered across the blocks, so that a few busy ones lie on
    // different SMs
    const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t nwarps = nth >> 5;
    const DevGraph& g = a.g;
    const uint32_t n = g.n;
    RunCounters* c = a.ctr;

    // ---- level 0: outputs and bitmaps reset, the source queued (the counters
    // were zeroed when they were made, or by the last run's last block)
    Run s{};
    {
        const uint32_t src = a.src;
        for (uint32_t v = tid; v < n; v += nth) {
            a.levels[v] = v == src ? 0u : kUnreached;
            if (PARENTS) a.parents[v] = v == src ? src : kUnreached;
        }
        const uint32_t sw = src >> 5, sb = 1u << (src & 31);
        for (uint32_t i = tid; i < a.words; i += nth) {
            a.visited[i] = i == sw ? sb : 0u;
            a.frontier0[i] = 0u;
            a.frontier1[i] = 0u;
            a.frontier2[i] = 0u;
        }
        for (uint32_t i = tid; i < a.sum_words; i += nth) {
            a.summary0[i] = 0u;
            a.summary1[i] = 0u;
            a.summary2[i] = 0u;
        }
        const uint32_t b = __ldg(&g.out_ptrs[src]), d = __ldg(&g.out_ptrs[src + 1]) - b;
        s.level = 1;
        if (tid == 0) {
            Span at{0u, 0u, 0u};
            put_entry(a, at, src, b, d);
        }
        s.size = d > kPiece ? Span{0u, 1u, pieces_of(d)} : Span{d ? 1u : 0u, 0u, 0u};
        s.D1 = 1;
        s.G1 = __ldg(&g.csr_ptrs[src + 1]) - __ldg(&g.csr_ptrs[src]);
        if (threadIdx.x == 0) reset_buffer(B);
    }
    if (!grid_barrier(c)) return;

    int dir = a.direction == BLEST_DIR_PULL ? BLEST_DIR_PULL : BLEST_DIR_PUSH;
    bool queued = true, mapped = false;  // the frontier is in the queue, in bitmap `gen` (or both)
    uint32_t gen = 0;    // bitmaps made; bitmap gen + 1 is zero (its clearing is part of making gen)
    const uint32_t W = (n + 31) / 32;
    auto clear_next = [&]() {
        uint32_t* f = bitmap_of(a, gen + 1);
        uint32_t* m = summary_of(a, gen + 1);
        for (uint32_t i = tid; i < a.words; i += nth) f[i] = 0u;
        for (uint32_t i = tid; i < a.sum_words; i += nth) m[i] = 0u;
    };

    for (;;) {
        const uint32_t level = s.level;
        const uint32_t nf = s.D1 - s.D2;  // discovered at level - 1
        const uint64_t mf = s.G1 - s.G2;  // their edges
        if (nf == 0 || level > n + 1) {
            if (tid == 0) {
                c->discovered = s.D1;
                c->degree = s.G1;
                c->push_levels = s.push;
                c->pull_levels = s.pull;
                if (nf == 0) {
                    c->levels = level - 1;  // max level + 1
                    trace_level(a, level, 0, 0, 0);
                }
            }
            if (nf != 0) set_error(c, BLEST_ERR_LEVEL_CAP);
            break;
        }
        if (a.direction == BLEST_DIR_AUTO) {
            // Beamer's switch in edge/vertex units: to pull when the new
            // frontier's edges m_f exceed the unvisited edges m_u / alpha and
            // the frontier grows; back to push when it has fewer than n / beta
            // vertices. Going to pull also needs m_f above 8 edges per
            // bitmap word, going back below that: a pull level visits every
            // word, so a grid's growing wavefront (4.6 edges a word at its
            // widest, which passes Beamer's test) is better off pushing.
            const double bar = 8.0 * (double)W;
            if (dir == BLEST_DIR_PUSH) {
                if ((double)mf * a.alpha > (double)(g.degree_total - s.G1) && nf > s.nf_prev && (double)mf > bar)
                    dir = BLEST_DIR_PULL;
            } else if ((double)nf * a.beta < (double)n && (double)mf < bar) {
                dir = BLEST_DIR_PUSH;
            }
        }
        if (tid == 0) trace_level(a, level, dir, nf, queued ? s.size.a + s.size.u : nf);
        unsigned long long* lvl = c->lvl[s.step % 3];
        // the next step's counters (their slot was last read two steps back)
        if (tid < kSlotWords) c->lvl[(s.step + 1) % 3][tid] = 0;
        // the queues end where the frontier's entries end
        const Span next{s.from.a + s.size.a, s.from.b + s.size.b, 0u};
        uint32_t disc = 0, deg = 0;

        // ---- the frontier in the form this direction reads
        if (dir == BLEST_DIR_PUSH && !queued) {
            const Tail tail{next, &lvl[3], &lvl[5]};
            const uint32_t* f = bitmap_of(a, gen);
            for (uint32_t base = warp * 32; base < W; base += nwarps * 32) {
                uint32_t bits = base + lane < W ? __ldcg(&f[base + lane]) : 0u;
                while (__any_sync(0xFFFFFFFFu, bits)) {
                    uint32_t v[4], b[4], d[4];
                    const uint32_t won = take_bits(g, (base + lane) * 32, bits, v, b, d);
                    emit(a, B, v, b, d, won, tail);
                }
            }
            flush(a, B, tail, nullptr, 0, 0, false);
            if (!level_end(a, B, lvl, false, 0, 0)) return;
            s.from = next;
            s.size = span_of(B.val[3], B.val[5]);
            queued = true;
        } else if (dir == BLEST_DIR_PULL && !mapped) {
            ++gen;
            clear_next();
            uint32_t* f = bitmap_of(a, gen);
            uint32_t* m = summary_of(a, gen);
            // a vertex without out-edges has no entry, and is nobody's in-neighbour
            for (uint32_t e = tid; e < s.size.a + s.size.b; e += nth) {
                const uint32_t at = e < s.size.a ? s.from.a + e : n + s.from.b + (e - s.size.a);
                const uint32_t v = __ldcg(&a.pieces[at].z);
                atomicOr(&f[v >> 5], 1u << (v & 31));
                // many vertices share a summary word: look before the atomic
                const uint32_t sb = (v >> 5) >> a.sum_shift;
                if (!((__ldcg(&m[sb >> 5]) >> (sb & 31)) & 1u)) atomicOr(&m[sb >> 5], 1u << (sb & 31));
            }
            if (!grid_barrier(c)) return;
            mapped = true;
        }

        if (dir == BLEST_DIR_PUSH) {
            const Span end{s.from.a + s.size.a, s.from.b + s.size.b, 0u};
            const Tail tail{end, &lvl[0], &lvl[4]};
            // mf counts in-edges, of which a directed graph's frontier with 65 k
            // out-edges may have few: its out-edges are summed first, as flush
            // does (5 levels of 500 x 128 out-edges: 154 -> 80 us; a sum takes
            // 1 us).
            bool alone = s.size.a + s.size.u <= kSoloPieces && mf <= kSoloEdges;
            if (alone && g.out_ptrs != g.csr_ptrs) alone = frontier_edges(a, B, s) <= kSoloEdges;
            if (alone) {
                if (blockIdx.x == 0) solo_levels<PARENTS>(a, B, s, tail);
                if (!level_end(a, B, c->solo[s.step % 2], false, 0, 0)) return;
                s.level = (uint32_t)B.val[0];
                s.nf_prev = (uint32_t)(B.val[0] >> 32);
                s.from = Span{(uint32_t)(B.val[1] >> 32), (uint32_t)(B.val[2] >> 32), 0u};
                s.size = Span{(uint32_t)B.val[1], (uint32_t)B.val[2], (uint32_t)B.val[3]};
                s.push = (uint32_t)(B.val[3] >> 32);
                s.D1 = (uint32_t)B.val[4];
                s.D2 = (uint32_t)(B.val[4] >> 32);
                s.G1 = (uint32_t)B.val[5];
                s.G2 = B.val[5] >> 32;
                mapped = false;
                ++s.step;
                continue;
            }
            // A large level looks before it claims, since most ends are visited;
            // below that the look is one more round trip (from 16 k edges on
            // instead, the grid of 2901 x 2801 took 1126 us against 1116).
            const bool precheck = mf > 131072;
            // Lazy level: when the frontier's edges exceed n / 4 the level
            // discovers a large part of the graph; then an edge only marks its
            // end (an atomic nobody waits for) and a word sweep keeps the
            // unvisited ones and writes their levels, coalesced. While under
            // an eighth of the graph is visited the look first would filter
            // little.
            if (!PARENTS && mf > (uint64_t)(n / 4)) {
                ++gen;
                clear_next();
                uint32_t* fcur = bitmap_of(a, gen);
                uint32_t* fsum = summary_of(a, gen);
                push_level<PARENTS, true>(a, B, s, warp, nwarps, s.D1 > n / 8, fcur, tail, disc, deg);
                if (!grid_barrier(c)) return;
                if (a.trace && tid == 0 && level <= BLEST_TRACE_CAPACITY) a.trace[level - 1].sweep_ns = global_ns();
                for (uint32_t base = warp * 32; base < W; base += nwarps * 32) {
                    const uint32_t wi = base + lane;
                    uint32_t nw = 0;
                    if (wi < W) {
                        const uint32_t cand = __ldcg(&fcur[wi]);
                        if (cand) {
                            const uint32_t vis = __ldcg(&a.visited[wi]);
                            nw = cand & ~vis;
                            fcur[wi] = nw;
                            if (nw) {
                                a.visited[wi] = vis | nw;
                                mark_summary(a, fsum, wi);
                            }
                        }
                    }
                    // 8 words at a time, a lane per vertex: all their degree
                    // loads are issued before any is added
                    const uint32_t words = __ballot_sync(0xFFFFFFFFu, nw != 0);
                    for (uint32_t j0 = 0; j0 < 32; j0 += 8) {
                        if (!((words >> j0) & 0xFFu)) continue;
                        uint32_t d0[8], d1[8], vb = 0;
#pragma unroll
                        for (uint32_t k = 0; k < 8; ++k) {
                            const uint32_t bits = __shfl_sync(0xFFFFFFFFu, nw, j0 + k);
                            const uint32_t v = (base + j0 + k) * 32 + lane;
                            d0[k] = d1[k] = 0u;
                            if ((bits >> lane) & 1u) {
                                vb |= 1u << k;
                                d0[k] = __ldg(&g.csr_ptrs[v]);
                                d1[k] = __ldg(&g.csr_ptrs[v + 1]);
                            }
                        }
#pragma unroll
                        for (uint32_t k = 0; k < 8; ++k) {
                            if ((vb >> k) & 1u) {
                                a.levels[(base + j0 + k) * 32 + lane] = level;
                                ++disc;
                                deg += d1[k] - d0[k];
                            }
                        }
                    }
                }
                queued = false;
                mapped = true;
                ++s.push;
                if (!level_end(a, B, lvl, true, disc, deg)) return;
                s.from = end;  // nothing was queued
                s.size = Span{0u, 0u, 0u};
            } else {
                push_level<PARENTS, false>(a, B, s, warp, nwarps, precheck, nullptr, tail, disc, deg);
                flush(a, B, tail, lvl, disc, deg, false);
                ++s.push;
                if (!level_end(a, B, lvl, false, 0, 0)) return;
                s.from = end;
                s.size = span_of(B.val[0], B.val[4]);
                mapped = false;
            }
        } else {
            const Frontier front{bitmap_of(a, gen), s_sum, a.sum_shift};
            const uint32_t* sprev = summary_of(a, gen);
            for (uint32_t i = threadIdx.x; i < a.sum_words; i += blockDim.x) s_sum[i] = __ldcg(&sprev[i]);
            ++gen;
            clear_next();
            uint32_t* fcur = bitmap_of(a, gen);
            uint32_t* fsum = summary_of(a, gen);
            __syncthreads();
            // With next to no edges left unvisited the level finds little and
            // the next one is a push: what this one finds is queued at once
            // (else a pass over the bitmap and a barrier later, 6 us).
            const bool queue_too = a.direction == BLEST_DIR_AUTO && g.degree_total - s.G1 < 8ull * W;
            const Tail tail{next, &lvl[0], &lvl[4]};
            pull_level<PARENTS>(a, B, level, warp, nwarps, fcur, fsum, lvl, front, queue_too, tail, disc, deg);
            if (queue_too) {
                __syncthreads();
                for (uint32_t i = threadIdx.x; i < min(B.win_cnt, B.win_end); i += blockDim.x) {
                    const uint32_t v = B.pulled[i], b = __ldg(&g.out_ptrs[v]);
                    B.win_v[i] = v;
                    B.win_b[i] = b;
                    B.win_d[i] = __ldg(&g.out_ptrs[v + 1]) - b;
                }
                flush(a, B, tail, nullptr, 0, 0, false);
            }
            ++s.pull;
            if (!level_end(a, B, lvl, true, disc, deg)) return;
            if (B.val[3]) {
                const uint64_t hq = B.val[3];
                disc = deg = 0;
                heavy_level<PARENTS>(a, hq, level, warp, nwarps, fcur, fsum, front, disc, deg);
                if (!level_end(a, B, lvl, true, disc, deg)) return;
            }
            // (the heavy lists' finds are in the bitmap only: the queued ones
            // are then dropped and their place used again)
            queued = queue_too && !B.val[3];
            mapped = true;
            s.from = next;
            s.size = queued ? span_of(B.val[0], B.val[4]) : Span{0u, 0u, 0u};
        }
        s.nf_prev = nf;
        s.D2 = s.D1;
        s.G2 = s.G1;
        s.D1 += (uint32_t)B.val[1];
        s.G1 += B.val[2];
        ++s.level;
        ++s.step;
    }
}

template <bool PARENTS>
__global__ void __launch_bounds__(512, 2) bfs_lists_kernel(BfsArgs a) {
    RunCounters* const c = a.ctr;
    if (blockIdx.x == 0 && threadIdx.x == 0) c->start_ns = global_ns();
    lists_run<PARENTS>(a);
    // The last block to leave writes the record and zeroes the counters, so
    // that the next run needs no memset before it and a host that sees the
    // record knows that nothing of this run is still to come.
    if (!last_block_out(c)) return;
    if (a.record) fill_record(a.record, a, ld_relaxed64(&c->start_ns));
    zero_counters(c);
    if (a.record) publish_record(a.record, a.seq);
}

}  // namespace
}  // namespace dev

namespace {

template <bool PARENTS>
void launch_lists(const blest_graph* g, const dev::BfsArgs& args, int blocks_per_sm, int threads, uint32_t grid_cap,
                  cudaStream_t s) {
    auto kern = dev::bfs_lists_kernel<PARENTS>;
    const size_t smem = 4ull * args.sum_words;
    // Per (device, block size, shared memory): the attribute is set once
    // (always the maximum, so concurrent calls for graphs of different sizes
    // agree) and the occupancy is asked once; both are fixed per device.
    static std::mutex mu;
    static std::map<std::tuple<int, int, size_t>, int> occupancy;
    int maxBlocks = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        const auto key = std::make_tuple(g->device, threads, smem);
        const auto it = occupancy.find(key);
        if (it != occupancy.end()) {
            maxBlocks = it->second;
        } else {
            BLEST_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)kSummaryMaxBytes));
            BLEST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxBlocks, kern, threads, smem));
            occupancy[key] = maxBlocks;
        }
    }
    if (maxBlocks < 1) throw Error(BLEST_ERR_CUDA, "BFS kernel cannot be resident with this block size");
    const int want = bfs_lists_blocks(g->d.n, g->d.nnz, g->sm_count, maxBlocks, blocks_per_sm, threads);
    const int grid = std::min(want, cooperative_grid(maxBlocks, g->sm_count, grid_cap));
    void* kargs[] = {(void*)&args};
    BLEST_CUDA(cudaLaunchCooperativeKernel((void*)kern, grid, threads, kargs, smem, s));
}

}  // namespace

void launch_bfs_lists(const blest_graph* g, const dev::BfsArgs& args, int blocks_per_sm, int threads,
                      uint32_t grid_cap, cudaStream_t s) {
    if (args.parents) launch_lists<true>(g, args, blocks_per_sm, threads, grid_cap, s);
    else launch_lists<false>(g, args, blocks_per_sm, threads, grid_cap, s);
}

}  // namespace blest
