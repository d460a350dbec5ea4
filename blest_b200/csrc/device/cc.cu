// Connected components, as ONE persistent cooperative kernel: union-find over
// the pull lists when the graph is symmetric (cc_union_kernel), min-label
// propagation over BVSS tiles otherwise (cc_persistent_kernel). Replaces the CC kernels of
// CC/BVSSCCKernel.cuh (:33-1045) and BVSSCCKernel::hostCode (:1067-1311).
//
// Same fixpoint as the reference in both. Label propagation: labels start as the vertex id; a slice
// (row, mask byte) whose columns include active vertices lowers the row's
// label to the minimum label of those active columns (CC/BVSSCCKernel.cuh:
// 106-220); a row whose label dropped is active in the next iteration; the
// run ends when an iteration lowers nothing. labels[v] is then the smallest
// id with a path to v. Scheduling follows the BFS kernel: active rsets are
// queued with running tile offsets (even split of tiles over warps), the
// active bitmaps are triple-buffered and cleared through the queue two
// iterations back, and each iteration ends in one bounded grid barrier
// (the reference sweeps all n/32 words and syncs three times). A warp
// works on 32 tiles of ONE rset at a time, so the rset's 8 column labels
// are read once (8 lanes, one sector) and shared by shuffle.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "../host/common.hpp"
#include "common.cuh"
#include "runtime.hpp"

namespace blest {
namespace dev {

struct CcArgs {
    DevGraph g;
    uint32_t* labels;
    uint32_t* active0;
    uint32_t* active1;
    uint32_t* active2;
    uint32_t* q_rset;  // 4 regions of qreg entries
    uint32_t* q_off;
    uint32_t qreg;
    RunCounters* ctr;
    unsigned long long* qctr;  // 4 packed counters (entries<<36 | tiles), in the workspace
    uint32_t words;
};

__device__ __forceinline__ uint32_t* active_buf(const CcArgs& a, uint32_t it) {
    const uint32_t m = it % 3;
    return m == 0 ? a.active0 : (m == 1 ? a.active1 : a.active2);
}

// Queue units of an rset: its 32-tile chunks.
__device__ __forceinline__ uint32_t tiles_of(const DevGraph& g, uint32_t r) {
    return (__ldg(&g.rset_tile[r + 1]) - __ldg(&g.rset_tile[r]) + 31) / 32;
}

struct CcEnqueue {
    uint32_t rset[4];
    uint32_t cnt;
    uint32_t units;
};

__device__ __forceinline__ void cc_flush(const CcArgs& a, uint32_t slot, CcEnqueue& q) {
    const uint32_t lane = threadIdx.x & 31;
    if (!__any_sync(0xFFFFFFFFu, q.cnt != 0)) return;
    const uint64_t mine = ((uint64_t)q.cnt << kQShift) | q.units;
    const uint64_t incl = warp_inclusive_scan64(mine);
    uint64_t base = 0;
    if (lane == 31) base = atomicAdd(&a.qctr[slot], (unsigned long long)incl);
    base = __shfl_sync(0xFFFFFFFFu, base, 31);
    const uint64_t excl = base + incl - mine;
    uint32_t e = (uint32_t)(excl >> kQShift);
    uint32_t u = (uint32_t)(excl & kQUnitMask);
    uint32_t* qr = a.q_rset + (size_t)slot * a.qreg;
    uint32_t* qo = a.q_off + (size_t)slot * a.qreg;
    for (uint32_t i = 0; i < q.cnt; ++i) {
        qr[e] = q.rset[i];
        qo[e] = u;
        ++e;
        u += tiles_of(a.g, q.rset[i]);
    }
    q.cnt = 0;
    q.units = 0;
}

// Labels = identity, all valid vertices active, every rset with tiles queued
// in slot 0 (iteration 0's output).
__global__ void cc_init_kernel(CcArgs a) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nth = gridDim.x * blockDim.x;
    const uint32_t n = a.g.n;
    for (uint32_t v = tid; v < n; v += nth) a.labels[v] = v;
    const uint32_t W = (n + 31) / 32;
    const uint32_t tail = (n & 31) ? ((1u << (n & 31)) - 1) : 0xFFFFFFFFu;
    for (uint32_t i = tid; i < a.words; i += nth) {
        a.active0[i] = i < W ? (i == W - 1 ? tail : 0xFFFFFFFFu) : 0u;
        a.active1[i] = 0u;
        a.active2[i] = 0u;
    }
}

__global__ void cc_seed_queue_kernel(CcArgs a) {
    // Whole warps (grid is a multiple of 32 threads); one atomic per warp.
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nth = gridDim.x * blockDim.x;
    const uint32_t R = a.g.no_real;
    for (uint32_t base = tid & ~31u; base < R; base += nth) {
        const uint32_t r = base + (threadIdx.x & 31);
        CcEnqueue q;
        q.cnt = 0;
        q.units = 0;
        if (r < R) {
            const uint32_t t = tiles_of(a.g, r);
            if (t) {
                q.rset[0] = r;
                q.cnt = 1;
                q.units = t;
            }
        }
        cc_flush(a, 0, q);
    }
}

__device__ __forceinline__ uint32_t cc_find_owner(const uint32_t* q_off, uint32_t lo, uint32_t hi, uint32_t pos) {
    const uint32_t lane = threadIdx.x & 31;
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + lane * step;
        const bool ok = idx < hi && __ldcg(&q_off[idx]) <= pos;
        const uint32_t cnt = __popc(__ballot_sync(0xFFFFFFFFu, ok));
        const uint32_t nlo = lo + (cnt - 1) * step;
        hi = min(hi, nlo + step);
        lo = nlo;
    }
    const uint32_t idx = lo + lane;
    const bool ok = idx < hi && __ldcg(&q_off[idx]) <= pos;
    return lo + __popc(__ballot_sync(0xFFFFFFFFu, ok)) - 1;
}

// Three blocks of 512 threads per SM: the register bound (42) keeps the
// pointer jump from costing a third of the resident threads.
__global__ void __launch_bounds__(512, 3) cc_persistent_kernel(CcArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nth = gridDim.x * blockDim.x;
    const uint32_t warp = tid >> 5;
    const uint32_t nwarps = nth >> 5;
    const DevGraph& g = a.g;
    RunCounters* c = a.ctr;

    for (uint32_t it = 1;; ++it) {
        const uint32_t inSlot = (it - 1) & 3, outSlot = it & 3, clrSlot = (it - 2) & 3;
        const uint64_t qin = ld_relaxed64(&a.qctr[inSlot]);
        const uint32_t Ein = (uint32_t)(qin >> kQShift), Uin = (uint32_t)(qin & kQUnitMask);
        if (Ein == 0) {
            if (tid == 0) c->iterations = it - 1;
            break;
        }
        if (it > g.n + 1) {
            set_error(c, BLEST_ERR_LEVEL_CAP);
            break;
        }
        if (tid == 0) a.qctr[(it + 1) & 3] = 0;  // slot of iteration it+1; last read at it-1
        const uint32_t* fprev = active_buf(a, it - 1);
        uint32_t* fcur = active_buf(a, it);
        uint8_t* fclr = reinterpret_cast<uint8_t*>(active_buf(a, it + 1));
        const uint32_t* qr = a.q_rset + (size_t)inSlot * a.qreg;
        const uint32_t* qo = a.q_off + (size_t)inSlot * a.qreg;

        CcEnqueue q;
        q.cnt = 0;
        q.units = 0;
        uint32_t changes = 0;
        const uint32_t k = (Uin + nwarps - 1) / nwarps;  // chunks per warp
        uint32_t s = warp * k;
        const uint32_t send = min(Uin, s + k);
        if (s < send) {
            uint32_t owner = cc_find_owner(qo, 0, Ein, s);
            for (; s < send; ++s) {
                // entries owner..owner+31 cover chunk s
                const uint32_t ei = owner + lane;
                const bool in = ei < Ein;
                const uint32_t eoff = in ? __ldcg(&qo[ei]) : 0xFFFFFFFFu;
                const uint32_t ers = in ? __ldcg(&qr[ei]) : 0u;
                const uint32_t my = __popc(__ballot_sync(0xFFFFFFFFu, eoff <= s)) - 1;
                const uint32_t r = __shfl_sync(0xFFFFFFFFu, ers, my);
                const uint32_t off = __shfl_sync(0xFFFFFFFFu, eoff, my);
                owner += my;
                const uint32_t t1 = __ldg(&g.rset_tile[r + 1]);
                const uint32_t tile = __ldg(&g.rset_tile[r]) + (s - off) * 32 + lane;
                const uint32_t fb = (__ldcg(&fprev[r >> 2]) >> (8 * (r & 3))) & 0xFFu;
                // the rset's column labels, lane k < 8 holds column r*8+k
                const uint32_t cv = r * 8 + (lane & 7);
                const uint32_t cl = (lane < 8 && cv < g.n) ? __ldcg(&a.labels[cv]) : 0xFFFFFFFFu;
                uint32_t col[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) col[j] = __shfl_sync(0xFFFFFFFFu, cl, j);
                if (tile < t1 && fb) {
                    const uint4 rows = ld_stream(&g.row4[tile]);
                    const uint32_t mask = ld_stream(&g.masks[tile]);
                    const uint32_t rowk[4] = {rows.x, rows.y, rows.z, rows.w};
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) {
                        const uint32_t hb = (mask >> (8 * kk)) & fb & 0xFFu;
                        if (!hb) continue;
                        const uint32_t row = rowk[kk];
                        if (row >= g.n) {
                            set_error(c, BLEST_ERR_DEVICE_INDEX);
                            continue;
                        }
                        uint32_t m = 0xFFFFFFFFu;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if ((hb >> j) & 1u) m = min(m, col[j]);
                        // labels only fall from the vertex id, so labels[row] <= row:
                        // m >= row lowers nothing and needs no label read (half the
                        // slices of the first iteration, where labels are the ids)
                        if (m >= row) continue;
                        if (m < __ldcg(&a.labels[row])) {
                            // one pointer jump: m is the id of a vertex of the
                            // same component, so its label is a valid, possibly
                            // smaller, label too (the fixpoint, the component's
                            // minimum id, is unchanged; long chains such as a
                            // grid numbered outward from a corner shrink by
                            // doubling instead of one hop per iteration).
                            m = min(m, __ldcg(&a.labels[m]));
                            const uint32_t old = atomicMin(&a.labels[row], m);
                            if (m < old) {
                                ++changes;
                                const uint32_t w = row >> 5, b = 1u << (row & 31);
                                const uint32_t oldF = atomicOr(&fcur[w], b);
                                if (((oldF >> (row & 24)) & 0xFFu) == 0) {
                                    const uint32_t rr = row >> 3;
                                    const uint32_t t = tiles_of(g, rr);
                                    if (t) {
                                        q.rset[q.cnt++] = rr;
                                        q.units += t;
                                    }
                                }
                            }
                        }
                    }
                }
                cc_flush(a, outSlot, q);
            }
        }
        // clear active bytes set two iterations back
        if (it >= 2) {
            const uint64_t qc = ld_relaxed64(&a.qctr[clrSlot]);
            const uint32_t Ec = (uint32_t)(qc >> kQShift);
            const uint32_t* qrc = a.q_rset + (size_t)clrSlot * a.qreg;
            for (uint32_t e = tid; e < Ec; e += nth) fclr[__ldcg(&qrc[e])] = 0;
        }
        const uint32_t wc = (uint32_t)warp_sum64(changes);
        if (lane == 0 && wc) atomicAdd(&a.qctr[4], (unsigned long long)wc);
        if (!grid_barrier(c)) return;
    }
}

// no_components = #{v : labels[v] == v}
__global__ void cc_count_kernel(const uint32_t* labels, uint32_t n, RunCounters* c) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nth = gridDim.x * blockDim.x;
    uint32_t cnt = 0;
    for (uint32_t v = tid; v < ((n + 31) & ~31u); v += nth) {
        const bool root = v < n && labels[v] == v;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, root);
        if ((threadIdx.x & 31) == 0) cnt += __popc(b);
    }
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd((unsigned long long*)&c->discovered, (unsigned long long)cnt);
}

// ---------------------------------------------------------------------------
// Symmetric graphs: labels[v] = the smallest id that reaches v is the minimum
// id of v's component, which union-find gives in a few passes over the
// vertices instead of one pass per hop of the label's way.
//
// The scheme is Afforest's (Sutton, Ben-Nun, Barak 2018): merge along a sample
// of the edges until one component holds most vertices, then let only the
// vertices outside it look at all their edges (the large component's edges to
// them are seen from their side, since the graph is symmetric):
//  A  every vertex hooks under one of its first two neighbours and keeps the
//     other one;
//  R  rounds over the kept edges: each vertex whose kept neighbour lies in
//     another tree tries ONCE to hook the one root under the other, until a
//     round hooks next to nothing;
//  C  trees are flattened and the most frequent root of 256 evenly spaced
//     vertices is taken as the large component;
//  D  the vertices outside it link all their edges;
//  E  trees are flattened again, each root's smallest vertex found;
//  F  labels written.
// Parents come before their children in the order (degree descending, mixed
// id): pull lists start with the neighbours of highest degree, so on a skewed
// graph A alone hangs almost everything under a few hubs, and among equal
// degrees the mixed id keeps trees a few hops deep whatever the numbering (a
// grid numbered row by row makes chains of thousands under plain ids).
//
// What bounds it: L2 round trips and the hot spot that one root's word is to
// one L2 slice (about one access a nanosecond). Hooking with retries instead
// of rounds took 90 us for RMAT-20 and 740 us for a 2048 x 2047 grid in one
// phase, nearly all of it failing compare-and-swaps on the growing tree's
// root; so a vertex tries once a round, lanes of a warp with the same root
// try once together, the largest degree is never the one that is hooked, and
// roots are read through L1 (a stale parent is an ancestor all the same).
// Label propagation and this, device time of one run: RMAT-20 (31 M edges)
// 584 -> 53 us, grid 2048 x 2047 3880 -> 303 us (phases A 30, R 212, C 26,
// D 10, E 9, F 5), uniform 1 M vertices x degree 32: 111 us.
struct CcUnionArgs {
    DevGraph g;
    uint32_t* labels;
    uint32_t* parent;  // n words of scratch
    uint32_t* kept;    // n words of scratch: the sampled edge not used in A, v itself when it is settled
    RunCounters* ctr;  // zero between runs (the last block out clears them)
    CcRecord* record;  // mapped host memory
    unsigned long long seq;
};

// Position of v in the trees' order, given its degree: degree descending,
// then a bijection of the ids (the 32-bit finaliser of MurmurHash3), so the
// order is total. Smaller = nearer to the root.
__device__ __forceinline__ uint64_t cc_key(uint32_t v, uint32_t degree) {
    v ^= v >> 16;
    v *= 0x85EBCA6Bu;
    v ^= v >> 13;
    v *= 0xC2B2AE35u;
    v ^= v >> 16;
    return ((uint64_t)~degree << 32) | v;
}

__device__ __forceinline__ uint64_t cc_key(const DevGraph& g, uint32_t v) {
    return cc_key(v, __ldg(&g.csr_ptrs[v + 1]) - __ldg(&g.csr_ptrs[v]));
}

// Unite the trees of u and v. Each round replaces the one of larger key by
// its parent (of smaller key) or hooks it, if it is a root, under the other:
// the larger of the two keys falls in every round, so the loop ends.
__device__ __forceinline__ void cc_link(const DevGraph& g, uint32_t* parent, uint32_t u, uint32_t v) {
    while (u != v) {
        const bool uh = cc_key(g, u) > cc_key(g, v);
        const uint32_t hi = uh ? u : v, lo = uh ? v : u;
        uint32_t p = __ldcg(&parent[hi]);
        if (p == hi) {
            p = atomicCAS(&parent[hi], hi, lo);
            if (p == hi) return;
        }
        u = p;
        v = lo;
    }
}

// The root above p, by plain loads: parents only ever move to further
// ancestors, so a value from L1 is an ancestor too (a root of a moment ago at
// the least), and every warp's reads of a large component's root stay off its
// one L2 slice.
__device__ __forceinline__ uint32_t cc_root(const uint32_t* parent, uint32_t p) {
    for (uint32_t q; (q = parent[p]) != p; p = q) {
    }
    return p;
}

// Roots above x[0..N), climbed in step so that the loads of one hop are in
// flight together; kUnreached entries stay.
template <int N>
__device__ __forceinline__ void cc_roots(const uint32_t* parent, uint32_t (&x)[N]) {
    for (bool more = true; more;) {
        uint32_t q[N];
#pragma unroll
        for (int j = 0; j < N; ++j) q[j] = x[j] != kUnreached ? parent[x[j]] : kUnreached;
        more = false;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            more |= q[j] != x[j];
            x[j] = q[j];
        }
    }
}

constexpr uint32_t kCcBatch = 4;    // vertices per thread and step in A and C: their loads are in flight together
constexpr uint32_t kCcRounds = 12;  // most rounds of R (one counter each in RunCounters::lvl)
constexpr uint32_t kCcSamples = 256;
static_assert(kCcRounds <= 12, "RunCounters::lvl has 12 counters");

__device__ __forceinline__ void cc_union_run(const CcUnionArgs& a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nth = gridDim.x * blockDim.x;
    const DevGraph& g = a.g;
    const uint32_t n = g.n;
    uint32_t* const parent = a.parent;
    RunCounters* c = a.ctr;
    // ids in the lists were checked against n when the graph was made

    // A
    for (uint64_t v0 = tid; v0 < n; v0 += (uint64_t)kCcBatch * nth) {
        uint32_t b[kCcBatch], e[kCcBatch], u[kCcBatch][2], d[kCcBatch][2];
#pragma unroll
        for (uint32_t j = 0; j < kCcBatch; ++j) {
            const uint64_t v = v0 + (uint64_t)j * nth;
            b[j] = v < n ? __ldg(&g.csr_ptrs[v]) : 0u;
            e[j] = v < n ? __ldg(&g.csr_ptrs[v + 1]) : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < kCcBatch; ++j)
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k)
                u[j][k] = b[j] + k < e[j] ? __ldg(&g.csr_ids[b[j] + k]) : kUnreached;
#pragma unroll
        for (uint32_t j = 0; j < kCcBatch; ++j)
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k)
                d[j][k] = u[j][k] != kUnreached ? __ldg(&g.csr_ptrs[u[j][k] + 1]) - __ldg(&g.csr_ptrs[u[j][k]]) : 0u;
#pragma unroll
        for (uint32_t j = 0; j < kCcBatch; ++j) {
            const uint64_t v = v0 + (uint64_t)j * nth;
            if (v >= n) break;
            const uint32_t self = (uint32_t)v;
            const uint64_t kv = cc_key(self, e[j] - b[j]);
            const uint64_t k0 = u[j][0] != kUnreached ? cc_key(u[j][0], d[j][0]) : ~0ull;
            const uint64_t k1 = u[j][1] != kUnreached ? cc_key(u[j][1], d[j][1]) : ~0ull;
            const bool first = k0 <= k1;
            const uint32_t best = first ? u[j][0] : u[j][1], rest = first ? u[j][1] : u[j][0];
            const bool hook = min(k0, k1) < kv;
            parent[self] = hook ? best : self;
            const uint32_t keep = hook ? rest : best;  // a local minimum keeps its best neighbour
            a.kept[self] = keep != kUnreached ? keep : self;
            a.labels[self] = self;
        }
    }
    if (!grid_barrier(c)) return;

    // R
    unsigned long long* const hooked = &c->lvl[0][0];
    __shared__ unsigned long long s_hooked;
    for (uint32_t round = 0; round < kCcRounds; ++round) {
        uint32_t mine = 0;
        for (uint64_t base = tid - lane; base < n; base += nth) {
            const uint64_t v = base + lane;
            uint32_t o = 0, ru = 0, rw = 0;
            bool differ = false;
            if (v < n) {
                o = a.kept[v];
                if (o != v) {
                    const uint32_t p = parent[v];
                    ru = cc_root(parent, p);
                    if (ru != p) parent[v] = ru;
                    rw = cc_root(parent, o);
                    differ = ru != rw;
                    if (!differ) a.kept[v] = (uint32_t)v;
                }
            }
            if (!__any_sync(0xFFFFFFFFu, differ)) continue;
            uint32_t hi = 0, lo = 0;
            if (differ) {
                const bool uh = cc_key(g, ru) > cc_key(g, rw);
                hi = uh ? ru : rw;
                lo = uh ? rw : ru;
            }
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, differ ? hi : kUnreached);
            if (differ && lane == (uint32_t)__ffs(same) - 1 && atomicCAS(&parent[hi], hi, lo) == hi) {
                ++mine;
                a.kept[v] = (uint32_t)v;
            }
        }
        mine = __reduce_add_sync(0xFFFFFFFFu, mine);
        if (lane == 0 && mine) atomicAdd(&hooked[round], (unsigned long long)mine);
        __syncthreads();
        if (threadIdx.x == 0) {
            const bool ok = (barrier_arrive_wait(c) & kArriveError) == 0;
            s_hooked = ok ? ld_relaxed64(&hooked[round]) : ~0ull;
            // passes over edges: A, the rounds so far, D
            if (blockIdx.x == 0) c->iterations = g.nnz ? round + 3 : 0;
        }
        __syncthreads();
        const uint64_t h = s_hooked;
        __syncthreads();
        if (h == ~0ull) return;  // an error is recorded
        if (h <= 16 + (n >> 16)) break;  // what is left costs D less than another round
    }

    // C: no hooks until the next barrier, so every block finds the same roots
    // for the samples and takes the same one
    __shared__ uint32_t s_root[kCcSamples];
    __shared__ unsigned long long s_best;
    if (threadIdx.x == 0) s_best = 0;
    for (uint32_t i = threadIdx.x; i < kCcSamples; i += blockDim.x)
        s_root[i] = cc_root(parent, (uint32_t)((uint64_t)i * n / kCcSamples));
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kCcSamples; i += blockDim.x) {
        uint32_t cnt = 0;
        for (uint32_t j = 0; j < kCcSamples; ++j) cnt += s_root[j] == s_root[i];
        atomicMax(&s_best, ((unsigned long long)cnt << 32) | s_root[i]);
    }
    for (uint64_t v0 = tid; v0 < n; v0 += (uint64_t)kCcBatch * nth) {
        uint32_t p[kCcBatch], x[kCcBatch];
#pragma unroll
        for (uint32_t j = 0; j < kCcBatch; ++j) {
            const uint64_t v = v0 + (uint64_t)j * nth;
            x[j] = p[j] = v < n ? parent[v] : kUnreached;
        }
        cc_roots(parent, x);
#pragma unroll
        for (uint32_t j = 0; j < kCcBatch; ++j)
            if (x[j] != p[j]) parent[v0 + (uint64_t)j * nth] = x[j];
    }
    if (!grid_barrier(c)) return;
    const uint32_t big = (uint32_t)s_best;
    // D: a vertex whose parent is `big` is in its component (phase C made it
    // so, or a hook since); lists over kPullChunk edges go by their pieces
    for (uint64_t v = tid; v < n; v += nth) {
        const uint32_t p = __ldcg(&parent[v]);
        if (p == big) continue;
        const uint32_t b = __ldg(&g.csr_ptrs[v]), e = __ldg(&g.csr_ptrs[v + 1]);
        if (e - b > kPullChunk) continue;
        for (uint32_t i = b; i < e; ++i) {
            const uint32_t q = __ldcg(&parent[__ldg(&g.csr_ids[i])]);
            if (q != p) cc_link(g, parent, p, q);
        }
    }
    for (uint32_t i = tid; i < g.no_pull_chunks; i += nth) {
        const uint4 piece = __ldg(&g.pull_chunks[i]);
        const uint32_t p = __ldcg(&parent[piece.x]);
        if (p == big) continue;
        for (uint32_t k = piece.y; k < piece.z; ++k) {
            const uint32_t q = __ldcg(&parent[__ldg(&g.csr_ids[k])]);
            if (q != p) cc_link(g, parent, p, q);
        }
    }
    if (!grid_barrier(c)) return;
    // E: the vertices under the large component's root keep their minimum in
    // a register (one atomic per block); elsewhere the first lane of each
    // root in the warp, which has the smallest id, lowers the root's label
    const uint32_t top = cc_root(parent, big);
    uint32_t low = 0xFFFFFFFFu, roots = 0;
    for (uint64_t base = tid - lane; base < n; base += nth) {
        const uint32_t v = (uint32_t)base + lane;
        const bool in = v < n;
        uint32_t r = 0xFFFFFFFFu;
        if (in) {
            const uint32_t p = parent[v];
            r = cc_root(parent, p);
            if (r != p) parent[v] = r;
            roots += r == v;
            if (r == top) low = min(low, v);
        }
        const bool other = in && r != top && r != v;
        if (__any_sync(0xFFFFFFFFu, other)) {
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, other ? r : 0xFFFFFFFFu);
            if (other && lane == (uint32_t)__ffs(same) - 1 && v < __ldcg(&a.labels[r])) atomicMin(&a.labels[r], v);
        }
    }
    low = __reduce_min_sync(0xFFFFFFFFu, low);
    roots = __reduce_add_sync(0xFFFFFFFFu, roots);
    __shared__ uint32_t s_low, s_roots;
    if (threadIdx.x == 0) {
        s_low = 0xFFFFFFFFu;
        s_roots = 0;
    }
    __syncthreads();
    if (lane == 0) {
        atomicMin(&s_low, low);
        atomicAdd(&s_roots, roots);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_low != 0xFFFFFFFFu) atomicMin(&a.labels[top], s_low);
        if (s_roots) atomicAdd(&c->discovered, (unsigned long long)s_roots);
    }
    if (!grid_barrier(c)) return;
    // F: a root's label is final, and only non-roots' labels are written
    for (uint64_t v = tid; v < n; v += nth) {
        const uint32_t r = parent[v];
        if (r != v) a.labels[v] = a.labels[r];
    }
}

__global__ void __launch_bounds__(512, 3) cc_union_kernel(CcUnionArgs a) {
    RunCounters* c = a.ctr;
    if (blockIdx.x == 0 && threadIdx.x == 0) c->start_ns = global_ns();
    cc_union_run(a);
    if (!last_block_out(c)) return;
    CcRecord* r = a.record;
    r->start_ns = ld_relaxed64(&c->start_ns);
    r->end_ns = global_ns();
    r->components = ld_relaxed64(&c->discovered);
    r->error = ld_relaxed(&c->error);
    r->iterations = ld_relaxed(&c->iterations);
    zero_counters(c);
    __threadfence_system();
    *(volatile unsigned long long*)&r->seq = a.seq;
}

}  // namespace dev

void launch_cc_union(const blest_graph* g, Workspace& w, uint32_t* labels, cudaStream_t s, uint64_t seq) {
    dev::CcUnionArgs a{};
    a.g = g->d;
    a.labels = labels;
    a.parent = w.cc_parent;
    a.kept = w.cc_parent + g->d.n;
    a.ctr = w.cc_counters;
    a.record = w.cc_record;
    a.seq = seq;
    const int threads = 512;
    // asked once per device (the query costs microseconds)
    static std::mutex mu;
    static std::map<int, int> occupancy;
    int maxBlocks = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        int& known = occupancy[g->device];
        if (!known)
            BLEST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&known, dev::cc_union_kernel, threads, 0));
        maxBlocks = known;
    }
    if (maxBlocks < 1) throw Error(BLEST_ERR_CUDA, "CC kernel cannot be resident");
    // no more blocks than vertices / threads: every block costs the barriers
    const int grid = std::min(cooperative_grid(maxBlocks, g->sm_count, w.grid_blocks),
                              (int)((g->d.n + threads - 1) / threads));
    void* kargs[] = {(void*)&a};
    BLEST_CUDA(cudaLaunchCooperativeKernel((void*)dev::cc_union_kernel, grid, threads, kargs, 0, s));
}

void launch_cc(const blest_graph* g, Workspace& w, uint32_t* labels, cudaStream_t s) {
    dev::CcArgs a{};
    a.g = g->d;
    a.labels = labels;
    a.active0 = w.frontier[0];
    a.active1 = w.frontier[1];
    a.active2 = w.frontier[2];
    a.qreg = w.qcap / 4;
    if (a.qreg < g->d.no_real) throw Error(BLEST_ERR_UNSUPPORTED, "workspace queue too small for CC");
    a.q_rset = w.q_rset;
    a.q_off = w.q_off;
    a.ctr = w.counters;
    a.qctr = w.counters->aux;  // device address inside the counters block
    a.words = w.words;
    const int threads = 512;
    int maxBlocks = 0;
    BLEST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxBlocks, dev::cc_persistent_kernel, threads, 0));
    if (maxBlocks < 1) throw Error(BLEST_ERR_CUDA, "CC kernel cannot be resident");
    const int grid = cooperative_grid(maxBlocks, g->sm_count, w.grid_blocks);
    w.trace_seq = -1;
    BLEST_CUDA(cudaMemsetAsync(w.counters, 0, sizeof(dev::RunCounters), s));
    dev::cc_init_kernel<<<g->sm_count * 4, 512, 0, s>>>(a);
    BLEST_CUDA(cudaGetLastError());
    dev::cc_seed_queue_kernel<<<g->sm_count * 4, 512, 0, s>>>(a);
    BLEST_CUDA(cudaGetLastError());
    void* kargs[] = {(void*)&a};
    BLEST_CUDA(cudaLaunchCooperativeKernel((void*)dev::cc_persistent_kernel, grid, threads, kargs, 0, s));
    dev::cc_count_kernel<<<g->sm_count * 4, 512, 0, s>>>(labels, g->d.n, w.counters);
    BLEST_CUDA(cudaGetLastError());
}

}  // namespace blest
