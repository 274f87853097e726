// Parallel iterative-deepening A* (IDA*) passes for the sliding-tile
// puzzles: the exact phase of the memory-bounded mode.
//
// One pass searches every path whose f = g + h stays at or below a threshold
// t (no dedup table).  Its first moves are searched level by level (k_ida_cut;
// move sequences without immediate reversal, as the search itself prunes)
// until a level has enough nodes to go round; then threads take those roots
// from a queue and search each one's subtree depth-first, with memory
// proportional to the depth, a stack of at most kMaxDepth levels in the
// thread's own local memory.  A pass that finds no goal proves the optimum
// above t and reports the least f it cut off, the next threshold (Korf,
// "Depth-first iterative-deepening: an optimal admissible tree search", 1985).
// With an admissible h the first pass that finds a goal finds an optimal
// solution.
//
// A pass lasts as long as its largest subtree (a chain of dependent pattern
// reads per node), so the roots are many and near the leaves.  57-move
// 15-puzzle, table capped at 2^18 slots: 189 ms with 2^18 roots of one depth
// cut on the host (10 ms of them the cut), 162 / 86 / 64 with 2^18 / 2^20 / 2^21
// cut here, 54 with 2^20 of a tree cut at the pass's threshold.
#pragma once
#include <cstdint>

#include "ga_device.cuh"
#include "ga_problems.cuh"

namespace uastar {

// A root of the cut tree: its board (narrow keys use lo only), depth, aux word
// (pattern parts and the move that reached it) and the moves from the start, 2
// bits each, first move in the lowest bits.
struct IdaRoot {
    unsigned long long lo, hi;
    uint32_t g;
    uint32_t aux;
    unsigned long long prefix;
};

// The cut: the first depth with kIdaRoots nodes (down to kIdaLeastRoots where the
// memory for more is not there), at most kIdaCutDepth (what a prefix holds).
constexpr uint32_t kIdaRoots = 1u << 20, kIdaLeastRoots = 1u << 12;
constexpr uint32_t kIdaCutDepth = 32;
// The levels follow each other in a ring of 4 records per root: a level that is
// expanded has fewer nodes than there are roots and at most three children each
// (the start four), so it and its children fit, whatever came before.
// 134 MB for 2^20 roots (two buffers of a level's children each took 268).
struct IdaCut {
    uint32_t count[kIdaCutDepth + 1];  // nodes per level; 0 past the last
    uint32_t first[kIdaCutDepth + 1];  // a level's first record (modulo the ring)
    uint32_t goal;                     // a goal's depth (0: none met)
    uint32_t min_exceed;               // least f above the threshold
    unsigned long long goal_prefix;    // the moves to the goal
};

constexpr uint32_t kIdaMaxMoves = 256;  // longest solution a pass records

// Pass state, zeroed by the host before each pass (min_exceed set to all ones).
struct IdaPass {
    uint32_t next_root;   // root queue
    uint32_t found;       // 1: a goal was reached (the first finder records it)
    uint32_t stopped;     // 1: the time limit cut the pass short; 2: a subtree was deeper than the stack
    uint32_t min_exceed;  // least f above the threshold among the cut-off nodes
    unsigned long long nodes;
    uint32_t found_root;
    uint32_t found_len;   // moves below the root
    uint8_t moves[kIdaMaxMoves];
};

template <class P> __device__ __forceinline__ typename P::Key ida_key(const IdaRoot &r) {
    if constexpr (P::kWide)
        return Key128{r.lo, r.hi};
    else
        return (uint64_t)r.lo;
}

// The start as the cut's first node.
template <class P> __global__ void k_ida_start(P prob, IdaRoot *out) {
    IdaRoot r;
    if constexpr (P::kWide) {
        r.lo = prob.start.lo;
        r.hi = prob.start.hi;
    } else {
        r.lo = prob.start;
        r.hi = 0;
    }
    r.g = 0;
    r.aux = prob.start_aux();
    r.prefix = 0;
    *out = r;
}

// One level of the cut: the children of level d's nodes with f <= t, appended
// behind it in the ring in any order, unless level d is the last.  `roots`: a
// power of two.
template <class P>
__global__ void __launch_bounds__(256) k_ida_cut(P prob, IdaRoot *ring, uint32_t roots, uint32_t d, uint32_t t,
                                                 IdaCut *cut) {
    const uint32_t n = ldcg_u32(&cut->count[d]);
    if (n == 0 || n >= roots) return;
    const uint32_t wrap = 4u * roots - 1u;
    const uint32_t first = ldcg_u32(&cut->first[d]);
    if (blockIdx.x == 0 && threadIdx.x == 0) cut->first[d + 1] = first + n;
    uint32_t minx = ~0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const IdaRoot r = ring[(first + i) & wrap];
        const typename P::Key key = ida_key<P>(r);
        const uint32_t mask = prob.moves(key, r.aux);
        typename P::Succ sc[4];
        uint32_t naux[4], keep = 0;
#pragma unroll
        for (int mv = 0; mv < 4; ++mv) {
            if (!(mask >> mv & 1u)) continue;
            prob.succ_key(key, d, mv, sc[mv]);
            prob.succ_rest(sc[mv]);
            uint64_t nf;
            prob.succ_end(sc[mv], r.aux, mv, naux[mv], nf);
            if (nf > t) {
                minx = min(minx, (uint32_t)nf);
                continue;
            }
            keep |= 1u << mv;
            if (prob.is_goal(sc[mv].key) && atomicCAS(&cut->goal, 0u, d + 1) == 0u)
                cut->goal_prefix = r.prefix | (unsigned long long)mv << (2 * d);
        }
        if (!keep) continue;
        uint32_t at = first + n + atomicAdd(&cut->count[d + 1], (uint32_t)__popc(keep));
#pragma unroll
        for (int mv = 0; mv < 4; ++mv) {
            if (!(keep >> mv & 1u)) continue;
            IdaRoot c;
            if constexpr (P::kWide) {
                c.lo = sc[mv].key.lo;
                c.hi = sc[mv].key.hi;
            } else {
                c.lo = sc[mv].key;
                c.hi = 0;
            }
            c.g = d + 1;
            c.aux = naux[mv];
            c.prefix = r.prefix | (unsigned long long)mv << (2 * d);
            ring[at++ & wrap] = c;
        }
    }
    if (minx != ~0u) atomicMin(&cut->min_exceed, minx);
}

template <class P, int kMaxDepth>
__global__ void __launch_bounds__(128) k_ida_pass(P prob, const IdaRoot *ring, uint32_t wrap, uint32_t first,
                                                  uint32_t nroots, uint32_t t, IdaPass *out,
                                                  unsigned long long budget_ns) {
    using Key = typename P::Key;
    // the pass ends budget_ns after this thread started (the threads of a
    // launch start together: the grid fits the GPU at once)
    const unsigned long long deadline_ns = globaltimer_ns() + budget_ns;
    Key ks[kMaxDepth + 1];
    uint32_t as[kMaxDepth + 1];
    uint8_t rem[kMaxDepth + 1];
    unsigned long long nodes = 0, next_check = 1024;
    uint32_t minx = ~0u;
    bool quit = false;
    while (!quit) {
        if (ldcg_u32(&out->found) || ldcg_u32(&out->stopped)) break;
        if (globaltimer_ns() > deadline_ns) {
            atomicCAS(&out->stopped, 0u, 1u);
            break;
        }
        const uint32_t i = atomicAdd(&out->next_root, 1u);
        if (i >= nroots) break;
        const IdaRoot r = ring[(first + i) & wrap];
        const uint32_t g0 = r.g;
        ks[0] = ida_key<P>(r);
        as[0] = r.aux;
        rem[0] = (uint8_t)prob.moves(ks[0], as[0]);
        int d = 0;
        while (d >= 0) {
            if (rem[d] == 0) {
                --d;
                continue;
            }
            const int mv = __ffs(rem[d]) - 1;
            rem[d] &= (uint8_t)(rem[d] - 1);
            typename P::Succ sc;
            prob.succ_key(ks[d], g0 + d, mv, sc);
            prob.succ_rest(sc);
            uint32_t naux;
            uint64_t nf;
            prob.succ_end(sc, as[d], mv, naux, nf);
            ++nodes;
            if (nf > t) {
                minx = min(minx, (uint32_t)nf);
                continue;
            }
            if (prob.is_goal(sc.key)) {
                if (atomicCAS(&out->found, 0u, 1u) == 0u) {
                    const uint32_t len = (uint32_t)d + 1;
                    out->found_root = i;
                    out->found_len = len;
                    for (int j = 1; j <= d; ++j) out->moves[j - 1] = (uint8_t)((as[j] >> P::kLastMoveShift) - 1);
                    out->moves[d] = (uint8_t)mv;
                }
                quit = true;
                break;
            }
            if (d + 1 >= kMaxDepth) {
                atomicCAS(&out->stopped, 0u, 2u);
                quit = true;
                break;
            }
            ++d;
            ks[d] = sc.key;
            as[d] = naux;
            rem[d] = (uint8_t)prob.moves(ks[d], naux);
            if (nodes >= next_check) {  // another thread's goal, or the time limit
                next_check = nodes + 1024;
                if (ldcg_u32(&out->found)) {
                    quit = true;
                    break;
                }
                if (globaltimer_ns() > deadline_ns) {
                    atomicCAS(&out->stopped, 0u, 1u);
                    quit = true;
                    break;
                }
            }
        }
    }
    if (nodes) atomicAdd(&out->nodes, nodes);
    if (minx != ~0u) atomicMin(&out->min_exceed, minx);
}

}  // namespace uastar
