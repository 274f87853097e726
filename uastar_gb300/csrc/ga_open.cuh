// The open list of a paused puzzle search (memory-bounded mode).
#pragma once
#include <cstdint>

#include "ga_device.cuh"
#include "ga_problems.cuh"
#include "ga_search.cuh"

namespace uastar {
namespace {

// The best open node of a paused puzzle search: the least entry (least f, then
// deepest) of all heaps that is current (its f still matches the node's g), as
// key << 32 | slot into *best by atomicMin.  Every entry is looked at, not only
// the heaps' tops: a current entry may lie under stale ones, and the caller
// takes this minimum for a bound that ends the search.  One warp per heap; an
// entry that cannot lower *best any more costs its read alone, so the pass is
// bound by the heaps' bytes (8 an entry).
template <int N>
__global__ void k_best_open(PuzzleProblem<N> prob, SearchMem<PuzzleEntry> m, uint32_t k,
                            unsigned long long *best) {
    using P = PuzzleProblem<N>;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t topn = (1u << m.L) - 1u;
    for (uint32_t h = warp; h < k; h += nwarps) {
        // a parked heap: its shared top at the head of its block, then its bricks
        PuzzleEntry *const gblock = m.heaps + (size_t)h * m.stride;
        const BrickHeap<P> bh{gblock + top_reserve<P>(m.L), nullptr, nullptr, m.L};
        const uint32_t sz = __ldcg(&m.heap_size[h]);
        for (uint32_t i = 1 + lane; i <= sz; i += 32) {
            const PuzzleEntry e = P::load(i <= topn ? gblock + i : bh.g + bh.off(i));
            const unsigned long long v = ((unsigned long long)e.key << 32) | e.slot;
            if (v >= ldcg_u64(best)) continue;
            typename P::Key key;
            uint64_t g;
            uint32_t aux;
            P::load_node(P::at(m.tab, e.slot), e, key, g, aux);
            if (prob.f_of(key, g, aux) != P::entry_cost(e)) continue;  // stale
            atomicMin(best, v);
        }
    }
}

}  // namespace
}  // namespace uastar
