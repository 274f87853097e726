// Moving a paused search to a larger dedup table (plain engine and serving
// loop).  A search paused by ga_search (it returned ST_RUNNING at a round
// boundary, its insertion buffers drained into its heaps) names slots in
// three places: the slots' prev links, the heap entries and the team's goal
// slot.  Growth re-inserts every occupied slot into the empty larger table,
// recording old -> new in `map`, then rewrites all three.  The kernels have
// internal linkage: each translation unit that launches them has its own.
#pragma once
#include <cstdint>

#include "ga_device.cuh"
#include "ga_search.cuh"

namespace uastar {
namespace {

// Re-insert the occupied slots of `src` (n slots) into `dst` (mask + 1
// empty slots).  Keys are unique, so an insert only races other keys for an
// empty slot; prev is copied as is and rewritten by k_grow_links.  Wide:
// 16-byte keys (WideSlot layout), claimed with one 16-byte CAS.  PrevInKey:
// the key word is cell | prev << 32 (grids), hashed on the cell.
template <bool Wide, bool PrevInKey>
__global__ void k_grow_move(const Slot *src, uint64_t n, Slot *dst, uint64_t mask, uint32_t *map) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x) {
        constexpr uint64_t words = Wide ? 2 : 1;  // of 16 bytes a slot
        const uint4 *from = reinterpret_cast<const uint4 *>(src) + s * words;
        const uint4 a = __ldcg(from);
        const unsigned long long key = ((unsigned long long)a.y << 32) | a.x;
        if (key == kEmptyKey) continue;
        uint64_t h;
        if constexpr (Wide) {
            const KeyG k{key, ((unsigned long long)a.w << 32) | a.z};
            const uint64_t home = key_hash(WideSlots::word_key(k)) & mask;
            h = home;
            for (uint32_t probe = 1; probe <= mask; ++probe) {
                const KeyG old = cas128(WideSlots::at(dst, h), KeyG{kEmptyKey, kEmptyKey}, k);
                if (old.key == kEmptyKey && old.g == kEmptyKey) break;
                h = probe_slot(home, probe, mask);
            }
        } else {
            const uint64_t home = mix64(PrevInKey ? key & 0xffffffffull : key) & mask;
            h = home;
            for (uint32_t probe = 1; probe <= mask; ++probe) {
                if (atomicCAS(&dst[h].key, kEmptyKey, key) == kEmptyKey) break;
                h = probe_slot(home, probe, mask);
            }
        }
        uint4 *d = reinterpret_cast<uint4 *>(dst) + h * words;
        d[0] = a;                                     // key and g
        if constexpr (Wide) d[1] = __ldcg(from + 1);  // aux, prev (old index)
        map[s] = (uint32_t)h;
    }
}

// Link: where the slots keep their parent link (SlotLink).
template <bool Wide, int Link>
__global__ void k_grow_links(const Slot *src, uint64_t n, Slot *dst, const uint32_t *map) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x) {
        const Slot *from = src + (Wide ? 2 * s : s);
        const uint64_t w = __ldcg(&from->key);
        if (w == kEmptyKey) continue;
        if constexpr (Link == LINK_IN_KEY) {
            const uint32_t p = (uint32_t)(w >> 32);
            dst[map[s]].key = (w & 0xffffffffull) | (uint64_t)(p == kNone ? kNone : map[p]) << 32;
        } else if constexpr (Link == LINK_IN_G) {
            const uint64_t gw = __ldcg(&from->g);
            const uint32_t p = (uint32_t)gw;
            dst[map[s]].g = (gw & ~0xffffffffull) | (p == kNone ? kNone : map[p]);
        } else {
            const uint32_t p = __ldcg(&WideSlots::w(from)->prev);
            WideSlots::w(WideSlots::at(dst, map[s]))->prev = p == kNone ? kNone : map[p];
        }
    }
}

// One warp per heap: entries 1..size, the saved shared top first (heap
// indices <= 2^L - 1 at the head of the heap's block), then the bricks.
template <class P>
__global__ void k_grow_heaps(typename P::Entry *heaps, uint32_t stride, uint32_t L, const uint32_t *heap_size,
                             uint32_t k, const uint32_t *map, TeamState *st) {
    using E = typename P::Entry;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t topn = (1u << L) - 1u;
    for (uint32_t h = warp; h < k; h += nwarps) {
        E *gblock = heaps + (size_t)h * stride;
        const BrickHeap<P> bh{gblock + top_reserve<P>(L), nullptr, nullptr, L};
        const uint32_t sz = heap_size[h];
        for (uint32_t i = 1 + lane; i <= sz; i += 32) {
            E *q = i <= topn ? gblock + i : bh.g + bh.off(i);
            E e = P::load(q);
            e.slot = map[e.slot];
            P::store(q, e);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (st->goal_slot != kNone) st->goal_slot = map[st->goal_slot];
        st->barrier = 0;  // a grid team's next launch counts barriers from zero
    }
}

}  // namespace
}  // namespace uastar
