// Reading a path out of a finished grid search: the prev chain from the goal
// to the start, by one CTA.
//
// Followed link by link, the chain is one dependent table read per cell (0.44 us
// each, 9.8 ms on the 20000^2 grid's 22 293 cells).  But the next cell is one of
// the eight neighbours, so the CTA looks up a whole window of cells around the
// current one at once (each by its own hash), finds every cell's parent among
// its neighbours in shared memory, and one thread then follows the chain there
// until it leaves the window.  The window lies on the side of the start, so a
// path that makes its way there stays in it for ~27 cells, at the price of
// about two memory trips.  Bound by these trips and the chain in shared memory
// (45 cycles a cell).  Walks of 1000^2, 700 x 1021 and 20000^2 cells in hashed
// slots: 490 -> 150, 390 -> 116 and 9800 -> 3130 us; in words (one look-up a
// cell, no neighbours to compare) 73 us for the second, 1670 for the third.
// Windows 64 wide took 215 us at 1000^2 where these, not yet trimmed, took 170:
// four times the look-ups, half of them for nothing.
#pragma once
#include <cstdint>

#include "ga_device.cuh"
#include "ga_problems.cuh"

namespace uastar {

struct GridWalkSmem {
    static constexpr uint32_t kSide = 32, kCells = kSide * kSide;
    static constexpr uint32_t kAhead = kSide - 5;  // cells of the window towards the start
    static constexpr uint16_t kOut = 0xFFFF, kEnd = 0xFFFE;
    uint32_t slot[kCells], prev[kCells];  // the cell's slot (kNone: not in the table) and its parent's
    uint16_t next[kCells];                // its parent's place in the window, kOut or kEnd
    uint16_t chain[kCells];               // the chain's places in the window, from its first cell on
    uint32_t links;                       // cells of it before the last
    uint16_t last;                        // the last one's next: kOut or kEnd
};

// Slot and parent slot of a cell; kNone if the table does not hold it.  Most
// cells are in their home slot or have it free: the other three of its group are
// read only for the rest.
__device__ __forceinline__ void find_cell(const Slot *tab, uint64_t mask, uint32_t cell, uint32_t &slot,
                                          uint32_t &prev) {
    const uint64_t home = mix64(cell) & mask;
    slot = prev = kNone;
    for (uint64_t i = 0; i <= mask; ++i) {
        const uint64_t at = probe_slot(home, i, mask);
        const unsigned long long w = __ldcg(&tab[at].key);
        if (w == kEmptyKey) return;
        if ((uint32_t)w == cell) {
            slot = (uint32_t)at;
            prev = (uint32_t)(w >> 32);
            return;
        }
    }
}

// Each window cell's parent's place, from hashed slots.  All threads of the CTA
// call it; the next barrier makes the result theirs.
__device__ __forceinline__ void window_links(const Slot *tab, uint64_t mask, const GridProblem &prob, int x0, int y0,
                                             GridWalkSmem &s) {
    constexpr int kSide = (int)GridWalkSmem::kSide;
    const uint32_t tid = threadIdx.x, T = blockDim.x;
    for (uint32_t w = tid; w < GridWalkSmem::kCells; w += T) {
        const int x = x0 + (int)(w / kSide), y = y0 + (int)(w % kSide);
        uint32_t slot = kNone, prev = kNone;
        if (x >= 0 && x < prob.H && y >= 0 && y < prob.W)
            find_cell(tab, mask, (uint32_t)x * (uint32_t)prob.W + (uint32_t)y, slot, prev);
        s.slot[w] = slot;
        s.prev[w] = prev;
    }
    __syncthreads();
    for (uint32_t w = tid; w < GridWalkSmem::kCells; w += T) {
        const uint32_t prev = s.prev[w];
        uint16_t to = prev == kNone ? GridWalkSmem::kEnd : GridWalkSmem::kOut;
        if (prev != kNone) {
            const int lx = (int)(w / kSide), ly = (int)(w % kSide);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int px = lx + GridProblem::c_dx(i), py = ly + GridProblem::c_dy(i);
                if (px < 0 || px >= kSide || py < 0 || py >= kSide) continue;
                if (s.slot[px * kSide + py] == prev) to = (uint16_t)(px * kSide + py);
            }
        }
        s.next[w] = to;
    }
}
// The same from one word per cell, which names the move that reached it.
__device__ __forceinline__ void window_links(const Slot *tab, uint64_t, const GridDirect &prob, int x0, int y0,
                                             GridWalkSmem &s) {
    constexpr int kSide = (int)GridWalkSmem::kSide;
    for (uint32_t w = threadIdx.x; w < GridWalkSmem::kCells; w += blockDim.x) {
        const int lx = (int)(w / kSide), ly = (int)(w % kSide), x = x0 + lx, y = y0 + ly;
        uint16_t to = GridWalkSmem::kEnd;  // unreached cells and the start
        if (x >= 0 && x < prob.H && y >= 0 && y < prob.W && !(x == prob.sx && y == prob.sy)) {
            const unsigned long long v = __ldcg(GridDirect::words(tab) + (uint64_t)x * prob.W + y);
            if (v != kInfCost) {
                const int px = lx - GridProblem::c_dx((int)(v & 7u)), py = ly - GridProblem::c_dy((int)(v & 7u));
                to = px < 0 || px >= kSide || py < 0 || py >= kSide ? GridWalkSmem::kOut : (uint16_t)(px * kSide + py);
            }
        }
        s.next[w] = to;
    }
}

// Calls store(i, cell) for the i-th cell of the chain from the goal, at most
// `cap` of them, each on some thread of the first warp; returns their number,
// or cap + 1 if the chain is longer.  All threads of the CTA call it and get
// the result.
template <class P, class Store>
__device__ unsigned long long walk_grid(const Slot *tab, uint64_t mask, const P &prob, uint64_t cap, GridWalkSmem &s,
                                        Store &&store) {
    constexpr int kSide = (int)GridWalkSmem::kSide;
    constexpr uint32_t kCells = GridWalkSmem::kCells;
    const uint32_t tid = threadIdx.x;
    int cx = prob.ex, cy = prob.ey;
    // n cells lie before (cx, cy), the first of the window's part of the chain
    for (unsigned long long n = 0;;) {
        const auto first = [](int at, int to) {
            return at - (to < at ? (int)GridWalkSmem::kAhead : to > at ? kSide - 1 - (int)GridWalkSmem::kAhead : kSide / 2);
        };
        const int x0 = first(cx, prob.sx), y0 = first(cy, prob.sy);
        window_links(tab, mask, prob, x0, y0, s);
        __syncthreads();
        if (tid < 32) {
            if (tid == 0) {
                uint32_t at = (uint32_t)((cx - x0) * kSide + (cy - y0)), k = 0;
                for (;;) {
                    s.chain[k] = (uint16_t)at;
                    const uint32_t to = s.next[at];
                    if (to >= kCells || k + 1 >= kCells) {  // (a chain visits no cell twice)
                        s.last = (uint16_t)to;
                        break;
                    }
                    ++k;
                    at = to;
                }
                s.links = k;
            }
            __syncwarp();
            // the last cell of a chain that leaves the window is the first of
            // the next one's, which has its whole neighbourhood
            const uint32_t links = s.links + (s.last == GridWalkSmem::kEnd ? 1u : 0u);
            for (uint32_t k = tid; k < links && n + k < cap; k += 32) {
                const uint32_t at = s.chain[k];
                store(n + k, (uint32_t)((x0 + (int)(at / kSide)) * prob.W + y0 + (int)(at % kSide)));
            }
        }
        __syncthreads();
        const uint32_t links = s.links, at = s.chain[links];
        n += links;
        if (s.last == GridWalkSmem::kEnd) return n + 1 <= cap ? n + 1 : cap + 1;
        if (n >= cap || links == 0) return cap + 1;
        cx = x0 + (int)(at / kSide);
        cy = y0 + (int)(at % kSide);
    }
}

}  // namespace uastar
