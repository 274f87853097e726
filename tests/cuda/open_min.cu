// k_best_open on hand-made parked heaps: the least current entry, wherever in a
// heap the stale ones lie, against a loop over all entries on the host.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "../../uastar_gb300/csrc/ga_open.cuh"

using namespace uastar;

static PuzzleEntry entry_of(int n, uint32_t f, uint32_t g, uint32_t slot) {
    // (4x4: one pattern part of the heuristic in the low byte)
    return {n == 5 ? f << 16 | (0xffffu - g) : f << 22 | (255u - g) << 14 | std::min(f - g, 7u), slot};
}

// Entry i of a parked heap: the shared top's L levels at the head of its block,
// then bricks of D levels, level by level (ga_search.cuh BrickHeap).
static uint32_t place(uint32_t i, uint32_t L, uint32_t D) {
    if (i < (1u << L)) return i;
    const uint32_t BE = 1u << D, reserve = ((1u << L) + BE - 1) / BE * BE;
    uint32_t l = 31;
    while (!(i >> l)) --l;
    const uint32_t bl = (l - L) / D, d = (l - L) % D;
    const uint32_t first = (((1u << bl * D) - 1) << L) / (BE - 1);
    return reserve + (first + (i >> d) - (1u << (L + bl * D))) * BE + ((1u << d) | (i & ((1u << d) - 1)));
}

// `stale`: how many of each heap's least entries are stale.
template <int N> static bool check(uint32_t L, uint32_t k, uint32_t size, uint32_t stale, uint32_t seed) {
    using P = PuzzleProblem<N>;
    const HeapGeometry<P> geo = heap_geometry<P>(L, std::max(size, 1u));
    if (size > geo.hcap) return true;
    std::mt19937 rng(seed);
    const uint32_t words = N == 5 ? 4u : 2u;  // 8-byte words of a slot
    const uint32_t slots = k * std::max(size, 1u);
    std::vector<unsigned long long> tab((size_t)slots * words, 0);
    std::vector<PuzzleEntry> heaps((size_t)k * geo.stride, PuzzleEntry{0, 0});
    std::vector<uint32_t> sizes(k, size);
    unsigned long long want = ~0ull;
    for (uint32_t h = 0; h < k; ++h) {
        std::vector<PuzzleEntry> es;
        for (uint32_t i = 0; i < size; ++i) {
            const uint32_t g = 2 + rng() % 60, f = g + rng() % 20;
            es.push_back(entry_of(N, f, g, h * size + i));
        }
        // in ascending order: a heap
        std::sort(es.begin(), es.end(), [](const PuzzleEntry &a, const PuzzleEntry &b) { return a.key < b.key; });
        for (uint32_t i = 1; i <= size; ++i) {
            const PuzzleEntry e = es[i - 1];
            heaps[(size_t)h * geo.stride + place(i, L, BrickHeap<P>::D)] = e;
            const bool old = i <= stale;
            uint64_t g = N == 5 ? 0xffffu - (e.key & 0xffffu) : 255u - (e.key >> 14 & 255u);
            const uint64_t hval = P::entry_cost(e) - g;
            if (old) g -= 1 + rng() % 2;  // the node was reached by fewer moves since
            unsigned long long *w = &tab[(size_t)e.slot * words];
            if (N == 5) {
                w[0] = 12345 | g << 60;
                w[1] = 54321 | g >> 4 << 60;
                w[3] = (unsigned)hval;  // aux: one pattern part
            } else {
                w[0] = 777 + e.slot;
                w[1] = g << 40;
            }
            if (!old) want = std::min(want, (unsigned long long)e.key << 32 | e.slot);
        }
    }
    unsigned long long *d_tab, *d_best, got = ~0ull;
    PuzzleEntry *d_heaps;
    uint32_t *d_sizes;
    cudaMalloc(&d_tab, tab.size() * 8);
    cudaMalloc(&d_heaps, heaps.size() * sizeof(PuzzleEntry));
    cudaMalloc(&d_sizes, k * 4);
    cudaMalloc(&d_best, 8);
    cudaMemcpy(d_tab, tab.data(), tab.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d_heaps, heaps.data(), heaps.size() * sizeof(PuzzleEntry), cudaMemcpyHostToDevice);
    cudaMemcpy(d_sizes, sizes.data(), k * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d_best, &got, 8, cudaMemcpyHostToDevice);
    SearchMem<PuzzleEntry> m{};
    m.tab = reinterpret_cast<Slot *>(d_tab);
    m.heaps = d_heaps;
    m.heap_size = d_sizes;
    m.stride = geo.stride;
    m.hcap = geo.hcap;
    m.L = L;
    P prob{};
    k_best_open<N><<<4, 64>>>(prob, m, k, d_best);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(&got, d_best, 8, cudaMemcpyDeviceToHost);
    cudaFree(d_tab);
    cudaFree(d_heaps);
    cudaFree(d_sizes);
    cudaFree(d_best);
    if (e == cudaSuccess && got == want) return true;
    std::printf("%dx%d L %u k %u size %u stale %u: %llx, want %llx (%s)\n", N, N, L, k, size, stale, got, want,
                cudaGetErrorString(e));
    return false;
}

int main() {
    int bad = 0, n = 0;
    for (uint32_t L : {1u, 3u, 5u})
        for (uint32_t k : {1u, 3u, 20u})
            for (uint32_t size : {0u, 1u, 7u, 31u, 32u, 200u, 3000u})
                for (uint32_t stale : {0u, 1u, 31u, 32u, 199u, 2999u, 3000u}) {
                    const uint32_t seed = ++n;
                    bad += !check<4>(L, k, size, stale, seed);
                    bad += !check<5>(L, k, size, stale, seed);
                }
    std::printf("%d of %d cases wrong\n", bad, 2 * n);
    return bad ? 1 : 0;
}
