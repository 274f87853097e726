// ga_search on an 8-puzzle a few moves from the goal, by one CTA: with a bound on
// f it is solved, without one it is refused before the search begins.
#include <cstdio>

#include "../../uastar_gb300/csrc/ga_problems.cuh"
#include "../../uastar_gb300/csrc/ga_search.cuh"

using namespace uastar;
using P = PuzzleProblem<3>;
constexpr uint32_t kHeaps = 16, kTop = 4, kSlots = 1u << 14;

__global__ void k_search(P prob, SearchMem<PuzzleEntry> m, uint32_t *status, unsigned long long *best) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ TeamState st;
    if (threadIdx.x == 0) team_state_init(&st);
    __syncthreads();
    BlockTeam team{&st};
    const uint32_t s = ga_search(prob, team, m, kHeaps, smem, 100000);
    __syncthreads();
    if (threadIdx.x == 0) {
        status[0] = s;
        status[1] = st.status;
        *best = st.goal_best;
    }
}

int main() {
    const HeapGeometry<P> geo = heap_geometry<P>(kTop, 4095);
    uint8_t *pdb;  // an admissible heuristic: nothing to go in every pattern
    Slot *tab;
    PuzzleEntry *heaps;
    uint32_t *sizes, *status, got[2];
    Cand *cand;
    unsigned long long *best, g;
    cudaMalloc(&pdb, 362880);
    cudaMalloc(&tab, kSlots * sizeof(Slot));
    cudaMalloc(&heaps, (size_t)kHeaps * geo.stride * sizeof(PuzzleEntry));
    cudaMalloc(&sizes, kHeaps * 4);
    cudaMalloc(&cand, cand_records<P>(1, kHeaps) * sizeof(Cand));
    cudaMalloc(&status, 8);
    cudaMalloc(&best, 8);
    cudaMemset(pdb, 0, 362880);
    const size_t smem = SearchSmem<P>::bytes(kHeaps, kTop);
    cudaFuncSetAttribute(k_search, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    P prob;
    prob.pdb = pdb;
    prob.goal = P::goal_key();
    // the blank up and left of its place: tiles 6 and 5 moved
    prob.start = prob.goal & ~(0xfull | 0xfull << 24 | 0xfull << 20);
    prob.start |= 4ull | 8ull << 24 | 5ull << 20;
    int bad = 0;
    for (const float slack : {0.5f, 0.f}) {
        cudaMemset(tab, 0xff, kSlots * sizeof(Slot));
        cudaMemset(sizes, 0, kHeaps * 4);
        SearchMem<PuzzleEntry> m;
        m.tab = tab;
        m.mask = kSlots - 1;
        m.max_inserted = kSlots / 2;
        m.max_probe = 4096;
        m.heaps = heaps;
        m.stride = geo.stride;
        m.hcap = geo.hcap;
        m.L = kTop;
        m.heap_size = sizes;
        m.cand = cand;
        m.max_rounds = 1000;
        m.slack = slack;
        k_search<<<1, 64, smem>>>(prob, m, status, best);
        const cudaError_t e = cudaDeviceSynchronize();
        cudaMemcpy(got, status, 8, cudaMemcpyDeviceToHost);
        cudaMemcpy(&g, best, 8, cudaMemcpyDeviceToHost);
        const bool ok = slack > 0.f ? got[0] == ST_OK && got[1] == ST_OK && g == 2
                                    : got[0] == ST_BAD_INPUT && got[1] == ST_BAD_INPUT;
        std::printf("slack %.1f: %u %u, %llu moves (%s)\n", slack, got[0], got[1], g, cudaGetErrorString(e));
        bad += !ok || e != cudaSuccess;
    }
    return bad;
}
