// The two search problems the engine instantiates GA* for.
//
// A problem supplies: the heap entry type and its order, the cost word
// (compared with cost_cmp), the start/goal keys, f = g + h, the valid-move
// mask of a popped node and the successor of one move.
//
// GridProblem   — 8-direction grid of uAstar's --pathway mode.  Costs are the
//                 exact pair (straight A, diagonal B) with value A + B*sqrt(2),
//                 packed A<<32 | B and compared with integer arithmetic only,
//                 so the search is exact where the reference accumulates float32.
// PuzzleProblem — n x n sliding tile of --puzzle with the additive disjoint
//                 pattern database; integer move counts.
#pragma once
#include <cstdint>

#include "ga_device.cuh"

namespace uastar {

// How far a whole-GPU search of k heaps expands beyond its pops
// (SearchMem::cont, cont_pops and slack).
struct Expansion {
    uint32_t cont, cont_pops;
    float slack;
};

// ----------------------------------------------------------------- grid ---
struct __align__(16) GridEntry {
    uint32_t fa, fb;  // f = fa + fb*sqrt(2)
    uint32_t slot;
    uint32_t cell;    // the node's cell: a pop reads its bitmap neighbourhood
                      // while the node record is still in flight
};

// sign(d - e*sqrt2), exact for |d|, |e| < 2^31.  In float32 first: the
// conversions, the constant and the multiply-add are each off by at most 2^-24
// of their terms, together less than 2^-21 (|d| + 2 |e|), so a larger result
// has the right sign; the rest (ties, and near misses of sqrt2 by d / e) takes
// 64-bit integers.  A heap compares entries ~10 times per pop, and the integer
// form alone is four times the instructions in branches (with the successor
// numbering of a round down from three CTA barriers to one: 20000^2 grid 177 ->
// 167 ms, 1000^2 8.7 -> 8.3, six queries on 1537 x 2049 32.9 -> 31.2).
__host__ __device__ __forceinline__ int sqrt2_sign(int32_t d, int32_t e) {
    const float fd = (float)d, fe = (float)e, v = fd - 1.41421356f * fe;
    if (fabsf(v) > 4.8e-7f * (fabsf(fd) + 2.f * fabsf(fe))) return v > 0.f ? 1 : -1;
    if (e == 0) return d > 0 ? 1 : (d < 0 ? -1 : 0);
    if (d >= 0 && e < 0) return 1;
    if (d <= 0 && e > 0) return -1;
    const uint64_t lhs = (uint64_t)((int64_t)d * d), rhs = 2ull * (uint64_t)((int64_t)e * e);
    const int s = lhs > rhs ? 1 : -1;  // never equal: sqrt(2) is irrational
    return d > 0 ? s : -s;
}

// sign((a1 + b1*sqrt2) - (a2 + b2*sqrt2)) for packed a<<32|b words; kInfCost
// is larger than every cost.  Exact for a, b < 2^31.
__host__ __device__ __forceinline__ int grid_cost_cmp(uint64_t p, uint64_t q) {
    if (p == q) return 0;
    if (p == kInfCost) return 1;
    if (q == kInfCost) return -1;
    return sqrt2_sign((int32_t)(p >> 32) - (int32_t)(q >> 32), (int32_t)(uint32_t)q - (int32_t)(uint32_t)p);
}

struct GridProblem : NarrowSlots {
    using Entry = GridEntry;
    static constexpr int kMoves = 8;
    // Slot key word = cell | prev << 32 (cells are < 2^32 - 1): the relax CAS
    // sets g and the parent link together, so no push-phase winner check.
    static constexpr bool kPrevInKey = true;
    static constexpr int kLink = LINK_IN_KEY;
    __device__ static KeyG cas_word(uint64_t key, uint64_t g, uint32_t prev, int) {
        return KeyG{key | (uint64_t)prev << 32, g};
    }
    __device__ static bool word_is(KeyG w, uint64_t key) {
        return (w.key & 0xffffffffull) == key && w.key != kEmptyKey;
    }
    __device__ static uint64_t word_g(KeyG w) { return w.g; }

    struct Succ {  // see succ_key
        uint64_t key, g, f;
        int x, y;
    };
    const uint32_t *bm;  // bitmap as 32-bit words (same bytes as the uint64 words)
    int32_t H, W;
    int32_t sx, sy, ex, ey;
    uint64_t w_inv;  // row_inverse(W)

    // c / W as one widening multiply: w_inv = ceil(2^64 / W) makes
    // floor(c * w_inv / 2^64) exact for every c < 2^32 (w_inv * W exceeds
    // 2^64 by less than W, so the product by less than c / 2^64 < 1 / W);
    // 0 stands for 2^64 (W = 1).
    __host__ __device__ static uint64_t row_inverse(int32_t W) {
        return W == 1 ? 0ull : ~0ull / (uint64_t)W + 1ull;
    }
    __device__ __forceinline__ uint32_t row_of(uint32_t c) const {
        return w_inv ? (uint32_t)__umul64hi((uint64_t)c, w_inv) : c;
    }

    __device__ static int cost_cmp(uint64_t a, uint64_t b) { return grid_cost_cmp(a, b); }
    // a cost as one number, to place the round's bound (no exact test uses it)
    __device__ static float cost_val(uint64_t c) {
        return (float)(uint32_t)(c >> 32) + 1.41421356f * (float)(uint32_t)c;
    }

    __device__ __forceinline__ bool open(int64_t id) const {
        return (__ldg(bm + (id >> 5)) >> (id & 31)) & 1u;
    }
    __device__ uint64_t start_key() const { return (uint64_t)sx * W + sy; }
    // a grid node's aux is its own cell (carried into its heap entries)
    __device__ uint32_t start_aux() const { return (uint32_t)start_key(); }
    __device__ bool is_goal(uint64_t key) const { return key == (uint64_t)ex * W + ey; }
    // The entry names its node's key: moves() can start before load_node().
    // On grids of at most 2^29 cells it also carries the move that reached
    // the node (bits 29-31 of the cell word), and the expansion skips every
    // successor that is the parent p or one of p's neighbours: one step from
    // p costs at most sqrt2, two steps through the node at least 2, so the
    // relax could never succeed.  (By induction along the parent chain this
    // holds although the ancestors skipped successors too: a neighbour n of
    // the node that is skipped was relaxed by the nearest ancestor that did
    // not skip it, at that ancestor's g + one step, while the node's g is at
    // least that g + 1 and the step from the node at least 1.)  The start
    // node has no incoming move.  Entries that are stale are not expanded, so
    // the move is always that of the node's current g and parent.
    static constexpr bool kEntryKey = true;
    static constexpr uint32_t kCellBits = 29;
    __device__ __forceinline__ bool dirs() const { return (uint64_t)(uint32_t)H * (uint32_t)W <= (1ull << kCellBits); }
    __device__ __forceinline__ uint64_t entry_key(const GridEntry &e) const {
        return dirs() ? (e.cell & ((1u << kCellBits) - 1u)) : e.cell;
    }
    // successors of the move that reached a node that can never improve
    // (bit j = move j), indexed by that move
    __device__ __forceinline__ static uint32_t pruned(uint32_t in) {
        return (uint32_t)(0x1529468a57ab3dceull >> (8 * in)) & 0xffu;
    }
    __device__ __forceinline__ uint32_t entry_moves(const GridEntry &e) const {
        const uint64_t key = entry_key(e);
        uint32_t m = moves(key, 0);
        if (dirs() && key != start_key()) m &= ~pruned(e.cell >> kCellBits);
        return m;
    }

    // Octile heuristic (src/pathway/CPU-solver.cpp:139-146): with dx, dy the
    // distances to the goal, h = min(dx,dy)*sqrt2 + |dx-dy| — as a pair.
    __device__ __forceinline__ uint64_t h_of(uint64_t key) const {
        const uint32_t c = (uint32_t)key;  // H*W < 2^32 is checked on the host
        const int x = (int)row_of(c), y = (int)(c - (uint32_t)x * (uint32_t)W);
        return h_at(x, y);
    }
    __device__ __forceinline__ uint64_t h_at(int x, int y) const {
        const int dx = abs(x - ex), dy = abs(y - ey);
        const int mn = min(dx, dy), mx = max(dx, dy);
        return ((uint64_t)(mx - mn) << 32) | (uint64_t)mn;
    }
    __device__ __forceinline__ uint64_t f_of(uint64_t key, uint64_t g, uint32_t) const {
        return g + h_of(key);  // field-wise: both halves stay below 2^31
    }

    // Open bits of the cells (r, y-1), (r, y), (r, y+1) as bits 0..2 (0 for a
    // row or column outside the grid).  Two 32-bit words cover the three
    // cells, and their addresses depend on the cell alone, so the three rows
    // of a node are read in one round trip of independent loads (look_begin)
    // and taken apart later (look_rows).
    struct Look {
        uint64_t v[3];
    };
    __device__ __forceinline__ uint64_t row_words(int r, int y) const {
        const int64_t c0 = (int64_t)r * W + y - 1;  // cell (r, y-1); -1 only for (0, 0)
        const uint64_t lo = c0 < 0 ? 0 : (uint64_t)c0;
        const uint64_t wlast = ((uint64_t)(uint32_t)H * (uint32_t)W + 63) / 64 * 2 - 1;  // last 32-bit word
        const uint64_t w0 = lo >> 5, w1 = w0 + 1 <= wlast ? w0 + 1 : wlast;
        return (uint64_t)__ldg(bm + w0) | ((uint64_t)__ldg(bm + w1) << 32);
    }
    __device__ __forceinline__ uint32_t row_bits(uint64_t v, int r, int y) const {
        if (r < 0 || r >= H) return 0;
        const int64_t c0 = (int64_t)r * W + y - 1;
        const uint64_t lo = c0 < 0 ? 0 : (uint64_t)c0;
        uint32_t bits = (uint32_t)(v >> (lo & 31u)) & 7u;
        if (c0 < 0) bits = (bits << 1) & 7u;  // the window starts one cell before the grid
        if (y == 0) bits &= ~1u;              // (r, -1) is no cell
        if (y == W - 1) bits &= ~4u;          // (r, W) is no cell (the next row's first)
        return bits;
    }
    __device__ __forceinline__ void look_begin(int x, int y, Look &k) const {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int r = x - 1 + i;
            k.v[i] = r < 0 || r >= H ? 0 : row_words(r, y);
        }
    }

    // Valid moves of a cell, bit i = direction i (4 straight, then 4
    // diagonal; src/utils.hpp:120-122).  Only an open cell moves
    // (CPU-solver.cpp:98-100).  A move into a blocked cell is legal in the
    // reference but such a cell has no out-moves, so it is generated only
    // when it is the goal: no path cost changes.
    __device__ __forceinline__ uint32_t rows_moves(int x, int y, const Look &k) const {
        const uint32_t rows[3] = {row_bits(k.v[0], x - 1, y), row_bits(k.v[1], x, y), row_bits(k.v[2], x + 1, y)};
        if (!(rows[1] & 2u)) return 0;
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int dx = c_dx(i), dy = c_dy(i);
            const bool goal = x + dx == ex && y + dy == ey;
            if (((rows[dx + 1] >> (dy + 1)) & 1u) || goal) m |= 1u << i;
        }
        return m;
    }
    __device__ __forceinline__ uint32_t moves(uint64_t key, uint32_t) const {
        const uint32_t c = (uint32_t)key;
        const int x = (int)row_of(c), y = (int)(c - (uint32_t)x * (uint32_t)W);
        Look k;
        look_begin(x, y, k);
        return rows_moves(x, y, k);
    }
    // Three passes a round, within 1/64 of the straight distance between the
    // query's ends, 1 to 16.  Measured on 20000^2 (distance 28283), hashed:
    // slack 4 / 8 / 16 / 32: 272 / 224 / 215 / 277 ms (narrow: more rounds;
    // wide: every state expanded again); on words: slack 12 / 16 / 24: 107 /
    // 107 / 112, passes 2 / 3 / 4 / 5 / 7 at 16: 108 / 107 / 112 / 115 / 138;
    // six queries on 1537 x 2049 with these passes 14.6 / 13.8 / 14.0 / 15.0 /
    // 16.8 ms; 61 x 67 (distance 84): slack 1 0.21 ms, 8 0.27, 32 0.32.
    __host__ __device__ Expansion expansion(uint32_t) const {
        const int dx = sx < ex ? ex - sx : sx - ex, dy = sy < ey ? ey - sy : sy - ey;
        const int mn = dx < dy ? dx : dy, mx = dx < dy ? dy : dx;
        const float slack = ((float)mx + 0.41421356f * (float)mn) / 64.f;
        return Expansion{3u, ~0u, slack < 1.f ? 1.f : slack > 16.f ? 16.f : slack};
    }
    // Continuation (ga_search): whether this successor is within the bound, and
    // the moves of one that is, reached by move mv (see entry_moves).
    __device__ __forceinline__ bool peek(const Succ &s, float bound) const { return cost_val(s.f) <= bound; }
    __device__ __forceinline__ uint32_t next_moves(const Succ &s, int mv) const {
        Look k;
        look_begin(s.x, s.y, k);
        uint32_t m = rows_moves(s.x, s.y, k);
        if (dirs()) m &= ~pruned((uint32_t)mv);
        return m;
    }
    __device__ __forceinline__ static int c_dx(int i) {
        return i == 0 ? 1 : i == 1 ? -1 : i < 4 ? 0 : (i < 6 ? 1 : -1);
    }
    __device__ __forceinline__ static int c_dy(int i) {
        return i < 2 ? 0 : i == 2 ? 1 : i == 3 ? -1 : ((i & 1) ? -1 : 1);
    }
    // Successor in three steps: its key and g, which its relax needs; the rest
    // (a grid's f, a puzzle's database load) beside the relax's memory trip; and
    // what waits for that load, after it.
    __device__ __forceinline__ void succ_place(uint64_t key, int mv, Succ &s) const {
        const uint32_t c = (uint32_t)key;
        const int x = (int)row_of(c), y = (int)(c - (uint32_t)x * (uint32_t)W);
        s.x = x + c_dx(mv);
        s.y = y + c_dy(mv);
        s.key = (uint64_t)s.x * W + (uint64_t)s.y;
    }
    __device__ __forceinline__ void succ_key(uint64_t key, uint64_t g, int mv, Succ &s) const {
        succ_place(key, mv, s);
        s.g = g + (mv < 4 ? (1ull << 32) : 1ull);
    }
    __device__ __forceinline__ void succ_rest(Succ &s) const { s.f = s.g + h_at(s.x, s.y); }
    __device__ __forceinline__ void succ_end(const Succ &s, uint32_t, int mv, uint32_t &naux, uint64_t &nf) const {
        naux = in_aux(s.key, mv);
        nf = s.f;
    }
    // a successor's entry cell word: its cell and, where it fits, the move
    __device__ __forceinline__ uint32_t in_aux(uint64_t nkey, int mv) const {
        return (uint32_t)nkey | (dirs() ? (uint32_t)mv << kCellBits : 0u);
    }
    __device__ __forceinline__ Entry make_entry(uint64_t f, uint64_t, uint32_t slot, uint32_t aux) const {
        Entry e;
        e.fa = (uint32_t)(f >> 32);
        e.fb = (uint32_t)f;
        e.slot = slot;
        e.cell = aux;
        return e;
    }
    __device__ __forceinline__ static uint64_t entry_cost(const Entry &e) {
        return ((uint64_t)e.fa << 32) | e.fb;
    }
    // Equal f: no preference (a deeper-first tie-break measured no change in
    // expansions or time on the 1000^2 and 20000^2 grids).
    __device__ __forceinline__ static bool less(const Entry &a, const Entry &b) {
        return sqrt2_sign((int32_t)a.fa - (int32_t)b.fa, (int32_t)b.fb - (int32_t)a.fb) < 0;
    }
    __device__ __forceinline__ static Entry load(const Entry *p) {
        const uint4 u = __ldcg(reinterpret_cast<const uint4 *>(p));
        Entry e;
        e.fa = u.x;
        e.fb = u.y;
        e.slot = u.z;
        e.cell = u.w;
        return e;
    }
    __device__ __forceinline__ static void store(Entry *p, const Entry &e) {
        *reinterpret_cast<uint4 *>(p) = make_uint4(e.fa, e.fb, e.slot, e.cell);
    }
    // Node record fields needed at pop time: key and g share the first 16 B.
    __device__ __forceinline__ static void load_node(const Slot *s, const Entry &, uint64_t &key, uint64_t &g,
                                                     uint32_t &aux) {
        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(s));
        key = v.x & 0xffffffffull;
        g = v.y;
        aux = (uint32_t)key;
    }
};

// x with x * odd = 1 modulo 2^64 (Newton's iteration: the correct low bits double).
__host__ __device__ constexpr uint64_t odd_inverse(uint64_t odd) {
    uint64_t x = odd;
    for (int i = 0; i < 6; ++i) x *= 2 - odd * x;
    return x;
}

// A grid search whose table is one 8-byte word per cell instead of hashed
// 16-byte slots: slot = cell, word = g << 3 | the move that reached the cell
// (all ones: unreached).  A relax is then one 64-bit atomicMin, one memory trip
// whatever it finds, where the hashed table's 16-byte CAS takes one to claim
// and two or more to improve or on a collision.  For that a cost has to be one
// number: g = A * 2^40 + B * kDiag for A straight and B diagonal steps, kDiag an
// odd number next to sqrt2 * 2^40.  Sums of costs are exact, (A, B) come back
// from the number (pair) and numbers compare as the costs do while B < 600000:
// two costs with B apart by n differ by at least 1 / (2 sqrt2 n + 1) and the
// number's error in the difference is at most n * 2^-40, less while n (2.83 n
// + 1) < 2^40.  Costs that could reach kLimit (800000, so B < 566000) end the
// search with ST_COST_RANGE, and the hashed search takes the problem over.
// Comparing two costs is one integer compare, and a map's words are no more bytes
// than hashed slots for half of its cells.  Kernels, hashed (32-byte slots) ->
// word: 20000^2 165 -> 103 ms (5.35 -> 3.34 us a step), six queries on 1537 x
// 2049 20.2 -> 13.3 ms, 61 x 67 0.24 -> 0.20 ms, the allocation-free 700 x 1021
// 7.1 -> 4.8 ms.  Still bound by the latency of a step's chain, not by bytes.
struct GridDirect : GridProblem {
    static constexpr bool kDirect = true;
    static constexpr int kFrac = 40;
    static constexpr uint64_t kStraight = 1ull << kFrac, kDiag = 1554944255987ull;
    static constexpr uint64_t kLimit = 800000ull << kFrac;
    // A cost as the pair A << 32 | B.
    __host__ __device__ static uint64_t pair(uint64_t c) {
        if (c == kInfCost) return c;
        constexpr uint64_t inv = odd_inverse(kDiag);
        const uint64_t b = (c * inv) & (kStraight - 1);
        return ((c - b * kDiag) >> kFrac << 32) | b;
    }
    __device__ __forceinline__ static int cost_cmp(uint64_t a, uint64_t b) { return a < b ? -1 : a > b ? 1 : 0; }
    __device__ __forceinline__ static float cost_val(uint64_t c) { return __ull2float_rn(c) * (1.f / (float)kStraight); }
    __device__ __forceinline__ static uint64_t number(uint64_t p) {  // of a cost as a pair
        return (p >> 32 << kFrac) + (uint64_t)(uint32_t)p * kDiag;
    }
    __device__ __forceinline__ uint64_t f_of(uint64_t key, uint64_t g, uint32_t) const { return g + number(h_of(key)); }
    __device__ __forceinline__ bool peek(const Succ &s, float bound) const { return cost_val(s.f) <= bound; }
    __device__ __forceinline__ void succ_key(uint64_t key, uint64_t g, int mv, Succ &s) const {
        succ_place(key, mv, s);
        s.g = g + (mv < 4 ? kStraight : kDiag);
    }
    __device__ __forceinline__ void succ_rest(Succ &s) const { s.f = s.g + number(h_at(s.x, s.y)); }
    __device__ __forceinline__ static bool less(const Entry &a, const Entry &b) { return entry_cost(a) < entry_cost(b); }
    __device__ __forceinline__ static const unsigned long long *words(const Slot *tab) {
        return reinterpret_cast<const unsigned long long *>(tab);
    }
};

// --------------------------------------------------------------- puzzle ---
struct __align__(8) PuzzleEntry {
    uint32_t key;   // min f, then max g: 5x5 f << 16 | (0xFFFF - g), else see PuzzleProblem::make_entry
    uint32_t slot;
};

// Disjoint pattern partitions of the reference (src/puzzle/CPU-solver.hpp:43-70)
// and the mixed-radix multipliers of its rank (src/puzzle/database.cpp:8-25):
// multiple[j] = prod_{i=j}^{k-1} (n*n - i), rank = sum_j v_j * multiple[j+1],
// v_j = cell of tracked tile j minus the number of earlier tracked tiles on
// lower cells (database.cpp:140-163).
template <int N> struct PuzzlePatterns;
template <> struct PuzzlePatterns<3> {
    static constexpr int kNum = 1;
    __host__ __device__ static constexpr int count(int) { return 8; }
    __host__ __device__ static constexpr int tile(int, int j) { return j + 1; }
    __host__ __device__ static constexpr uint64_t offset(int) { return 0; }
};
template <> struct PuzzlePatterns<4> {
    static constexpr int kNum = 2;
    __host__ __device__ static constexpr int count(int p) { return p == 0 ? 8 : 7; }
    __host__ __device__ static constexpr int tile(int p, int j) {
        return p == 0 ? (j < 6 ? j + 1 : (j == 6 ? 9 : 13))
                      : (j < 2 ? j + 7 : (j < 5 ? j + 8 : j + 9));
    }
    __host__ __device__ static constexpr uint64_t offset(int p) { return p == 0 ? 0ull : 518918400ull; }
};

// 5x5: the four 6-tile partitions, in the reference's tracked order (the
// order fixes the rank; src/puzzle/CPU-solver.hpp:71-102).
template <> struct PuzzlePatterns<5> {
    static constexpr int kNum = 4;
    __host__ __device__ static constexpr int count(int) { return 6; }
    __host__ __device__ static constexpr int tile(int p, int j) {
        constexpr int t[4][6] = {{3, 4, 5, 10, 15, 20}, {2, 1, 6, 11, 16, 21}, {7, 8, 9, 12, 17, 22},
                                 {13, 14, 18, 19, 23, 24}};
        return t[p][j];
    }
    __host__ __device__ static constexpr uint64_t offset(int p) { return (uint64_t)p * 127512000ull; }
};

template <int N> __host__ __device__ constexpr uint32_t pattern_mult(int p, int j) {
    // prod_{i=j}^{k-1} (N*N - i)
    uint32_t m = 1;
    for (int i = j; i < PuzzlePatterns<N>::count(p); ++i) m *= (uint32_t)(N * N - i);
    return m;
}
template <int N> __host__ __device__ constexpr int pattern_of_tile(int t) {
    for (int p = 0; p < PuzzlePatterns<N>::kNum; ++p)
        for (int j = 0; j < PuzzlePatterns<N>::count(p); ++j)
            if (PuzzlePatterns<N>::tile(p, j) == t) return p;
    return -1;
}

// the pattern of every tile, 2 bits per tile
template <int N> __host__ __device__ constexpr uint64_t pattern_bits() {
    uint64_t m = 0;
    for (int t = 1; t < N * N; ++t) m |= (uint64_t)pattern_of_tile<N>(t) << (2 * t);
    return m;
}

template <int N> struct PuzzleProblem : NarrowSlots {
    using Entry = PuzzleEntry;
    static constexpr int kMoves = 4;
    static constexpr int NN = N * N;
    // The slot's g word is g << 40 | (last move + 1) << 32 | prev: the relax
    // CAS sets the cost and the path link together, so the push phase checks
    // no winner (a candidate that lost is a stale entry, dropped at its pop).
    // The pattern parts depend on the board alone and travel in its entries
    // (make_entry).
    static constexpr int kLink = LINK_IN_G;
    static constexpr bool kNeedsBound = true;  // see make_entry
    __device__ static KeyG cas_word(uint64_t key, uint64_t g, uint32_t prev, int mv) {
        return KeyG{key, g << 40 | (uint64_t)(uint32_t)(mv + 1) << 32 | prev};
    }
    __device__ static bool word_is(KeyG w, uint64_t key) { return w.key == key; }
    __device__ static uint64_t word_g(KeyG w) { return w.g >> 40; }

    // The key is the board's inverse: nibble t = cell of tile t (tile 0 = the
    // blank), nibbles past the last tile all ones (no cell has that number).
    // Ranks read tiles' cells, so a successor's rank needs no inversion of its
    // board, and a move swaps two nibbles (two tiles trade cells).
    static constexpr uint64_t kPad = NN < 16 ? (~0ull << (4 * (NN < 16 ? NN : 0))) : 0ull;

    const uint8_t *pdb;   // concatenated tables
    uint64_t start;
    uint64_t goal;

    __device__ static int cost_cmp(uint64_t a, uint64_t b) { return a < b ? -1 : (a > b ? 1 : 0); }
    __device__ static float cost_val(uint64_t c) { return (float)c; }

    __host__ __device__ static uint64_t goal_key() {
        uint64_t k = kPad | (uint64_t)(NN - 1);
        for (int t = 1; t < NN; ++t) k |= (uint64_t)(t - 1) << (4 * t);
        return k;
    }
    // Rank of pattern p's tiles (the reference's mixed-radix code in Horner
    // form: digit j counts the cells below tile j's that no earlier tile of
    // the pattern holds).  Both patterns of the 4x4 board take the same
    // instructions, each tile's cell selected by p: lanes of a warp move tiles
    // of both, and the two ranks in diverged branches would add up.
    __device__ __forceinline__ static uint32_t rank(int p, uint64_t key) {
        constexpr int K = PuzzlePatterns<N>::count(0);
        uint32_t used = 0, code = 0, shorter = 0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            uint32_t pos = (uint32_t)(key >> (4 * PuzzlePatterns<N>::tile(0, j))) & 15u;
            if constexpr (PuzzlePatterns<N>::kNum > 1) {
                if (j < PuzzlePatterns<N>::count(1)) {
                    const uint32_t pos1 = (uint32_t)(key >> (4 * PuzzlePatterns<N>::tile(1, j))) & 15u;
                    pos = p ? pos1 : pos;
                }
            }
            code = code * (uint32_t)(NN - j) + pos - __popc(used & ((1u << pos) - 1u));
            used |= 1u << pos;
            if constexpr (PuzzlePatterns<N>::kNum > 1)
                if (j + 1 == PuzzlePatterns<N>::count(1)) shorter = code;
        }
        return PuzzlePatterns<N>::kNum > 1 && p ? shorter : code;
    }
    __device__ __forceinline__ uint32_t part(int p, uint64_t key) const {
        uint32_t off = 0;
        if constexpr (PuzzlePatterns<N>::kNum > 1) off = p ? (uint32_t)PuzzlePatterns<N>::offset(1) : 0u;
        return __ldg(pdb + (off + rank(p, key)));
    }
    // aux = part0 | part1 << 8 | (last move + 1) << 16
    static constexpr uint32_t kLastMoveShift = 16;
    __device__ static uint32_t hsum(uint32_t aux) { return (aux & 0xff) + ((aux >> 8) & 0xff); }

    __device__ uint64_t start_key() const { return start; }
    __device__ uint32_t start_aux() const {
        uint32_t a = part(0, start);
        if (PuzzlePatterns<N>::kNum > 1) a |= part(1, start) << 8;
        return a;
    }
    __device__ bool is_goal(uint64_t key) const { return key == goal; }
    __host__ bool start_is_goal() const { return start == goal; }
    __device__ __forceinline__ uint64_t f_of(uint64_t, uint64_t g, uint32_t aux) const {
        return g + hsum(aux);
    }
    __device__ __forceinline__ static int blank(uint64_t key) { return (int)(key & 15u); }
    // The tile on cell q: the one nibble equal to q (lowest zero nibble of the
    // difference; the test is exact up to the first one).
    __device__ __forceinline__ static int tile_on(uint64_t key, int q) {
        const uint64_t x = key ^ ((uint64_t)q * 0x1111111111111111ull);
        const uint64_t z = (x - 0x1111111111111111ull) & ~x & 0x8888888888888888ull;
        return (__ffsll((long long)z) - 1) >> 2;
    }
    // Blank moves 0..3 = DX/DY[0..3] of src/utils.hpp:120-121.  The move that
    // would undo the parent's move is skipped: it leads back to the parent,
    // whose g is already lower, so it never improves a slot.
    __device__ uint32_t moves(uint64_t key, uint32_t aux) const {
        const int b = blank(key), bx = b / N, by = b % N;
        uint32_t m = 0;
        if (bx + 1 < N) m |= 1u;
        if (bx > 0) m |= 2u;
        if (by + 1 < N) m |= 4u;
        if (by > 0) m |= 8u;
        const uint32_t last = aux >> 16;
        if (last) m &= ~(1u << ((last - 1) ^ 1));
        return m;
    }
    // Successor in three steps (see GridProblem): the board; the load of the
    // moved tile's pattern entry; and what follows from it, aux and f.
    struct Succ {
        uint64_t key, g;
        uint32_t part;  // the loaded pattern entry
        uint32_t which; // its pattern
    };
    static constexpr uint64_t kPatternOf = pattern_bits<N>();
    __device__ __forceinline__ void succ_key(uint64_t key, uint64_t g, int mv, Succ &s) const {
        const int b = blank(key);
        const int q = b + (mv == 0 ? N : mv == 1 ? -N : mv == 2 ? 1 : -1);
        const int t = tile_on(key, q);
        const uint64_t swap = (uint64_t)(b ^ q);  // tile t and the blank trade cells
        s.key = key ^ swap ^ (swap << (4 * t));
        s.g = g + 1;
        s.which = (uint32_t)(kPatternOf >> (2 * t)) & 3u;
    }
    __device__ __forceinline__ void succ_rest(Succ &s) const { s.part = part((int)s.which, s.key); }
    __device__ __forceinline__ void succ_end(const Succ &s, uint32_t aux, int mv, uint32_t &naux,
                                             uint64_t &nf) const {
        uint32_t a = aux & 0xffffu;
        if (s.which == 0)
            a = (a & 0xff00u) | s.part;
        else
            a = (a & 0x00ffu) | (s.part << 8);
        naux = a | ((uint32_t)(mv + 1) << 16);
        nf = s.g + hsum(naux);
    }
    // An 8-puzzle's search never fills the heaps: many passes, least f first
    // (four boards: 0.70 ms without, 0.44 / 0.36 / 0.31 with 1 / 2 / 4 passes).
    // A 15-puzzle does within ~25 rounds, and then a pass more is a longer round
    // of the same expansions (60-move board: 6.2 ms without, 7.5 with two
    // throughout, 6.3 with two while less than a quarter of the heaps pop); a
    // slack of two f levels (4), since a strict order leaves most heaps idle
    // (eight boards 16.3 ms against 19.0 with the least f only).
    __host__ __device__ Expansion expansion(uint32_t k) const {
        return N == 3 ? Expansion{4u, ~0u, 0.5f} : Expansion{2u, k / 4u, 4.f};
    }
    // Continuation (see GridProblem): f is known only once the pattern entry
    // has arrived (ga_search tests it then), and the moves follow from the
    // board alone.
    __device__ __forceinline__ bool peek(const Succ &, float) const { return true; }
    __device__ __forceinline__ uint32_t next_moves(const Succ &s, int mv) const {
        return moves(s.key, (uint32_t)(mv + 1) << kLastMoveShift);
    }
    static constexpr bool kEntryKey = false;
    // f in 10 bits, 255 - g in 8 from bit 14 on, the first pattern's part in the
    // low 8: with h = f - g it gives the second's, so a slot needs no more than
    // its CAS word.  g fits because every board searched is solvable and the
    // search bounded: it expands nothing whose f is above the optimum (80 moves at
    // most on 4x4, 208 on 5x5, where the slot has 8 bits for g) plus the slack.
    // ga_search refuses a puzzle without a bound.
    __device__ __forceinline__ Entry make_entry(uint64_t f, uint64_t g, uint32_t slot, uint32_t aux) const {
        Entry e;
        e.key = (uint32_t)f << 22 | (255u - (uint32_t)g) << 14 | (aux & 0xffu);
        e.slot = slot;
        return e;
    }
    __host__ __device__ __forceinline__ static uint64_t entry_cost(const Entry &e) { return e.key >> 22; }
    __device__ __forceinline__ static bool less(const Entry &a, const Entry &b) { return a.key < b.key; }
    __device__ __forceinline__ static Entry load(const Entry *p) {
        const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(p));
        Entry e;
        e.key = u.x;
        e.slot = u.y;
        return e;
    }
    __device__ __forceinline__ static void store(Entry *p, const Entry &e) {
        *reinterpret_cast<uint2 *>(p) = make_uint2(e.key, e.slot);
    }
    __device__ __forceinline__ static void load_node(const Slot *s, const Entry &e, uint64_t &key, uint64_t &g,
                                                     uint32_t &aux) {
        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(s));
        key = v.x;
        g = v.y >> 40;
        const uint32_t part0 = e.key & 0xffu, h = (e.key >> 22) - (255u - ((e.key >> 14) & 0xffu));
        aux = part0 | (h - part0) << 8 | ((uint32_t)(v.y >> 32) & 0xffu) << kLastMoveShift;
    }
};

// ------------------------------------------------------- 24-puzzle ---
// 5x5 board, 128-bit key: the cells of tiles 0 (the blank) .. 11 in `lo` and
// 12 .. 23 in `hi`, 5 bits each; tile 24's cell is implied (the cells sum to
// 300), so every state has one key and bits 60..63 of both words are left for g
// (WideSlots; the all-ones empty key is never a board).  With g in the CAS that
// claims the key, a relax of a new board takes one memory trip instead of two
// and of an old one two instead of three: a step of three boards of 60 random
// moves 7.2 / 7.9 / 5.3 -> 5.9 / 6.9 / 4.5 us.  aux = the four pattern parts, 7
// bits each, | (last move + 1) << 28.
template <> struct PuzzleProblem<5> : WideSlots {
    using Entry = PuzzleEntry;
    static constexpr int kMoves = 4;
    static constexpr int N = 5;
    static constexpr int NN = 25;
    static constexpr bool kNeedsBound = true;  // 8 bits of g (PuzzleProblem::make_entry)
    static constexpr uint64_t kFieldLow = 0x0084210842108421ull;  // bit 0 of each of 12 fields

    const uint8_t *pdb;  // four concatenated tables
    Key128 start;
    Key128 goal;

    __device__ static int cost_cmp(uint64_t a, uint64_t b) { return a < b ? -1 : (a > b ? 1 : 0); }
    __device__ static float cost_val(uint64_t c) { return (float)c; }

    // sum of the 12 fields of a word
    __host__ __device__ static uint32_t field_sum(uint64_t w) {
        constexpr uint64_t even = 0x007c1f07c1f07c1full;  // fields 0, 2, .. 10
        const uint64_t s = (w & even) + ((w >> 5) & even);  // six sums, 10 bits apart
        const uint64_t t = s + (s >> 30);                   // three of them
        return (uint32_t)((t & 1023u) + (t >> 10 & 1023u) + (t >> 20 & 1023u));
    }
    // cell of tile t
    __host__ __device__ static uint32_t cell(const Key128 &k, int t) {
        if (t < 12) return (uint32_t)(k.lo >> (5 * t)) & 31u;
        if (t < 24) return (uint32_t)(k.hi >> (5 * (t - 12))) & 31u;
        return 300u - field_sum(k.lo) - field_sum(k.hi);
    }
    __host__ __device__ static Key128 pack(const uint8_t *tiles) {
        Key128 k{0, 0};
        for (int i = 0; i < 25; ++i) {
            const int t = tiles[i];
            if (t < 12)
                k.lo |= (uint64_t)i << (5 * t);
            else if (t < 24)
                k.hi |= (uint64_t)i << (5 * (t - 12));
            // tile 24 is implied
        }
        return k;
    }
    __host__ __device__ static Key128 goal_key() {
        uint8_t tiles[25] = {};
        for (int i = 0; i < 24; ++i) tiles[i] = (uint8_t)(i + 1);
        return pack(tiles);
    }
    __device__ __forceinline__ static int blank(const Key128 &k) { return (int)((uint32_t)k.lo & 31u); }
    // index of the field of a 60-bit word equal to q (12 if none)
    __device__ __forceinline__ static int field_of(uint64_t w, int q) {
        const uint64_t x = w ^ ((uint64_t)q * kFieldLow);
        const uint64_t z = (x - kFieldLow) & ~x & (kFieldLow << 4);
        return z ? (__ffsll((long long)z) - 1) / 5 : 12;
    }
    __device__ __forceinline__ static int tile_on(const Key128 &k, int q) {
        const int a = field_of(k.lo, q);
        return a < 12 ? a : 12 + field_of(k.hi, q);  // 24 if neither word names the cell
    }
    // Rank of pattern p's six tiles (see PuzzleProblem::rank); the tile's cell
    // is selected by p, so that the lanes of a warp rank their four patterns
    // together.
    __device__ __forceinline__ static uint32_t rank(int p, const Key128 &k) {
        uint32_t used = 0, code = 0;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const uint32_t c0 = cell(k, PuzzlePatterns<5>::tile(0, j)), c1 = cell(k, PuzzlePatterns<5>::tile(1, j));
            const uint32_t c2 = cell(k, PuzzlePatterns<5>::tile(2, j)), c3 = cell(k, PuzzlePatterns<5>::tile(3, j));
            const uint32_t pos = p < 2 ? (p == 0 ? c0 : c1) : (p == 2 ? c2 : c3);
            code = code * (uint32_t)(NN - j) + pos - __popc(used & ((1u << pos) - 1u));
            used |= 1u << pos;
        }
        return code;
    }
    __device__ __forceinline__ uint32_t part(int p, const Key128 &k) const {
        return __ldg(pdb + ((uint32_t)p * (uint32_t)PuzzlePatterns<5>::offset(1) + rank(p, k)));
    }
    // aux = four 7-bit pattern parts | (last move + 1) << 28
    static constexpr uint32_t kLastMoveShift = 28;
    __device__ static uint32_t hsum(uint32_t aux) {
        return (aux & 127u) + ((aux >> 7) & 127u) + ((aux >> 14) & 127u) + ((aux >> 21) & 127u);
    }

    __device__ Key128 start_key() const { return start; }
    __device__ uint32_t start_aux() const {
        return part(0, start) | part(1, start) << 7 | part(2, start) << 14 | part(3, start) << 21;
    }
    __device__ bool is_goal(const Key128 &k) const { return k.lo == goal.lo && k.hi == goal.hi; }
    __host__ bool start_is_goal() const { return start.lo == goal.lo && start.hi == goal.hi; }
    __device__ __forceinline__ uint64_t f_of(const Key128 &, uint64_t g, uint32_t aux) const { return g + hsum(aux); }
    // Blank moves 0..3 = DX/DY[0..3]; the move undoing the parent's is skipped.
    __device__ uint32_t moves(const Key128 &k, uint32_t aux) const {
        const int b = blank(k), bx = b / N, by = b % N;
        uint32_t m = 0;
        if (bx + 1 < N) m |= 1u;
        if (bx > 0) m |= 2u;
        if (by + 1 < N) m |= 4u;
        if (by > 0) m |= 8u;
        const uint32_t last = aux >> 28;
        if (last) m &= ~(1u << ((last - 1) ^ 1));
        return m;
    }
    struct Succ {
        Key128 key;
        uint64_t g;
        uint32_t part;   // the moved tile's pattern entry
        uint32_t which;  // its pattern
    };
    static constexpr uint64_t kPatternOf = pattern_bits<5>();
    __device__ __forceinline__ void succ_key(const Key128 &key, uint64_t g, int mv, Succ &s) const {
        const int b = blank(key);
        const int q = b + (mv == 0 ? N : mv == 1 ? -N : mv == 2 ? 1 : -1);
        const int t = tile_on(key, q);
        const uint64_t swap = (uint64_t)(b ^ q);  // tile t and the blank trade cells
        s.key.lo = key.lo ^ swap ^ (t < 12 ? swap << (5 * t) : 0ull);
        s.key.hi = key.hi ^ (t >= 12 && t < 24 ? swap << (5 * (t - 12)) : 0ull);
        s.g = g + 1;
        s.which = (uint32_t)(kPatternOf >> (2 * t)) & 3u;
    }
    __device__ __forceinline__ void succ_rest(Succ &s) const { s.part = part((int)s.which, s.key); }
    __device__ __forceinline__ void succ_end(const Succ &s, uint32_t aux, int mv, uint32_t &naux,
                                             uint64_t &nf) const {
        const uint32_t sh = 7u * s.which;
        uint32_t a = (aux & 0x0fffffffu & ~(127u << sh)) | (s.part << sh);
        naux = a | ((uint32_t)(mv + 1) << 28);
        nf = s.g + hsum(naux);
    }
    // (three boards of 60 random moves: 1.51 ms without, 1.09 ms)
    __host__ __device__ Expansion expansion(uint32_t k) const { return Expansion{2u, k / 4u, 4.f}; }
    // Continuation (see GridProblem): f is known only once the pattern entry
    // has arrived (ga_search tests it then), and the moves follow from the
    // board alone.
    __device__ __forceinline__ bool peek(const Succ &, float) const { return true; }
    __device__ __forceinline__ uint32_t next_moves(const Succ &s, int mv) const {
        return moves(s.key, (uint32_t)(mv + 1) << 28);
    }
    static constexpr bool kEntryKey = false;
    __device__ __forceinline__ Entry make_entry(uint64_t f, uint64_t g, uint32_t slot, uint32_t) const {
        Entry e;
        e.key = ((uint32_t)f << 16) | (0xffffu - (uint32_t)g);
        e.slot = slot;
        return e;
    }
    __host__ __device__ __forceinline__ static uint64_t entry_cost(const Entry &e) { return e.key >> 16; }
    __device__ __forceinline__ static bool less(const Entry &a, const Entry &b) { return a.key < b.key; }
    __device__ __forceinline__ static Entry load(const Entry *p) {
        const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(p));
        Entry e;
        e.key = u.x;
        e.slot = u.y;
        return e;
    }
    __device__ __forceinline__ static void store(Entry *p, const Entry &e) {
        *reinterpret_cast<uint2 *>(p) = make_uint2(e.key, e.slot);
    }
    __device__ __forceinline__ static void load_node(const Slot *s, const Entry &, Key128 &key, uint64_t &g,
                                                     uint32_t &aux) {
        const KeyG v = cas_half(s);
        key = word_key(v);
        g = word_g(v);
        aux = __ldcg(&w(s)->aux);
    }
};

}  // namespace uastar
