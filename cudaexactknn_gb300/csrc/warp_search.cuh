// One query per warp: exact depth-first search of a k-d or ball tree, the 32 lanes testing 32
// descendants (five levels down) of a node at once and scanning 32 leaf slots at once.
//
// Why a warp per query: a thread per query leaves most lanes idle as neighbouring queries' paths
// part, keeps its top-k in a chain of compares (or local memory) and needs tens of thousands of
// queries before every SM has work.  Here every load of a step is in flight at once, no lane
// waits for another query, the top-k is one key per lane and rank, and a few thousand queries
// already fill the GPU.
//
// The search.  The tree is cut into steps of five levels (the first step takes the remainder), the
// last one ending at the buckets: subtrees of `bucket` slots.  A step's row holds, one per lane, a
// lower bound for each of the up-to-32 descendants; the best one whose bound is within the k-th
// distance is entered next (nearest first, chosen by a warp-wide minimum), and a row with none
// left is done.  A row waits in shared memory while the search is below it, so the state is one
// row per step (at most 7) and never overflows.  At the last step the nearest buckets are scanned
// together, 32 slots at a time.  A subtree is skipped only when its bound exceeds the k-th
// distance, so ties are kept: the answer is brute force's.
#pragma once

#include <type_traits>

#include "tree_query.cuh"

namespace knn {

constexpr uint32_t kWarpFan = 5;    // levels per step: up to 32 descendants, one per lane
constexpr uint32_t kWarpRows = 7;   // steps of a tree of at most 32 levels
constexpr uint32_t kFullMask = 0xFFFFFFFFu;
constexpr uint32_t kWarpsPerBlock = 2;  // queries of a block (4: 2% slower, 8: 5%, as a block waits for its slowest)
constexpr size_t kMaxBlockSmem = 232448;      // most shared memory a block can ask for
constexpr size_t kL2Bytes = 128u << 20;       // this GPU's L2
constexpr uint32_t kWarpOrderMin = 1u << 18;  // fewest queries worth an order on an index beyond L2

__device__ __forceinline__ uint64_t shfl_xor64(uint64_t v, uint32_t m) {
    const uint32_t lo = __shfl_xor_sync(kFullMask, static_cast<uint32_t>(v), m);
    const uint32_t hi = __shfl_xor_sync(kFullMask, static_cast<uint32_t>(v >> 32), m);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

__device__ __forceinline__ uint64_t shfl64(uint64_t v, uint32_t src) {
    const uint32_t lo = __shfl_sync(kFullMask, static_cast<uint32_t>(v), src);
    const uint32_t hi = __shfl_sync(kFullMask, static_cast<uint32_t>(v >> 32), src);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

__device__ __forceinline__ uint64_t shfl_up64(uint64_t v) {
    const uint32_t lo = __shfl_up_sync(kFullMask, static_cast<uint32_t>(v), 1);
    const uint32_t hi = __shfl_up_sync(kFullMask, static_cast<uint32_t>(v >> 32), 1);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Ascending bitonic sort of 32 keys, one per lane.
__device__ __forceinline__ uint64_t warp_sort64(uint64_t v, uint32_t lane) {
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const uint64_t o = shfl_xor64(v, j);
            const bool up = (lane & k) == 0, lower = (lane & j) == 0;
            v = (lower == up) ? (v < o ? v : o) : (v < o ? o : v);
        }
    }
    return v;
}

// Ascending order of a bitonic sequence of 32 keys, one per lane.
__device__ __forceinline__ uint64_t warp_bitonic_merge64(uint64_t v, uint32_t lane) {
#pragma unroll
    for (uint32_t j = 16; j > 0; j >>= 1) {
        const uint64_t o = shfl_xor64(v, j);
        v = (lane & j) == 0 ? (v < o ? v : o) : (v < o ? o : v);
    }
    return v;
}

// The k smallest keys seen, ascending over (register, lane): rank r is register r / 32 of lane r % 32.
// KR = 1 takes k <= 32, 2 k in (32, 64], 4 k in (64, 128].
template <int KR>
struct WarpTopK {
    uint64_t v[KR];
    uint64_t kth;   // key at rank k - 1, in every lane
    uint32_t k, lane;
    bool empty;     // nothing inserted yet

    __device__ __forceinline__ void init(uint32_t k_, float r2, uint32_t lane_) {
        k = k_;
        lane = lane_;
        kth = make_key(r2, -1);
        empty = true;
#pragma unroll
        for (int j = 0; j < KR; ++j) v[j] = kth;
    }
    __device__ __forceinline__ float radius() const { return key_dist(kth); }
    __device__ __forceinline__ void refresh() {
        // (Rank k - 1 is in the last register, or with four in the third: k > 16 KR beyond 32.)
        kth = shfl64(KR == 4 && k <= 96 ? v[KR - 2 + (KR == 1)] : v[KR - 1], (k - 1) & 31u);
    }
    // Inserts a key every lane holds.
    __device__ __forceinline__ void insert(uint64_t x) {
        uint64_t carry = 0;  // the key of the rank before lane 0's (below every key at rank 0)
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            uint64_t up = shfl_up64(v[j]);
            const uint64_t next = KR > 1 ? shfl64(v[j], 31) : 0;
            if (lane == 0) up = carry;
            const uint64_t put = up > x ? up : x;
            v[j] = v[j] > x ? put : v[j];
            carry = next;
        }
    }
    // Offers one key per lane (where `cand`): few are inserted one by one, more are sorted and merged.
    __device__ __forceinline__ void offer(bool cand, uint64_t key) {
        uint32_t m = __ballot_sync(kFullMask, cand && key < kth);
        if (!m) return;
        if (__popc(m) <= (KR == 1 ? 8 : 6)) {
            do {
                insert(shfl64(key, static_cast<uint32_t>(__ffs(m) - 1)));
                m &= m - 1u;
            } while (m);
        } else {
            uint64_t x = warp_sort64((m >> lane) & 1u ? key : ~0ull, lane);
            if (empty) {
                v[0] = v[0] < x ? v[0] : x;
            } else {
#pragma unroll
                for (int j = 0; j < KR; ++j) {
                    const uint64_t rx = shfl64(x, 31 - lane);
                    const uint64_t lo = v[j] < rx ? v[j] : rx, hi = v[j] < rx ? rx : v[j];
                    v[j] = warp_bitonic_merge64(lo, lane);
                    if (j + 1 < KR) x = warp_bitonic_merge64(hi, lane);
                }
            }
        }
        empty = false;
        refresh();
    }
    __device__ __forceinline__ void emit_keys(uint64_t* __restrict__ out) const {
#pragma unroll
        for (int j = 0; j < KR; ++j)
            if (32u * j + lane < k) out[32u * j + lane] = v[j];
    }
    __device__ __forceinline__ void emit(int32_t* __restrict__ idx, float* __restrict__ dist) const {
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            const uint32_t r = 32u * j + lane;
            if (r < k) {
                idx[r] = key_index(v[j]);
                dist[r] = key_dist(v[j]);
            }
        }
    }
};

// Groups of four dimensions a search of `dims` dimensions padded to dp reads: known at compile time
// up to 32 dims (3 or 4 of 16, 6 or 8 of 32: a loop that ends early instead kept the loads from being
// in flight together, 4.5 against 3.6 ms at 16 dims), counted at run time beyond.  (500,000 uniform 11-d
// points, 10,000 queries: 1.81 ms with 3, 2.0 with 4.)
__host__ __device__ constexpr int warp_quads(int dp, int dims) {
    return dp == 16 ? (dims <= 12 ? 3 : 4) : dp == 32 ? (dims <= 24 ? 6 : 8) : (dp + 3) / 4;
}
template <int DP, class F>
void with_quads(uint32_t dims, F&& f) {
    constexpr int kLess = warp_quads(DP, DP == 16 ? 12 : DP == 32 ? 24 : DP), kAll = warp_quads(DP, DP);
    if (kLess != kAll && warp_quads(DP, static_cast<int>(dims)) == kLess) f(std::integral_constant<int, kLess>{});
    else f(std::integral_constant<int, kAll>{});
}

// Shared memory of one warp: the waiting rows (bounds; where the tree's visit order is not the
// bound's, order keys; and for a seeded search over balls the bounds as they were tested).
template <bool KEYS>
struct WarpRows {
    float bound[kWarpRows][32];
    uint32_t key[KEYS ? kWarpRows : 1][32];
    float tested[KEYS ? kWarpRows : 1][32];
};

struct WarpTree {
    const float* leaf;
    uint32_t leaf_stride, bucket, stop;  // bucket slots (a power of two), depth of the buckets
};

// Searches one query with the whole warp, within r2.  View::test(node, &bound, &key) gives a node's
// lower bound and its visit order (smaller first); View::dist(slot, &id) a slot's distance.  `lc`
// counts the nodes whose bound was within the radius when tested, the buckets and the slots scanned
// (uniform over the warp).
//
// SEEDED: subtrees are first entered only within r < r2 as well (scanned slots are offered all the
// same).  A row left behind keeps its least remaining bound in its parent's, so that a seed that held
// fewer than k points costs no second search: r goes to r2 and the search goes on from there, past the
// buckets it has scanned.  (A ball's bound can be below its parent's: which buckets were scanned is
// told by the largest bound on their path, `tested`.)  Returns whether it had to.
template <class View, int KR, bool SEEDED>
__device__ __forceinline__ bool warp_search(const View& view, const WarpTree& t, WarpRows<View::kKeys>& sm,
                                            WarpTopK<KR>& top, LocalCounters& lc, float r, float r2) {
    const uint32_t lane = top.lane;
    const uint32_t steps = t.stop ? (t.stop + kWarpFan - 1) / kWarpFan : 1u;
    const uint32_t lv0 = t.stop - kWarpFan * (steps - 1);  // levels of the first step (0: the root is a bucket)
    uint32_t row = 0, par = 0, depth = lv0, lv = lv0;      // par: index, within its depth, of the row's parent
    float bound = __int_as_float(0x7fc00000);              // NaN: never within a radius (absent, or taken)
    uint32_t key = 0;
    constexpr bool kTrack = SEEDED && View::kKeys;
    float tested = 0.0f, above = 0.0f;                     // kTrack: this lane's path bound, the row's parent's
    float scanned = -1.0f;                                 // SEEDED: buckets within this are done
    auto radius = [&]() { return SEEDED ? fminf(r, top.radius()) : top.radius(); };
    auto expand = [&]() {
        bound = __int_as_float(0x7fc00000);
        if (lane < (1u << lv)) view.test((1u << depth) - 1u + (par << lv) + lane, &bound, &key);
        if (kTrack && bound < above) bound = above;
        tested = bound;
        if (SEEDED && row + 1 == steps && bound <= scanned) bound = __int_as_float(0x7fc00000);
        lc.nodes += __popc(__ballot_sync(kFullMask, bound <= radius()));
    };
    // Takes the row's best descendant within the k-th distance; false when there is none.
    auto take = [&](uint32_t* child) -> bool {
        const bool want = bound <= radius();
        uint32_t m = __ballot_sync(kFullMask, want);
        if (!m) return false;
        if (m & (m - 1u)) {
            const uint32_t k = View::kKeys ? key : __float_as_uint(bound);
            const uint32_t best = __reduce_min_sync(kFullMask, want ? k : kFullMask);
            m = __ballot_sync(kFullMask, want && k == best);
        }
        const uint32_t src = static_cast<uint32_t>(__ffs(m) - 1);
        if constexpr (kTrack) above = __shfl_sync(kFullMask, tested, src);
        if (lane == src) bound = __int_as_float(0x7fc00000);
        *child = (par << lv) + src;
        return true;
    };
    expand();
    for (;;) {
        uint32_t child;
        if (!take(&child)) {
            if (row == 0) {
                if (!SEEDED || !(r < r2) || !(r < top.radius())) return SEEDED && scanned >= 0.0f;
                scanned = r;
                r = r2;
                continue;
            }
            uint32_t rest = 0;
            if constexpr (SEEDED) rest = __reduce_min_sync(kFullMask, __float_as_uint(bound));
            --row;
            lv = row ? kWarpFan : lv0;
            const uint32_t src = par & ((1u << lv) - 1u);
            par >>= lv;
            depth -= kWarpFan;
            bound = sm.bound[row][lane];
            if (SEEDED && lane == src) bound = __uint_as_float(rest);
            if constexpr (View::kKeys) key = sm.key[row][lane];
            if constexpr (kTrack) tested = sm.tested[row][lane];
            continue;
        }
        if (row + 1 < steps) {
            sm.bound[row][lane] = bound;
            if constexpr (View::kKeys) sm.key[row][lane] = key;
            if constexpr (kTrack) sm.tested[row][lane] = tested;
            ++row;
            par = child;
            lv = kWarpFan;
            depth += kWarpFan;
            expand();
            continue;
        }
        // Buckets: as many of the nearest as 32 lanes hold, or one of more slots in several passes.
        ++lc.leaves;
        if (t.bucket >= 32) {
            for (uint32_t s = lane; s < t.bucket; s += 32) {
                int32_t id;
                const float d2 = view.dist(t.leaf + (static_cast<size_t>(child) * t.bucket + s) * t.leaf_stride, &id);
                lc.points += 32;
                top.offer(id >= 0, make_key(d2, id));
            }
        } else {
            uint32_t mine = child, filled = 1;
            const uint32_t groups = 32 / t.bucket, g = lane / t.bucket;
            while (filled < groups && take(&child)) {
                if (g >= filled) mine = child;
                ++filled;
                ++lc.leaves;
            }
            int32_t id = -1;
            float d2 = 0.0f;
            if (g < filled)
                d2 = view.dist(t.leaf + (static_cast<size_t>(mine) * t.bucket + (lane & (t.bucket - 1u))) * t.leaf_stride, &id);
            lc.points += filled * t.bucket;
            top.offer(id >= 0, make_key(d2, id));
        }
    }
}

}  // namespace knn
