// Ball tree query kernels, one translation unit per padded dimension count (KNN_DP).
//
// Replaces BallTreeKernels::knnDevice and its four storage variants (src/BallTreeGpu.cuh:36-200),
// a depth-first search per thread: at each internal node the distance to both child balls, the closer
// one entered, the farther one pushed when it can still hold a neighbour (src/BallTreeGpu.cuh:82-92).
// Here each query gets a warp (ball_warp_query_kernel, warp_search.cuh), or a thread where very many
// queries have very few dims (ball_knn_kernel); traversal 1 walks 32 neighbouring queries together.
// The reference's border distance sqrt(d2) - r (with -use_fast_math's approximate sqrt) can
// round above a point's own float distance and prune a true neighbour; here knn::ball_bound
// uses directed rounding and relative margins so it never exceeds the float dist2 of any point
// in the ball, and a ball is pruned only when its bound > the k-th distance.

#include <algorithm>
#include <cstring>

#include "tree_query.cuh"
#include "warp_search.cuh"

#ifndef KNN_DP
#error "compile with -DKNN_DP=<padded dims>"
#endif

namespace knn {

struct BallParams {
    const float* ball;     // node i: centre (DP floats), radius at [DP]
    uint32_t ball_stride;
    const float* leaf;
    uint32_t leaf_stride;
    uint32_t node_count;
    uint32_t node_depth;
    uint32_t stop_depth;
    uint32_t leaf_slots;
    float margin;
    const float* queries;
    uint32_t dims;
    uint32_t nq;
    const uint32_t* order;
    const uint32_t* count_dev;
    uint32_t order_base;  // subtracted from order entries (batched orders hold batch-wide ids)
    float max_d2;
    const float* radii;
    const float* seeds;   // warp-per-query search: per query radius to start from (x seed_scale), or null
    float seed_scale;
    uint32_t k;
    int32_t* out_idx;
    float* out_dist;
    DevCounters* counters;
};

// Float dist2 from q to a ball's centre; the radius comes back through *r.
template <int DP>
__device__ __forceinline__ float centre_dist(const float (&q)[DP], const float* __restrict__ b, float* r) {
    if constexpr (DP < 4) {
        const float4 v = *reinterpret_cast<const float4*>(b);
        const float w[4] = {v.x, v.y, v.z, v.w};
        *r = w[DP];
        float acc = 0.0f;
#pragma unroll
        for (int d = 0; d < DP; ++d) {
            const float t = __fsub_rn(q[d], w[d]);
            acc = __fmaf_rn(t, t, acc);
        }
        return acc;
    } else {
        *r = b[DP];
        return dist2_vec4<DP>(q, reinterpret_cast<const float4*>(b));
    }
}

// One thread's search: query slot t of the batch (its query is p.order[t] - p.order_base, or t).
template <int DP, int KMAX>
__device__ __forceinline__ void ball_search_thread(const BallParams& p, uint32_t t, uint2* sh_stack) {
    const uint32_t qi = p.order ? p.order[t] - p.order_base : t;
    float q[DP];
    load_query<DP>(p.queries, p.dims, qi, q);
    const float r2 = p.radii ? p.radii[qi] : p.max_d2;

    Tracker<KMAX, false, false> tr;
    tr.init(p.k, r2, nullptr, 0);
    LevelStack st{sh_stack + threadIdx.x, blockDim.x, p.stop_depth + 1, 0};
    st.push(0, 0.0f);
    LocalCounters lc;
    bool overflow = false;

    while (st.top) {
        uint32_t node;
        float bound;
        st.pop(&node, &bound);
        if (bound > tr.radius()) continue;
        uint32_t depth = heap_depth(node);
        bool within = true;
        // (One condition and no early exit: with one, the compiler had a warp's threads go on apart for
        // 1.5 times the instructions.)
        while (within && depth < p.stop_depth) {
            const uint32_t l = 2 * node + 1;
            float rl, rr;
            const float sl = centre_dist<DP>(q, p.ball + static_cast<size_t>(l) * p.ball_stride, &rl);
            const float sr = centre_dist<DP>(q, p.ball + static_cast<size_t>(l + 1) * p.ball_stride, &rr);
            const float bl = ball_bound(sl, rl, p.margin);
            const float br = ball_bound(sr, rr, p.margin);
            ++lc.nodes;
            const bool left_first = sqrtf(sl) - rl < sqrtf(sr) - rr;
            const float close_b = left_first ? bl : br, far_b = left_first ? br : bl;
            const bool close_in = close_b <= tr.radius(), far_in = far_b <= tr.radius();
            const uint32_t close_child = left_first ? l : l + 1, far_child = left_first ? l + 1 : l;
            if (close_in && far_in) overflow |= !st.push(far_child, far_b);
            node = close_in ? close_child : far_child;
            within = close_in || far_in;
            ++depth;
        }
        if (!within) continue;
        const SlotRange r = subtree_slots(node, depth, p.node_depth, p.node_count, p.leaf_slots);
        const float* slot = p.leaf + r.first * p.leaf_stride;
        ++lc.leaves;
        for (uint32_t s = 0; s < r.count; ++s, slot += p.leaf_stride) {
            int32_t id;
            const float d2 = slot_dist<DP>(q, slot, &id);
            lc.points += id >= 0 ? 1u : 0u;
            tr.offer(id >= 0 ? make_key(d2, id) : ~0ull);
        }
    }
    tr.emit(p.k, p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
    if (p.counters) {
        lc.flush(p.counters);
        if (overflow) atomicExch(&p.counters->error, 1);
    }
}

template <int DP, int KMAX>
__global__ void __launch_bounds__(128) ball_knn_kernel(const BallParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < p.nq) ball_search_thread<DP, KMAX>(p, t, reinterpret_cast<uint2*>(smem));
}

// Warp-coherent variant (see kd_knn_warp_kernel): the warp's queries walk the tree together,
// descending first into the child most still-interested lanes are closer to; each lane's bound
// for a child is max(its inherited bound, its rigorous bound to the child's ball).
// One warp's search over slots t (this lane) of the batch; `live` slots exist.
template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
__device__ __forceinline__ void ball_search_warp(const BallParams& p, uint32_t t, uint32_t live, unsigned char* smem) {
    if ((t & ~31u) >= live) return;
    const bool active = t < live;
    uint64_t* sh_nn = reinterpret_cast<uint64_t*>(smem);
    uint32_t* sh_st = reinterpret_cast<uint32_t*>(smem + tracker_smem_bytes(SHNN, KMAX, blockDim.x));

    const uint32_t qi = active ? (p.order ? p.order[t] - p.order_base : t) : 0u;
    float q[DP];
    load_query<DP>(p.queries, p.dims, qi, q);
    const float r2 = active ? (p.radii ? p.radii[qi] : p.max_d2) : 0.0f;

    Tracker<KMAX, HEAP, SHNN> tr;
    tr.init(p.k, r2, sh_nn + threadIdx.x, blockDim.x);
    Stack<SHST> st;
    st.init(sh_st, blockDim.x);
    st.push(0, active ? 0.0f : INFINITY);
    LocalCounters lc;
    bool overflow = false;

    while (st.top) {
        uint32_t node;
        float bound;
        st.pop(&node, &bound);
        if (!__any_sync(0xFFFFFFFFu, bound <= tr.radius())) continue;
        uint32_t depth = heap_depth(node);
        bool pruned = false;
        while (depth < p.stop_depth) {
            const uint32_t l = 2 * node + 1;
            float rl, rr;
            const float sl = centre_dist<DP>(q, p.ball + static_cast<size_t>(l) * p.ball_stride, &rl);
            const float sr = centre_dist<DP>(q, p.ball + static_cast<size_t>(l + 1) * p.ball_stride, &rr);
            const float bl = fmaxf(bound, ball_bound(sl, rl, p.margin));
            const float br = fmaxf(bound, ball_bound(sr, rr, p.margin));
            const bool want = bound <= tr.radius();
            const bool left_near = sqrtf(sl) - rl < sqrtf(sr) - rr;
            const uint32_t left_votes = __popc(__ballot_sync(0xFFFFFFFFu, want && left_near));
            const uint32_t right_votes = __popc(__ballot_sync(0xFFFFFFFFu, want && !left_near));
            const bool first_left = left_votes >= right_votes;
            const float b_first = first_left ? bl : br;
            const float b_second = first_left ? br : bl;
            ++lc.nodes;
            if (__any_sync(0xFFFFFFFFu, b_second <= tr.radius())) overflow |= !st.push(first_left ? l + 1 : l, b_second);
            node = first_left ? l : l + 1;
            bound = b_first;
            ++depth;
            if (!__any_sync(0xFFFFFFFFu, bound <= tr.radius())) {
                pruned = true;
                break;
            }
        }
        if (pruned) continue;
        const SlotRange r = subtree_slots(node, depth, p.node_depth, p.node_count, p.leaf_slots);
        const float* slot = p.leaf + r.first * p.leaf_stride;
        const bool want = bound <= tr.radius();
        lc.leaves += want ? 1u : 0u;
        for (uint32_t s = 0; s < r.count; ++s, slot += p.leaf_stride) {
            int32_t id;
            const float d2 = slot_dist<DP>(q, slot, &id);
            if (id < 0) continue;
            if (want) {
                ++lc.points;
                tr.offer(make_key(d2, id));
            }
        }
    }
    if (!active) return;
    tr.emit(p.k, p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
    if (p.counters) {
        lc.flush(p.counters);
        if (overflow) atomicExch(&p.counters->error, 1);
    }
}

template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
__global__ void __launch_bounds__(256) ball_knn_warp_kernel(const BallParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t live = p.count_dev ? *p.count_dev : p.nq;
    ball_search_warp<DP, KMAX, HEAP, SHNN, SHST>(p, t, live, smem);
}

// One query per warp (warp_search.cuh) over the balls: a node's bound is its ball's, the visit order
// the distance to the ball's border (overlapping balls have equal bounds of zero).  65,536 queries, k
// 32, on 262,144 points near a 4-d subspace of 16 dims: 3.7 ms (a thread per query with its stack and
// top-k in local memory: 15.6; 4,000 uniform 32-d queries, k 64, on 30,000: 3.4 and 177).  Bound by the
// L1 reads of balls and slots, about 10,000 rows of 80 bytes per query there: each lane reads its own
// row, a line per lane and 16 bytes.  (Rows staged through shared memory by coalesced asynchronous
// copies: 5.3 ms, as the staging takes the room in which L1 keeps the rows.)
template <int DP, int NQ>
struct BallWarpView {
    static constexpr bool kKeys = true;
    static constexpr bool kShared = DP > 32;  // wide queries are read from shared memory (broadcast)
    float q[kShared ? 1 : DP];
    const float4* sq;
    const float* ball;
    uint32_t ball_stride, quads;  // quads: groups of four dimensions in use (NQ where known at compile time)
    float margin;
    __device__ __forceinline__ float dist2_to(const float* row, float* last) const {
        if constexpr (kShared) {
            *last = row[DP];
            return dist2_shared(sq, reinterpret_cast<const float4*>(row), quads);
        } else if constexpr (DP == 16 || DP == 32) {
            *last = row[DP];
            return dist2_vec4<4 * NQ>(reinterpret_cast<const float(&)[4 * NQ]>(q), reinterpret_cast<const float4*>(row));
        } else {
            return centre_dist<DP>(q, row, last);
        }
    }
    __device__ __forceinline__ void test(uint32_t node, float* bound, uint32_t* key) const {
        float r;
        const float s = dist2_to(ball + static_cast<size_t>(node) * ball_stride, &r);
        *bound = ball_bound(s, r, margin);
        *key = min(orderable(sqrtf(s) - r), 0xFFFFFFFEu);
    }
    __device__ __forceinline__ float dist(const float* slot, int32_t* id) const {
        float last;
        const float d2 = dist2_to(slot, &last);
        *id = __float_as_int(last);
        return d2;
    }
};

template <int DP>
struct BallWarpSmem {
    WarpRows<true> rows;
    float4 q[DP > 32 ? DP / 4 : 1];
};

// One warp's search of query qi within r2; its row goes to the query's result slots.
template <int DP, int NQ, int KR, bool SEEDED>
__device__ __forceinline__ void ball_warp_query(const BallParams& p, uint32_t qi, float r2, BallWarpSmem<DP>& sm) {
    const uint32_t lane = threadIdx.x & 31u;
    BallWarpView<DP, NQ> view;
    if constexpr (DP > 32) {
        stage_query<DP>(p.queries, p.dims, qi, lane, sm.q);
        view.sq = sm.q;
    } else {
        load_query<DP>(p.queries, p.dims, qi, view.q);
    }
    view.ball = p.ball;
    view.ball_stride = p.ball_stride;
    view.margin = p.margin;
    view.quads = (p.dims + 3) / 4;
    const WarpTree t{p.leaf, p.leaf_stride, p.leaf_slots << (p.node_depth - p.stop_depth), p.stop_depth};
    WarpTopK<KR> top;
    LocalCounters lc;
    bool missed = false;
    top.init(p.k, r2, lane);
    if constexpr (SEEDED) {
        const float r = p.seeds[qi] * p.seed_scale;
        missed = warp_search<BallWarpView<DP, NQ>, KR, true>(view, t, sm.rows, top, lc, r < r2 ? r : r2, r2);
    } else {
        warp_search<BallWarpView<DP, NQ>, KR, false>(view, t, sm.rows, top, lc, r2, r2);
    }
    top.emit(p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
    if (p.counters && lane == 0) {
        lc.flush(p.counters);
        if (missed) atomicAdd(&p.counters->fallback, 1ull);
    }
}

template <int DP, int NQ, int KR, bool SEEDED>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) ball_warp_query_kernel(const BallParams p) {
    __shared__ BallWarpSmem<DP> sm[kWarpsPerBlock];
    const uint32_t w = threadIdx.x >> 5, t = blockIdx.x * kWarpsPerBlock + w;
    if (t >= (p.count_dev ? *p.count_dev : p.nq)) return;  // no block-wide barriers
    const uint32_t qi = p.order ? p.order[t] : t;
    ball_warp_query<DP, NQ, KR, SEEDED>(p, qi, p.radii ? p.radii[qi] : p.max_d2, sm[w]);
}

// Sort key of a query: the node reached after `levels` steps towards the nearer child centre.
template <int DP>
__global__ void ball_leaf_key_kernel(const float* __restrict__ ball, uint32_t ball_stride, uint32_t levels,
                                     const float* __restrict__ queries, uint32_t dims, uint32_t nq,
                                     uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nq) return;
    float q[DP];
    load_query<DP>(queries, dims, t, q);
    uint32_t node = 0;
    for (uint32_t d = 0; d < levels; ++d) {
        const uint32_t l = 2 * node + 1;
        float rl, rr;
        const float sl = centre_dist<DP>(q, ball + static_cast<size_t>(l) * ball_stride, &rl);
        const float sr = centre_dist<DP>(q, ball + static_cast<size_t>(l + 1) * ball_stride, &rr);
        node = sl <= sr ? l : l + 1;
    }
    keys[t] = node - ((1u << levels) - 1u);
    vals[t] = t;
}

// A query batch's search parameters: its tree, buckets of `bucket` slots (0 = the tree's leaves).
inline BallParams ball_params(const knn_index* ix, const QueryArgs& a, const uint32_t* order, uint32_t bucket) {
    BallParams p{};
    p.ball = ix->ball.as<float>();
    p.ball_stride = ix->ball_stride;
    p.leaf = ix->leaf.as<float>();
    p.leaf_stride = ix->leaf_stride;
    p.node_count = ix->node_count;
    p.node_depth = ix->node_depth;
    p.stop_depth = scan_depth_for(ix->node_depth, ix->leaf_slots, bucket);
    p.leaf_slots = ix->leaf_slots;
    p.margin = rel_margin(ix->dims);
    p.queries = a.queries;
    p.dims = ix->dims;
    p.nq = a.count;
    p.order = order;
    p.count_dev = a.count_dev;
    p.max_d2 = a.max_d2;
    p.radii = a.radii;
    p.seeds = a.seeds;
    p.seed_scale = a.seed_scale;
    p.k = a.k;
    p.out_idx = a.out_idx;
    p.out_dist = a.out_dist;
    p.counters = a.counters;
    return p;
}

// Whether a batch's queries get a thread each, in locality order, instead of a warp each (kd_by_thread says
// when that pays; a ball's bound is the same either way, so queries far from the points cost a thread no
// more than a warp).  1,000,000 queries, a warp and a thread each, us: 30,000 1-d points, k 1, 656 and 186;
// 20,000 3-d points, k 8, 1,702 and 1,197; 300 4-d points, k 16, 1,527 and 1,617, 600 3-d ones 1,477 and 1,258;
// 1,000,000 uniform 3-d points, k 1, 1,524 and 970, clustered ones 6,150 and 6,700, with k 4 7,115 and 8,600: from
// k 3 on the line also asks for many queries a point.
constexpr bool kBallThreadDims(int dp) { return dp <= 4; }
inline bool ball_by_thread(int dp, uint32_t n, const QueryArgs& a, const QueryPlan& p) {
    if (!p.reorder || a.order || a.count_dev || a.seeds || a.k > 16) return false;
    const uint64_t q = a.count;
    if (n <= 64 && a.k <= 4) return q >= 200000;
    if (dp == 1) return q >= (a.k <= 8 ? 250000u : 500000u);
    if (dp <= 3 && a.k <= 2) return q >= 500000;
    if (a.k <= 8) return dp <= 3 ? q >= 400000 && q >= 8ull * n : q >= 1000000 && q >= 8ull * n;
    return q >= 1000000 && q >= (dp <= 3 ? 32ull : 128ull) * n;
}

template <int DP>
int launch_ball_thread(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order, cudaStream_t s) {
    const BallParams p = ball_params(ix, a, order, plan.leaf_scan);
    auto kern = a.k <= 8 ? ball_knn_kernel<DP, 8> : ball_knn_kernel<DP, 16>;
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    kern<<<ceil_div(a.count, 128), 128, (p.stop_depth + 1) * 128 * sizeof(uint2), s>>>(p);
    KNN_LAUNCHED();
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return KNN_OK;
}

// Warp-coherent search (traversal 1).
template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
static int launch_ball(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order,
                       cudaStream_t s) {
    const uint32_t block = plan.block ? plan.block : 128;
    const size_t smem = tracker_smem_bytes(SHNN, KMAX, block) + stack_smem_bytes(SHST, block);
    auto kern = ball_knn_warp_kernel<DP, KMAX, HEAP, SHNN, SHST>;
    if (smem > 48 * 1024)
        KNN_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    const BallParams p = ball_params(ix, a, order, plan.leaf_scan);
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    kern<<<ceil_div(a.count, block), block, smem, s>>>(p);
    KNN_LAUNCHED();
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return KNN_OK;
}

template <int DP, int KMAX>
static int launch_ball_variant(knn_index* ix, const QueryArgs& a, const QueryPlan& p, const uint32_t* order,
                               cudaStream_t s) {
#define KNN_BALL_CASE(H, N, S)                                          \
    if (p.heap == H && p.sh_nn == N && p.sh_stack == S)                 \
        return launch_ball<DP, KMAX, H, N, S>(ix, a, p, order, s);
    KNN_BALL_CASE(false, false, false)
    KNN_BALL_CASE(false, false, true)
    KNN_BALL_CASE(false, true, false)
    KNN_BALL_CASE(false, true, true)
    KNN_BALL_CASE(true, false, false)
    KNN_BALL_CASE(true, false, true)
    KNN_BALL_CASE(true, true, false)
    KNN_BALL_CASE(true, true, true)
#undef KNN_BALL_CASE
    return fail(KNN_ERR_INVALID_ARGUMENT, "bad query plan");
}

// Query order for locality: queries sorted by the node they reach after up to 24 greedy
// descent steps (stable radix sort on the path bits).  The order lives in the index workspace
// until the next query.
template <uint32_t DP>
int ball_order_dp(knn_index* ix, const QueryArgs& a, cudaStream_t s, const uint32_t** order) {
    *order = nullptr;
    const uint32_t levels = std::min<uint32_t>(ix->node_depth, 24);
    if (levels == 0) return KNN_OK;
    const size_t nq = a.count;
    KNN_TRY(ix->workspace.reserve(order_bytes(a.count)));
    Carver c(ix->workspace.ptr);
    uint32_t* keys = c.take<uint32_t>(nq);
    uint32_t* vals = c.take<uint32_t>(nq);
    uint32_t* keys_alt = c.take<uint32_t>(nq);
    uint32_t* vals_alt = c.take<uint32_t>(nq);
    void* temp = c.take<uint8_t>(radix_sort_temp_bytes(a.count));
    ball_leaf_key_kernel<DP><<<ceil_div(a.count, 256), 256, 0, s>>>(ix->ball.as<float>(), ix->ball_stride, levels,
                                                       a.queries, ix->dims, a.count, keys, vals);
    KNN_LAUNCHED();
    bool in_alt = false;
    KNN_TRY(radix_sort_pairs(keys, vals, keys_alt, vals_alt, a.count, static_cast<int>(levels), temp, s, &in_alt));
    *order = in_alt ? vals_alt : vals;
    return KNN_OK;
}

// Bucket slots at least (plans may ask for more): 16 up to 16 dims (16 dims, 262,144 points: 4.16 to
// 4.39 ms with 8, 16 and 32), 8 beyond, where smaller balls prune more than larger scans save (24
// dims: 3.06 ms with 8, 3.46 with 32; 100 dims: 4.7 and 6.4).
inline uint32_t ball_warp_bucket(uint32_t dims) { return dims <= 16 ? 16u : 8u; }

// A warp per query over the balls (traversal 0).
template <uint32_t DP>
int ball_warp_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order, cudaStream_t s) {
    const BallParams p = ball_params(ix, a, order, std::max(plan.leaf_scan, ball_warp_bucket(ix->dims)));
    const uint32_t grid = ceil_div(a.count, kWarpsPerBlock), threads = 32 * kWarpsPerBlock;
    void (*kern)(const BallParams) = nullptr;
    with_quads<DP>(ix->dims, [&](auto nq) {
        constexpr int NQ = decltype(nq)::value;
        if (p.seeds)
            kern = a.k <= 32 ? ball_warp_query_kernel<DP, NQ, 1, true> : a.k <= 64 ? ball_warp_query_kernel<DP, NQ, 2, true> : ball_warp_query_kernel<DP, NQ, 4, true>;
        else
            kern = a.k <= 32 ? ball_warp_query_kernel<DP, NQ, 1, false> : a.k <= 64 ? ball_warp_query_kernel<DP, NQ, 2, false> : ball_warp_query_kernel<DP, NQ, 4, false>;
    });
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    kern<<<grid, threads, 0, s>>>(p);
    KNN_LAUNCHED();
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return KNN_OK;
}

template <uint32_t DP>
int ball_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& p, cudaStream_t s) {
    const uint32_t* order = a.order;
    if (!p.warp) {
        // The storage options do not matter to a warp's search; sizes no block can hold stay refused.
        const uint32_t block = p.block ? p.block : 128;
        const size_t storage = tracker_smem_bytes(p.sh_nn, k_class(a.k), block) + stack_smem_bytes(p.sh_stack, block);
        if (storage > kMaxBlockSmem)
            return fail(KNN_ERR_CUDA, "storage options: %zu bytes of shared memory per block of %u", storage, block);
        if constexpr (kBallThreadDims(DP)) {
            if (ball_by_thread(DP, ix->n, a, p)) {
                bool room = false;
                KNN_TRY(order_room(ix, a.count, s, &room));
                if (room) KNN_TRY(ball_order_dp<DP>(ix, a, s, &order));
                if (order) return launch_ball_thread<DP>(ix, a, p, order, s);
            }
        }
        // Neighbouring queries share the rows they read through the caches: an order pays where rows are
        // wide (the search then lives on L2 reads; 16 dims, 65,536 queries on 262,144 points: 4.14 ms
        // sorted, 4.39 not) or the index outgrows L2, and costs otherwise (3 dims, 25,000 queries on
        // 200,000: 0.25 and 0.17).
        const bool wide = DP >= 16 && a.count >= 16384, large = a.count >= kWarpOrderMin && ix->leaf.bytes > kL2Bytes;
        if (!order && p.reorder && (wide || large)) KNN_TRY(ball_order_dp<DP>(ix, a, s, &order));
        return ball_warp_query_dp<DP>(ix, a, p, order, s);
    }
    if (!order && p.reorder && a.count >= 4096) KNN_TRY(ball_order_dp<DP>(ix, a, s, &order));
    switch (k_class(a.k)) {
        case 8: return launch_ball_variant<DP, 8>(ix, a, p, order, s);
        case 16: return launch_ball_variant<DP, 16>(ix, a, p, order, s);
        case 32: return launch_ball_variant<DP, 32>(ix, a, p, order, s);
        case 64: return launch_ball_variant<DP, 64>(ix, a, p, order, s);
        default: return launch_ball_variant<DP, 128>(ix, a, p, order, s);
    }
}

template int ball_query_dp<KNN_DP>(knn_index*, const QueryArgs&, const QueryPlan&, cudaStream_t);
template int ball_order_dp<KNN_DP>(knn_index*, const QueryArgs&, cudaStream_t, const uint32_t**);


// ---- batches of independent sets (one persistent kernel per class of sets) -----------------------
struct BallBatchSet {
    BallParams p;                 // the set's search parameters; p.order is the class order, p.order_base its offset
    uint32_t first_block;  // first work block of this set in the class
    uint32_t query_offset; // first query of this set in the class-wide numbering
    uint32_t levels;       // descent depth of the locality key
};

__device__ __forceinline__ uint32_t ball_find_set(const BallBatchSet* sets, uint32_t nsets, uint32_t item, bool by_query) {
    uint32_t lo = 0, hi = nsets;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if ((by_query ? sets[mid].query_offset : sets[mid].first_block) <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Locality key of every query of the class: (set << 24) | descent path scaled to 24 bits.
template <int DP>
__global__ void ball_batch_key_kernel(const BallBatchSet* __restrict__ sets, uint32_t nsets, uint32_t total,
                                     uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const uint32_t si = ball_find_set(sets, nsets, g, true);
    const BallParams& p = sets[si].p;
    float q[DP];
    load_query<DP>(p.queries, p.dims, g - sets[si].query_offset, q);
    const uint32_t levels = sets[si].levels;
    uint32_t node = 0;
    for (uint32_t d = 0; d < levels; ++d) {
        const uint32_t l = 2 * node + 1;
        float rl, rr;
        const float sl = centre_dist<DP>(q, p.ball + static_cast<size_t>(l) * p.ball_stride, &rl);
        const float sr = centre_dist<DP>(q, p.ball + static_cast<size_t>(l + 1) * p.ball_stride, &rr);
        node = sl <= sr ? l : l + 1;
    }
    keys[g] = (si << 24) | ((node - ((1u << levels) - 1u)) << (24 - levels));
    vals[g] = g;
}

// Warp-coherent search: blocks take work blocks (blockDim queries of one set) from a shared counter
// until the class is done; sets of very different sizes share the GPU without a launch each.
template <int DP, int KMAX>
__global__ void __launch_bounds__(256) ball_batch_kernel(const BallBatchSet* __restrict__ sets, uint32_t nsets,
                                                        uint32_t total_blocks, uint32_t* __restrict__ counter) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t item_s;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) item_s = atomicAdd(counter, 1u);
        __syncthreads();
        const uint32_t item = item_s;
        if (item >= total_blocks) break;
        const uint32_t si = ball_find_set(sets, nsets, item, false);
        const BallParams& p = sets[si].p;
        const uint32_t t = (item - sets[si].first_block) * blockDim.x + threadIdx.x;
        ball_search_warp<DP, KMAX, false, false, false>(p, t, p.nq, smem);
    }
}

// A warp per query: persistent warps take the class's queries one by one.
template <int DP, int KR>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) ball_batch_warp_kernel(const BallBatchSet* __restrict__ sets,
                                                                             uint32_t nsets, uint32_t total_queries,
                                                                             uint32_t* __restrict__ counter) {
    __shared__ BallWarpSmem<DP> sm[kWarpsPerBlock];
    for (;;) {
        uint32_t g = 0;
        if ((threadIdx.x & 31u) == 0) g = atomicAdd(counter, 1u);
        g = __shfl_sync(kFullMask, g, 0);
        if (g >= total_queries) break;  // no block-wide barriers
        const uint32_t si = ball_find_set(sets, nsets, g, true);
        const BallParams& p = sets[si].p;
        const uint32_t t = g - sets[si].query_offset;
        const uint32_t qi = p.order ? p.order[t] - p.order_base : t;
        ball_warp_query<DP, warp_quads(DP, DP), KR, false>(p, qi, p.max_d2, sm[threadIdx.x >> 5]);
        __syncwarp();
    }
}

template <uint32_t DP>
int ball_batch_launch(const void* sets, uint32_t nsets, uint32_t total_queries, uint32_t total_blocks, uint32_t kmax,
                       uint32_t mode, uint32_t block, uint32_t* counter, uint32_t* keys, uint32_t* vals, bool key_pass,
                       cudaStream_t s) {
    using Set = BallBatchSet;
    const Set* d_sets = static_cast<const Set*>(sets);
    if (key_pass) {
        ball_batch_key_kernel<DP><<<ceil_div(total_queries, 256), 256, 0, s>>>(d_sets, nsets, total_queries, keys, vals);
        KNN_LAUNCHED();
        return KNN_OK;
    }
#define KNN_BATCH(KM)                                                                                 \
    if (kmax == KM && mode == 1) {                                                                    \
        auto kern = ball_batch_kernel<DP, KM>;                                                       \
        int per_sm = 0;                                                                               \
        KNN_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0));         \
        const uint32_t grid = std::max(1, per_sm) * static_cast<uint32_t>(sm_count());                \
        kern<<<std::min(grid, total_blocks), block, 0, s>>>(d_sets, nsets, total_blocks, counter);   \
        KNN_LAUNCHED();                                                                               \
        return KNN_OK;                                                                                \
    }
    KNN_BATCH(8) KNN_BATCH(16) KNN_BATCH(32) KNN_BATCH(64) KNN_BATCH(128)
#undef KNN_BATCH
    if (mode == 2) {
        auto kern = kmax <= 32 ? ball_batch_warp_kernel<DP, 1> : kmax <= 64 ? ball_batch_warp_kernel<DP, 2> : ball_batch_warp_kernel<DP, 4>;
        int per_sm = 0;
        KNN_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kWarpsPerBlock, 0));
        const uint32_t grid = std::max(1, per_sm) * static_cast<uint32_t>(sm_count());
        kern<<<std::min(grid, ceil_div(total_queries, kWarpsPerBlock)), 32 * kWarpsPerBlock, 0, s>>>(d_sets, nsets, total_queries, counter);
        KNN_LAUNCHED();
        return KNN_OK;
    }
    return fail(KNN_ERR_INVALID_ARGUMENT, "batch class k %u", kmax);
}

#if KNN_DP == 1
// Fills the search parameters of one batch set from its index and item.
size_t ball_batch_set_bytes() { return sizeof(BallBatchSet); }

void ball_batch_set_fill(void* out, const knn_index* ix, const QueryArgs& a, const QueryPlan& plan,
                        const uint32_t* order, uint32_t order_base, uint32_t first_block, uint32_t query_offset) {
    BallBatchSet bs{};
    bs.p = ball_params(ix, a, order, plan.warp ? plan.leaf_scan : std::max(plan.leaf_scan, ball_warp_bucket(ix->dims)));
    bs.p.order_base = order_base;
    bs.first_block = first_block;
    bs.query_offset = query_offset;
    bs.levels = std::min<uint32_t>(ix->node_depth, 24);
    std::memcpy(out, &bs, sizeof(bs));
}
#endif

template int ball_batch_launch<KNN_DP>(const void*, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t*,
                                      uint32_t*, uint32_t*, bool, cudaStream_t);

}  // namespace knn
