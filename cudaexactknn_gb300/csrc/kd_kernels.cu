// k-d tree query kernels, one translation unit per padded dimension count (KNN_DP).
//
// Replaces KdTreeKernels::knnDevice and its four storage variants (src/KdTreeGpu.cuh:37-184).
// Same depth-first search: descend to the closer child, push the farther child with the squared
// distance to its splitting plane, scan leaves, pop.  Differences:
//   * queries are reordered so that neighbouring threads descend to neighbouring leaves (sorted
//     by the leaf each query reaches), which keeps a warp's node and leaf loads together;
//   * the plane bound fl((q[dim]-split)^2) never exceeds the float distance of any point
//     beyond the plane (float subtraction and rounding are monotone and every term of the
//     fused sum is non-negative), and nodes are pruned only when bound > k-th distance, so no
//     point whose key could enter the top-k is skipped, ties included;
//   * k-th key cached in a register; tracker/stack storage chosen by the plan.
//
// That per-thread search is what the engine runs where the tight node boxes are not to be had (no
// memory for them when the index was made, nor since), and for very many queries of very few dims
// (kd_by_thread; with the boxes as a second bound).  Otherwise each query gets a warp (kd_warp_query_kernel, warp_search.cuh), bounded by the boxes.

#include <algorithm>
#include <cstring>

#include "tree_query.cuh"
#include "warp_search.cuh"

#ifndef KNN_DP
#error "compile with -DKNN_DP=<padded dims>"
#endif

namespace knn {

struct KdParams {
    const float* split;
    const float* leaf;
    uint32_t leaf_stride;
    uint32_t node_count;
    uint32_t node_depth;
    uint32_t stop_depth;  // descend to this depth, then scan the subtree's slots
    uint32_t leaf_slots;
    uint32_t aux;
    const float* queries;
    uint32_t dims;
    uint32_t nq;
    const uint32_t* order;  // thread -> query, or null
    const uint32_t* count_dev;  // when set, *count_dev threads are live (nq is an upper bound)
    uint32_t order_base;  // subtracted from order entries (batched orders hold batch-wide ids)
    float max_d2;
    const float* radii;
    const float* box;     // tight node boxes, per node lo[], hi[], down to depth box_depth, or null
    uint32_t box_stride;  // floats per box
    uint32_t box_depth;
    const float* seeds;   // warp-per-query search: per query radius to start from (x seed_scale), or null
    float seed_scale;
    uint32_t k;
    int32_t* out_idx;
    float* out_dist;
    DevCounters* counters;
};

// Floats per coordinate set of a node box.
__host__ __device__ constexpr int box_qs(int dp) { return dp < 4 ? 4 : dp; }

// Lower bound on the float dist2 from q to any point of the box (lo, hi): per dimension the gap
// o = max(fl(lo - q), fl(q - hi), 0), then the same fused sum as dist2 in dimension order.  For a
// point p of the box, |fl(q - p)| >= o (p lies beyond lo or hi, and rounding is monotone), and
// fma(t, t, acc) is non-decreasing in |t| and acc >= 0, so the bound never exceeds dist2(q, p).
// An empty box (lo = +inf, hi = -inf) gives +inf.
template <int DP>
__device__ __forceinline__ float box_bound(const float (&q)[DP], const float4* __restrict__ lo4,
                                           const float4* __restrict__ hi4, float acc) {
#pragma unroll
    for (int v = 0; v < (DP + 3) / 4; ++v) {
        const float4 lo = __ldg(lo4 + v), hi = __ldg(hi4 + v);
        const float l[4] = {lo.x, lo.y, lo.z, lo.w};
        const float h[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (4 * v + c < DP) {
                const float o = fmaxf(fmaxf(__fsub_rn(l[c], q[4 * v + c]), __fsub_rn(q[4 * v + c], h[c])), 0.0f);
                acc = __fmaf_rn(o, o, acc);
            }
        }
    }
    return acc;
}

template <int DP>
__device__ __forceinline__ float box_bound(const float (&q)[DP], const float* __restrict__ box) {
    return box_bound<DP>(q, reinterpret_cast<const float4*>(box), reinterpret_cast<const float4*>(box + box_qs(DP)), 0.0f);
}

// Whether a batch's queries get a thread each, in locality order, instead of a warp each: in very few
// dims, for few neighbours, where the queries are so many that neighbouring threads walk the same path
// (a warp's search has some 500 instructions even then).  The sort and the divergence of fewer queries
// cost more, the more so for queries far from the points.  1,000,000 queries, a warp and a thread each, us:
// 30,000 1-d points, k 1, 470 and 142; 30,000 2-d points, k 4, 571 and 386; 2,000 3-d points, k 1, 557 and
// 386; but 1,000,000 2-d points, k 8, 745 and 750, and 400,000 queries far from them, k 1, 414 and 1,492.
// And on trees so small that a search reads most of them: 200,000 queries, 300 50-d points, k 10, 2,295 and
// 1,479; 20 3-d points, k 1, 1.5 times a thread's time.
constexpr bool kd_by_thread_dims(int dp) { return dp <= 3; }
inline bool kd_by_thread(int dp, uint32_t n, const QueryArgs& a, const QueryPlan& p) {
    if (!p.reorder || a.order || a.count_dev || a.seeds || a.k > 16) return false;
    const uint64_t q = a.count;
    if (n <= 64 && q >= (dp <= 4 && a.k <= 4 ? 200000u : 1000000u)) return true;
    if (dp >= 32 && n <= 320 && q >= 200000) return true;
    if (!kd_by_thread_dims(dp)) return false;
    if (dp == 1) return q >= (a.k <= 8 ? 250000u : 500000u);
    if (dp == 2) return a.k <= 4 && q >= 800000 && q >= 4ull * n;
    return a.k <= 2 && q >= 1000000 && q >= 128ull * n;
}

// One thread's search: query slot t of the batch (its query is p.order[t] - p.order_base, or t).
template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
__device__ __forceinline__ void kd_search_thread(const KdParams& p, uint32_t t, unsigned char* smem) {
    uint64_t* sh_nn = reinterpret_cast<uint64_t*>(smem);
    uint32_t* sh_st = reinterpret_cast<uint32_t*>(smem + tracker_smem_bytes(SHNN, KMAX, blockDim.x));

    const uint32_t qi = p.order ? p.order[t] - p.order_base : t;
    float q[DP];
    load_query<DP>(p.queries, p.dims, qi, q);
    const float r2 = p.radii ? p.radii[qi] : p.max_d2;

    Tracker<KMAX, HEAP, SHNN> tr;
    tr.init(p.k, r2, sh_nn + threadIdx.x, blockDim.x);
    Stack<SHST> st;
    st.init(sh_st, blockDim.x);
    st.push(0, 0.0f);
    LocalCounters lc;
    bool overflow = false;

    while (st.top) {
        uint32_t node;
        float bound;
        st.pop(&node, &bound);
        if (bound > tr.radius()) continue;
        uint32_t depth = heap_depth(node);
        while (depth < p.stop_depth) {
            const uint32_t dim = depth % p.aux;
            const float diff = __fsub_rn(pick<DP>(q, dim), __ldg(p.split + node));
            const uint32_t l = 2 * node + 1;
            const uint32_t close_child = diff < 0.0f ? l : l + 1;
            const uint32_t far_child = diff < 0.0f ? l + 1 : l;
            float b = __fmul_rn(diff, diff);
            if (b <= tr.radius()) {
                // (The plane alone says little to a query far from the points.)
                if constexpr (kd_by_thread_dims(DP))
                    if (depth < p.box_depth) b = fmaxf(b, box_bound<DP>(q, p.box + static_cast<size_t>(far_child) * p.box_stride));
                if (b <= tr.radius()) overflow |= !st.push(far_child, b);
            }
            node = close_child;
            ++depth;
            ++lc.nodes;
        }
        const SlotRange r = subtree_slots(node, depth, p.node_depth, p.node_count, p.leaf_slots);
        const float* slot = p.leaf + r.first * p.leaf_stride;
        ++lc.leaves;
        for (uint32_t s = 0; s < r.count; ++s, slot += p.leaf_stride) {
            int32_t id;
            const float d2 = slot_dist<DP>(q, slot, &id);
            if (id < 0) continue;  // padding of a partly filled leaf
            ++lc.points;
            tr.offer(make_key(d2, id));
        }
    }
    tr.emit(p.k, p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
    if (p.counters) {
        lc.flush(p.counters);
        if (overflow) atomicExch(&p.counters->error, 1);
    }
}

template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
__global__ void __launch_bounds__(256) kd_knn_kernel(const KdParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (p.count_dev ? *p.count_dev : p.nq)) return;  // no block-wide barriers below
    kd_search_thread<DP, KMAX, HEAP, SHNN, SHST>(p, t, smem);
}

// Warp-coherent variant: the 32 queries of a warp (neighbours after the leaf-order sort) walk the
// tree together.  Each node's split is one broadcast load; the warp descends first into the
// child most of its still-interested lanes are closer to; every lane keeps its own lower bound
// for each stacked subtree, max(bound inherited from the parent, its squared distance to the
// plane), and a subtree is skipped only when no lane's bound is within that lane's radius.
// Leaf buckets are scanned by all lanes against the same slots (broadcast loads).  Control flow
// is uniform across the warp; only the (rare) top-k insertions diverge.
// One warp's search over slots t (this lane) of the batch; `live` slots exist.
template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
__device__ __forceinline__ void kd_search_warp(const KdParams& p, uint32_t t, uint32_t live, unsigned char* smem) {
    const uint32_t warp_first = t & ~31u;
    if (warp_first >= live) return;  // whole warp idle; no block-wide barriers below
    const bool active = t < live;
    uint64_t* sh_nn = reinterpret_cast<uint64_t*>(smem);
    uint32_t* sh_st = reinterpret_cast<uint32_t*>(smem + tracker_smem_bytes(SHNN, KMAX, blockDim.x));

    const uint32_t qi = active ? (p.order ? p.order[t] - p.order_base : t) : 0u;
    float q[DP];
    load_query<DP>(p.queries, p.dims, qi, q);
    // Idle lanes (past the end of the batch) search with radius -1: they never want a node.
    const float r2 = active ? (p.radii ? p.radii[qi] : p.max_d2) : 0.0f;

    Tracker<KMAX, HEAP, SHNN> tr;
    tr.init(p.k, r2, sh_nn + threadIdx.x, blockDim.x);
    Stack<SHST> st;
    st.init(sh_st, blockDim.x);
    st.push(0, active ? 0.0f : INFINITY);
    LocalCounters lc;
    bool overflow = false;

    while (st.top) {  // st.top is warp-uniform: every lane pushes and pops together
        uint32_t node;
        float bound;
        st.pop(&node, &bound);
        if (!__any_sync(0xFFFFFFFFu, bound <= tr.radius())) continue;
        uint32_t depth = heap_depth(node);
        bool pruned = false;
        while (depth < p.stop_depth) {
            const uint32_t dim = depth % p.aux;
            const float diff = __fsub_rn(pick<DP>(q, dim), __ldg(p.split + node));
            const float b = fmaxf(bound, __fmul_rn(diff, diff));
            const bool want = bound <= tr.radius();
            const bool go_left = diff < 0.0f;
            const uint32_t left_votes = __popc(__ballot_sync(0xFFFFFFFFu, want && go_left));
            const uint32_t right_votes = __popc(__ballot_sync(0xFFFFFFFFu, want && !go_left));
            const bool first_left = left_votes >= right_votes;
            const uint32_t l = 2 * node + 1;
            // This lane's bound for each child: its inherited bound on its own side, the plane
            // bound on the other.
            const float b_left = go_left ? bound : b;
            const float b_right = go_left ? b : bound;
            const float b_first = first_left ? b_left : b_right;
            const float b_second = first_left ? b_right : b_left;
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
__global__ void __launch_bounds__(256) kd_knn_warp_kernel(const KdParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t live = p.count_dev ? *p.count_dev : p.nq;
    kd_search_warp<DP, KMAX, HEAP, SHNN, SHST>(p, t, live, smem);
}

// Sort key of a query: the node it reaches after `levels` closer-child steps (path bits).
template <int DP>
__global__ void kd_leaf_key_kernel(const float* __restrict__ split, uint32_t aux, uint32_t levels,
                                   const float* __restrict__ queries, uint32_t dims, uint32_t nq,
                                   uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nq) return;
    float q[DP];
    load_query<DP>(queries, dims, t, q);
    uint32_t node = 0;
    for (uint32_t d = 0; d < levels; ++d) {
        const float diff = pick<DP>(q, d % aux) - __ldg(split + node);
        node = 2 * node + (diff < 0.0f ? 1u : 2u);
    }
    keys[t] = node - ((1u << levels) - 1u);
    vals[t] = t;
}

// A query batch's search parameters: its tree, buckets of `bucket` slots (0 = the tree's leaves).
inline KdParams kd_params(const knn_index* ix, const QueryArgs& a, const uint32_t* order, uint32_t bucket) {
    KdParams p{};
    p.split = ix->split.as<float>();
    p.leaf = ix->leaf.as<float>();
    p.leaf_stride = ix->leaf_stride;
    p.node_count = ix->node_count;
    p.node_depth = ix->node_depth;
    p.stop_depth = scan_depth_for(ix->node_depth, ix->leaf_slots, bucket);
    p.leaf_slots = ix->leaf_slots;
    p.aux = ix->aux_dims;
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

// The same for a search over node boxes.
inline KdParams kd_box_params(const knn_index* ix, const knn_index::KdBoxes& boxes, const QueryArgs& a,
                              const uint32_t* order, uint32_t bucket) {
    KdParams p = kd_params(ix, a, order, bucket);
    p.stop_depth = std::min(p.stop_depth, boxes.depth);
    p.box = boxes.buf.as<float>();
    p.box_stride = 2 * box_qs(static_cast<int>(ix->dp));
    p.box_depth = boxes.depth;
    return p;
}

template <int DP, int KMAX, bool HEAP, bool SHNN, bool SHST>
static int launch_kd(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order,
                     cudaStream_t s) {
    const uint32_t block = plan.block ? plan.block : 128;
    const size_t smem = tracker_smem_bytes(SHNN, KMAX, block) + stack_smem_bytes(SHST, block);
    auto kern = plan.warp ? kd_knn_warp_kernel<DP, KMAX, HEAP, SHNN, SHST> : kd_knn_kernel<DP, KMAX, HEAP, SHNN, SHST>;
    if (smem > 48 * 1024)
        KNN_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    KdParams p = kd_params(ix, a, order, plan.leaf_scan);
    if (ix->kd_box.buf.ptr) {
        p.box = ix->kd_box.buf.as<float>();
        p.box_stride = 2 * box_qs(DP);
        p.box_depth = ix->kd_box.depth;
    }
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    kern<<<ceil_div(a.count, block), block, smem, s>>>(p);
    KNN_LAUNCHED();
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return KNN_OK;
}

template <int DP, int KMAX>
static int launch_kd_variant(knn_index* ix, const QueryArgs& a, const QueryPlan& p, const uint32_t* order,
                             cudaStream_t s) {
#define KNN_KD_CASE(H, N, S)                                            \
    if (p.heap == H && p.sh_nn == N && p.sh_stack == S)                 \
        return launch_kd<DP, KMAX, H, N, S>(ix, a, p, order, s);
    KNN_KD_CASE(false, false, false)
    KNN_KD_CASE(false, false, true)
    KNN_KD_CASE(false, true, false)
    KNN_KD_CASE(false, true, true)
    KNN_KD_CASE(true, false, false)
    KNN_KD_CASE(true, false, true)
    KNN_KD_CASE(true, true, false)
    KNN_KD_CASE(true, true, true)
#undef KNN_KD_CASE
    return fail(KNN_ERR_INVALID_ARGUMENT, "bad query plan");
}

// Query order for locality: queries sorted by the node they reach after up to 24 greedy
// descent steps (stable radix sort on the path bits).  The order lives in the index workspace
// until the next query.
template <uint32_t DP>
int kd_order_dp(knn_index* ix, const QueryArgs& a, cudaStream_t s, const uint32_t** order) {
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
    kd_leaf_key_kernel<DP><<<ceil_div(a.count, 256), 256, 0, s>>>(ix->split.as<float>(), ix->aux_dims, levels,
                                                       a.queries, ix->dims, a.count, keys, vals);
    KNN_LAUNCHED();
    bool in_alt = false;
    KNN_TRY(radix_sort_pairs(keys, vals, keys_alt, vals_alt, a.count, static_cast<int>(levels), temp, s, &in_alt));
    *order = in_alt ? vals_alt : vals;
    return KNN_OK;
}

template <uint32_t DP>
int kd_group_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order, cudaStream_t s);

template <uint32_t DP>
int kd_warp_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order, cudaStream_t s);

template <uint32_t DP>
int kd_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& p, cudaStream_t s) {
    if (p.box && DP > 16) return fail(KNN_ERR_INVALID_ARGUMENT, "box search: dims above 16");
    const uint32_t* order = a.order;
    if (!p.warp && !(p.group && !a.count_dev)) {
        // A warp per query, where its node boxes are at hand.  The per-thread search's storage options
        // do not matter to it, but sizes that search refuses stay refused (by the launch below).
        const uint32_t block = p.block ? p.block : 128;
        const bool fits = tracker_smem_bytes(p.sh_nn, k_class(a.k), block) + stack_smem_bytes(p.sh_stack, block) <= kMaxBlockSmem;
        bool ready = false;
        if (fits || p.box) KNN_TRY(kd_boxes_ready(ix, s, &ready));
        if (ready) {
            if (kd_by_thread(DP, ix->n, a, p)) {
                bool room = false;
                KNN_TRY(order_room(ix, a.count, s, &room));
                if (room) KNN_TRY(kd_order_dp<DP>(ix, a, s, &order));
                if (order) return a.k <= 8 ? launch_kd_variant<DP, 8>(ix, a, p, order, s) : launch_kd_variant<DP, 16>(ix, a, p, order, s);
            }
            // Neighbouring queries share the boxes and slots they read only through the caches: an
            // order pays once the index outgrows L2 (16 M clustered 3-d points, 2 M queries: 3.74 ms
            // sorted, 3.96 unsorted; 40 M and 4 M: 7.59 and 8.48) and costs before (4.19 M and 1 M:
            // 1.92 and 1.83).
            if (!order && p.reorder && a.count >= kWarpOrderMin && ix->leaf.bytes > kL2Bytes)
                KNN_TRY(kd_order_dp<DP>(ix, a, s, &order));
            return kd_warp_query_dp<DP>(ix, a, p, order, s);
        }
    }
    if (!order && p.reorder && a.count >= 4096) KNN_TRY(kd_order_dp<DP>(ix, a, s, &order));
    if (p.group && !a.count_dev) return kd_group_query_dp<DP>(ix, a, p, order, s);
    switch (k_class(a.k)) {
        case 8: return launch_kd_variant<DP, 8>(ix, a, p, order, s);
        case 16: return launch_kd_variant<DP, 16>(ix, a, p, order, s);
        case 32: return launch_kd_variant<DP, 32>(ix, a, p, order, s);
        case 64: return launch_kd_variant<DP, 64>(ix, a, p, order, s);
        default: return launch_kd_variant<DP, 128>(ix, a, p, order, s);
    }
}

// ---- warp-group search ---------------------------------------------------------------------------
//
// The 32 lanes of a warp hold 32 neighbouring queries (locality order) and a radius each (a seed
// from the radius model or from the query's own subtree, never below its k-th distance for most
// queries).  The warp walks the tree once for all of them, bounding every node by the distance
// from each lane's query to the node's tight bounding box; a node is entered when some lane's
// bound is within that lane's radius.  Leaf buckets are collected as (bucket, lanes) entries,
// and the (bucket, query) pairs are then dealt out over the warp's lanes one pair per lane, so a
// warp does the sum of its queries' bucket scans rather than their union.  A point within its
// query's radius is appended to that query's candidate list in shared memory; at the end each
// lane sorts its query's list.  A query with fewer than k candidates inside a radius below the
// caller's grows its radius by the density it saw and walks again; one whose list overflows, or
// that is still short after a few rounds, goes to a list that the warp-per-query search answers.  Every
// answer is exact: a bucket is skipped only when its box bound exceeds the radius, and the box
// bound is a rigorous lower bound on the float distance of every point inside (below).
constexpr uint32_t kGroupWarps = 4;
constexpr uint32_t kGroupList = 64;   // bucket entries collected before they are scanned
constexpr uint32_t kGroupFan = 3;     // levels the walk descends per step (up to 8 boxes tested at once)
constexpr uint32_t kGroupStack = 96;  // node stack (at most 7 net entries per step, 11 steps deep)
constexpr uint32_t kGroupRounds = 6;  // radius growth rounds before a query is left over

__host__ __device__ constexpr uint32_t group_cap(int kmax) { return kmax <= 8 ? 32u : (kmax <= 16 ? 48u : 80u); }

template <int DP, int KMAX>
struct GroupWarpSmem {
    uint32_t buf[group_cap(KMAX)][32];  // candidates' leaf slots, slot-major (entry i of lane l at [i][l])
    uint64_t list[kGroupList];          // (bucket node << 32) | lanes
    float qv[32][box_qs(DP)];           // the warp's queries
    float rad[32];                      // radius of each lane this round (-1: none)
    uint32_t cnt[32];                   // candidates appended per lane
    uint32_t pre[32];                   // inclusive prefix of pairs per list entry
    uint32_t stack[kGroupStack];
};

template <int DP, int KMAX>
constexpr size_t group_smem_bytes() { return kGroupWarps * sizeof(GroupWarpSmem<DP, KMAX>); }

struct KdGroupParams {
    KdParams p;              // tree, queries, locality order, caller's radius (max_d2 / radii), outputs
    float* seeds;            // per query radius to start from (<= the caller's); leftover's radius on exit
    uint32_t* fb_list;       // queries left to the warp-per-query search
    uint32_t* fb_count;
    uint32_t* group_counter; // next group of 32 queries (zero before the launch)
};

template <int DP, int KMAX>
__global__ void __launch_bounds__(kGroupWarps * 32) kd_group_kernel(const KdGroupParams gp) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Sm = GroupWarpSmem<DP, KMAX>;
    constexpr uint32_t C = group_cap(KMAX);
    constexpr int QS = box_qs(DP);
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    Sm& sm = reinterpret_cast<Sm*>(smem_raw)[threadIdx.x >> 5];
    const KdParams& p = gp.p;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stop = p.stop_depth;
    const uint32_t bucket_slots = p.leaf_slots << (p.node_depth - stop);
    uint32_t nodes = 0, pairs = 0;
    bool stack_error = false;
    // Persistent warps: each takes the next group of 32 queries from a counter until the batch is
    // done, so that no partial last wave of blocks is left and regions of uneven cost balance.
    for (;;) {
        uint32_t grp = 0;
        if (lane == 0) grp = atomicAdd(gp.group_counter, 1u);
        const uint32_t g = __shfl_sync(FULL, grp, 0) * 32u;
        if (g >= p.nq) break;
        const uint32_t t = g + lane;
        const bool active = t < p.nq;
        const uint32_t qi = active ? (p.order ? p.order[t] : t) : 0u;
        float q[DP];
        load_query<DP>(p.queries, p.dims, qi, q);
#pragma unroll
        for (int d = 0; d < QS; ++d) sm.qv[lane][d] = d < DP ? q[d] : 0.0f;
        const float R = active ? (p.radii ? p.radii[qi] : p.max_d2) : -1.0f;
        float r = active ? gp.seeds[qi] : -1.0f;
        if (!(r <= R)) r = R;  // a seed above the caller's radius (or NaN) starts at the caller's
        bool pending = active;

        // Scans the collected (bucket, lanes) entries, one (bucket, query) pair per lane at a time.
        auto scan = [&](uint32_t n) {
            for (uint32_t base = 0; base < n; base += 32) {
                const uint32_t e = base + lane;
                const uint32_t m = e < n ? static_cast<uint32_t>(sm.list[e]) : 0u;
                uint32_t incl = __popc(m);
#pragma unroll
                for (uint32_t o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += v;
                }
                const uint32_t total = __shfl_sync(FULL, incl, 31);
                sm.pre[lane] = incl;
                __syncwarp();
                for (uint32_t it = lane; it < total; it += 32) {
                    uint32_t j = 0;  // first entry whose inclusive prefix exceeds it
#pragma unroll
                    for (uint32_t step = 16; step; step >>= 1)
                        if (sm.pre[j + step - 1] <= it) j += step;
                    const uint64_t ent = sm.list[base + j];
                    const uint32_t excl = j ? sm.pre[j - 1] : 0u;
                    const uint32_t ql = nth_set_bit(static_cast<uint32_t>(ent), it - excl);
                    float qq[DP];
#pragma unroll
                    for (int d = 0; d < DP; ++d) qq[d] = sm.qv[ql][d];
                    const float rq = sm.rad[ql];
                    const uint32_t bucket = static_cast<uint32_t>(ent >> 32);
                    if (heap_depth(bucket) != stop) {  // cannot happen (the walk lists buckets only); recorded
                        stack_error = true;
                        continue;
                    }
                    const SlotRange sr = subtree_slots(bucket, stop, p.node_depth, p.node_count, p.leaf_slots);
                    const float* slot = p.leaf + sr.first * p.leaf_stride;
#pragma unroll 4
                    for (uint32_t s = 0; s < bucket_slots; ++s, slot += p.leaf_stride) {
                        int32_t id;
                        const float d2 = slot_dist<DP>(qq, slot, &id);
                        if (id >= 0 && d2 <= rq) {
                            // The slot is kept, not the key: half the shared memory, and the owner lane
                            // recomputes the same distance from it when it sorts its list.
                            const uint32_t pos = atomicAdd(&sm.cnt[ql], 1u);
                            if (pos < C) sm.buf[pos][ql] = static_cast<uint32_t>(sr.first) + s;
                        }
                    }
                    ++pairs;
                }
                __syncwarp();
            }
        };

        for (uint32_t round = 0; __any_sync(FULL, pending); ++round) {
            const float rl = pending ? r : -1.0f;
            sm.cnt[lane] = 0;
            sm.rad[lane] = rl;
            __syncwarp();
            uint32_t top = 0, nlist = 0;
            const uint32_t m0 = __ballot_sync(FULL, box_bound<DP>(q, p.box) <= rl);
            if (m0) {
                if (stop == 0) {
                    if (lane == 0) sm.list[0] = m0;
                    nlist = 1;
                } else {
                    if (lane == 0) sm.stack[0] = 0;
                    top = 1;
                }
            }
            while (top) {
                __syncwarp();
                const uint32_t node = sm.stack[--top];
                // The node's descendants `levels` below (up to 8, contiguous in the heap order) are
                // tested at once: their box loads are independent, so they overlap in flight.
                const uint32_t levels = min(kGroupFan, stop - heap_depth(node));
                const uint32_t fan = 1u << levels;
                const uint32_t first = ((node + 1) << levels) - 1;
                uint32_t want[1u << kGroupFan];
#pragma unroll
                for (uint32_t j = 0; j < (1u << kGroupFan); ++j) {
                    // (j < fan first: with an unbounded radius an infinite bound is still "within".)
                    const bool in = j < fan && box_bound<DP>(q, p.box + static_cast<size_t>(first + j) * p.box_stride) <= rl;
                    want[j] = __ballot_sync(FULL, in);
                }
                ++nodes;
                if (heap_depth(node) + levels == stop) {
#pragma unroll
                    for (uint32_t j = 0; j < (1u << kGroupFan); ++j) {
                        if (want[j]) {
                            if (lane == 0) sm.list[nlist] = (static_cast<uint64_t>(first + j) << 32) | want[j];
                            ++nlist;
                        }
                    }
                    if (nlist + (1u << kGroupFan) > kGroupList) {
                        __syncwarp();
                        scan(nlist);
                        nlist = 0;
                    }
                } else {
                    if (top + (1u << kGroupFan) > kGroupStack) {  // cannot happen (see kGroupStack); recorded
                        stack_error = true;
                        continue;
                    }
#pragma unroll
                    for (uint32_t j = (1u << kGroupFan); j-- > 0;) {
                        if (want[j]) {
                            if (lane == 0) sm.stack[top] = first + j;
                            ++top;
                        }
                    }
                }
            }
            if (nlist) {
                __syncwarp();
                scan(nlist);
            }
            __syncwarp();
            if (pending) {
                const uint32_t c = sm.cnt[lane];
                // The k smallest keys among the first n listed candidates (their distances
                // recomputed from the slots, four loads in flight).
                auto select = [&](Tracker<KMAX, false, false>& tr, uint32_t n) {
                    uint32_t i = 0;
                    for (; i + 4 <= n; i += 4) {
                        int32_t id[4];
                        float d2[4];
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u)
                            d2[u] = slot_dist<DP>(q, p.leaf + static_cast<size_t>(sm.buf[i + u][lane]) * p.leaf_stride, &id[u]);
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) tr.offer(make_key(d2[u], id[u]));
                    }
                    for (; i < n; ++i) {
                        int32_t id;
                        const float d2 = slot_dist<DP>(q, p.leaf + static_cast<size_t>(sm.buf[i][lane]) * p.leaf_stride, &id);
                        tr.offer(make_key(d2, id));
                    }
                };
                if (c > C) {
                    // More candidates than the list holds.  The k-th smallest distance among the C
                    // kept bounds the k-th neighbour's (k real points lie within it): its
                    // own search starts from it.  (Walking again with a radius shrunk by the
                    // density was tried: the extra rounds cost more than the searches they save.)
                    Tracker<KMAX, false, false> tr;
                    tr.init(p.k, r, nullptr, 0);
                    select(tr, C);
                    const uint32_t pos = atomicAdd(gp.fb_count, 1u);
                    gp.fb_list[pos] = qi;
                    gp.seeds[qi] = fminf(tr.radius(), r);
                    if (p.counters) atomicAdd(&p.counters->fallback, 1ull);
                    pending = false;
                } else if (c >= p.k || !(r < R)) {
                    Tracker<KMAX, false, false> tr;
                    tr.init(p.k, R, nullptr, 0);
                    select(tr, c);
                    tr.emit(p.k, p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
                    pending = false;
                } else if (round + 1 >= kGroupRounds) {
                    const uint32_t pos = atomicAdd(gp.fb_count, 1u);
                    gp.fb_list[pos] = qi;
                    gp.seeds[qi] = R;
                    if (p.counters) atomicAdd(&p.counters->fallback, 1ull);
                    pending = false;
                } else {
                    // Fewer than k within r: grow r^2 by the volume ratio k points need at the density
                    // seen, (1.5 k / c)^(2 / dims), between 1.25 and 16.
                    const float ce = fmaxf(static_cast<float>(c), 0.5f);
                    const float grow = fminf(fmaxf(exp2f(log2f(1.5f * static_cast<float>(p.k) / ce) * (2.0f / p.dims)),
                                                   1.25f), 16.0f);
                    r = fminf(R, fmaxf(r * grow, 1e-30f));
                }
            }
            __syncwarp();
        }
    }
    if (p.counters) {
        // nodes: walk steps (each tests up to 8 descendants); leaves: (bucket, query) pairs.
        if (lane == 0) {
            atomicAdd(&p.counters->nodes, static_cast<unsigned long long>(nodes));
            if (stack_error) atomicExch(&p.counters->error, 1);
        }
        if (pairs) {
            atomicAdd(&p.counters->leaves, static_cast<unsigned long long>(pairs));
            atomicAdd(&p.counters->points, static_cast<unsigned long long>(pairs) * bucket_slots);
        }
    }
}

// One query per warp (warp_search.cuh) against the tight node boxes: the default search, and the
// group search's leftovers.  1,048,576 queries, k 16, on 4.19 M clustered 3-d points: 1.76 ms, 8.5
// boxes of 32 tested and 7.5 buckets of 32 slots scanned per query; a thread per query took 3.2 ms
// over the same boxes and 38 to 60 ms with splitting planes only (their bound prunes little in the
// space between clusters).  10,000 uniform 11-d queries within a radius on 500,000 points: 1.8 ms
// (28 and 145 ms).  Bound by the instructions of the top-k insertions and box tests at C2's shape,
// by L2 reads of boxes and slots in more dimensions.
template <int DP, int NQ>
struct KdWarpView {
    static constexpr bool kKeys = false;      // the nearest box first
    static constexpr bool kShared = DP > 32;  // wide queries are read from shared memory (broadcast)
    float q[kShared ? 1 : DP];
    const float4* sq;
    const float* box;
    uint32_t box_stride, quads;  // quads: groups of four dimensions in use, NQ at most where that is known
                                 // at compile time (the padding beyond adds exactly 0)
    __device__ __forceinline__ void test(uint32_t node, float* bound, uint32_t*) const {
        const float* b = box + static_cast<size_t>(node) * box_stride;
        if constexpr (DP == 16 || DP == 32) {
            const float4* lo4 = reinterpret_cast<const float4*>(b);
            *bound = box_bound<4 * NQ>(reinterpret_cast<const float(&)[4 * NQ]>(q), lo4, lo4 + DP / 4, 0.0f);
        } else if constexpr (kShared) {
            const float4* lo4 = reinterpret_cast<const float4*>(b);
            const float4* hi4 = reinterpret_cast<const float4*>(b + DP);
            float acc = 0.0f;
#pragma unroll 4
            for (uint32_t v = 0; v < quads; ++v) {
                const float4 a = sq[v];
                const float qq[4] = {a.x, a.y, a.z, a.w};
                acc = box_bound<4>(qq, lo4 + v, hi4 + v, acc);
            }
            *bound = acc;
        } else {
            *bound = box_bound<DP>(q, b);
        }
    }
    __device__ __forceinline__ float dist(const float* slot, int32_t* id) const {
        if constexpr (kShared) {
            *id = __float_as_int(slot[DP]);
            return dist2_shared(sq, reinterpret_cast<const float4*>(slot), quads);
        } else if constexpr (DP == 16 || DP == 32) {
            *id = __float_as_int(slot[DP]);
            return dist2_vec4<4 * NQ>(reinterpret_cast<const float(&)[4 * NQ]>(q), reinterpret_cast<const float4*>(slot));
        } else {
            return slot_dist<DP>(q, slot, id);
        }
    }
};

template <int DP>
struct KdWarpSmem {
    WarpRows<false> rows;
    float4 q[DP > 32 ? DP / 4 : 1];
};

// One warp's search of query qi within r2; its row goes to the query's result slots.
template <int DP, int NQ, int KR, bool SEEDED>
__device__ __forceinline__ void kd_warp_query(const KdParams& p, uint32_t qi, float r2, KdWarpSmem<DP>& sm) {
    const uint32_t lane = threadIdx.x & 31u;
    KdWarpView<DP, NQ> view;
    if constexpr (DP > 32) {
        stage_query<DP>(p.queries, p.dims, qi, lane, sm.q);
        view.sq = sm.q;
    } else {
        load_query<DP>(p.queries, p.dims, qi, view.q);
    }
    view.box = p.box;
    view.box_stride = p.box_stride;
    view.quads = (p.dims + 3) / 4;
    const WarpTree t{p.leaf, p.leaf_stride, p.leaf_slots << (p.node_depth - p.stop_depth), p.stop_depth};
    WarpTopK<KR> top;
    LocalCounters lc;
    bool missed = false;
    top.init(p.k, r2, lane);
    if constexpr (SEEDED) {
        const float r = p.seeds[qi] * p.seed_scale;
        missed = warp_search<KdWarpView<DP, NQ>, KR, true>(view, t, sm.rows, top, lc, r < r2 ? r : r2, r2);
    } else {
        warp_search<KdWarpView<DP, NQ>, KR, false>(view, t, sm.rows, top, lc, r2, r2);
    }
    top.emit(p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
    if (p.counters && lane == 0) {
        lc.flush(p.counters);
        if (missed) atomicAdd(&p.counters->fallback, 1ull);
    }
}

template <int DP, int NQ, int KR, bool SEEDED>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) kd_warp_query_kernel(const KdParams p) {
    __shared__ KdWarpSmem<DP> sm[kWarpsPerBlock];
    const uint32_t w = threadIdx.x >> 5, t = blockIdx.x * kWarpsPerBlock + w;
    if (t >= (p.count_dev ? *p.count_dev : p.nq)) return;  // no block-wide barriers
    const uint32_t qi = p.order ? p.order[t] : t;
    kd_warp_query<DP, NQ, KR, SEEDED>(p, qi, p.radii ? p.radii[qi] : p.max_d2, sm[w]);
}

// The group search's leftovers, each within its radius in `seeds`; warps stride over the list.
template <int DP>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) kd_leftover_kernel(const KdGroupParams gp) {
    __shared__ KdWarpSmem<DP> sm[kWarpsPerBlock];
    const uint32_t w = threadIdx.x >> 5, n = *gp.fb_count;
    for (uint32_t t = blockIdx.x * kWarpsPerBlock + w; t < n; t += gridDim.x * kWarpsPerBlock) {
        const uint32_t qi = gp.fb_list[t];
        kd_warp_query<DP, warp_quads(DP, DP), 1, false>(gp.p, qi, gp.seeds[qi], sm[w]);
        __syncwarp();
    }
}

// Self seeds: each query's k-th distance among the points of the subtree of at least
// max(4k, 32) slots it descends to -- an upper bound on its k-th neighbour distance (those
// points are real points), capped by the caller's radius.  The caller's radius where the
// subtree holds fewer than k points.
template <int DP, int KMAX>
__global__ void __launch_bounds__(128) kd_self_seed_kernel(const KdParams p, uint32_t seed_depth, float* __restrict__ seeds) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p.nq) return;
    const uint32_t qi = p.order ? p.order[t] : t;
    float q[DP];
    load_query<DP>(p.queries, p.dims, qi, q);
    const float R = p.radii ? p.radii[qi] : p.max_d2;
    uint32_t node = 0;
    for (uint32_t depth = 0; depth < seed_depth; ++depth) {
        const float diff = pick<DP>(q, depth % p.aux) - __ldg(p.split + node);
        node = 2 * node + (diff < 0.0f ? 1u : 2u);
    }
    Tracker<KMAX, false, false> tr;
    tr.init(p.k, R, nullptr, 0);
    const SlotRange sr = subtree_slots(node, seed_depth, p.node_depth, p.node_count, p.leaf_slots);
    const float* slot = p.leaf + sr.first * p.leaf_stride;
    for (uint32_t s = 0; s < sr.count; ++s, slot += p.leaf_stride) {
        int32_t id;
        const float d2 = slot_dist<DP>(q, slot, &id);
        if (id >= 0) tr.offer(make_key(d2, id));
    }
    seeds[qi] = tr.radius();  // the caller's radius while fewer than k points were offered
}

// Tight boxes of the nodes at `depth` (per node lo[QS], hi[QS]; padding slots excluded).  Up to 16 dims
// min(32, slots) lanes share a node, a slot each at a time, and fold their corners by shuffles; beyond,
// a warp goes through a node's slots with its lanes over the dimensions.  Either way neighbouring lanes
// read neighbouring memory and no thread has more than a 32nd of a large node's slots or dimensions.
template <int DP>
__global__ void __launch_bounds__(128) kd_box_bottom_kernel(const float* __restrict__ leaf, uint32_t leaf_stride,
                                                            uint32_t depth, uint32_t slots, float* __restrict__ box) {
    constexpr int QS = box_qs(DP);
    const uint32_t lanes = DP > 16 ? 32u : min(slots, 32u);  // powers of two
    const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t l = threadIdx.x & (lanes - 1u);
    const uint64_t i = t / lanes;
    const bool live = i < (1u << depth);
    const float* slot = leaf + static_cast<size_t>(live ? i : 0) * slots * leaf_stride;
    float* out = box + ((static_cast<size_t>(1) << depth) - 1 + i) * (2 * QS);
    if constexpr (DP > 16) {
        constexpr int N = DP / 32;
        float lo[N], hi[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            lo[j] = INFINITY;
            hi[j] = -INFINITY;
        }
        if (!live) return;
#pragma unroll 4
        for (uint32_t s = 0; s < slots; ++s, slot += leaf_stride) {
            const bool point = __float_as_int(slot[DP]) >= 0;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const float x = slot[32 * j + l];
                lo[j] = point ? fminf(lo[j], x) : lo[j];
                hi[j] = point ? fmaxf(hi[j], x) : hi[j];
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            out[32 * j + l] = lo[j];
            out[QS + 32 * j + l] = hi[j];
        }
    } else {
        float lo[DP], hi[DP];
#pragma unroll
        for (int d = 0; d < DP; ++d) {
            lo[d] = INFINITY;
            hi[d] = -INFINITY;
        }
        for (uint32_t s = l; live && s < slots; s += lanes) {
            const float* x = slot + static_cast<size_t>(s) * leaf_stride;
            if (__float_as_int(x[DP]) < 0) continue;  // padding
#pragma unroll
            for (int d = 0; d < DP; ++d) {
                lo[d] = fminf(lo[d], x[d]);
                hi[d] = fmaxf(hi[d], x[d]);
            }
        }
        for (uint32_t m = lanes / 2; m; m /= 2) {
#pragma unroll
            for (int d = 0; d < DP; ++d) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xFFFFFFFFu, lo[d], m));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xFFFFFFFFu, hi[d], m));
            }
        }
        if (!live || l) return;
#pragma unroll
        for (int d = 0; d < QS; ++d) {
            out[d] = d < DP ? lo[d < DP ? d : 0] : 0.0f;
            out[QS + d] = d < DP ? hi[d < DP ? d : 0] : 0.0f;
        }
    }
}

// Nodes whose boxes one block of kd_box_up_kernel folds (a power of two; 32 KB of shared memory at most).
constexpr uint32_t box_up_nodes(uint32_t qs) { return qs <= 16 ? 256u : 4096u / qs; }

// Boxes of up to log2(T) levels above `depth`: a block loads the boxes of T neighbouring nodes there
// and folds them pairwise in shared memory (one launch instead of one per level, whose tiny grids
// near the root each cost a launch).
template <int QS>
__global__ void kd_box_up_kernel(float* __restrict__ box, uint32_t depth, uint32_t levels) {
    constexpr uint32_t T = box_up_nodes(QS);
    __shared__ float sb[T][2 * QS];
    const uint32_t t = threadIdx.x, first = blockIdx.x * T;
    uint32_t nodes = min(T, (1u << depth) - first);
    if (t < nodes) {
        const float* in = box + ((1u << depth) - 1u + first + t) * static_cast<size_t>(2 * QS);
#pragma unroll 8
        for (int d = 0; d < 2 * QS; ++d) sb[t][d] = in[d];
    }
    for (uint32_t l = 1; l <= levels; ++l) {
        nodes >>= 1;
        for (int d = 0; d < QS; ++d) {
            __syncthreads();
            float lo = 0.0f, hi = 0.0f;
            if (t < nodes) {
                lo = fminf(sb[2 * t][d], sb[2 * t + 1][d]);
                hi = fmaxf(sb[2 * t][QS + d], sb[2 * t + 1][QS + d]);
            }
            __syncthreads();
            if (t < nodes) {
                sb[t][d] = lo;
                sb[t][QS + d] = hi;
                float* out = box + ((1u << (depth - l)) - 1u + (first >> l) + t) * static_cast<size_t>(2 * QS);
                out[d] = lo;
                out[QS + d] = hi;
            }
        }
    }
}

template <int DP, int KMAX>
static int launch_kd_group(knn_index* ix, const knn_index::KdBoxes& boxes, const QueryArgs& a, const QueryPlan& plan,
                           const uint32_t* order, float* seeds, uint32_t* fb_list, uint32_t* fb_count, cudaStream_t s) {
    KdGroupParams gp{};
    gp.p = kd_box_params(ix, boxes, a, order, plan.leaf_scan ? plan.leaf_scan : 8u);
    gp.seeds = seeds;
    gp.fb_list = fb_list;
    gp.fb_count = fb_count;
    gp.group_counter = fb_count + 1;  // the count's scratch slot holds 256 bytes
    KNN_TRY_CUDA(cudaMemsetAsync(fb_count, 0, 2 * sizeof(uint32_t), s));
    // Self seeds from a subtree of at least max(4k, 32) slots.
    const uint32_t want = std::max<uint32_t>(32u, 4u * a.k);
    uint32_t sd = ix->node_depth;
    while (sd > 0 && (static_cast<uint64_t>(ix->leaf_slots) << (ix->node_depth - sd)) < want) --sd;
    kd_self_seed_kernel<DP, KMAX><<<ceil_div(a.count, 128), 128, 0, s>>>(gp.p, sd, seeds);
    KNN_LAUNCHED();
    constexpr size_t smem = group_smem_bytes<DP, KMAX>();
    auto kern = kd_group_kernel<DP, KMAX>;
    KNN_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    int per_sm = 0;
    KNN_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kGroupWarps, smem));
    const uint32_t grid = std::min<uint32_t>(ceil_div(a.count, 32 * kGroupWarps),
                                             static_cast<uint32_t>(std::max(per_sm, 1) * sm_count()));
    kern<<<grid, 32 * kGroupWarps, smem, s>>>(gp);
    KNN_LAUNCHED();
    kd_leftover_kernel<DP><<<8 * static_cast<uint32_t>(sm_count()), 32 * kWarpsPerBlock, 0, s>>>(gp);
    KNN_LAUNCHED();
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return KNN_OK;
}

// Bucket slots at least (plans may ask for more).  A warp scans 32 slots at once, and the fewer, larger
// buckets of 32 are the cheapest in few dimensions (4.19 M 3-d points: 1.76 ms, 8% more with 8); in more
// the boxes of smaller ones prune more (11 dims: 1.8 ms with 16, a fifth more with 32).
inline uint32_t kd_warp_bucket(uint32_t dims) { return dims <= 8 ? 32u : 16u; }

// Enqueues the build of the node boxes down to subtrees of at most `bucket` slots (0: the default
// search's) into boxes of their own.
template <uint32_t DP>
int kd_box_build_dp(const knn_index* ix, uint32_t bucket, knn_index::KdBoxes* boxes, cudaStream_t s) {
    constexpr uint32_t QS = box_qs(DP), T = box_up_nodes(QS);
    boxes->depth = scan_depth_for(ix->node_depth, ix->leaf_slots, bucket ? bucket : kd_warp_bucket(ix->dims));
    // Leaves beyond 256 slots are read in parts, levels below the tree's that only this build knows: two
    // leaves of 65,536 slots and 40 dims would take two warps 7 ms.
    uint32_t bottom = boxes->depth, slots = ix->leaf_slots << (ix->node_depth - bottom);
    for (; slots > 256; slots /= 2) ++bottom;
    KNN_TRY(boxes->buf.alloc(((static_cast<size_t>(2) << bottom) - 1) * 2 * QS * sizeof(float)));
    float* box = boxes->buf.as<float>();
    const uint64_t threads = static_cast<uint64_t>(DP > 16 ? 32u : std::min(slots, 32u)) << bottom;
    kd_box_bottom_kernel<DP><<<static_cast<uint32_t>((threads + 127) / 128), 128, 0, s>>>(
        ix->leaf.as<float>(), ix->leaf_stride, bottom, slots, box);
    KNN_LAUNCHED();
    for (uint32_t depth = bottom, levels = 0; depth; depth -= levels) {
        for (levels = 0; levels < depth && (2u << levels) <= T; ++levels) {}
        kd_box_up_kernel<QS><<<ceil_div(1u << depth, T), T, 0, s>>>(box, depth, levels);
        KNN_LAUNCHED();
    }
    return KNN_OK;
}

template <uint32_t DP>
int kd_warp_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order, cudaStream_t s) {
    const KdParams p = kd_box_params(ix, ix->kd_box, a, order, std::max(plan.leaf_scan, kd_warp_bucket(ix->dims)));
    const uint32_t grid = ceil_div(a.count, kWarpsPerBlock), threads = 32 * kWarpsPerBlock;
    void (*kern)(const KdParams) = nullptr;
    with_quads<DP>(ix->dims, [&](auto nq) {
        constexpr int NQ = decltype(nq)::value;
        if (p.seeds)
            kern = a.k <= 32 ? kd_warp_query_kernel<DP, NQ, 1, true> : a.k <= 64 ? kd_warp_query_kernel<DP, NQ, 2, true> : kd_warp_query_kernel<DP, NQ, 4, true>;
        else
            kern = a.k <= 32 ? kd_warp_query_kernel<DP, NQ, 1, false> : a.k <= 64 ? kd_warp_query_kernel<DP, NQ, 2, false> : kd_warp_query_kernel<DP, NQ, 4, false>;
    });
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    kern<<<grid, threads, 0, s>>>(p);
    KNN_LAUNCHED();
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return KNN_OK;
}

// Warp-group search (plan.group) from each query's own subtree: its boxes built on first use, the group
// kernel in the batch's locality order, then the leftovers.
template <uint32_t DP>
int kd_group_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, const uint32_t* order, cudaStream_t s) {
    if constexpr (DP > 16) {
        return fail(KNN_ERR_INVALID_ARGUMENT, "group search: dims above 16");
    } else {
        if (a.k > 32) return fail(KNN_ERR_INVALID_ARGUMENT, "group search: k above 32");
        // Boxes of subtrees of 4 slots, as its plans may scan; a tree whose leaves are as large as the
        // default search's buckets has one set of boxes for both.
        knn_index::KdBoxes& boxes = ix->leaf_slots >= kd_warp_bucket(ix->dims) ? ix->kd_box : ix->kd_fine_box;
        KNN_TRY(kd_box_ensure(ix, boxes, 4, s));
        const size_t n = a.count;
        KNN_TRY(ix->group_ws.reserve(carve_bytes({n * 4, n * 4, 256})));
        Carver c(ix->group_ws.ptr);
        float* seeds = c.take<float>(n);
        uint32_t* fb_list = c.take<uint32_t>(n);
        uint32_t* fb_count = c.take<uint32_t>(1);
        switch (k_class(a.k)) {
            case 8: return launch_kd_group<DP, 8>(ix, boxes, a, plan, order, seeds, fb_list, fb_count, s);
            case 16: return launch_kd_group<DP, 16>(ix, boxes, a, plan, order, seeds, fb_list, fb_count, s);
            default: return launch_kd_group<DP, 32>(ix, boxes, a, plan, order, seeds, fb_list, fb_count, s);
        }
    }
}

template int kd_query_dp<KNN_DP>(knn_index*, const QueryArgs&, const QueryPlan&, cudaStream_t);
template int kd_box_build_dp<KNN_DP>(const knn_index*, uint32_t, knn_index::KdBoxes*, cudaStream_t);
template int kd_order_dp<KNN_DP>(knn_index*, const QueryArgs&, cudaStream_t, const uint32_t**);


// ---- batches of independent sets (one persistent kernel per class of sets) -----------------------
struct KdBatchSet {
    KdParams p;                 // the set's search parameters; p.order is the class order, p.order_base its offset
    uint32_t first_block;  // first work block of this set in the class
    uint32_t query_offset; // first query of this set in the class-wide numbering
    uint32_t levels;       // descent depth of the locality key
};

__device__ __forceinline__ uint32_t kd_find_set(const KdBatchSet* sets, uint32_t nsets, uint32_t item, bool by_query) {
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
__global__ void kd_batch_key_kernel(const KdBatchSet* __restrict__ sets, uint32_t nsets, uint32_t total,
                                     uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const uint32_t si = kd_find_set(sets, nsets, g, true);
    const KdParams& p = sets[si].p;
    float q[DP];
    load_query<DP>(p.queries, p.dims, g - sets[si].query_offset, q);
    const uint32_t levels = sets[si].levels;
    uint32_t node = 0;
    for (uint32_t d = 0; d < levels; ++d) {
        const float diff = pick<DP>(q, d % p.aux) - __ldg(p.split + node);
        node = 2 * node + (diff < 0.0f ? 1u : 2u);
    }
    keys[g] = (si << 24) | ((node - ((1u << levels) - 1u)) << (24 - levels));
    vals[g] = g;
}

// Persistent kernel: blocks take work blocks (blockDim queries of one set) from a shared counter
// until the class is done; sets of very different sizes share the GPU without a launch each.
// MODE: 0 per-thread search, 1 warp-coherent search.
template <int DP, int KMAX, int MODE>
__global__ void __launch_bounds__(256) kd_batch_kernel(const KdBatchSet* __restrict__ sets, uint32_t nsets,
                                                        uint32_t total_blocks, uint32_t* __restrict__ counter) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t item_s;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) item_s = atomicAdd(counter, 1u);
        __syncthreads();
        const uint32_t item = item_s;
        if (item >= total_blocks) break;
        const uint32_t si = kd_find_set(sets, nsets, item, false);
        const KdParams& p = sets[si].p;
        const uint32_t t = (item - sets[si].first_block) * blockDim.x + threadIdx.x;
        if constexpr (MODE == 1) {
            kd_search_warp<DP, KMAX, false, false, false>(p, t, p.nq, smem);
        } else {
            if (t < p.nq) kd_search_thread<DP, KMAX, false, false, false>(p, t, smem);
        }
    }
}

// A warp per query over the sets' node boxes: persistent warps take the class's queries one by one.
template <int DP, int KR>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) kd_batch_warp_kernel(const KdBatchSet* __restrict__ sets,
                                                                           uint32_t nsets, uint32_t total_queries,
                                                                           uint32_t* __restrict__ counter) {
    __shared__ KdWarpSmem<DP> sm[kWarpsPerBlock];
    for (;;) {
        uint32_t g = 0;
        if ((threadIdx.x & 31u) == 0) g = atomicAdd(counter, 1u);
        g = __shfl_sync(kFullMask, g, 0);
        if (g >= total_queries) break;  // no block-wide barriers
        const uint32_t si = kd_find_set(sets, nsets, g, true);
        const KdParams& p = sets[si].p;
        const uint32_t t = g - sets[si].query_offset;
        const uint32_t qi = p.order ? p.order[t] - p.order_base : t;
        kd_warp_query<DP, warp_quads(DP, DP), KR, false>(p, qi, p.max_d2, sm[threadIdx.x >> 5]);
        __syncwarp();
    }
}

template <uint32_t DP>
int kd_batch_launch(const void* sets, uint32_t nsets, uint32_t total_queries, uint32_t total_blocks, uint32_t kmax,
                       uint32_t mode, uint32_t block, uint32_t* counter, uint32_t* keys, uint32_t* vals, bool key_pass,
                       cudaStream_t s) {
    using Set = KdBatchSet;
    const Set* d_sets = static_cast<const Set*>(sets);
    if (key_pass) {
        kd_batch_key_kernel<DP><<<ceil_div(total_queries, 256), 256, 0, s>>>(d_sets, nsets, total_queries, keys, vals);
        KNN_LAUNCHED();
        return KNN_OK;
    }
#define KNN_BATCH(KM, W)                                                                              \
    if (kmax == KM && mode == W) {                                                                    \
        auto kern = kd_batch_kernel<DP, KM, W>;                                                    \
        int per_sm = 0;                                                                               \
        KNN_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, 0));         \
        const uint32_t grid = std::max(1, per_sm) * static_cast<uint32_t>(sm_count());                \
        kern<<<std::min(grid, total_blocks), block, 0, s>>>(d_sets, nsets, total_blocks, counter);   \
        KNN_LAUNCHED();                                                                               \
        return KNN_OK;                                                                                \
    }
    KNN_BATCH(8, 0) KNN_BATCH(16, 0) KNN_BATCH(32, 0) KNN_BATCH(64, 0) KNN_BATCH(128, 0)
    KNN_BATCH(8, 1) KNN_BATCH(16, 1) KNN_BATCH(32, 1) KNN_BATCH(64, 1) KNN_BATCH(128, 1)
#undef KNN_BATCH
    if (mode == 2) {
        auto kern = kmax <= 32 ? kd_batch_warp_kernel<DP, 1> : kmax <= 64 ? kd_batch_warp_kernel<DP, 2> : kd_batch_warp_kernel<DP, 4>;
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
// Fills the search parameters of one batch set from its index and item (plan.box: a warp per query).
size_t kd_batch_set_bytes() { return sizeof(KdBatchSet); }

void kd_batch_set_fill(void* out, const knn_index* ix, const QueryArgs& a, const QueryPlan& plan,
                        const uint32_t* order, uint32_t order_base, uint32_t first_block, uint32_t query_offset) {
    KdBatchSet bs{};
    // (A class of warp-per-query searches has every index's boxes.)
    bs.p = plan.box ? kd_box_params(ix, ix->kd_box, a, order, std::max(plan.leaf_scan, kd_warp_bucket(ix->dims)))
                    : kd_params(ix, a, order, plan.leaf_scan);
    bs.p.order_base = order_base;
    bs.first_block = first_block;
    bs.query_offset = query_offset;
    bs.levels = std::min<uint32_t>(ix->node_depth, 24);
    std::memcpy(out, &bs, sizeof(bs));
}
#endif

template int kd_batch_launch<KNN_DP>(const void*, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t*,
                                      uint32_t*, uint32_t*, bool, cudaStream_t);

}  // namespace knn
