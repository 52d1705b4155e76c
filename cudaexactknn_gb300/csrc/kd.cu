// k-d tree: construction and the query dispatcher over padded dimension counts.
//
// Replaces KdTreeGpu's constructor and mSplitPoints (src/KdTreeGpu.cuh:297-385).  Same tree:
// node_depth = log2Ceil(n) - skips levels of internal nodes in an implicit heap, split
// dimension = depth % aux_dims, a node of n points sends ceil(n/2) to the left child, the split
// value is the largest left value along the split dimension (src/KdTreeGpu.cuh:229-238), and
// leaves hold 2^skips slots padded with index -1 (src/KdTreeGpu.cuh:354-363).  The
// construction is the presorted-orders scheme of tree_build.cuh: aux_dims radix sorts up front,
// then per level one split kernel and one stable partition of the other orders.

#include <algorithm>
#include <vector>

#include "tree_build.cuh"

namespace knn {

template <uint32_t DP>
int kd_query_dp(knn_index*, const QueryArgs&, const QueryPlan&, cudaStream_t);
template <uint32_t DP>
int kd_order_dp(knn_index*, const QueryArgs&, cudaStream_t, const uint32_t**);
template <uint32_t DP>
int kd_box_build_dp(const knn_index*, uint32_t, knn_index::KdBoxes*, cudaStream_t);

namespace {

// Split value and side flags of level `level` from the split dimension's order.
__global__ void kd_split_kernel(const uint32_t* __restrict__ ord, const float* __restrict__ pts, uint32_t n,
                                uint32_t dims, uint32_t dim, const uint32_t* __restrict__ node_of,
                                const uint32_t* __restrict__ off, const uint32_t* __restrict__ size,
                                float* __restrict__ split_level, uint8_t* __restrict__ side) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint32_t j = node_of[p];
    const uint32_t rel = p - off[j], left = (size[j] + 1) / 2;
    const uint32_t id = ord[p];
    side[id] = rel >= left ? 1 : 0;
    if (rel + 1 == left) split_level[j] = pts[static_cast<size_t>(id) * dims + dim];
}

// Leaf slots: coordinates (zero padded to the leaf stride) then the index bits; empty slots
// carry index -1.
__global__ void write_leaves_kernel(const uint32_t* __restrict__ ord, const float* __restrict__ pts,
                                    uint32_t dims, uint32_t slots, uint32_t leaves,
                                    const uint32_t* __restrict__ off, const uint32_t* __restrict__ size,
                                    uint32_t stride, uint32_t id_at, float* __restrict__ leaf) {
    const uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= static_cast<uint64_t>(slots) * leaves) return;
    const uint32_t j = static_cast<uint32_t>(s / slots), r = static_cast<uint32_t>(s % slots);
    float* out = leaf + s * stride;
    int32_t id = -1;
    if (r < size[j]) id = static_cast<int32_t>(ord[off[j] + r]);
    for (uint32_t d = 0; d < stride; ++d) out[d] = 0.0f;
    if (id >= 0)
        for (uint32_t d = 0; d < dims; ++d) out[d] = pts[static_cast<size_t>(id) * dims + d];
    out[id_at] = __int_as_float(id);
}

__global__ void init_root_kernel(uint32_t* off, uint32_t* size, uint32_t n, uint32_t* node_of, uint32_t count) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) {
        off[0] = 0;
        size[0] = n;
    }
    if (p < count) node_of[p] = 0;
}

// ---- the lower levels: whole subtrees in shared memory -----------------------------------------------
// Once a node holds at most `cap` points (4,096 up to 16 orders), one block takes it and splits it down to
// the leaves: its segment of every order is read once, as local indices (16 bits) into its points, and
// every further level partitions the orders in shared memory.  A level over all n points in global
// memory took six launches and about 195 us at 4.19 M 3-d points, most of it streaming and gathering ids;
// twelve of its 22 levels run here instead, in 470 us.
// Bound by the barriers of two block scans a level.
constexpr uint32_t kSubItems = 8;      // positions per thread
constexpr uint32_t kSubCap = 4096;     // most points of a subtree

struct SubtreeParams {
    const uint32_t* ord[kMaxDims];  // the level's orders; ord[0] is rewritten in leaf order into out0
    uint32_t orders;                // orders in use
    uint32_t aux;                   // split dimension = depth % aux
    uint32_t level, depth;          // the subtrees' roots, the leaves
    uint32_t cap;
    const uint32_t* off;            // per root: first position, points
    const uint32_t* size;
    const float* pts;
    uint32_t dims;
    uint32_t* local;                // per point: its index within its subtree (scratch)
    float* split;
    uint32_t* out0;
    uint32_t* leaf_off;             // per leaf (leaf_size zero before the launch: an empty leaf is not written)
    uint32_t* leaf_size;
};

inline size_t subtree_smem(uint32_t cap, uint32_t orders) {
    return static_cast<size_t>(cap) * (2 * orders + 2 + 2 + 4 + 1) + 128;
}

__global__ void __launch_bounds__(kSubCap / kSubItems) kd_subtree_kernel(const SubtreeParams t) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    __shared__ uint32_t warp_sum[kSubCap / kSubItems / 32];
    const uint32_t cap = t.cap, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t* gid = reinterpret_cast<uint32_t*>(sub_smem);           // global id of each local index
    uint16_t* ord = reinterpret_cast<uint16_t*>(gid + cap);          // [orders][cap]
    uint16_t* next = ord + static_cast<size_t>(t.orders) * cap;
    uint16_t* pre = next + cap;                                      // left flags before each position
    uint8_t* right = reinterpret_cast<uint8_t*>(pre + cap);          // side of each local index
    const uint32_t base = t.off[blockIdx.x], m = t.size[blockIdx.x];
    for (uint32_t p = tid; p < m; p += blockDim.x) {
        const uint32_t id = t.ord[0][base + p];
        gid[p] = id;
        t.local[id] = p;
        ord[p] = static_cast<uint16_t>(p);
    }
    __threadfence();  // (they are read back past L1, below)
    __syncthreads();
    // (Past L1: a line there may hold another subtree's entries from before this block wrote its own.)
    for (uint32_t a = 1; a < t.orders; ++a)
        for (uint32_t p = tid; p < m; p += blockDim.x)
            ord[a * cap + p] = static_cast<uint16_t>(__ldcg(t.local + t.ord[a][base + p]));
    // This thread's positions and, for each, its node: first position, points, index within the level.
    uint32_t off[kSubItems], size[kSubItems], node[kSubItems];
    const uint32_t p0 = tid * kSubItems;
#pragma unroll
    for (uint32_t i = 0; i < kSubItems; ++i) {
        off[i] = 0;
        size[i] = m;
        node[i] = blockIdx.x;
    }
    for (uint32_t d = t.level; d < t.depth; ++d) {
        const uint32_t dim = d % t.aux;
        const uint16_t* by = ord + static_cast<size_t>(dim) * cap;
        __syncthreads();  // the orders are complete
#pragma unroll
        for (uint32_t i = 0; i < kSubItems; ++i) {
            const uint32_t p = p0 + i;
            if (p >= m) continue;
            const uint32_t left = (size[i] + 1) / 2, id = by[p];
            right[id] = p - off[i] >= left ? 1 : 0;
            if (p - off[i] + 1 == left)
                t.split[(1u << d) - 1u + node[i]] = t.pts[static_cast<size_t>(gid[id]) * t.dims + dim];
        }
        __syncthreads();
        for (uint32_t a = 0; a < t.orders; ++a) {
            // An order that no level below splits by is not needed (the first one: the leaves).
            if (a == dim) continue;
            uint32_t again = d + 1 + (a + t.aux - (d + 1) % t.aux) % t.aux;
            if (a && again >= t.depth) continue;
            uint16_t* o = ord + static_cast<size_t>(a) * cap;
            uint32_t id[kSubItems], f = 0, c = 0;
#pragma unroll
            for (uint32_t i = 0; i < kSubItems; ++i) {
                const bool in = p0 + i < m;
                id[i] = in ? o[p0 + i] : 0u;
                const uint32_t l = in && right[id[i]] == 0 ? 1u : 0u;
                f |= l << i;
                c += l;
            }
            uint32_t incl = c;
#pragma unroll
            for (uint32_t s = 1; s < 32; s <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, s);
                if (lane >= s) incl += v;
            }
            if (lane == 31) warp_sum[warp] = incl;
            __syncthreads();
            uint32_t run = incl - c;
            for (uint32_t w = 0; w < warp; ++w) run += warp_sum[w];
            uint32_t mine[kSubItems];
#pragma unroll
            for (uint32_t i = 0; i < kSubItems; ++i) {
                mine[i] = run;
                if (p0 + i < m) pre[p0 + i] = static_cast<uint16_t>(run);
                run += f >> i & 1u;
            }
            __syncthreads();
#pragma unroll
            for (uint32_t i = 0; i < kSubItems; ++i) {
                const uint32_t p = p0 + i;
                if (p >= m) continue;
                const uint32_t lr = mine[i] - pre[off[i]];  // left entries of its node before it
                const uint32_t dst = f >> i & 1u ? off[i] + lr : off[i] + (size[i] + 1) / 2 + (p - off[i] - lr);
                next[dst] = static_cast<uint16_t>(id[i]);
            }
            __syncthreads();
#pragma unroll
            for (uint32_t i = 0; i < kSubItems; ++i)
                if (p0 + i < m) o[p0 + i] = next[p0 + i];
            // (The next writes to warp_sum and pre come after a barrier that follows this copy.)
        }
#pragma unroll
        for (uint32_t i = 0; i < kSubItems; ++i) {
            const uint32_t left = (size[i] + 1) / 2;
            const bool r = p0 + i - off[i] >= left;
            off[i] += r ? left : 0u;
            size[i] = r ? size[i] - left : left;
            node[i] = 2 * node[i] + (r ? 1u : 0u);
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < kSubItems; ++i) {
        const uint32_t p = p0 + i;
        if (p >= m) continue;
        t.out0[base + p] = gid[ord[p]];
        if (p == off[i]) {
            t.leaf_off[node[i]] = base + p;
            t.leaf_size[node[i]] = size[i];
        }
    }
}

int kd_box_build(const knn_index* ix, uint32_t bucket, knn_index::KdBoxes* boxes, cudaStream_t s) {
    switch (ix->dp) {
        case 1: return kd_box_build_dp<1>(ix, bucket, boxes, s);
        case 2: return kd_box_build_dp<2>(ix, bucket, boxes, s);
        case 3: return kd_box_build_dp<3>(ix, bucket, boxes, s);
        case 4: return kd_box_build_dp<4>(ix, bucket, boxes, s);
        case 8: return kd_box_build_dp<8>(ix, bucket, boxes, s);
        case 16: return kd_box_build_dp<16>(ix, bucket, boxes, s);
        case 32: return kd_box_build_dp<32>(ix, bucket, boxes, s);
        case 64: return kd_box_build_dp<64>(ix, bucket, boxes, s);
        case 128: return kd_box_build_dp<128>(ix, bucket, boxes, s);
        default: return fail(KNN_ERR_UNSUPPORTED, "dims %u", ix->dims);
    }
}

// The index takes boxes that the device has finished.
void kd_box_hold(knn_index* ix, knn_index::KdBoxes& held, knn_index::KdBoxes& boxes) {
    held.depth = boxes.depth;
    held.buf.swap(boxes.buf);
    ix->device_bytes += held.buf.bytes;
}

}  // namespace

// Leaf slot stride (floats) and position of the index within a slot.
void leaf_layout(uint32_t dp, uint32_t* stride, uint32_t* id_at) {
    if (dp < 4) {
        *stride = 4;
        *id_at = dp;
    } else {
        *stride = dp + 4;
        *id_at = dp;
    }
}

int kd_build(knn_index* ix, const float* d_points, uint32_t, cudaStream_t s) {
    const uint32_t n = ix->n, A = ix->aux_dims, nd = ix->node_depth;
    const uint32_t leaves = 1u << nd;
    leaf_layout(ix->dp, &ix->leaf_stride, &ix->leaf_id_at);
    KNN_TRY(ix->split.alloc(sizeof(float) * std::max<uint32_t>(ix->node_count, 1)));
    KNN_TRY(ix->leaf.alloc(sizeof(float) * static_cast<size_t>(leaves) * ix->leaf_slots * ix->leaf_stride));
    ix->device_bytes = ix->split.bytes + ix->leaf.bytes;

    // Orders are needed for the dimensions that some level splits by (and the first, the leaves' order).
    const uint32_t used = std::max(1u, std::min(A, nd));
    DevBuf scratch_buf;
    KNN_TRY(scratch_buf.alloc(build::scratch_bytes(n, used, leaves)));
    build::Scratch sc{};
    build::carve_scratch(sc, scratch_buf.ptr, n, used, leaves);

    for (uint32_t a = 0; a < used; ++a) KNN_TRY(build::sort_dimension(sc, d_points, n, ix->dims, a, a, s));

    init_root_kernel<<<ceil_div(n, 256), 256, 0, s>>>(sc.off[0], sc.size[0], n, sc.node_of[0], n);
    KNN_LAUNCHED();
    // Levels over all points until a node fits a block, then whole subtrees.
    uint32_t cap = kSubCap;
    while (cap * used > kSubCap * 16) cap /= 2;
    uint32_t top = 0;
    while (top < nd && (static_cast<uint64_t>(n) + (1u << top) - 1) >> top > cap) ++top;
    int cur = 0, tab = 0, nof = 0;
    std::vector<uint32_t> others;
    for (uint32_t level = 0; level < top; ++level) {
        const uint32_t count = 1u << level;
        const uint32_t dim = level % A;
        kd_split_kernel<<<ceil_div(n, 256), 256, 0, s>>>(sc.ord[cur][dim], d_points, n, ix->dims, dim,
                                                         sc.node_of[nof], sc.off[tab], sc.size[tab],
                                                         ix->split.as<float>() + (count - 1), sc.side);
        KNN_LAUNCHED();
        others.clear();
        for (uint32_t b = 0; b < used; ++b)
            if (b != dim) others.push_back(b);
        KNN_TRY(build::partition_orders(sc, others.data(), static_cast<uint32_t>(others.size()), cur,
                                        sc.node_of[nof], sc.off[tab], sc.size[tab], n, s));
        // The split order is already partitioned: its left entries lead each segment.
        std::swap(sc.ord[0][dim], sc.ord[1][dim]);
        build::next_node_of_kernel<<<ceil_div(n, 256), 256, 0, s>>>(sc.node_of[nof], sc.off[tab], sc.size[tab], n,
                                                                    sc.node_of[nof ^ 1]);
        build::children_kernel<<<ceil_div(count, 256), 256, 0, s>>>(sc.off[tab], sc.size[tab], count,
                                                                    sc.off[tab ^ 1], sc.size[tab ^ 1]);
        KNN_LAUNCHED_N(2);
        cur ^= 1;
        tab ^= 1;
        nof ^= 1;
    }
    const uint32_t* leaf_order = sc.ord[cur][0];
    if (top < nd) {
        SubtreeParams t{};
        for (uint32_t a = 0; a < used; ++a) t.ord[a] = sc.ord[cur][a];
        t.orders = used;
        t.aux = A;
        t.level = top;
        t.depth = nd;
        t.cap = cap;
        t.off = sc.off[tab];
        t.size = sc.size[tab];
        t.pts = d_points;
        t.dims = ix->dims;
        t.local = sc.node_of[nof ^ 1];
        t.split = ix->split.as<float>();
        t.out0 = sc.ord[cur ^ 1][0];
        t.leaf_off = sc.off[tab ^ 1];
        t.leaf_size = sc.size[tab ^ 1];
        KNN_TRY_CUDA(cudaMemsetAsync(t.leaf_size, 0, leaves * sizeof(uint32_t), s));
        const size_t smem = subtree_smem(cap, used);
        KNN_TRY_CUDA(cudaFuncSetAttribute(kd_subtree_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        kd_subtree_kernel<<<1u << top, cap / kSubItems, smem, s>>>(t);
        KNN_LAUNCHED();
        leaf_order = t.out0;
        tab ^= 1;
    }
    const uint64_t total_slots = static_cast<uint64_t>(leaves) * ix->leaf_slots;
    write_leaves_kernel<<<static_cast<uint32_t>((total_slots + 255) / 256), 256, 0, s>>>(
        leaf_order, d_points, ix->dims, ix->leaf_slots, leaves, sc.off[tab], sc.size[tab], ix->leaf_stride,
        ix->leaf_id_at, ix->leaf.as<float>());
    KNN_LAUNCHED();
    // The node boxes are part of the tree: whatever searches it later, on any stream, finds them finished.
    // Without memory for them the index is made all the same (the first query tries again).
    knn_index::KdBoxes boxes;
    const int rc = kd_box_build(ix, 0, &boxes, s);
    if (rc != KNN_OK && rc != KNN_ERR_OUT_OF_MEMORY) return rc;
    KNN_TRY_CUDA(cudaStreamSynchronize(s));  // scratch is freed on return
    if (rc == KNN_OK) kd_box_hold(ix, ix->kd_box, boxes);
    return KNN_OK;
}

int kd_query(knn_index* ix, const QueryArgs& a, const QueryPlan& p, cudaStream_t s) {
    switch (ix->dp) {
        case 1: return kd_query_dp<1>(ix, a, p, s);
        case 2: return kd_query_dp<2>(ix, a, p, s);
        case 3: return kd_query_dp<3>(ix, a, p, s);
        case 4: return kd_query_dp<4>(ix, a, p, s);
        case 8: return kd_query_dp<8>(ix, a, p, s);
        case 16: return kd_query_dp<16>(ix, a, p, s);
        case 32: return kd_query_dp<32>(ix, a, p, s);
        case 64: return kd_query_dp<64>(ix, a, p, s);
        case 128: return kd_query_dp<128>(ix, a, p, s);
        default: return fail(KNN_ERR_UNSUPPORTED, "dims %u", ix->dims);
    }
}

// Boxes built after the index was made.  It holds them only once the device has finished them: batch
// graphs, training and captured queries read them without waiting for the stream of the query that
// built them, and a build that failed leaves none.
int kd_box_ensure(knn_index* ix, knn_index::KdBoxes& held, uint32_t bucket, cudaStream_t s) {
    if (held.buf.ptr) return KNN_OK;
    knn_index::KdBoxes boxes;
    KNN_TRY(kd_box_build(ix, bucket, &boxes, s));
    KNN_TRY_CUDA(cudaStreamSynchronize(s));
    kd_box_hold(ix, held, boxes);
    return KNN_OK;
}

int kd_boxes_ready(knn_index* ix, cudaStream_t s, bool* ready) {
    *ready = ix->kd_box.buf.ptr != nullptr;
    if (*ready) return KNN_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    KNN_TRY_CUDA(cudaStreamIsCapturing(s, &cs));
    if (cs != cudaStreamCaptureStatusNone) return KNN_OK;
    const int rc = kd_box_ensure(ix, ix->kd_box, 0, s);
    *ready = rc == KNN_OK;
    return rc == KNN_ERR_OUT_OF_MEMORY ? KNN_OK : rc;
}

int kd_order(knn_index* ix, const QueryArgs& a, cudaStream_t s, const uint32_t** order) {
    switch (ix->dp) {
        case 1: return kd_order_dp<1>(ix, a, s, order);
        case 2: return kd_order_dp<2>(ix, a, s, order);
        case 3: return kd_order_dp<3>(ix, a, s, order);
        case 4: return kd_order_dp<4>(ix, a, s, order);
        case 8: return kd_order_dp<8>(ix, a, s, order);
        case 16: return kd_order_dp<16>(ix, a, s, order);
        case 32: return kd_order_dp<32>(ix, a, s, order);
        case 64: return kd_order_dp<64>(ix, a, s, order);
        case 128: return kd_order_dp<128>(ix, a, s, order);
        default: return fail(KNN_ERR_UNSUPPORTED, "dims %u", ix->dims);
    }
}

}  // namespace knn
