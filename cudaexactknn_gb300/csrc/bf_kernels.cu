// Brute-force exact kNN, one translation unit per padded dimension count (KNN_DP): the launch of
// bf_warp_kernel or bf_thread_kernel (bf_kernels.cuh) on an index's padded points.

#include "bf_kernels.cuh"

#ifndef KNN_DP
#error "compile with -DKNN_DP=<padded dims>"
#endif

namespace knn {

template <int DP, int KR>
static int launch_bf(knn_index* ix, const BfParams& args, const QueryPlan& plan, cudaStream_t s) {
    BfParams p = args;
    const BfShape shape = bf_shape<DP, KR>(p.n, p.nq, ~0ull, plan.bf_warps);
    if (shape.splits > 1) {
        KNN_TRY(ix->workspace.reserve(static_cast<size_t>(shape.splits) * p.nq * p.k * sizeof(uint64_t) + 256));
        p.partial = ix->workspace.as<uint64_t>();
    }
    if (plan.timing) KNN_TRY(ix->timing.begin(s));
    KNN_TRY((bf_launch<DP, KR, false>(p, shape, s)));
    if (plan.timing) KNN_TRY(ix->timing.end(s));
    return shape.splits > 1 ? bf_launch_merge<KR>(p, shape.splits, s) : KNN_OK;
}

template <uint32_t DP>
int bf_query_dp(knn_index* ix, const QueryArgs& a, const QueryPlan& plan, cudaStream_t s) {
    // The storage options do not matter to this search; sizes no block can hold (with the 32 KB of
    // points beside them) stay refused.
    const uint32_t block = plan.block ? plan.block : 128;
    const size_t storage = 32768 + tracker_smem_bytes(plan.sh_nn, k_class(a.k), block);
    if (storage > kMaxBlockSmem)
        return fail(KNN_ERR_CUDA, "storage options: %zu bytes of shared memory per block of %u", storage, block);
    BfParams p{};
    p.points = ix->points.as<float>();
    p.n = ix->n;
    p.queries = a.queries;
    p.dims = ix->dims;
    p.nq = a.count;
    p.max_d2 = a.max_d2;
    p.radii = a.radii;
    p.order = a.order;
    p.count_dev = a.count_dev;
    p.k = a.k;
    p.out_idx = a.out_idx;
    p.out_dist = a.out_dist;
    if (!a.count_dev) {  // (a list whose length the device knows may be short)
        bool ran = false;
        if (plan.timing) KNN_TRY(ix->timing.begin(s));
        KNN_TRY((bf_thread_query<DP, false>(p, ~0ull, [&](uint32_t splits, uint64_t** out) -> int {
            KNN_TRY(ix->workspace.reserve(static_cast<size_t>(splits) * p.nq * p.k * sizeof(uint64_t)));
            *out = ix->workspace.as<uint64_t>();
            return KNN_OK;
        }, s, &ran)));
        if (ran) return plan.timing ? ix->timing.end(s) : KNN_OK;
    }
    if (a.k <= 32) return launch_bf<DP, 1>(ix, p, plan, s);
    if (a.k <= 64) return launch_bf<DP, 2>(ix, p, plan, s);
    return launch_bf<DP, 4>(ix, p, plan, s);
}

template int bf_query_dp<KNN_DP>(knn_index*, const QueryArgs&, const QueryPlan&, cudaStream_t);

}  // namespace knn
