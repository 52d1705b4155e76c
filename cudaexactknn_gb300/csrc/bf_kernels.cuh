// Brute-force kernels, shared by bf_kernels.cu (one translation unit per padded dimension count)
// and bf_noalloc.cu (the allocation-free entry point).
//
// Replaces BruteForceKernels::knnKernel / knnShKernel (src/BruteForceGpu.cuh:9-50), where one
// thread scans all n points for its query straight from global memory.  Here, but for few points or
// many queries with small k (the thread-per-query form at the end), a warp holds Q
// queries and its lanes take 32 points at a time:
//   * every pair's distance is the reference's sequential fused sum, two queries per packed
//     instruction (sub/fma.rn.f32x2 round each half as the scalar instructions do);
//   * a first look at every eighth tile of points (every fourth below 32 tiles, all of them below 8)
//     keeps only the least distance per lane (and, for k > 32, per turn of KR); the k-th smallest of
//     those is the distance of a point with
//     k - 1 others at or below it, an upper bound on the query's k-th distance.  The scan proper
//     then appends the few points within the bound to a buffer, and only a full buffer (or the end)
//     is sorted into the k smallest keys.  A list per thread, as
//     before, diverged at every insertion of any of a warp's 32 queries;
//   * the block stages tiles of points in shared memory (rows of more than 4 dims padded to an odd
//     number of 16-byte units: no bank conflicts), the next tile's copies in flight while one is
//     scanned; queries of more than 4 dims are read there by broadcast;
//   * where queries are few, a query's points are split over the warps of a block (which share
//     the bound and merge their lists in shared memory) and over blocks (merged by a second kernel).
// Keys, ties and results equal the reference's brute force bit for bit.
//
// Measured (before: a thread per query at all sizes, list in registers or local memory): 65,536 3-d points,
// 4,096 queries, k 8: 268 us (455; 1,335 with heap tracking); 4,096 points, 16 queries: 46 us with its
// launches (200, one block); 128 dims, 256 queries on 262,144 points, k 100: 1.64 ms (46.6).  At the first
// of these 54% of the issue slots are used, with 5 warps per scheduler; the largest stall is the barrier
// between staged tiles.
#pragma once

#include <algorithm>

#include "knn_internal.h"
#include "tracker.cuh"
#include "warp_search.cuh"

namespace knn {

struct BfParams {
    const float* points;  // [n][ps], zero padded (RAW: the caller's [n][dims])
    uint32_t n;
    const float* queries;  // [nq][dims]
    uint32_t dims;
    uint32_t nq;
    float max_d2;
    const float* radii;
    const uint32_t* order;      // list position -> query, or null
    const uint32_t* count_dev;  // live list length on the device, or null
    uint32_t k;
    uint32_t chunk;  // points per split (grid row)
    uint32_t parts;  // warps of a block that share a query group's points (a power of two)
    uint64_t* partial;  // [splits][nq][k] sorted keys, or null (single split)
    int32_t* out_idx;
    float* out_dist;
};

constexpr uint32_t kBfWarps = 8;   // warps per block
constexpr uint32_t kBfSample = 8;  // every how many tiles the first look takes one, of many

// Queries per warp, by top-k registers.
__host__ __device__ constexpr uint32_t bf_queries(int kr) { return kr == 1 ? 8u : kr == 2 ? 4u : 2u; }
__host__ __device__ constexpr bool bf_wide(int dp) { return dp >= 8; }
__host__ __device__ constexpr uint32_t bf_row(int dp) { return dp < 4 ? 4u : static_cast<uint32_t>(dp); }
// Points per staged tile (two tiles of at most 70 KB), so the most parts a block can have is a 32nd.
__host__ __device__ constexpr uint32_t bf_tile(int dp) { return dp <= 4 ? 512u : dp <= 64 ? 256u : 128u; }
__host__ __device__ constexpr uint32_t bf_max_parts(int dp) { return std::min(bf_tile(dp) / 32, kBfWarps); }

template <int DP, int KR>
struct BfSmem {
    static constexpr uint32_t Q = bf_queries(KR);
    static constexpr uint32_t kStride = bf_row(DP) + (bf_wide(DP) ? 4 : 0);  // floats of a staged row
    uint64_t list[kBfWarps][Q][32 * KR];                          // the k smallest keys flushed so far
    union {
        uint64_t buf[kBfWarps][Q][64];                             // keys within the bound, not yet sorted
        uint32_t least[kBfWarps * Q * KR * 32];                    // the first look's minima, query by query
    };
    uint32_t count[kBfWarps][Q];                                   // keys left in a buffer at the end, and (top bit) whether its list holds any
    uint4 limit[kBfWarps][Q >= 4 ? Q / 4 : 1];                     // per warp and query: see bf_limits
    float2 q[kBfWarps][Q / 2][bf_wide(DP) ? DP : 1];            // pairs of queries, by dimension
    float4 tile[2 * bf_tile(DP) * kStride / 4];
};

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    return (static_cast<uint64_t>(__float_as_uint(b)) << 32) | __float_as_uint(a);
}
// The distance bits that a warp's next points have to be below, as they stand (other warps lower them): one
// more than the bound on the k-th distance that any warp of the query has found, or its own list's k-th
// distance once that is a point's.  A warp meets its points by ascending index, so one at that distance
// comes after all in its list: with equal distances left to the keys, data of many of them filled and
// flushed buffers to no end (32,880 equal points, 16,237 queries: 1,661 us, a thread per query 374).
template <uint32_t Q>
__device__ __forceinline__ void bf_limits(const uint4* at, uint32_t (&out)[Q]) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(at));
    if constexpr (Q == 2) {
        asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(out[0]), "=r"(out[1]) : "r"(a));
    } else {
#pragma unroll
        for (uint32_t j = 0; j < Q; j += 4)
            asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(out[j]), "=r"(out[j + 1]), "=r"(out[j + 2]), "=r"(out[j + 3])
                         : "r"(a + 4 * j));
    }
}
__device__ __forceinline__ uint32_t bf_above(uint32_t bits) { return bits + (bits != 0xFFFFFFFFu ? 1u : 0u); }

// Sorts a buffer of n <= 64 keys into a list in shared memory; returns the list's k-th key.
template <int KR>
__device__ __noinline__ uint64_t bf_flush(uint64_t* list, const uint64_t* buf, uint32_t n, uint32_t k, uint32_t lane) {
    WarpTopK<KR> top;
    top.k = k;
    top.lane = lane;
    top.empty = false;
#pragma unroll
    for (int j = 0; j < KR; ++j) top.v[j] = list[32 * j + lane];
    top.refresh();
    for (uint32_t i = 0; i < n; i += 32) top.offer(i + lane < n, i + lane < n ? buf[i + lane] : ~0ull);
#pragma unroll
    for (int j = 0; j < KR; ++j) list[32 * j + lane] = top.v[j];
    return top.kth;
}

__device__ __forceinline__ void bf_copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

// Block: warp w has part w / groups of the points of query group w % groups (groups = warps / parts).
// R rows per lane at a time: their sums are independent, and share the reads of wide queries.
template <int DP, int KR, int R, bool RAW>
__global__ void __launch_bounds__(32 * kBfWarps, R == 1 ? 3 : 2) bf_warp_kernel(const BfParams p) {
    using Sm = BfSmem<DP, KR>;
    constexpr uint32_t Q = Sm::Q, PS = bf_row(DP), T = bf_tile(DP), S4 = Sm::kStride / 4;
    extern __shared__ __align__(16) unsigned char bf_smem[];
    Sm& sm = *reinterpret_cast<Sm*>(bf_smem);
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t parts = p.parts, groups = kBfWarps / parts, g = w % groups, part = w / groups;
    const uint32_t live = p.count_dev ? *p.count_dev : p.nq;
    const uint32_t block_first = blockIdx.x * groups * Q;
    if (block_first >= live) return;  // the whole block is past the live list
    const uint32_t first = block_first + g * Q;
    auto query_of = [&](uint32_t t) { return p.order ? p.order[t] : t; };
    // The group's queries in pairs, their lists and bounds.  A slot past the live list holds key 0:
    // nothing is below it.
    uint64_t qr[bf_wide(DP) ? 1 : Q / 2][bf_wide(DP) ? 1 : DP];
    auto limit_of = [&](uint32_t of_warp, uint32_t j) { return reinterpret_cast<uint32_t*>(sm.limit[of_warp]) + j; };
#pragma unroll
    for (uint32_t j = 0; j < Q; ++j) {
        const uint32_t t = first + j;
        const uint64_t fill = t < live ? make_key(p.radii ? p.radii[query_of(t)] : p.max_d2, -1) : 0ull;
#pragma unroll
        for (int r = 0; r < KR; ++r) sm.list[w][j][32 * r + lane] = fill;
        if (lane == 0) *limit_of(w, j) = t < live ? bf_above(static_cast<uint32_t>(fill >> 32)) : 0u;
    }
#pragma unroll
    for (uint32_t h = 0; h < Q / 2; ++h) {
        const uint32_t ta = first + 2 * h, tb = ta + 1;
        const float* a = p.queries + static_cast<size_t>(ta < live ? query_of(ta) : 0u) * p.dims;
        const float* b = p.queries + static_cast<size_t>(tb < live ? query_of(tb) : 0u) * p.dims;
        if constexpr (bf_wide(DP)) {
            if (part == 0)
                for (uint32_t d = lane; d < DP; d += 32)
                    sm.q[g][h][d] = make_float2(d < p.dims ? a[d] : 0.0f, d < p.dims ? b[d] : 0.0f);
        } else {
#pragma unroll
            for (int d = 0; d < DP; ++d)
                qr[h][d] = pack2(static_cast<uint32_t>(d) < p.dims ? a[d] : 0.0f, static_cast<uint32_t>(d) < p.dims ? b[d] : 0.0f);
        }
    }
    __syncthreads();

    const uint32_t lo = blockIdx.y * p.chunk, hi = min(p.n, lo + p.chunk);
    // Takes every `every`-th step (or tile) of the chunk; look(sums, index, live_point, turn) sees one
    // point per lane (`live_point`: there is one) with its pairs' sums.
    auto scan = [&](uint32_t every, auto&& look) {
        auto stage = [&](uint32_t base, uint32_t b) {
            float4* tile = sm.tile + b * T * S4;
            const uint32_t rows = min(T, hi - base);
            if constexpr (RAW) {
                for (uint32_t i = threadIdx.x; i < rows * PS; i += blockDim.x) {
                    const uint32_t r = i / PS, d = i % PS;
                    reinterpret_cast<float*>(tile)[r * 4 * S4 + d] =
                        d < p.dims ? p.points[static_cast<size_t>(base + r) * p.dims + d] : 0.0f;
                }
            } else {
                const float4* src = reinterpret_cast<const float4*>(p.points) + static_cast<size_t>(base) * (PS / 4);
                for (uint32_t i = threadIdx.x; i < rows * (PS / 4); i += blockDim.x)
                    bf_copy16(tile + i / (PS / 4) * S4 + i % (PS / 4), src + i);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        const uint32_t step = T * every;
        uint32_t b = 0, turn = 0;
        __syncthreads();  // the tiles of the scan before this one are read to the end
        if (lo < hi) stage(lo, 0);
        for (uint32_t base = lo; base < hi; base += step, b ^= 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();  // this tile has landed for every thread, and the other one is read to the end
            if (base + step < hi) stage(base + step, b ^ 1);
            const uint32_t rows = min(T, hi - base);
            for (uint32_t r0 = 32 * part; r0 < rows; r0 += 32 * R * parts) {
                const float4* row[R];
                uint64_t acc[R][Q / 2];
#pragma unroll
                for (uint32_t u = 0; u < static_cast<uint32_t>(R); ++u) {
                    // (A lane past the tile's rows reads some row of the tile and is not looked at.)
                    row[u] = sm.tile + b * T * S4 + min(r0 + 32 * parts * u + lane, rows - 1) * S4;
#pragma unroll
                    for (uint32_t h = 0; h < Q / 2; ++h) acc[u][h] = 0ull;
                }
                if constexpr (!bf_wide(DP)) {
#pragma unroll
                    for (uint32_t u = 0; u < static_cast<uint32_t>(R); ++u) {
                        const float4 v = row[u][0];
                        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int d = 0; d < DP; ++d) {
                            const uint64_t xx = pack2(x[d], x[d]);
#pragma unroll
                            for (uint32_t h = 0; h < Q / 2; ++h) acc[u][h] = sqr_add2(sub2(qr[h][d], xx), acc[u][h]);
                        }
                    }
                } else {
                    const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(&sm.q[g][0][0]);
#pragma unroll 2
                    for (uint32_t v = 0; v < DP / 4; ++v) {
                        float4 x[R];
#pragma unroll
                        for (uint32_t u = 0; u < static_cast<uint32_t>(R); ++u) x[u] = row[u][v];
#pragma unroll
                        for (uint32_t h = 0; h < Q / 2; ++h) {
                            const ulonglong2 a = q2[h * (DP / 2) + 2 * v], c = q2[h * (DP / 2) + 2 * v + 1];
#pragma unroll
                            for (uint32_t u = 0; u < static_cast<uint32_t>(R); ++u) {
                                acc[u][h] = sqr_add2(sub2(a.x, pack2(x[u].x, x[u].x)), acc[u][h]);
                                acc[u][h] = sqr_add2(sub2(a.y, pack2(x[u].y, x[u].y)), acc[u][h]);
                                acc[u][h] = sqr_add2(sub2(c.x, pack2(x[u].z, x[u].z)), acc[u][h]);
                                acc[u][h] = sqr_add2(sub2(c.y, pack2(x[u].w, x[u].w)), acc[u][h]);
                            }
                        }
                    }
                }
#pragma unroll
                for (uint32_t u = 0; u < static_cast<uint32_t>(R); ++u) {
                    const uint32_t r = r0 + 32 * parts * u + lane;
                    if (r - lane < rows) look(acc[u], base + r, r < rows, turn);
                    ++turn;
                }
            }
        }
    };
    auto bits_of = [](const uint64_t (&acc)[Q / 2], uint32_t j) { return static_cast<uint32_t>(acc[j / 2] >> (32 * (j & 1))); };

    // The first look: the least distance per lane and turn, and from the k-th smallest of a query's the
    // bound.  A few steps are all looked at twice.
    {
        const uint32_t tiles = (hi - lo + T - 1) / T;
        uint32_t least[Q][KR];
#pragma unroll
        for (uint32_t j = 0; j < Q; ++j)
#pragma unroll
            for (int c = 0; c < KR; ++c) least[j][c] = 0xFFFFFFFFu;
        scan(tiles >= 4 * kBfSample ? kBfSample : tiles >= 8 ? 4u : 1u, [&](const uint64_t (&acc)[Q / 2], uint32_t, bool live_point, uint32_t turn) {
#pragma unroll
            for (uint32_t j = 0; j < Q; ++j)
#pragma unroll
                for (int c = 0; c < KR; ++c)
                    if (live_point && (KR == 1 || turn % KR == static_cast<uint32_t>(c))) least[j][c] = min(least[j][c], bits_of(acc, j));
        });
        const uint32_t per_query = parts * KR * 32;
#pragma unroll
        for (uint32_t j = 0; j < Q; ++j)
#pragma unroll
            for (int c = 0; c < KR; ++c) sm.least[(g * Q + j) * per_query + (part * KR + c) * 32 + lane] = least[j][c];
        __syncthreads();
        for (uint32_t e = w; e < groups * Q; e += kBfWarps) {
            WarpTopK<KR> top;
            const uint32_t within = *limit_of(e / Q, e % Q);  // (the query's radius, in every part's row)
            if (!within) continue;
            top.init(p.k, __uint_as_float(within - 1u), lane);
            for (uint32_t s = 0; s < per_query; s += 32)
                top.offer(true, static_cast<uint64_t>(sm.least[e * per_query + s + lane]) << 32);
            if (lane < parts) *limit_of(lane * groups + e / Q, e % Q) = bf_above(static_cast<uint32_t>(top.kth >> 32));
        }
        __syncthreads();
    }

    uint32_t count[Q], limit[Q], flushed = 0;  // keys in each buffer; bf_limits; lists that hold any (bit j)
#pragma unroll
    for (uint32_t j = 0; j < Q; ++j) count[j] = 0;
    // Lane s tells part s of a new k-th distance.  (The address is kept beyond 4 dims only: there the loop is
    // 11% slower without, 6 dims, 65,536 points, 16,000 queries, k 32; up to 4 dims 15% slower with it.)
    const uint32_t peer = static_cast<uint32_t>(__cvta_generic_to_shared(limit_of(lane < parts ? lane * groups + g : w, 0)));
    bf_limits(sm.limit[w], limit);
    scan(1, [&](const uint64_t (&acc)[Q / 2], uint32_t index, bool live_point, uint32_t) {
        bool hit = false;
#pragma unroll
        for (uint32_t j = 0; j < Q; ++j) hit |= bits_of(acc, j) < limit[j];
        if (!__any_sync(kFullMask, hit && live_point)) return;
#pragma unroll
        for (uint32_t j = 0; j < Q; ++j) {
            const bool cand = live_point && bits_of(acc, j) < limit[j];
            const uint32_t m = __ballot_sync(kFullMask, cand);
            if (!m) continue;
            uint64_t* buf = sm.buf[w][j];
            if (cand) buf[count[j] + __popc(m & ((1u << lane) - 1u))] = (static_cast<uint64_t>(bits_of(acc, j)) << 32) | index;
            count[j] += __popc(m);
            if (count[j] <= 32) continue;  // room for the next step's 32
            __syncwarp();
            const uint64_t now = bf_flush<KR>(sm.list[w][j], buf, count[j], p.k, lane);
            count[j] = 0;
            flushed |= 1u << j;
            // (Its k points lie within the list's k-th distance, whichever part holds them.)
            if (lane < parts && key_index(now) >= 0) {
                const uint32_t to = static_cast<uint32_t>(now >> 32) + (lane == part ? 0u : 1u);
                if constexpr (bf_wide(DP)) asm volatile("red.shared.min.u32 [%0], %1;" ::"r"(peer + 4 * j), "r"(to) : "memory");
                else atomicMin(limit_of(lane * groups + g, j), to);
            }
            __syncwarp();
        }
        bf_limits(sm.limit[w], limit);  // (read here, not at every step: shared memory returns 128 bytes a clock)
    });
#pragma unroll
    for (uint32_t j = 0; j < Q; ++j)
        if (lane == 0) sm.count[w][j] = count[j] | ((flushed >> j & 1u) << 31);
    __syncthreads();
    // A warp per query merges its parts' lists.
    for (uint32_t e = w; e < groups * Q; e += kBfWarps) {
        const uint32_t t = block_first + e;
        if (t >= live) break;
        const uint32_t eg = e / Q, ej = e % Q, qi = query_of(t);
        WarpTopK<KR> top;
        top.init(p.k, p.radii ? p.radii[qi] : p.max_d2, lane);
        for (uint32_t s = 0; s < parts; ++s) {
            const uint32_t ew = s * groups + eg, n = sm.count[ew][ej] & 0x7FFFFFFFu;
            if (sm.count[ew][ej] >> 31) {
#pragma unroll
                for (int j = 0; j < KR; ++j) top.offer(true, sm.list[ew][ej][32 * j + lane]);
            }
            for (uint32_t i = 0; i < n; i += 32) top.offer(i + lane < n, i + lane < n ? sm.buf[ew][ej][i + lane] : ~0ull);
        }
        if (p.partial)
            top.emit_keys(p.partial + (static_cast<size_t>(blockIdx.y) * p.nq + t) * p.k);
        else
            top.emit(p.out_idx + static_cast<size_t>(qi) * p.k, p.out_dist + static_cast<size_t>(qi) * p.k);
    }
}

// Combines the per-split sorted key lists of each query into its final row, a warp per query.
template <int KR>
__global__ void __launch_bounds__(128) bf_merge_kernel(const uint64_t* __restrict__ partial, uint32_t splits,
                                                       uint32_t nq, uint32_t k, float max_d2,
                                                       const float* __restrict__ radii,
                                                       const uint32_t* __restrict__ order,
                                                       const uint32_t* __restrict__ count_dev,
                                                       int32_t* __restrict__ out_idx,
                                                       float* __restrict__ out_dist) {
    const uint32_t t = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31u;
    if (t >= (count_dev ? *count_dev : nq)) return;
    const uint32_t qi = order ? order[t] : t;
    WarpTopK<KR> top;
    top.init(k, radii ? radii[qi] : max_d2, lane);
    for (uint32_t s = 0; s < splits; ++s) {
        const uint64_t* row = partial + (static_cast<size_t>(s) * nq + t) * k;
        for (uint32_t i = 0; i < k; i += 32) {
            const uint64_t key = i + lane < k ? row[i + lane] : ~0ull;
            if (!__any_sync(kFullMask, key < top.kth)) break;  // rows are ascending
            top.offer(true, key);
        }
    }
    top.emit(out_idx + static_cast<size_t>(qi) * k, out_dist + static_cast<size_t>(qi) * k);
}

// How the points of `count` queries are shared out: parts (warps of a block), splits (blocks), and the
// rows a lane takes at a time.
struct BfShape {
    uint32_t parts, splits, chunk, grid, rows;
};

// As many warps as keep every SM's schedulers fed (32 per SM), each with at least 4 steps of 32
// points.  Up to 4 dims the warps of a block share a group's points first: they share the bound and
// need no second kernel.  Beyond, a block's warps take different queries wherever there are
// enough of them, so that each staged tile serves 64, and a lane takes four rows for every read of
// a query (shared memory returns 128 bytes a clock, broadcast or not): 2,048 queries of 128 dims on
// 100,000 points, k 10: 2.3 ms (3.4 with the block's warps on the same queries, one row a lane).
template <int DP, int KR>
BfShape bf_shape(uint32_t n, uint32_t count, uint64_t max_splits, uint32_t per_sm = 0) {
    const uint32_t query_groups = ceil_div(count, bf_queries(KR));
    const uint32_t want = ceil_div((per_sm ? per_sm : 32u) * static_cast<uint32_t>(sm_count()), query_groups);
    const uint32_t share = std::max(1u, std::min(want, n / 128));
    BfShape s{};
    const bool many = bf_wide(DP) && query_groups >= kBfWarps;
    s.rows = many ? 4 : 1;
    s.parts = 1;
    uint32_t room = many ? 1u : bf_max_parts(DP);
    if (bf_wide(DP))  // few queries: parts for the warps without any
        while (room > 1 && (room / 2) * query_groups >= kBfWarps) room /= 2;
    while (2 * s.parts <= std::min(share, room)) s.parts *= 2;
    const uint32_t splits = static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>({share / s.parts, max_splits, 0xFFFFu})));
    s.chunk = ceil_div(ceil_div(n, splits), bf_tile(DP)) * bf_tile(DP);
    s.splits = ceil_div(n, s.chunk);
    s.grid = ceil_div(count, kBfWarps / s.parts * bf_queries(KR));
    return s;
}

// Launches the search (and the merge, where the points are split over blocks) with the shape `s`.
template <int DP, int KR, bool RAW>
int bf_launch(BfParams p, const BfShape& s, cudaStream_t stream) {
    auto kern = bf_warp_kernel<DP, KR, 1, RAW>;
    if constexpr (bf_wide(DP))
        if (s.rows == 4) kern = bf_warp_kernel<DP, KR, 4, RAW>;
    constexpr size_t smem = sizeof(BfSmem<DP, KR>);
    if (smem > 48 * 1024)
        KNN_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    p.parts = s.parts;
    p.chunk = s.chunk;
    if (s.splits == 1) p.partial = nullptr;
    kern<<<dim3(s.grid, s.splits), 32 * kBfWarps, smem, stream>>>(p);
    KNN_LAUNCHED();
    return KNN_OK;
}

template <int KR>
int bf_launch_merge(const BfParams& p, uint32_t splits, cudaStream_t stream) {
    bf_merge_kernel<KR><<<ceil_div(p.nq, 4), 128, 0, stream>>>(p.partial, splits, p.nq, p.k, p.max_d2, p.radii, p.order,
                                                               p.count_dev, p.out_idx, p.out_dist);
    KNN_LAUNCHED();
    return KNN_OK;
}

// ---- a thread per query ---------------------------------------------------------------------------
// The plain form: a thread holds its query and its top-k in registers and goes through the tiles a block
// stages, all threads reading the same point.  No lists in shared memory, no first look, no merge
// over warps: nothing to pay per query but the insertions themselves.  bf_by_thread says where that wins.
// `kk` of the k places can be filled (min(k, n)); the others are written as they start.
template <int DP>
struct BfThreadTile {
    static constexpr uint32_t PS = (DP + 3) / 4 * 4, kRows = 8192 / PS;  // 32 KB
    static constexpr uint32_t kChunk = 4 * kRows;                        // least points of a split
};
constexpr uint32_t kBfThreads = 128;

template <int DP, int KMAX, bool RAW>
__global__ void __launch_bounds__(kBfThreads) bf_thread_kernel(const BfParams p, uint32_t kk) {
    constexpr uint32_t PS = BfThreadTile<DP>::PS, T = BfThreadTile<DP>::kRows;
    __shared__ float4 tile[T * PS / 4];
    const uint32_t t = blockIdx.x * kBfThreads + threadIdx.x;
    const bool active = t < p.nq;
    const uint32_t qi = active ? (p.order ? p.order[t] : t) : 0u;
    float q[PS];
#pragma unroll
    for (uint32_t d = 0; d < PS; ++d)
        q[d] = active && d < p.dims ? p.queries[static_cast<size_t>(qi) * p.dims + d] : 0.0f;
    const float r2 = active && p.radii ? p.radii[qi] : p.max_d2;
    Tracker<KMAX, false, false> tr;
    tr.init(kk, r2, nullptr, 0);
    const uint32_t lo = blockIdx.y * p.chunk, hi = min(p.n, lo + p.chunk);
    for (uint32_t base = lo; base < hi; base += T) {
        const uint32_t rows = min(T, hi - base);
        __syncthreads();
        if constexpr (RAW) {
            for (uint32_t i = threadIdx.x; i < rows * PS; i += kBfThreads) {
                const uint32_t r = i / PS, d = i % PS;
                reinterpret_cast<float*>(tile)[i] = d < p.dims ? p.points[static_cast<size_t>(base + r) * p.dims + d] : 0.0f;
            }
        } else {
            const float4* src = reinterpret_cast<const float4*>(p.points) + static_cast<size_t>(base) * (PS / 4);
            for (uint32_t i = threadIdx.x; i < rows * (PS / 4); i += kBfThreads) tile[i] = src[i];
        }
        __syncthreads();
        if (!active) continue;
        uint32_t r = 0;
        for (; r + 1 < rows; r += 2) {  // two chains at a time
            const float d0 = dist2_vec4<PS>(q, tile + r * (PS / 4));
            const float d1 = dist2_vec4<PS>(q, tile + (r + 1) * (PS / 4));
            tr.offer(make_key(d0, static_cast<int32_t>(base + r)));
            tr.offer(make_key(d1, static_cast<int32_t>(base + r + 1)));
        }
        if (r < rows) tr.offer(make_key(dist2_vec4<PS>(q, tile + r * (PS / 4)), static_cast<int32_t>(base + r)));
    }
    if (!active) return;
    if (p.partial) {
        tr.emit_keys(kk, p.partial + (static_cast<size_t>(blockIdx.y) * p.nq + t) * p.k);
        return;
    }
    int32_t* idx = p.out_idx + static_cast<size_t>(qi) * p.k;
    float* dist = p.out_dist + static_cast<size_t>(qi) * p.k;
    tr.emit(kk, idx, dist);
    for (uint32_t i = kk; i < p.k; ++i) {
        idx[i] = -1;
        dist[i] = r2;
    }
}

// Splits of a thread per query's scan: until the blocks cover the GPU about four times, at least kChunk
// points each.
template <int DP, int KMAX, bool RAW>
uint32_t bf_thread_splits(uint32_t n, uint32_t count, uint64_t max_splits) {
    static const int per_sm = [] {
        int v = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, bf_thread_kernel<DP, KMAX, RAW>, kBfThreads, 0) == cudaSuccess
                   ? std::max(v, 1) : 1;
    }();
    const uint32_t want = ceil_div(4u * static_cast<uint32_t>(sm_count() * per_sm), ceil_div(count, kBfThreads));
    return static_cast<uint32_t>(std::max<uint64_t>(
        1, std::min<uint64_t>({want, ceil_div(n, BfThreadTile<DP>::kChunk), max_splits, 0xFFFFu})));
}

// Whether a thread per query answers a call faster than the warps do.  Measured over 1 to 128 dims, 4 to
// 262,144 points, 1 to 200,000 queries, k 1 to 100; the line is where the two take the same time.
//   * Very few points: a thread's scan is over before a warp's lists are set up (3 dims, 32 points, k 8,
//     100,000 queries: 15 us, a warp 60).
//   * Beyond, once the threads fill the GPU (12,288: 81 per SM; with fewer the scan's latency shows:
//     2,048 points of 32 dims, k 8, 8,000 queries 134 us against 60 with a warp, 32,000 queries 195
//     against 295) up to a number of points that grows with the dimensions, as the warps' staging leaves
//     one block per SM there, and falls with k, as every insertion holds up 32 queries.
// (For k beyond 16 the line is a multiple of k or its square: that many of the points are insertions.)
inline bool bf_by_thread(int dp, uint32_t k, uint32_t n, uint32_t count, uint32_t splits, uint32_t chunk) {
    if (k > 32) return n <= 16 && dp >= 64 && count >= 16384;
    if (n <= 16) return true;
    if (count < 64) return false;
    if (n <= (k > 16 ? 32u : k <= 8 && dp <= 16 ? 128u : 64u)) return true;
    const uint64_t threads = static_cast<uint64_t>(count) * splits;
    if (threads < (count < 128 && dp >= 32 ? 8192u : dp == 128 ? 10000u : 12288u)) return false;
    switch (dp) {
        case 8:
        case 16: {
            const uint32_t most = threads < 30000 ? 1024u : dp == 8 ? 32768u : 4096u;
            return n <= (k <= 8 ? most : k <= 16 ? 128u : k * k / 8);
        }
        case 32: return k <= 8 || n <= (k <= 16 ? 1024u : k * k / 4);
        case 64: return k <= 8 || n <= (k <= 16 ? 2048u : k * k / 2);
        case 128:
            // (More work than this is the warps' again: the thread's registers leave two blocks per SM.)
            return (n <= 512 || static_cast<uint64_t>(count) * ceil_div(n, chunk) <= 200000) &&
                   n <= (k <= 8 ? 65536u : k <= 16 ? 16384u : k * k);
        default:
            return n <= (k <= 8 ? 256u : k <= 16 ? 64u : 2 * k) ||
                   (static_cast<uint64_t>(n) * k <= (dp == 4 ? 2048u : 1024u) && 60ull * n * k <= threads);
    }
}

// Launches a thread per query (and the merge, where the points are split); *ran is false where the warps
// are to answer.  `scratch(splits)` gives the room for the splits' lists in p.partial.
template <int DP, int KMAX, bool RAW, class Scratch>
int bf_launch_thread(BfParams p, uint64_t max_splits, Scratch&& scratch, cudaStream_t stream, bool* ran) {
    uint32_t splits = bf_thread_splits<DP, KMAX, RAW>(p.n, p.nq, max_splits);
    *ran = bf_by_thread(DP, p.k, p.n, p.nq, splits, BfThreadTile<DP>::kChunk);
    if (!*ran) return KNN_OK;
    p.chunk = ceil_div(ceil_div(p.n, splits), BfThreadTile<DP>::kRows) * BfThreadTile<DP>::kRows;
    splits = ceil_div(p.n, p.chunk);
    if (splits > 1) KNN_TRY(scratch(splits, &p.partial));
    else p.partial = nullptr;
    bf_thread_kernel<DP, KMAX, RAW><<<dim3(ceil_div(p.nq, kBfThreads), splits), kBfThreads, 0, stream>>>(p, std::min(p.k, p.n));
    KNN_LAUNCHED();
    return splits > 1 ? bf_launch_merge<1>(p, splits, stream) : KNN_OK;
}

// The same by the places there are to fill.
template <int DP, bool RAW, class Scratch>
int bf_thread_query(const BfParams& p, uint64_t max_splits, Scratch&& scratch, cudaStream_t stream, bool* ran) {
    const uint32_t kk = std::min(p.k, p.n);
    *ran = false;
    if (kk <= 8) return bf_launch_thread<DP, 8, RAW>(p, max_splits, scratch, stream, ran);
    if (kk <= 16) return bf_launch_thread<DP, 16, RAW>(p, max_splits, scratch, stream, ran);
    if (kk <= 32) return bf_launch_thread<DP, 32, RAW>(p, max_splits, scratch, stream, ran);
    return KNN_OK;
}

}  // namespace knn
