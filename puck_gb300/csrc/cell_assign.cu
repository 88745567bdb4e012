// Exact nearest-cell assignment of the build (HierarchicalClusterIndex::
// nearest_cell_assign, puck/hierarchical_cluster/hierarchical_cluster_index.cpp:
// 1042-1085, driven by assign :1087-1138): for each point x the cell c * F + f
// with the smallest
//     score = ((0.5|c|^2 - x.c) + 0.5|x|^2 - x.f) + stationary[c][f],
// walking the coarse clusters in ascending (coarse term, id) order and, inside
// each, the fine clusters in index order (descending norm at train time), with the
// reference's break test sqrt(best) - fneg[f] < sqrt(coarse term)
// (fneg[f] = -sqrt(0.5|f|^2)) and its strict-< update (first minimum wins).
//
// Every dot product is the reference's sequential FP32 sum (k_centroid_scores), so
// cells and distances are bit-identical to the sequential walk. One warp per point finds the
// walk's result without walking:
//   * g, the smallest score over ALL cells: in float arithmetic score = (t - x.f) + stat is
//     non-decreasing in t, -x.f and stat, so (t - max x.f) + min stat over a group of cells
//     bounds the group's scores from below exactly, roundings included, and a group whose
//     bound is above the best score so far is passed over. Groups are a cluster's cells and
//     32 consecutive fine ids of it;
//   * the walk's best is never below g, and it visits g's cell if the break tests up to that
//     cell pass with best = g (they are monotone in best, and best is larger until then).
//     They are one test against the largest fneg up to the cell. If that holds for every cell
//     with that score, the walk's result is g and the first of them in its order;
//   * otherwise (the test fails, no finite score) the warp walks in order:
//     the first cluster (the smallest term) in full; after it best can only decrease, so a
//     cluster whose f = 0 test already breaks changes nothing, and the remaining clusters are
//     walked by (term, id), 32 fine ids per step: each lane's break test uses the best before
//     it, the exclusive prefix minimum over the earlier lanes' scores, so the first breaking
//     lane and the update are the sequential walk's.
// On 100k points of a 96-dimensional mixture, 500 x 500 cells, the walk visits 51k cells per
// point and the bounds leave 170 (unit vectors) to 3800 (integers): the walk took 43.2 ms, the
// search 0.9. With the exact dot products (0.95 ms of k_centroid_scores) the call went from
// 43.9 to 2.5 ms.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "device_common.cuh"
#include "pgpu_internal.h"

namespace pgpu {
namespace {

constexpr int kWalkWarps = 8;
constexpr uint32_t kGroup = 32;    // fine ids per group
constexpr uint32_t kMaxNear = 64;  // collected clusters per point before the slow path

// (value, id) as one ordered 64-bit key: float order, then id.
__device__ __forceinline__ uint64_t term_key(float v, uint32_t id) {
    return ((uint64_t)ordered_key(v) << 32) | id;
}

// Walks coarse cluster c (term t) from fine id 0 in order, with the reference's
// break test and strict-< update; best / best_id on every lane.
__device__ __forceinline__ void walk_cluster(uint32_t c, float t, const float* __restrict__ fip,
                                             const float* __restrict__ fneg,
                                             const float* __restrict__ stat, uint32_t F,
                                             float& best, int32_t& best_id) {
    const int lane = threadIdx.x & 31;
    const float st = __fsqrt_rn(t);
    const float* srow = stat + (uint64_t)c * F;
    for (uint32_t f0 = 0; f0 < F; f0 += 32) {
        const uint32_t f = f0 + lane;
        const bool valid = f < F;
        // fip holds -x.f (k_centroid_scores MODE 1): negation is exact
        const float score = valid ? __fadd_rn(__fsub_rn(t, -fip[f]), srow[f]) : FLT_MAX;
        // best before this lane: min(best, scores of the earlier lanes)
        float pre = score;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre = fminf(pre, u);
        }
        float before = __shfl_up_sync(0xffffffffu, pre, 1);
        before = lane == 0 ? best : fminf(best, before);
        const bool brk = valid && __fsub_rn(__fsqrt_rn(before), fneg[f]) < st;
        const unsigned bb = __ballot_sync(0xffffffffu, brk);
        const int stop = bb ? __ffs(bb) - 1 : 32;  // lanes < stop are walked
        const bool walked = valid && lane < stop;
        float m = walked ? score : FLT_MAX;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (m < best) {
            // the first walked lane reaching the minimum sets best (strict <)
            const unsigned at = __ballot_sync(0xffffffffu, walked && score == m);
            best = m;
            best_id = (int32_t)(c * F + f0 + (__ffs(at) - 1));
        }
        if (bb) return;
    }
}

// The sequential walk for one point by a warp (cr, fr: the point's rows of ctm and fip).
__device__ __noinline__ void walk_in_order(const float* __restrict__ cr, const float* __restrict__ fr,
                                           float q, uint32_t C, uint32_t F,
                                           const float* __restrict__ fneg,
                                           const float* __restrict__ stat, uint64_t* near,
                                           float& best_out, int32_t& id_out) {
    const int lane = threadIdx.x & 31;
    // the first cluster: smallest (term, id)
    uint64_t kmin = ~0ull;
    for (uint32_t c = lane; c < C; c += 32) {
        const uint64_t k = term_key(__fadd_rn(cr[c], q), c);
        kmin = k < kmin ? k : kmin;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t u = __shfl_xor_sync(0xffffffffu, kmin, o);
        kmin = u < kmin ? u : kmin;
    }
    float best = FLT_MAX;
    int32_t best_id = -1;
    const uint32_t c1 = (uint32_t)kmin;
    walk_cluster(c1, key_to_float((uint32_t)(kmin >> 32)), fr, fneg, stat, F, best, best_id);
    // the clusters whose f = 0 test does not break with this best
    const float th = __fsub_rn(__fsqrt_rn(best), fneg[0]);
    uint32_t cnt = 0;
    for (uint32_t c0 = 0; c0 < C; c0 += 32) {
        const uint32_t c = c0 + lane;
        bool in = false;
        uint64_t k = 0;
        if (c < C && c != c1) {
            const float t = __fadd_rn(cr[c], q);
            in = !(th < __fsqrt_rn(t));
            k = term_key(t, c);
        }
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) {
            const uint32_t pos = cnt + __popc(b & ((1u << lane) - 1));
            if (pos < kMaxNear) near[pos] = k;
        }
        cnt += __popc(b);
    }
    __syncwarp();
    if (cnt <= kMaxNear) {
        // sort the collected keys (at most kMaxNear; odd-even transposition over lanes)
        for (uint32_t r = 0; r < cnt; ++r) {
            for (uint32_t j = 2 * lane + (r & 1); j + 1 < cnt; j += 64) {
                const uint64_t a = near[j], b = near[j + 1];
                if (b < a) {
                    near[j] = b;
                    near[j + 1] = a;
                }
            }
            __syncwarp();
        }
        for (uint32_t r = 0; r < cnt; ++r) {
            const uint64_t k = near[r];
            walk_cluster((uint32_t)k, key_to_float((uint32_t)(k >> 32)), fr, fneg, stat, F, best,
                         best_id);
        }
    } else {
        // many near clusters: take them in order by repeated selection
        uint64_t prev = kmin;
        for (uint32_t r = 0; r < cnt; ++r) {
            uint64_t next = ~0ull;
            for (uint32_t c = lane; c < C; c += 32) {
                const float t = __fadd_rn(cr[c], q);
                const uint64_t k = term_key(t, c);
                if (k > prev && !(th < __fsqrt_rn(t))) next = k < next ? k : next;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const uint64_t u = __shfl_xor_sync(0xffffffffu, next, o);
                next = u < next ? u : next;
            }
            walk_cluster((uint32_t)next, key_to_float((uint32_t)(next >> 32)), fr, fneg, stat, F,
                         best, best_id);
            prev = next;
        }
    }
    best_out = best;
    id_out = best_id;
}

// One warp per point; see the file comment. ctm: [rows][C] 0.5|c|^2 - x.c; fip: [rows][F]
// -x.f; qn: [rows] 0.5|x|^2 (all in the reference's sequential order); smin: [C][G + 1] the
// smallest stationary term of each group of kGroup fine ids, then of the cluster; fmax: [F]
// the largest fneg up to f. Shared memory: the G group minima of -x.f per warp.
__global__ __launch_bounds__(kWalkWarps * 32) void k_cell_walk(
    const float* __restrict__ ctm, const float* __restrict__ fip, const float* __restrict__ qn,
    uint32_t rows, uint32_t C, uint32_t F, uint32_t G, const float* __restrict__ fneg,
    const float* __restrict__ fmax, const float* __restrict__ stat, const float* __restrict__ smin,
    uint32_t* __restrict__ cell, float* __restrict__ dist) {
    extern __shared__ float gmin_s[];
    __shared__ uint64_t near[kWalkWarps][kMaxNear];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t i = blockIdx.x * kWalkWarps + warp;
    if (i >= rows) return;  // whole warps only
    const float* cr = ctm + (uint64_t)i * C;
    const float* fr = fip + (uint64_t)i * F;
    const float q = qn[i];
    if (G == 0) {
        float b;
        int32_t id;
        walk_in_order(cr, fr, q, C, F, fneg, stat, near[warp], b, id);
        if (lane == 0) {
            cell[i] = (uint32_t)id;
            dist[i] = b;
        }
        return;
    }
    float* gmin = gmin_s + (uint64_t)warp * G;
    // -x.f per group (fminf: a value that is not a number bounds nothing) and over all
    uint32_t kall = 0xFFFFFFFFu;
    for (uint32_t g = 0; g < G; ++g) {
        const uint32_t f = g * kGroup + lane;
        const float v = f < F ? fr[f] : FLT_MAX;
        const uint32_t k = __reduce_min_sync(0xffffffffu, v == v ? ordered_key(v) : 0xFFFFFFFFu);
        if (lane == 0) gmin[g] = key_to_float(k);
        kall = k < kall ? k : kall;
    }
    const float all = key_to_float(kall);
    __syncwarp();
    uint32_t bkey = ordered_key(FLT_MAX), bcell = 0;
    uint64_t border = 0;  // the best cell's cluster in the walk's order
    uint32_t without = 0xFFFFFFFFu;  // a cell left out
    bool sure = false;    // the walk visits every cell that has the best score
    // group g of cluster c with term t: the scores of its cells
    auto measure = [&](uint32_t c, float t, uint32_t g) {
        const uint32_t f = g * kGroup + lane;
        uint32_t k = 0xFFFFFFFFu;
        if (f < F && c * F + f != without) {
            const float s = __fadd_rn(__fsub_rn(t, -fr[f]), __ldg(stat + (uint64_t)c * F + f));
            if (s == s) k = ordered_key(s + 0.0f);  // -0 and 0 are equal scores
        }
        const uint32_t m = __reduce_min_sync(0xffffffffu, k);
        if (m > bkey || m == 0xFFFFFFFFu) return;
        // rounding can leave a best below 0: the walk has a best above it (the test holds with
        // 0) or one below 0, whose square root is no number and breaks nothing
        const unsigned at = __ballot_sync(0xffffffffu, k == m);
        const uint32_t f0 = g * kGroup + (__ffs(at) - 1), f1 = g * kGroup + (31 - __clz(at));
        const bool seen =
            !(__fsub_rn(__fsqrt_rn(fmaxf(key_to_float(m), 0.0f)), __ldg(fmax + f1)) < __fsqrt_rn(t));
        const uint64_t order = term_key(t, c);
        const bool lower = m < bkey;
        if (lower || order < border) {  // groups of a cluster ascend: the first stays
            bcell = c * F + f0;
            border = order;
        }
        sure = lower ? seen : sure && seen;
        bkey = m;
    };
    // cluster c: the groups whose bound is not above the best
    auto cluster = [&](uint32_t c, float t) {
        for (uint32_t g0 = 0; g0 < G; g0 += 32) {
            const uint32_t g = g0 + lane;
            bool live = false;
            if (g < G) {
                const float lb = __fadd_rn(__fsub_rn(t, -gmin[g]), __ldg(smin + (uint64_t)c * (G + 1) + g));
                live = !(lb > key_to_float(bkey));
            }
            unsigned todo = __ballot_sync(0xffffffffu, live);
            while (todo) {
                const uint32_t b = __ffs(todo) - 1;
                todo &= todo - 1;
                measure(c, t, g0 + b);
            }
        }
    };
    // the cluster with the smallest (term, id) first: its best cell bounds the others
    uint64_t kmin = ~0ull;
    for (uint32_t c = lane; c < C; c += 32) {
        const uint64_t k = term_key(__fadd_rn(cr[c], q), c);
        kmin = k < kmin ? k : kmin;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t u = __shfl_xor_sync(0xffffffffu, kmin, o);
        kmin = u < kmin ? u : kmin;
    }
    const uint32_t c1 = (uint32_t)kmin;
    float best = FLT_MAX;
    int32_t best_id = 0;
    for (;;) {
        cluster(c1, __fadd_rn(cr[c1], q));
        for (uint32_t c0 = 0; c0 < C; c0 += 32) {
            const uint32_t c = c0 + lane;
            float t = 0.0f;
            bool live = false;
            if (c < C && c != c1) {
                t = __fadd_rn(cr[c], q);
                const float lb = __fadd_rn(__fsub_rn(t, -all), __ldg(smin + (uint64_t)c * (G + 1) + G));
                live = !(lb > key_to_float(bkey));
            }
            unsigned todo = __ballot_sync(0xffffffffu, live);
            while (todo) {
                const uint32_t b = __ffs(todo) - 1;
                todo &= todo - 1;
                cluster(c0 + b, __shfl_sync(0xffffffffu, t, b));
            }
        }
        if (without != 0xFFFFFFFFu) {
            // the walk's best before the cell is one of the others': test with theirs
            const uint32_t c = without / F, f = without - c * F;
            sure = !(__fsub_rn(__fsqrt_rn(fmaxf(key_to_float(bkey), 0.0f)), fmax[f]) <
                     __fsqrt_rn(__fadd_rn(cr[c], q)));
            break;
        }
        best = key_to_float(bkey);
        best_id = (int32_t)bcell;
        if (sure || !(best < FLT_MAX)) break;
        // a point at a cell's very centre (its own cluster's only point, say): the test is
        // decided by roundings, with the smallest score of the other cells it is not
        without = bcell;
        bkey = ordered_key(FLT_MAX);
    }
    if (!sure || !(best < FLT_MAX)) walk_in_order(cr, fr, q, C, F, fneg, stat, near[warp], best, best_id);
    if (lane == 0) {
        cell[i] = (uint32_t)best_id;
        dist[i] = best;
    }
}

// smin (see k_cell_walk): one warp per coarse cluster.
__global__ __launch_bounds__(256) void k_group_min(const float* __restrict__ stat, uint32_t C,
                                                   uint32_t F, uint32_t G, float* __restrict__ smin) {
    const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (c >= C) return;
    float all = FLT_MAX;
    for (uint32_t g = 0; g < G; ++g) {
        const uint32_t f = g * kGroup + lane;
        float v = f < F ? stat[(uint64_t)c * F + f] : FLT_MAX;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) smin[(uint64_t)c * (G + 1) + g] = v;
        all = fminf(all, v);
    }
    if (lane == 0) smin[(uint64_t)c * (G + 1) + G] = all;
}


// fneg[f] = 0 - sqrt(0.5|f|^2) (hierarchical_cluster_index.cpp:1186-1194), and the largest
// one up to each f (one block).
__global__ __launch_bounds__(1024) void k_fneg(const float* __restrict__ fn, uint32_t F,
                                               float* __restrict__ fneg, float* __restrict__ fmax) {
    __shared__ float wmax[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float run = -FLT_MAX;
    for (uint32_t f0 = 0; f0 < F; f0 += 1024) {
        const uint32_t f = f0 + threadIdx.x;
        const float v = f < F ? 0.0f - __fsqrt_rn(fn[f]) : -FLT_MAX;
        float m = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, m, o);
            if (lane >= o) m = fmaxf(m, u);
        }
        if (lane == 31) wmax[warp] = m;
        __syncthreads();
        float before = run;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before = fmaxf(before, wmax[w]);
            run = fmaxf(run, wmax[w]);
        }
        if (f < F) {
            fneg[f] = v;
            fmax[f] = fmaxf(m, before);
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_nearest_cell_assign(uint32_t dim, const float* coarse, uint32_t C,
                                       const float* fine, uint32_t F, const float* x, uint64_t n,
                                       uint32_t* cell, float* dist, cudaStream_t stream,
                                       const float* stat_in) {
    if (n == 0) return cudaSuccess;
    // per-chunk scratch of about 64 MiB for the two term matrices: they stay in L2 between
    // the kernels that write and read them
    // (4096 rows at least, unless they take more than 512 MiB)
    const uint64_t row = 4ull * ((uint64_t)C + F) + 4;
    uint64_t chunk = std::max<uint64_t>((64ull << 20) / row, std::min<uint64_t>(4096, (512ull << 20) / row));
    chunk = chunk < 128 ? std::max<uint64_t>(chunk / 32 * 32, 32) : (chunk / 128) * 128;
    if (chunk > n) chunk = n;
    if (chunk > 65535ull * 64) chunk = 65535ull * 64;  // the score kernels' grid.y
    // group minima of a block's points in shared memory; none (G = 0) for fine counts whose
    // minima do not fit: every point is walked in order
    uint32_t G = (F + kGroup - 1) / kGroup;
    if (sizeof(float) * kWalkWarps * G > 200 * 1024) G = 0;
    float *cn = nullptr, *fn = nullptr, *fneg = nullptr, *fmax = nullptr, *stat = nullptr,
          *smin = nullptr, *ctm = nullptr, *fip = nullptr, *qn = nullptr;
    cudaError_t e = cudaMallocAsync(&cn, sizeof(float) * C, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&fn, sizeof(float) * F, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&fneg, sizeof(float) * F, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&fmax, sizeof(float) * F, stream);
    if (e == cudaSuccess && stat_in == nullptr)
        e = cudaMallocAsync(&stat, sizeof(float) * (uint64_t)C * F, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&smin, sizeof(float) * (uint64_t)C * (G + 1), stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&ctm, sizeof(float) * chunk * C, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&fip, sizeof(float) * chunk * F, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&qn, sizeof(float) * chunk, stream);
    if (e == cudaSuccess) e = launch_half_norms(coarse, C, dim, cn, stream);
    if (e == cudaSuccess) e = launch_half_norms(fine, F, dim, fn, stream);
    if (e == cudaSuccess) {
        k_fneg<<<1, 1024, 0, stream>>>(fn, F, fneg, fmax);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && stat_in == nullptr)
        e = launch_stationary(coarse, C, fine, F, dim, fn, stat, stream);
    const float* sp = stat_in ? stat_in : stat;
    if (e == cudaSuccess) {
        k_group_min<<<(C + 7) / 8, 256, 0, stream>>>(sp, C, F, G, smin);
        e = cudaGetLastError();
    }
    const size_t smem = sizeof(float) * kWalkWarps * G;
    ensure_max_dynamic_smem(k_cell_walk, 200 * 1024);
    for (uint64_t r0 = 0; e == cudaSuccess && r0 < n; r0 += chunk) {
        const uint32_t rows = (uint32_t)(n - r0 < chunk ? n - r0 : chunk);
        const float* xr = x + r0 * dim;
        e = launch_centroid_scores(xr, rows, coarse, C, dim, cn, false, ctm, C, stream);
        if (e == cudaSuccess)
            e = launch_centroid_scores(xr, rows, fine, F, dim, nullptr, true, fip, F, stream);
        if (e == cudaSuccess) e = launch_half_norms(xr, rows, dim, qn, stream);
        if (e == cudaSuccess) {
            k_cell_walk<<<(rows + kWalkWarps - 1) / kWalkWarps, kWalkWarps * 32, smem, stream>>>(
                ctm, fip, qn, rows, C, F, G, fneg, fmax, sp, smin, cell + r0, dist + r0);
            e = cudaGetLastError();
        }
    }
    for (float* p : {cn, fn, fneg, fmax, stat, smin, ctm, fip, qn})
        if (p) cudaFreeAsync(p, stream);
    return e;
}

}  // namespace pgpu
