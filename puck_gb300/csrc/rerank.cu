// k_rerank: rank_topN_points, Puck-Flat branch (puck/puck/puck_index.cpp:428-457):
// the exact FP32 squared L2 of every filter survivor against its original vector,
// then MaxHeap(topk) fed in the order the survivors are given, then reorder().
//
// One block per query. Each warp computes one candidate at a time with coalesced
// row loads; the sum follows the AVX build of L2Sqr16Ext / L2SqrExt
// (puck/tinker/method/hnsw_distfunc_opt_impl_inline.h:41-122): per 16-dim chunk,
// lane i<8 holds d_i^2 + d_{i+8}^2, the 8 lanes are added left to right, chunks
// are added to the running total in order; a tail under 16 dims uses 4 lane
// accumulators, ((l0+l1)+l2)+l3, then a scalar loop. The early abandon of the
// reference only ever rejects candidates the heap would reject, so full sums give
// the same result.
//
// Selection: when no two of the topk+1 smallest distances are equal the heap's
// output is just the ascending order, found by a bitonic sort of
// (distance, position); otherwise a warp replays the heap exactly.
//
// k_rerank_screen (precision form): the same result from fewer bytes. Each
// candidate is first measured on a BF16 copy of its vector; with |x~ - x| <=
// 2^-8 |x| per row and both sums in FP32, |d~ - d| <= E (see screen_bound), so
// every candidate whose exact distance can reach the topk-th lies in
// W = { j : d~_j - E_j <= U }, U = the topk-th smallest d~_j + E_j. Only W is
// recomputed with the exact FP32 order above, sorted and tie-checked like
// k_rerank; a tie sends the block to the full exact heap replay.
#include <cuda_bf16.h>

#include "device_common.cuh"
#include "pgpu_internal.h"

namespace pgpu {
namespace {

// Block shapes (compile-time; -D overrides for tuning sweeps). The exact FP32
// rerank runs 256 threads per query. The screen runs 128 with eight blocks per SM,
// so one block's select and sort overlap other blocks' row gathers.
#ifndef PGPU_RERANK_THREADS
#define PGPU_RERANK_THREADS 256
#endif
#ifndef PGPU_RERANK_SCREEN_THREADS
#define PGPU_RERANK_SCREEN_THREADS 128
#endif
#ifndef PGPU_RERANK_SCREEN_MIN_BLOCKS
#define PGPU_RERANK_SCREEN_MIN_BLOCKS 8
#endif
constexpr int kThreads = PGPU_RERANK_THREADS;
constexpr int kPqThreads = 512;  // the PQ table leaves two blocks per SM
constexpr int kScreenThreads = PGPU_RERANK_SCREEN_THREADS;
constexpr int kScreenWarps = kScreenThreads / 32;
constexpr int kRows = 8;  // candidate rows per warp in flight (rows8_l2_exact)

struct RerankParams {
    const float* q;
    const float* qnorm;
    const int32_t* status;
    const uint32_t* order;  // query of each block (scan mode: queries of one cluster together), or null
    const float* hdist;
    int sort_ties;  // scan mode: replay ties in the filter's (t, memory id) order
    const uint32_t* htag;
    const uint32_t* hcnt;
    const float* feat;
    const uint32_t* mem2local;
    float* out_dist;
    uint32_t* out_ids;
    int32_t* out_status;
    uint32_t d, T, Tp, topk;
    // second-level PQ (whether_pq)
    const float* pq_codebook;
    const float* pq_offsets;
    const uint8_t* pq_codes;
    uint32_t pq_nsq, pq_lsq, pq_code_stride;
    uint32_t work_bytes;  // PQ: shared memory before the query: sort arrays, before them the table
    int pq_table;         // the PQ table is in shared memory
    // a realtime index (RealtimeInsertPuckIndex) sums the PQ table subspace by
    // subspace in order (realtime_insert_puck_index.cpp:466-499), not in
    // lookup_dist_table's four partials
    int pq_sequential;
};

// Exact-order squared L2 of G rows against q (shared memory), computed by one
// warp with the G rows' loads in flight together; results on every lane.
template <int G>
__device__ __forceinline__ void warp_l2_exact(const float* const* rows, const float* q, uint32_t d,
                                              int lane, float* out) {
    const uint32_t d16 = d & ~15u;
    float t[G];
#pragma unroll
    for (int u = 0; u < G; ++u) t[u] = 0.0f;
    const int grp = lane & 16;
    for (uint32_t base = 0; base < d16; base += 32) {
        const uint32_t e = base + lane;
        float sq[G];
#pragma unroll
        for (int u = 0; u < G; ++u) {
            sq[u] = 0.0f;
            if (e < d16) {
                const float a = __fsub_rn(__ldg(rows[u] + e), q[e]);
                sq[u] = __fmul_rn(a, a);
            }
        }
#pragma unroll
        for (int u = 0; u < G; ++u) {
            // lanes 0-7 (chunk at base) and 16-23 (chunk at base+16): d_i^2 + d_{i+8}^2
            const float s = __fadd_rn(sq[u], __shfl_down_sync(0xffffffffu, sq[u], 8));
            float acc = __shfl_sync(0xffffffffu, s, grp);
#pragma unroll
            for (int i = 1; i < 8; ++i) acc = __fadd_rn(acc, __shfl_sync(0xffffffffu, s, grp + i));
            const float acc_b = __shfl_sync(0xffffffffu, acc, 16);
            float tu = __fadd_rn(t[u], acc);               // chunk at base (lane 0's acc)
            tu = __shfl_sync(0xffffffffu, tu, 0);
            if (base + 16 < d16) tu = __fadd_rn(tu, acc_b);  // chunk at base + 16
            t[u] = tu;
        }
    }
    if (d16 < d) {  // L2SqrExt on the last d - d16 < 16 dims, serially
        const uint32_t qty = d - d16;
#pragma unroll
        for (int u = 0; u < G; ++u) {
            const float* x = rows[u] + d16;
            const float* qq = q + d16;
            float l0 = 0.0f, l1 = 0.0f, l2 = 0.0f, l3 = 0.0f;
            uint32_t i = 0;
            for (; i + 4 <= qty; i += 4) {
                const float a0 = __fsub_rn(__ldg(x + i), qq[i]);
                const float a1 = __fsub_rn(__ldg(x + i + 1), qq[i + 1]);
                const float a2 = __fsub_rn(__ldg(x + i + 2), qq[i + 2]);
                const float a3 = __fsub_rn(__ldg(x + i + 3), qq[i + 3]);
                l0 = __fadd_rn(l0, __fmul_rn(a0, a0));
                l1 = __fadd_rn(l1, __fmul_rn(a1, a1));
                l2 = __fadd_rn(l2, __fmul_rn(a2, a2));
                l3 = __fadd_rn(l3, __fmul_rn(a3, a3));
            }
            float sum = __fadd_rn(__fadd_rn(__fadd_rn(l0, l1), l2), l3);
            for (; i < qty; ++i) {
                const float a = __fsub_rn(__ldg(x + i), qq[i]);
                sum = __fadd_rn(sum, __fmul_rn(a, a));
            }
            t[u] = __fadd_rn(t[u], sum);
        }
    }
#pragma unroll
    for (int u = 0; u < G; ++u) out[u] = t[u];
}

// The same sums as warp_l2_exact for G = 8 rows, d % 4 == 0 and 16-byte aligned
// rows and q: each group of 8 lanes measures two rows with 16-byte loads (lane l
// holds the float4s l, l + 8, ...), so a warp load instruction covers four whole
// 128-byte row segments. In one 16-dim chunk the four lanes holding float4s
// 0..3 pair dims i and i + 8 by one exchange (lane u <-> u + 2), lane 0 sums
// s0..s3 left to right and lane 1 continues with s4..s7 after one more
// exchange, so each chunk sum keeps the L2Sqr16Ext order; the running total is
// kept on lane 1 of the group, chunk by chunk in order. Results on every lane.
__device__ __forceinline__ void warp_l2_exact_vec(const float* const* rows, const float* q,
                                                  uint32_t d, int lane, float* out) {
    constexpr int R = 2;  // rows per group of 8 lanes
    const int g = lane >> 3, l = lane & 7;
    const uint32_t d16 = d & ~15u;
    const uint32_t nf4 = d16 >> 2;
    const float4* q4 = reinterpret_cast<const float4*>(q);
    // this group's rows g and g + 4 (selects on constant indices keep them in registers)
    const float* mine[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
        mine[r] = g == 0 ? rows[4 * r] : g == 1 ? rows[4 * r + 1] : g == 2 ? rows[4 * r + 2] : rows[4 * r + 3];
    float t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) t[r] = 0.0f;
    for (uint32_t f0 = 0; f0 < nf4; f0 += 8) {
        const uint32_t f = f0 + l;
        const bool in = f < nf4;
        float4 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            x[r] = in ? __ldg(reinterpret_cast<const float4*>(mine[r]) + f)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 qq = in ? q4[f] : make_float4(0.f, 0.f, 0.f, 0.f);
        const bool second = f0 + 4 < nf4;  // this step holds two chunks
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float a0 = __fsub_rn(x[r].x, qq.x), a1 = __fsub_rn(x[r].y, qq.y);
            const float a2 = __fsub_rn(x[r].z, qq.z), a3 = __fsub_rn(x[r].w, qq.w);
            const float q0 = __fmul_rn(a0, a0), q1 = __fmul_rn(a1, a1);
            const float q2 = __fmul_rn(a2, a2), q3 = __fmul_rn(a3, a3);
            // lanes u = 0, 1 of a chunk: d_i^2 + d_{i+8}^2 with the partner u + 2
            const float s0 = __fadd_rn(q0, __shfl_xor_sync(0xffffffffu, q0, 2));
            const float s1 = __fadd_rn(q1, __shfl_xor_sync(0xffffffffu, q1, 2));
            const float s2 = __fadd_rn(q2, __shfl_xor_sync(0xffffffffu, q2, 2));
            const float s3 = __fadd_rn(q3, __shfl_xor_sync(0xffffffffu, q3, 2));
            const float a = __fadd_rn(__fadd_rn(__fadd_rn(s0, s1), s2), s3);   // lane u = 0
            const float b = __shfl_xor_sync(0xffffffffu, a, 1);                 // to lane u = 1
            const float chunk = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(b, s0), s1), s2), s3);
            const float hi = __shfl_down_sync(0xffffffffu, chunk, 4);           // lane 5 -> 1
            float tr = __fadd_rn(t[r], chunk);
            if (second) tr = __fadd_rn(tr, hi);
            t[r] = tr;
        }
    }
    if (d16 < d && l == 1) {  // L2SqrExt on the last d - d16 (a multiple of 4) dims
        const uint32_t qty = d - d16;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float* xr = mine[r] + d16;
            const float* qr = q + d16;
            float l0 = 0.0f, l1 = 0.0f, l2 = 0.0f, l3 = 0.0f;
            for (uint32_t i = 0; i + 4 <= qty; i += 4) {
                const float a0 = __fsub_rn(__ldg(xr + i), qr[i]);
                const float a1 = __fsub_rn(__ldg(xr + i + 1), qr[i + 1]);
                const float a2 = __fsub_rn(__ldg(xr + i + 2), qr[i + 2]);
                const float a3 = __fsub_rn(__ldg(xr + i + 3), qr[i + 3]);
                l0 = __fadd_rn(l0, __fmul_rn(a0, a0));
                l1 = __fadd_rn(l1, __fmul_rn(a1, a1));
                l2 = __fadd_rn(l2, __fmul_rn(a2, a2));
                l3 = __fadd_rn(l3, __fmul_rn(a3, a3));
            }
            t[r] = __fadd_rn(t[r], __fadd_rn(__fadd_rn(__fadd_rn(l0, l1), l2), l3));
        }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) out[u] = __shfl_sync(0xffffffffu, t[u >> 2], 8 * (u & 3) + 1);
}

// Dispatch: the vector form when d % 4 == 0 and q is 16-byte aligned (rows then
// are: the vectors start 256-byte aligned with d * 4 bytes per row).
__device__ __forceinline__ void rows8_l2_exact(const float* const* rows, const float* q, uint32_t d,
                                               int lane, float* out) {
    if ((d & 3u) == 0 && (reinterpret_cast<uintptr_t>(q) & 15u) == 0)
        warp_l2_exact_vec(rows, q, d, lane, out);
    else
        warp_l2_exact<8>(rows, q, d, lane, out);
}

// The exact MaxHeap(topk) fed with cnt distances in the given order (null: as they are), then
// reorder(), written out; by one warp (heap: topk + 2 entries, 16-byte aligned). One thread
// doing all, with each tag fetched from memory, took 0.2 ms for 1100 candidates and topk 100
// (a query in that path ended a whole batch's launch). A distance that is not a number (of a
// stored vector that is not finite) is no result.
__device__ __forceinline__ void heap_replay(uint2* heap, const float* dist, const uint32_t* order,
                                         uint32_t cnt, uint32_t topk, const uint32_t* tags,
                                         const uint32_t* mem2local, float* od, uint32_t* oi) {
    const uint32_t rn = warp_heap_replay<true>(heap, dist, order, cnt, topk);
    for (uint32_t i = threadIdx.x & 31; i < topk; i += 32) {
        od[i] = __uint_as_float(heap[i + 1].x);
        oi[i] = i < rn ? mem2local[tags[heap[i + 1].y]] : kNoLabel;
    }
}

// PQ: the second-level PQ branch of rank_topN_points (puck_index.cpp:402-427): per
// candidate (filter distance - |q|^2) + pq offset, then + lookup_dist_table over
// the PQ table (get_dist_table, quantization.cpp:260-270), in the reference's
// float order; the same heap semantics as the Puck-Flat branch. Bound by the lookups: the
// table in shared memory (random banks, about 3.4 wavefronts per warp-wide lookup) and code
// rows by 16-byte loads; one-dimensional entries formed from the codebook at each lookup, and
// the rows read a word at a time, took 0.62 ms for 1537 queries of 1100 candidates and 96 entries
// each, with the heap by one thread; this form takes 0.23.
template <bool PQ>
__global__ __launch_bounds__(PQ ? kPqThreads : kThreads) void k_rerank(RerankParams p) {
    constexpr int NT = PQ ? kPqThreads : kThreads;
    extern __shared__ __align__(16) unsigned char smem[];
    // Sort keys, later a replayed heap of topk + 2 entries. PQ: with the other sort arrays they
    // take the table's place once the distances are there. Else query and distances follow the
    // keys and the ids come last: in the PQ order the rows of odd dimensions took 4% longer
    // (10000 queries of 300 rows, 30 dimensions: 1.50 ms a call, 1.55).
    unsigned long long* okey = reinterpret_cast<unsigned long long*>(smem);  // [Tp + 2]
    float* pq_lut = reinterpret_cast<float*>(smem);                          // [pq_nsq * 256] (PQ)
    float* after = reinterpret_cast<float*>(okey + p.Tp + 2);
    float* qv = PQ ? reinterpret_cast<float*>(smem + p.work_bytes) : after;  // [d]
    float* dist = qv + p.d;                                                  // [T]
    float* sv = PQ ? after : dist + p.T;                                     // [Tp]
    uint32_t* si = reinterpret_cast<uint32_t*>(sv + p.Tp);                   // [Tp]
    uint32_t* opos = si + p.Tp;                                              // [Tp]
    uint32_t* stag = PQ ? reinterpret_cast<uint32_t*>(dist + p.T) : opos + p.Tp;  // [T]
    __shared__ uint32_t sel_hist[256];
    __shared__ uint32_t sel_state[2];
    __shared__ uint32_t sel_count;
    const uint32_t qi = p.order ? p.order[blockIdx.x] : blockIdx.x, topk = p.topk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* od = p.out_dist + (uint64_t)qi * topk;
    uint32_t* oi = p.out_ids + (uint64_t)qi * topk;
    const int32_t stq = p.status[qi];
    if (p.out_status && tid == 0) p.out_status[qi] = stq;
    if (stq != 0) {
        for (uint32_t i = tid; i < topk; i += NT) {
            od[i] = sentinel_f();
            oi[i] = kNoLabel;
        }
        return;
    }
    const uint32_t cnt = p.hcnt[qi];
    const uint32_t* tags = p.htag + (uint64_t)qi * p.T;
    for (uint32_t i = tid; i < p.d; i += NT) qv[i] = p.q[(uint64_t)qi * p.d + i];
    // the candidates' memory ids in shared memory (one coalesced load)
    for (uint32_t i = tid; i < cnt; i += NT) {
        const uint32_t mi = tags[i];
        stag[i] = mi;
        if (PQ) {  // the candidates' rows are on their way while the table is built
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pq_codes + (uint64_t)mi * p.pq_code_stride));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pq_offsets + mi));
        }
    }
    tags = stag;
    __syncthreads();
    if (PQ && p.pq_table) {
        if (p.pq_lsq == 1) {  // entries (q_m - c)^2: l2sqr_sse of one dimension
            const float4* cb4 = reinterpret_cast<const float4*>(p.pq_codebook);
#pragma unroll 4
            for (uint32_t e = tid; e < p.pq_nsq * 64; e += NT) {
                const float4 c = __ldg(cb4 + e);
                const float x = qv[e >> 6];
                const float d0 = __fsub_rn(x, c.x), d1 = __fsub_rn(x, c.y);
                const float d2 = __fsub_rn(x, c.z), d3 = __fsub_rn(x, c.w);
                reinterpret_cast<float4*>(pq_lut)[e] = make_float4(
                    __fmul_rn(d0, d0), __fmul_rn(d1, d1), __fmul_rn(d2, d2), __fmul_rn(d3, d3));
            }
        } else {
            for (uint32_t e = tid; e < p.pq_nsq * 256; e += NT)
                pq_lut[e] = l2sqr_sse(qv + (e >> 8) * p.pq_lsq,
                                      p.pq_codebook + (uint64_t)e * p.pq_lsq, p.pq_lsq);
        }
        __syncthreads();
    }
    if (PQ) {
        const float qn = p.qnorm[qi];
        const float* hd = p.hdist + (uint64_t)qi * p.T;
        const bool wide = ((p.pq_code_stride | p.pq_nsq) & 15u) == 0;
        auto start = [&](uint32_t j) {
            return __fadd_rn(__fsub_rn(hd[j], qn), __ldg(p.pq_offsets + tags[j]));
        };
        auto row = [&](uint32_t j) { return p.pq_codes + (uint64_t)tags[j] * p.pq_code_stride; };
        if (p.pq_table && wide && !p.pq_sequential) {
            // rows of whole 16-byte words; lookup_dist_table's order, 16 entries at a time
            for (uint32_t j = tid; j < cnt; j += NT) {
                const uint4* w = reinterpret_cast<const uint4*>(row(j));
                const float t = start(j);
                float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                uint4 c = __ldg(w);
                const float* col = pq_lut;
                for (uint32_t m0 = 0; m0 < p.pq_nsq; m0 += 16, col += 16 * 256) {
                    const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
                    if (m0 + 16 < p.pq_nsq) c = __ldg(w + (m0 >> 4) + 1);
                    float x[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        x[k] = col[k * 256 + ((cw[k >> 2] >> (8 * (k & 3))) & 255u)];
#pragma unroll
                    for (int k = 0; k < 16; ++k) a[k & 3] = __fadd_rn(a[k & 3], x[k]);
                }
                dist[j] = __fadd_rn(t, __fadd_rn(__fadd_rn(a[0], a[1]), __fadd_rn(a[2], a[3])));
            }
        } else if (p.pq_table) {
            for (uint32_t j = tid; j < cnt; j += NT) {
                const uint8_t* code = row(j);
                float t = start(j);
                if (p.pq_sequential) {
                    for (uint32_t m = 0; m < p.pq_nsq; ++m)
                        t = __fadd_rn(t, pq_lut[m * 256 + code[m]]);
                } else {
                    t = __fadd_rn(t, lut_sum(code, pq_lut, p.pq_nsq));
                }
                dist[j] = t;
            }
        } else {
            // one-dimensional subspaces whose table does not fit: each entry (q_m - c)^2 is
            // formed when it is looked up (the same bits), in the same order
            for (uint32_t j = tid; j < cnt; j += NT) {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(row(j));
                float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                float t = start(j);
                for (uint32_t m0 = 0; m0 < p.pq_nsq; m0 += 4) {
                    const uint32_t c4 = __ldg(w + (m0 >> 2));
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t m = m0 + k;
                        if (m < p.pq_nsq) {
                            const float y = __ldg(p.pq_codebook + (uint64_t)m * 256 + ((c4 >> (8 * k)) & 255u));
                            const float df = __fsub_rn(qv[m], y);
                            if (p.pq_sequential) t = __fadd_rn(t, __fmul_rn(df, df));
                            else a[k] = __fadd_rn(a[k], __fmul_rn(df, df));
                        }
                    }
                }
                if (!p.pq_sequential)
                    t = __fadd_rn(t, __fadd_rn(__fadd_rn(a[0], a[1]), __fadd_rn(a[2], a[3])));
                dist[j] = t;
            }
        }
    }
    // kRows rows per warp with their loads in flight together
    for (uint32_t j0 = warp * kRows; !PQ && j0 < cnt; j0 += (NT / 32) * kRows) {
        const float* rows[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const uint32_t j = j0 + u;
            rows[u] = p.feat + (uint64_t)tags[j < cnt ? j : j0] * p.d;
        }
        float v[kRows];
        rows8_l2_exact(rows, qv, p.d, lane, v);
        if (lane == 0) {
#pragma unroll
            for (int u = 0; u < kRows; ++u)
                if (j0 + u < cnt) dist[j0 + u] = v[u];
        }
    }
    __syncthreads();
    // (distance, position) pairs, ascending. Only the topk+1 smallest matter (result
    // and tie check): with more candidates, keep every one at or below the
    // (topk+1)-th smallest distance (ties included) and sort just those.
    uint32_t m2 = p.Tp;
    if (cnt > topk + 1) {
        const float U = key_to_float(block_kth_key<NT>(dist, cnt, topk + 1, sel_hist, sel_state));
        if (tid == 0) sel_count = 0;
        __syncthreads();
        for (uint32_t i = tid; i < cnt; i += NT)
            if (dist[i] <= U) {
                const uint32_t pos = atomicAdd(&sel_count, 1u);
                sv[pos] = dist[i];
                si[pos] = i;
            }
        __syncthreads();
        const uint32_t m = sel_count;
        m2 = 2;
        while (m2 < m) m2 <<= 1;
        for (uint32_t i = m + tid; i < m2; i += NT) {
            sv[i] = __int_as_float(0x7f800000);
            si[i] = 0xFFFFFFFFu;
        }
    } else {
        for (uint32_t i = tid; i < p.Tp; i += NT) {
            sv[i] = i < cnt ? dist[i] : __int_as_float(0x7f800000);
            si[i] = i < cnt ? i : 0xFFFFFFFFu;
        }
    }
    __syncthreads();
    for (uint32_t size = 2; size <= m2; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t t = tid; t < m2 / 2; t += NT) {
                const uint32_t lo = 2 * t - (t & (stride - 1));
                const uint32_t hi = lo + stride;
                const bool asc = (lo & size) == 0;
                const float a = sv[lo], b = sv[hi];
                const uint32_t ia = si[lo], ib = si[hi];
                const bool gt = (a > b) || (a == b && ia > ib);
                if (gt == asc) {
                    sv[lo] = b;
                    sv[hi] = a;
                    si[lo] = ib;
                    si[hi] = ia;
                }
            }
            __syncthreads();
        }
    }
    const uint32_t keep = cnt < topk ? cnt : topk;
    // ties that the heap could resolve differently: among the topk+1 smallest, or
    // anywhere among the results when there are no more candidates than topk
    const uint32_t check = cnt <= topk ? (cnt > 0 ? cnt - 1 : 0) : topk;
    int tie = 0;
    for (uint32_t i = tid; i < check; i += NT)
        if (sv[i] == sv[i + 1]) tie = 1;
    tie = __syncthreads_or(tie);
    if (!tie) {
        for (uint32_t i = tid; i < topk; i += NT) {
            od[i] = i < keep ? sv[i] : sentinel_f();
            oi[i] = i < keep ? p.mem2local[tags[si[i]]] : kNoLabel;
        }
        return;
    }
    __syncthreads();
    if (p.sort_ties)
        order_by_filter_key<NT>(p.hdist + (uint64_t)qi * p.T, tags, cnt, p.Tp, okey, opos);
    // (the sort keys are no longer read)
    if (warp == 0)
        heap_replay(reinterpret_cast<uint2*>(okey), dist, p.sort_ties ? opos : nullptr, cnt, topk, tags,
                    p.mem2local, od, oi);
}

// Bound on |d~ - d| for a row with |x| <= xabs and screened distance d~ (d dims).
__device__ __forceinline__ float screen_bound(float dt, float xabs, uint32_t d) {
    const float ta = sqrtf(fmaxf(dt, 0.0f)) * 1.0009765625f + 1e-20f;
    const float dx = 0.00390625f * xabs * 1.0009765625f;
    const float tb = ta + dx;
    return dx * (2.0f * ta + dx) + (float)(3 * d + 8) * 1.1920928955078125e-07f * tb * tb + 1e-30f;
}

struct ScreenParams {
    const float* q;
    const int32_t* status;
    const uint32_t* order;
    const float* hdist;
    const uint32_t* htag;
    const uint32_t* hcnt;
    const float* feat;
    const uint16_t* feat_bf16;
    const float* feat_abs;
    const uint32_t* mem2local;
    float* out_dist;
    uint32_t* out_ids;
    int32_t* out_status;
    uint32_t d, T, Tp, topk;
};

__global__ __launch_bounds__(kScreenThreads, PGPU_RERANK_SCREEN_MIN_BLOCKS) void k_rerank_screen(ScreenParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    // [Tp + 2]: a heap replayed here has topk + 2 entries
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem);
    float* qv = reinterpret_cast<float*>(keys + p.Tp + 2);                   // [d]
    float* approx = qv + p.d;                                                // [T]
    float* hi = approx + p.T;                                                // [T] d~ + E, then exact
    float* bnd = hi + p.T;                                                   // [T]
    uint32_t* opos = reinterpret_cast<uint32_t*>(bnd + p.T);                 // [Tp]
    __shared__ uint32_t hist[256];
    __shared__ uint32_t state[2];
    __shared__ uint32_t wcount;
    const uint32_t qi = p.order ? p.order[blockIdx.x] : blockIdx.x, topk = p.topk, d = p.d;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* od = p.out_dist + (uint64_t)qi * topk;
    uint32_t* oi = p.out_ids + (uint64_t)qi * topk;
    const int32_t stq = p.status[qi];
    if (p.out_status && tid == 0) p.out_status[qi] = stq;
    if (stq != 0) {
        for (uint32_t i = tid; i < topk; i += kScreenThreads) {
            od[i] = sentinel_f();
            oi[i] = kNoLabel;
        }
        return;
    }
    const uint32_t cnt = p.hcnt[qi];
    const uint32_t* tags = p.htag + (uint64_t)qi * p.T;
    for (uint32_t i = tid; i < d; i += kScreenThreads) qv[i] = p.q[(uint64_t)qi * d + i];
    // the candidates' memory ids in shared memory: one coalesced load, then every row
    // gather below starts from a shared-memory read
    uint32_t* stag = opos + p.Tp;  // [T]
    for (uint32_t i = tid; i < cnt; i += kScreenThreads) stag[i] = tags[i];
    tags = stag;
    if (tid == 0) wcount = 0;
    __syncthreads();
    bool full = cnt <= topk;
    if (!full) {
        if ((d & 7u) == 0 && d <= 128) {
            // screen, vector form: a half warp per row, 8 dimensions (one 16-byte
            // load) per lane, kRows rows per half warp in flight
            const int half = lane >> 4, hl = lane & 15;
            const bool active = (uint32_t)hl * 8 < d;
            float qr[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) qr[t] = active ? qv[hl * 8 + t] : 0.0f;
            // the loop runs the same iterations on both half warps (the shuffles below
            // take the full mask): a warp owns 2 * kRows rows per iteration
            for (uint32_t jw = warp * 2 * kRows; jw < cnt; jw += kScreenWarps * 2 * kRows) {
                const uint32_t j0 = jw + half * kRows;
                uint4 x[kRows];
#pragma unroll
                for (int u = 0; u < kRows; ++u) {
                    const uint32_t j = j0 + u < cnt ? j0 + u : jw;
                    x[u] = active ? __ldg(reinterpret_cast<const uint4*>(
                                        p.feat_bf16 + (uint64_t)tags[j] * d) + hl)
                                  : make_uint4(0, 0, 0, 0);
                }
                float acc[kRows];
#pragma unroll
                for (int u = 0; u < kRows; ++u) {
                    const uint32_t w[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
                    float a = 0.0f;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const float lo = __uint_as_float(w[t] << 16);
                        const float hi2 = __uint_as_float(w[t] & 0xFFFF0000u);
                        const float d0 = qr[2 * t] - lo, d1 = qr[2 * t + 1] - hi2;
                        a += d0 * d0 + d1 * d1;
                    }
                    acc[u] = active ? a : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < kRows; ++u)
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
                if (hl < kRows) {
                    float mine = acc[0];
#pragma unroll
                    for (int u = 1; u < kRows; ++u)
                        if (hl == u) mine = acc[u];
                    const uint32_t j = j0 + hl;
                    if (j < cnt) {
                        const float e = screen_bound(mine, p.feat_abs[tags[j]], d);
                        approx[j] = mine;
                        bnd[j] = e;
                        hi[j] = mine + e;
                    }
                }
            }
        } else {
        // screen: kRows BF16 rows per warp in flight
        for (uint32_t j0 = warp * kRows; j0 < cnt; j0 += kScreenWarps * kRows) {
            float acc[kRows];
            const uint16_t* rows[kRows];
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                const uint32_t j = j0 + u;
                rows[u] = p.feat_bf16 + (uint64_t)tags[j < cnt ? j : j0] * d;
                acc[u] = 0.0f;
            }
            for (uint32_t k = lane; k < d; k += 32) {
                const float qk = qv[k];
#pragma unroll
                for (int u = 0; u < kRows; ++u) {
                    const float x = __bfloat162float(__ushort_as_bfloat16(__ldg(rows[u] + k)));
                    const float df = qk - x;
                    acc[u] += df * df;
                }
            }
#pragma unroll
            for (int u = 0; u < kRows; ++u)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
            if (lane < kRows) {
                float mine = acc[0];
#pragma unroll
                for (int u = 1; u < kRows; ++u)
                    if (lane == u) mine = acc[u];
                const uint32_t j = j0 + lane;
                if (j < cnt) {
                    const float e = screen_bound(mine, p.feat_abs[tags[j]], d);
                    approx[j] = mine;
                    bnd[j] = e;
                    hi[j] = mine + e;
                }
            }
        }
        }
        __syncthreads();
        const float U = key_to_float(block_kth_key<kScreenThreads>(hi, cnt, topk, hist, state));
        for (uint32_t j = tid; j < cnt; j += kScreenThreads)
            if (approx[j] - bnd[j] <= U) keys[atomicAdd(&wcount, 1u)] = j;
        __syncthreads();
        const uint32_t m = wcount;
        // exact FP32 distances of the window, in the reference's order
        for (uint32_t i0 = warp * kRows; i0 < m; i0 += kScreenWarps * kRows) {
            const float* rows[kRows];
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                const uint32_t i = i0 + u;
                rows[u] = p.feat + (uint64_t)tags[(uint32_t)keys[i < m ? i : i0]] * d;
            }
            float v[kRows];
            rows8_l2_exact(rows, qv, d, lane, v);
            __syncwarp();
            if (lane == 0) {
#pragma unroll
                for (int u = 0; u < kRows; ++u) {
                    const uint32_t i = i0 + u;
                    if (i < m) {
                        const uint32_t j = (uint32_t)keys[i];
                        keys[i] = ((unsigned long long)ordered_key(v[u]) << 32) | j;
                    }
                }
            }
        }
        __syncthreads();
        uint32_t mp = 2;
        while (mp < m) mp <<= 1;
        for (uint32_t i = m + tid; i < mp; i += kScreenThreads) keys[i] = ~0ull;
        __syncthreads();
        bitonic_sort_u64<kScreenThreads>(keys, mp);
        const uint32_t check = m - 1 < topk ? m - 1 : topk;
        int tie = 0;
        for (uint32_t i = tid; i < check; i += kScreenThreads)
            if ((uint32_t)(keys[i] >> 32) == (uint32_t)(keys[i + 1] >> 32)) tie = 1;
        tie = __syncthreads_or(tie);
        if (!tie) {
            for (uint32_t i = tid; i < topk; i += kScreenThreads) {
                od[i] = key_to_float((uint32_t)(keys[i] >> 32));
                oi[i] = p.mem2local[tags[(uint32_t)keys[i]]];
            }
            return;
        }
        full = true;
    }
    // every candidate exactly, then MaxHeap(topk) in candidate order and reorder()
    for (uint32_t j0 = warp * kRows; j0 < cnt; j0 += kScreenWarps * kRows) {
        const float* rows[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const uint32_t j = j0 + u;
            rows[u] = p.feat + (uint64_t)tags[j < cnt ? j : j0] * d;
        }
        float v[kRows];
        rows8_l2_exact(rows, qv, d, lane, v);
        if (lane == 0) {
#pragma unroll
            for (int u = 0; u < kRows; ++u)
                if (j0 + u < cnt) hi[j0 + u] = v[u];
        }
    }
    __syncthreads();
    // the heap is fed in the filter's (t, memory id) order
    order_by_filter_key<kScreenThreads>(p.hdist + (uint64_t)qi * p.T, tags, cnt, p.Tp, keys, opos);
    if (warp == 0)
        heap_replay(reinterpret_cast<uint2*>(keys), hi, opos, cnt, topk, tags, p.mem2local, od, oi);
}

uint32_t pow2_at_least(uint32_t v) {
    uint32_t p = 2;
    while (p < v) p <<= 1;
    return p;
}

}  // namespace

// The limit on filter_topk and topk is checked against this size (the launch may take less).
size_t rerank_smem_bytes(const DeviceIndex& ix, uint32_t T, uint32_t topk) {
    const uint32_t Tp = pow2_at_least(T > topk ? T : topk);
    // the PQ table is only held for subspaces of more than one dimension
    const size_t pq_table = ix.pq_lsq > 1 ? sizeof(float) * ix.pq_nsq * 256 : 0;
    return sizeof(float) * (ix.d + T) + (sizeof(float) + 2 * sizeof(uint32_t) + 8) * Tp + pq_table +
           sizeof(uint32_t) * T;
}

cudaError_t launch_rerank(const DeviceIndex& ix, const SearchConfig& cfg, uint32_t n,
                          uint32_t topk, const Scratch& s, float* out_dist, uint32_t* out_ids,
                          int32_t* out_status, cudaStream_t stream) {
    RerankParams p;
    p.q = s.q;
    p.qnorm = s.qnorm;
    p.status = s.status;
    p.order = s.order;
    p.hdist = s.hdist;
    p.sort_ties = cfg.mode == PGPU_MODE_SCAN ? 1 : 0;
    p.pq_codebook = ix.pq_codebook;
    p.pq_offsets = ix.pq_offsets;
    p.pq_codes = ix.pq_codes;
    p.pq_nsq = ix.pq_nsq;
    p.pq_lsq = ix.pq_lsq;
    p.pq_code_stride = ix.pq_code_stride;
    p.pq_sequential = ix.ins_cap > 0 ? 1 : 0;
    p.htag = s.htag;
    p.hcnt = s.hcnt;
    p.feat = ix.feat;
    p.mem2local = ix.mem2local;
    p.out_dist = out_dist;
    p.out_ids = out_ids;
    p.out_status = out_status;
    p.d = ix.d;
    p.T = s.T;
    p.Tp = pow2_at_least(s.T > topk ? s.T : topk);
    p.topk = topk;
    // the sort arrays, or the PQ table while the distances are formed; and query, distances
    // and ids. The table of one-dimensional subspaces is left out where it does not fit.
    const size_t sort = (sizeof(float) + 2 * sizeof(uint32_t) + 8) * (size_t)p.Tp + 16;
    const size_t table = sizeof(float) * 256 * (size_t)ix.pq_nsq;
    const size_t rest = sizeof(float) * (ix.d + (size_t)s.T) + sizeof(uint32_t) * (size_t)s.T;
    p.pq_table = ix.pq_nsq && (ix.pq_lsq > 1 || table + rest + 16 <= 220 * 1024);
    const size_t work = p.pq_table && table > sort ? table : sort;
    p.work_bytes = (uint32_t)((work + 15) / 16 * 16);
    const size_t smem = p.work_bytes + rest;
    if (ix.pq_nsq) {
        ensure_max_dynamic_smem(k_rerank<true>, 220 * 1024);
        k_rerank<true><<<n, kPqThreads, smem, stream>>>(p);
    } else {
        ensure_max_dynamic_smem(k_rerank<false>, 220 * 1024);
        k_rerank<false><<<n, kThreads, smem, stream>>>(p);
    }
    return cudaGetLastError();
}

size_t rerank_screen_smem_bytes(const DeviceIndex& ix, uint32_t T) {
    const uint32_t Tp = pow2_at_least(T);
    return sizeof(unsigned long long) * (Tp + 2) + sizeof(float) * (ix.d + 3ull * T) +
           sizeof(uint32_t) * (Tp + T);
}

cudaError_t launch_rerank_screen(const DeviceIndex& ix, uint32_t n, uint32_t topk, const Scratch& s,
                                 float* out_dist, uint32_t* out_ids, int32_t* out_status,
                                 cudaStream_t stream) {
    if (ix.feat_bf16 == nullptr || ix.feat_abs == nullptr) return cudaErrorInvalidValue;
    ScreenParams p;
    p.q = s.q;
    p.status = s.status;
    p.order = s.order;
    p.hdist = s.hdist;
    p.htag = s.htag;
    p.hcnt = s.hcnt;
    p.feat = ix.feat;
    p.feat_bf16 = ix.feat_bf16;
    p.feat_abs = ix.feat_abs;
    p.mem2local = ix.mem2local;
    p.out_dist = out_dist;
    p.out_ids = out_ids;
    p.out_status = out_status;
    p.d = ix.d;
    p.T = s.T;
    p.Tp = pow2_at_least(s.T);
    p.topk = topk;
    const size_t smem = rerank_screen_smem_bytes(ix, s.T);
    ensure_max_dynamic_smem(k_rerank_screen, 220 * 1024);
    k_rerank_screen<<<n, kScreenThreads, smem, stream>>>(p);
    return cudaGetLastError();
}

}  // namespace pgpu
