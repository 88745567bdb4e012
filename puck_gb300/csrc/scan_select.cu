// The throughput-mode filter stage (scan mode). For one query it streams every
// filter record of its probed coarse clusters (each cluster is one contiguous
// range in memory order) and keeps the filter_topk smallest ADC distances. Three
// kernels: the split scan (k_scan_score, "split scan" below), which answers every
// query whose candidates fit its key buffer; the fused k_scan_il
// (interleaved layout) for the rest; k_scan_select for nsq not a multiple of 4.
//
// Per record the distance is the reference's own expression for a scanned point
// (puck/puck/puck_index.cpp:360-368 with cell_dist from :539-540):
//     cell_dist = (coarse_term + stationary[c][f]) + fine_term[f]
//     t         = (float)(2 * cell_dist + offset) + lookup_dist_table(codes)
// so every t is bit-identical to the value PuckIndex::search would compute for
// that point. Unlike the reference's pivot-pruned cell walk, no cell of a probed
// cluster is skipped: the result is the exact top-filter_topk by (t, memory id)
// over all records of the probed clusters, a superset search of the same cells.
//
// Table: each block builds its query's table in shared memory
// (get_dist_table, quantization.cpp:260-270, in the reference's lane order):
// thread j computes codeword j of every subspace from one coalesced 16-byte
// codebook load per subspace (the codebook stays in L2).
//
// Selection: a buffer of (t, id) keys in shared memory, sized from filter_topk,
// with a running threshold tau, a key with at least filter_topk kept keys below
// it; records whose (2*cell_dist + offset, id) key is not below tau are dropped
// before the table lookups (t can only grow). When the buffer could not take
// another round, one histogram pass over the buffer's float values (1024 linear
// bins between the smallest and the largest) finds the bin holding the
// filter_topk-th key; the keys above that bin are dropped and tau becomes the
// bin's upper edge. A last exact radix select leaves the set of the filter_topk
// smallest (t, id) keys, unordered.
//
// Blocks start in launch order longest scan first, queries of neighbouring clusters
// together (k_scan_work, k_scan_order), one block per query.
//
// Precision form (FP16 tables): the table is stored in FP16, scaled per query by a
// power of two 2^e chosen from the bound (|q| + max |codeword|)^2 >= every entry
// so that all entries stay below 32768; lookups are accumulated in FP32 and the
// sum is multiplied by 2^-e. Entries are non-negative, so t >= t0 still holds and
// the threshold test before the lookups stays valid.
//
// Interleaved kernel (k_scan_il; nsq a multiple of 4, at most 32: every index
// the library builds for its configurations). The codes come from the interleaved
// copy (DeviceIndex::codes_il, pgpu_internal.h): record r's codes rotated by
// l = r & 31, its lane in a block of 32 records. Thread t of a round takes the
// records whose memory id is congruent to t mod 32, so every 8-byte code load of a
// warp reads one whole 256-byte line, and at lookup step s lane l reads table
// column s + l. The table holds, for each code c (a row) and each column
// m' < nsq + 31, the entry of subspace m' mod nsq at word c * 64 + m' (FP32) or
// half c * 64 + m' (FP16): the 32 lanes of a warp read 32 distinct banks at every
// lookup, whatever the codes (the reference's [subspace][code] table costs about
// 3.4 shared-memory wavefronts per warp-wide lookup of random codes). A lookup is
// one PRMT (the address (c << 8) | 4l from the code word and the lane), one load
// and one add. The sum runs in the rotated order: lookup step s goes to partial
// s mod 4, and t = t0 + ((a0 + a1) + (a2 + a3)), FP32 throughout; the oracle's
// scan mode restates that order (the reference's own order, partial m mod 4 over
// subspaces m, holds for the other kernel, k_scan_select). This kernel has no
// threshold test before the lookups: t0 lacks the table's |q|^2 share, so the test
// passes for almost every record. Loads are double-buffered: a round's records are
// fetched while the previous round is scored.
#include <cuda_fp16.h>

#include <type_traits>

#include "device_common.cuh"
#include "pgpu_internal.h"

namespace pgpu {
namespace {

// Block shape of the scan (compile-time; -D overrides for tuning sweeps).
#ifndef PGPU_SCAN_THREADS
#define PGPU_SCAN_THREADS 256
#endif
#ifndef PGPU_SCAN_RECORDS
#define PGPU_SCAN_RECORDS 4
#endif
#ifndef PGPU_SCAN_MIN_BLOCKS
#define PGPU_SCAN_MIN_BLOCKS 3
#endif
constexpr int kThreads = PGPU_SCAN_THREADS;
constexpr int kRecPerThread = PGPU_SCAN_RECORDS;
constexpr int kRound = kThreads * kRecPerThread;  // records per round
// Candidate buffer: at most kMaxCap keys (kCapPer per thread in the compaction);
// sized per launch from filter_topk (scan_cap).
constexpr int kCapPer = 16;
constexpr uint32_t kMaxCap = kThreads * kCapPer;
constexpr uint32_t kHistBins = 1024;  // bins of the cut-back histogram
static_assert(kHistBins % kThreads == 0, "bins split evenly over the threads");

// Buffer size for filter_topk T: T + a round + room for max(1024, T) more keys
// before the next cut, in whole multiples of the block, at most kMaxCap.
__host__ __device__ inline uint32_t scan_cap(uint32_t T) {
    uint32_t room = T > 1024 ? T : 1024;
    uint32_t c = T + kRound + room;
    c = (c + kThreads - 1) / kThreads * kThreads;
    return c > kMaxCap ? kMaxCap : c;
}

struct ScanParams {
    const float* q;
    const float* qnorm;
    const int32_t* status;
    const float* cdist;
    const uint32_t* ctag;
    const float* fd_by_fine;  // [B][F]
    float* hdist;
    uint32_t* htag;
    uint32_t* hcnt;
    const float* stationary;  // [C][F]
    const uint32_t* cell_start;
    const uint16_t* rec_fine; // [n] fine id of each record
    const float* offsets;
    const uint8_t* codes;
    const uint8_t* codes_il;    // interleaved copy (k_scan_il)
    const float* codebook;
    unsigned long long* counters;
    const uint32_t* order;      // [B] query of each block
    int* err;                   // set when a bulk copy's wait expired
    const uint32_t* ins_cl_start;  // realtime: [C+1] inserted records per cluster, or null
    const uint32_t* ins_cl_ids;    // their memory ids
    const uint32_t* todo;          // k_scan_il: the queries the split scan left, or null (all, in order)
    const uint32_t* ntodo;         // their number (device)
    uint32_t n;
    uint32_t d, C, F, nsq, lsq, code_stride, P, T, cap;
    float codebook_max;
};

// Power-of-two scale of the FP16 table: 2^e with every entry * 2^e < 32768, from
// the bound (|q| + max |codeword|)^2 on |q_m - c|^2.
__device__ __forceinline__ int half_lut_exponent(float qnorm, float codebook_max) {
    const float qa = sqrtf(qnorm) + codebook_max;
    const float bound = qa * qa * 1.0001f + 1e-30f;
    int e = (int)floorf(log2f(32768.0f / bound));
    return e < -60 ? -60 : (e > 60 ? 60 : e);
}

// get_dist_table (quantization.cpp:260-270) for one query into shared memory:
// thread j computes codeword j of every subspace (one coalesced 16-byte codebook
// load per subspace when lsq = 4), in the reference's lane order (l2sqr_sse).
// Table variants: FP32 (the reference's values and order), FP16 in the same
// layout, FP16 in the rotated one-bank-per-subspace layout.
enum { kTabF32 = 0, kTabF16 = 1 };

template <int TAB>
__device__ __forceinline__ void build_table(void* lut, const float* qv,
                                            const float* __restrict__ cb, uint32_t nsq,
                                            uint32_t lsq, float scale) {
    for (uint32_t j = threadIdx.x; j < 256; j += kThreads) {
        auto store = [&](uint32_t m, float v) {
            if (TAB == kTabF16)
                reinterpret_cast<__half*>(lut)[m * 256 + j] = __float2half_rn(v * scale);
            else
                reinterpret_cast<float*>(lut)[m * 256 + j] = v;
        };
        if (lsq == 4) {
            const float4* cb4 = reinterpret_cast<const float4*>(cb);
            for (uint32_t m0 = 0; m0 < nsq; m0 += 8) {
                float4 y[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (m0 + u < nsq) y[u] = __ldg(cb4 + (uint64_t)(m0 + u) * 256 + j);
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t m = m0 + u;
                    if (m >= nsq) break;
                    const float* x = qv + m * 4;
                    const float t0 = __fsub_rn(x[0], y[u].x), t1 = __fsub_rn(x[1], y[u].y);
                    const float t2 = __fsub_rn(x[2], y[u].z), t3 = __fsub_rn(x[3], y[u].w);
                    store(m, __fadd_rn(__fadd_rn(__fmul_rn(t0, t0), __fmul_rn(t1, t1)),
                                       __fadd_rn(__fmul_rn(t2, t2), __fmul_rn(t3, t3))));
                }
            }
        } else {
            for (uint32_t m = 0; m < nsq; ++m)
                store(m, l2sqr_sse(qv + m * lsq, cb + ((uint64_t)m * 256 + j) * lsq, lsq));
        }
    }
}

template <int NW>
__device__ __forceinline__ float lut_sum_words_half(const uint32_t (&w)[NW], const __half* lut,
                                                    uint32_t nsq) {
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const uint32_t m = 4u * i;
        if (m >= nsq) break;
        const uint32_t c = w[i];
        a0 += __half2float(lut[(m + 0) * 256 + (c & 0xff)]);
        if (m + 1 < nsq) a1 += __half2float(lut[(m + 1) * 256 + ((c >> 8) & 0xff)]);
        if (m + 2 < nsq) a2 += __half2float(lut[(m + 2) * 256 + ((c >> 16) & 0xff)]);
        if (m + 3 < nsq) a3 += __half2float(lut[(m + 3) * 256 + (c >> 24)]);
    }
    return (a0 + a1) + (a2 + a3);
}

__device__ __forceinline__ float key_value(uint64_t k) {
    uint32_t b = (uint32_t)(k >> 32);
    b = (b & 0x80000000u) ? (b & 0x7fffffffu) : ~b;
    return __uint_as_float(b);
}

constexpr uint64_t kKeyMax = ~0ull;

// The K-th smallest (1-based) of keys[0..count), all distinct: MSB-first radix
// select with 8-bit digits, stopping as soon as the chosen digit's bucket holds
// one key (usually after the 2nd or 3rd digit of the float). `hist` has 256
// slots, `sel` 4. All threads call it.
template <int NT>
__device__ uint64_t block_select_kth(const uint64_t* keys, uint32_t count, uint32_t K,
                                     uint32_t* hist, uint64_t* sel) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the leading bits every key shares need no pass: start at the digit where the
    // smallest and the largest key first differ
    uint64_t lo = ~0ull, hi = 0;
    for (uint32_t i = tid; i < count; i += NT) {
        const uint64_t x = keys[i];
        lo = x < lo ? x : lo;
        hi = x > hi ? x : hi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t a = __shfl_xor_sync(0xffffffffu, lo, o);
        const uint64_t b = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    __shared__ uint64_t red_lo[NT / 32], red_hi[NT / 32];
    if (lane == 0) {
        red_lo[warp] = lo;
        red_hi[warp] = hi;
    }
    __syncthreads();
    lo = red_lo[0];
    hi = red_hi[0];
    for (int w = 1; w < NT / 32; ++w) {
        lo = red_lo[w] < lo ? red_lo[w] : lo;
        hi = red_hi[w] > hi ? red_hi[w] : hi;
    }
    __syncthreads();
    int top = 56;
    if (lo != hi) {
        const int msb = 63 - __clzll((long long)(lo ^ hi));
        top = (msb / 8) * 8;
    } else {
        top = 0;
    }
    uint64_t mask = top >= 56 ? 0ull : ~((1ull << (top + 8)) - 1);
    uint64_t prefix = lo & mask;
    uint32_t k = K;
    for (int shift = top; shift >= 0; shift -= 8) {
        for (int i = tid; i < 256; i += NT) hist[i] = 0;
        __syncthreads();
        for (uint32_t i0 = 0; i0 < count; i0 += NT) {
            const uint32_t i = i0 + tid;
            bool in = false;
            uint32_t digit = 0;
            if (i < count) {
                const uint64_t key = keys[i];
                in = (key & mask) == prefix;
                digit = (uint32_t)(key >> shift) & 255u;
            }
            // one atomic per distinct digit in the warp
            const unsigned active = __ballot_sync(0xffffffffu, in);
            if (in) {
                const unsigned same = __match_any_sync(active, digit);
                if (lane == __ffs(same) - 1) atomicAdd(&hist[digit], (uint32_t)__popc(same));
            }
        }
        __syncthreads();
        if (tid < 32) {
            // digit d with (count below d) < k <= (count up to d)
            uint32_t c[8], run = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                c[j] = hist[tid * 8 + j];
                run += c[j];
            }
            uint32_t incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            uint32_t below = incl - run;
            if (below < k && k <= incl) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (below < k && k <= below + c[j]) {
                        sel[0] = (uint64_t)(tid * 8 + j);
                        sel[1] = k - below;
                        sel[2] = c[j];
                    }
                    below += c[j];
                }
            }
        }
        __syncthreads();
        prefix |= sel[0] << shift;
        mask |= 255ull << shift;
        k = (uint32_t)sel[1];
        const bool unique = sel[2] == 1;
        __syncthreads();
        if (unique && shift > 0) {
            // the one key under this prefix is the K-th
            for (uint32_t i = tid; i < count; i += NT)
                if ((keys[i] & mask) == prefix) sel[3] = keys[i];
            __syncthreads();
            const uint64_t r = sel[3];
            __syncthreads();
            return r;
        }
    }
    return prefix;
}

// Cut-back bound of the buffer: keys[0..count) hold at least K keys. One pass
// of a kHistBins-bin histogram of the keys' float parts, linear between the
// smallest and the largest, finds the bin holding the K-th smallest; the result
// is the (exclusive) upper edge of that bin as a key: at least K keys lie below
// it, and only the keys of that one bin above the K-th are kept in excess.
// Returns kKeyMax when the float parts are all equal (no cut possible). `hist`
// has kHistBins slots, `red` 2 * (kThreads / 32) + 2. All threads call it.
template <int NT>
__device__ uint64_t block_cut_bound(const uint64_t* keys, uint32_t count, uint32_t K,
                                    uint32_t* hist, uint32_t* red) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kW = NT / 32;
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
    for (uint32_t i = tid; i < count; i += NT) {
        const uint32_t h = (uint32_t)(keys[i] >> 32);
        lo = h < lo ? h : lo;
        hi = h > hi ? h : hi;
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
        red[warp] = lo;
        red[kW + warp] = hi;
    }
    for (uint32_t b = tid; b < kHistBins; b += NT) hist[b] = 0;
    __syncthreads();
    lo = red[0];
    hi = red[kW];
#pragma unroll
    for (int w = 1; w < kW; ++w) {
        lo = red[w] < lo ? red[w] : lo;
        hi = red[kW + w] > hi ? red[kW + w] : hi;
    }
    if (lo == hi) {
        __syncthreads();
        return kKeyMax;
    }
    int shift = 0;
    while (((hi - lo) >> shift) >= kHistBins) ++shift;
    for (uint32_t i = tid; i < count; i += NT)
        atomicAdd(&hist[((uint32_t)(keys[i] >> 32) - lo) >> shift], 1u);
    __syncthreads();
    // thread t owns bins [t * per, (t + 1) * per): the bin where the running count reaches K
    constexpr uint32_t per = kHistBins / NT;
    uint32_t c[per], run = 0;
#pragma unroll
    for (uint32_t j = 0; j < per; ++j) {
        c[j] = hist[tid * per + j];
        run += c[j];
    }
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) red[warp] = incl;  // red's min/max were read before the histogram barrier
    __syncthreads();
    uint32_t below = incl - run;
    for (int w = 0; w < warp; ++w) below += red[w];
    if (below < K && K <= below + run) {
#pragma unroll
        for (uint32_t j = 0; j < per; ++j) {
            if (below < K && K <= below + c[j]) red[2 * kW + 1] = tid * per + j;
            below += c[j];
        }
    }
    __syncthreads();
    const uint32_t bin = red[2 * kW + 1];
    __syncthreads();
    const uint64_t edge = (uint64_t)lo + ((uint64_t)(bin + 1) << shift);
    return edge > 0xFFFFFFFFull ? kKeyMax : (edge << 32);
}

// The K-th smallest (1-based) of keys[0..count), all distinct, K <= count: one
// histogram pass of kHistBins linear bins over the keys' float parts (as
// block_cut_bound) finds the bin holding the K-th; the keys of that bin (at most
// kHistBins / 2 of them: `hist` then holds them as 64-bit keys) are ranked by
// counting, and the one of rank K - (keys below the bin) is the result. A bin
// holding more keys, or all float parts equal, goes to block_select_kth. `red` has
// 2 * (NT / 32) + 2 slots, `cnt` is a shared counter. All threads call it.
template <int NT>
__device__ uint64_t block_kth_hist(const uint64_t* keys, uint32_t count, uint32_t K, uint32_t* hist,
                                   uint32_t* red, uint32_t* cnt, uint32_t* hist256, uint64_t* sel) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kW = NT / 32;
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
    for (uint32_t i = tid; i < count; i += NT) {
        const uint32_t h = (uint32_t)(keys[i] >> 32);
        lo = h < lo ? h : lo;
        hi = h > hi ? h : hi;
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
        red[warp] = lo;
        red[kW + warp] = hi;
    }
    for (uint32_t b = tid; b < kHistBins; b += NT) hist[b] = 0;
    if (tid == 0) *cnt = 0;
    __syncthreads();
    lo = red[0];
    hi = red[kW];
#pragma unroll
    for (int w = 1; w < kW; ++w) {
        lo = red[w] < lo ? red[w] : lo;
        hi = red[kW + w] > hi ? red[kW + w] : hi;
    }
    if (lo == hi) {
        __syncthreads();
        return block_select_kth<NT>(keys, count, K, hist256, sel);
    }
    int shift = 0;
    while (((hi - lo) >> shift) >= kHistBins) ++shift;
    for (uint32_t i = tid; i < count; i += NT)
        atomicAdd(&hist[((uint32_t)(keys[i] >> 32) - lo) >> shift], 1u);
    __syncthreads();
    constexpr uint32_t per = kHistBins / NT;
    uint32_t c[per], run = 0;
#pragma unroll
    for (uint32_t j = 0; j < per; ++j) {
        c[j] = hist[tid * per + j];
        run += c[j];
    }
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) red[warp] = incl;
    __syncthreads();
    uint32_t below = incl - run;
    for (int w = 0; w < warp; ++w) below += red[w];
    if (below < K && K <= below + run) {
#pragma unroll
        for (uint32_t j = 0; j < per; ++j) {
            if (below < K && K <= below + c[j]) {
                red[2 * kW] = tid * per + j;  // the bin
                red[2 * kW + 1] = below;      // keys below it
                sel[0] = c[j];                // keys in it
            }
            below += c[j];
        }
    }
    __syncthreads();
    const uint32_t bin = red[2 * kW], nbelow = red[2 * kW + 1], m = (uint32_t)sel[0];
    if (m > kHistBins / 2) {
        __syncthreads();
        return block_select_kth<NT>(keys, count, K, hist256, sel);
    }
    // the bin's keys into hist (as 64-bit keys), then the one of rank K - nbelow
    uint64_t* bk = reinterpret_cast<uint64_t*>(hist);
    for (uint32_t i = tid; i < count; i += NT) {
        const uint64_t k = keys[i];
        if ((((uint32_t)(k >> 32) - lo) >> shift) == bin) bk[atomicAdd(cnt, 1u)] = k;
    }
    __syncthreads();
    const uint32_t want = K - nbelow - 1;  // 0-based rank in the bin
    for (uint32_t i = tid; i < m; i += NT) {
        const uint64_t k = bk[i];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < m; ++j) rank += bk[j] < k ? 1u : 0u;
        if (rank == want) sel[1] = k;
    }
    __syncthreads();
    const uint64_t r = sel[1];
    __syncthreads();
    return r;
}

// Keeps the keys < bound at the front (in arbitrary order); returns their count.
// `cnt` is a shared counter. All threads call it.
template <int NT, int PER = (int)(kMaxCap / NT)>
__device__ uint32_t block_compact_lt(uint64_t* keys, uint32_t count, uint64_t bound, uint32_t* cnt) {
    const int tid = threadIdx.x, lane = tid & 31;
    uint64_t mine[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t i = tid + j * NT;
        mine[j] = i < count ? keys[i] : ~0ull;
    }
    if (tid == 0) *cnt = 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const bool keep = mine[j] < bound;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        uint32_t base = 0;
        if (b) {
            if (lane == __ffs(b) - 1) base = atomicAdd(cnt, (uint32_t)__popc(b));
            base = __shfl_sync(0xffffffffu, base, __ffs(b) - 1);
        }
        if (keep) keys[base + __popc(b & ((1u << lane) - 1))] = mine[j];
    }
    __syncthreads();
    const uint32_t r = *cnt;
    __syncthreads();
    return r;
}

// Diagnostic counters (pgpu_walk_counters slots, summed per launch): 0 records
// evaluated, 1 records past the cell-distance test (table lookups), 2 records kept, 3 compactions, 5 max records of one query, and
// thread-0 clock cycles: 6 prologue (table, query), 7 whole block, 8 record
// rounds, 9 compactions, 10 final select + output.
enum { kScRecords = 0, kScLookups = 1, kScKept = 2, kScCompactions = 3, kScMaxRecords = 5, kScCycPrologue = 6,
       kScCycTotal = 7, kScCycRounds = 8, kScCycCompact = 9, kScCycFinal = 10 };

struct ScanState {
    uint64_t tau;
    uint64_t sel[4];
    uint32_t hist[256];
    uint32_t red[2 * (512 / 32) + 2];  // for blocks of up to 512 threads
    uint32_t ccount;
    uint32_t count;
    uint32_t c;
    float cdl;
    uint32_t r0, r1, i0, i1;
    unsigned long long evaluated, looked, passed;
    unsigned long long cyc_rounds, cyc_compact, n_compact, n_records;
};

// Slot l of query qi's probed clusters into st (all threads; barriers on both
// sides): false when the slot is empty (the probed clusters fill a prefix).
__device__ __forceinline__ bool scan_cluster_begin(const ScanParams& p, ScanState& st, uint32_t qi,
                                                   uint32_t l) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t c = p.ctag[(uint64_t)qi * p.P + l];
        st.c = c;
        st.cdl = p.cdist[(uint64_t)qi * p.P + l];
        st.i0 = st.i1 = 0;
        st.r0 = st.r1 = 0;
        if (c < p.C) {
            st.r0 = p.cell_start[(uint64_t)c * p.F];
            st.r1 = p.cell_start[(uint64_t)c * p.F + p.F];
            if (p.ins_cl_start) {
                st.i0 = p.ins_cl_start[c];
                st.i1 = p.ins_cl_start[c + 1];
            }
        }
    }
    __syncthreads();
    return st.c < p.C;
}

// srow[f] = 2 * cell_dist of cluster c's cell f, cell_dist = (cd + stationary) + fd
// (puck_index.cpp:539-540); all threads, barrier after.
__device__ __forceinline__ void scan_fill_srow(const ScanParams& p, float* srow, const float* fdk,
                                               uint32_t c, float cdl) {
    const uint32_t F = p.F;
    if ((F & 3u) == 0) {
        // 16-byte rows (F % 4 == 0): one float4 of each row per step
        const float4* st4 = reinterpret_cast<const float4*>(p.stationary + (uint64_t)c * F);
        const float4* fd4 = reinterpret_cast<const float4*>(fdk);
        float4* s4 = reinterpret_cast<float4*>(srow);
        for (uint32_t i = threadIdx.x; i < (F >> 2); i += blockDim.x) {
            const float4 a = __ldg(st4 + i), b = __ldg(fd4 + i);
            s4[i] = make_float4(2.0f * __fadd_rn(__fadd_rn(cdl, a.x), b.x),
                                2.0f * __fadd_rn(__fadd_rn(cdl, a.y), b.y),
                                2.0f * __fadd_rn(__fadd_rn(cdl, a.z), b.z),
                                2.0f * __fadd_rn(__fadd_rn(cdl, a.w), b.w));
        }
    } else {
        for (uint32_t i = threadIdx.x; i < F; i += blockDim.x)
            srow[i] = 2.0f * __fadd_rn(__fadd_rn(cdl, p.stationary[(uint64_t)c * F + i]), fdk[i]);
    }
    __syncthreads();
}

// Buffer insert of one round slot: the kept keys of the warp take consecutive
// slots (one shared atomic per warp). The capacity is kept >= count + a round by
// the cut in scan_after_round.
__device__ __forceinline__ void scan_insert(ScanState& st, uint64_t* keys, bool keep, uint64_t key,
                                            unsigned long long& my_pass) {
    const unsigned ballot = __ballot_sync(0xffffffffu, keep);
    if (ballot) {
        const int lane = threadIdx.x & 31;
        uint32_t base_slot = 0;
        if (lane == __ffs(ballot) - 1) base_slot = atomicAdd(&st.count, (uint32_t)__popc(ballot));
        base_slot = __shfl_sync(0xffffffffu, base_slot, __ffs(ballot) - 1);
        if (keep) {
            keys[base_slot + __popc(ballot & ((1u << lane) - 1))] = key;
            ++my_pass;
        }
    }
}

// After a round (all threads): cut the buffer back when it could not take another
// round of `round` keys. One histogram pass gives a bound with at least T keys below
// it (the final select is exact); tau = that bound. If the cut kept too many to take
// another round, cut exactly to T.
template <int NT>
__device__ __forceinline__ void scan_after_round(ScanState& st, uint64_t* keys, uint32_t* hist,
                                                 uint32_t cap, uint32_t round, uint32_t T,
                                                 uint64_t tau, long long t_round) {
    __syncthreads();
    const long long t_round_end = clock64();
    if (threadIdx.x == 0) st.cyc_rounds += (unsigned long long)(t_round_end - t_round);
    if (st.count > cap - round) {
        const uint32_t cnt = st.count;
        uint64_t bound = block_cut_bound<NT>(keys, cnt, T, hist, st.red);
        uint32_t kept = bound == kKeyMax ? cnt : block_compact_lt<NT>(keys, cnt, bound, &st.ccount);
        if (kept > cap - round) {
            const uint64_t kth = block_select_kth<NT>(keys, kept, T, st.hist, st.sel);
            bound = kth + 1;  // kth < kKeyMax: keys are distinct by id
            kept = block_compact_lt<NT>(keys, kept, bound, &st.ccount);
        }
        if (threadIdx.x == 0) {
            st.count = kept;
            st.tau = bound < tau ? bound : tau;
            st.n_compact += 1;
            st.cyc_compact += (unsigned long long)(clock64() - t_round_end);
        }
        __syncthreads();
    }
}

// The block's last steps: the exact T smallest keys of the buffer, written out
// unordered (only the rerank's tie path needs their (t, id) order, and it sorts
// them itself), and the diagnostic counters.
template <int NT>
__device__ void scan_finish(const ScanParams& p, ScanState& st, uint64_t* keys, uint32_t* hist,
                            uint32_t qi,
                            unsigned long long my_eval, unsigned long long my_look,
                            unsigned long long my_pass, long long t_start, long long t_pro) {
    const int tid = threadIdx.x;
    const uint32_t T = p.T;
    __syncthreads();
    const long long t_final = clock64();
    uint32_t count = st.count;
    if (count > T) {
        const uint64_t kth =
            block_kth_hist<NT>(keys, count, T, hist, st.red, &st.ccount, st.hist, st.sel);
        block_compact_lt<NT>(keys, count, kth + 1, &st.ccount);
        count = T;
    }
    const uint32_t out = count < T ? count : T;
    for (uint32_t i = tid; i < T; i += NT) {
        p.hdist[(uint64_t)qi * T + i] = i < out ? key_value(keys[i]) : sentinel_f();
        p.htag[(uint64_t)qi * T + i] = i < out ? (uint32_t)keys[i] : kNoLabel;
    }
    if (tid == 0) p.hcnt[qi] = out;
    if (p.counters) {
        // records evaluated / looked up / kept: summed over the block first, so each
        // counter takes one global atomic per block (the counters share one sector,
        // and atomics on it from every thread of the grid serialise in L2)
        const unsigned we = __reduce_add_sync(0xffffffffu, (unsigned)my_eval);
        const unsigned wl = __reduce_add_sync(0xffffffffu, (unsigned)my_look);
        const unsigned wp = __reduce_add_sync(0xffffffffu, (unsigned)my_pass);
        if ((tid & 31) == 0) {
            atomicAdd(&st.evaluated, (unsigned long long)we);
            atomicAdd(&st.looked, (unsigned long long)wl);
            atomicAdd(&st.passed, (unsigned long long)wp);
        }
        __syncthreads();
        if (tid == 0) {
            const long long t_end = clock64();
            atomicAdd(p.counters + kScRecords, st.evaluated);
            atomicAdd(p.counters + kScLookups, st.looked);
            atomicAdd(p.counters + kScKept, st.passed);
            atomicAdd(p.counters + kScCompactions, st.n_compact);
            atomicMax(p.counters + kScMaxRecords, st.n_records);
            atomicAdd(p.counters + kScCycPrologue, (unsigned long long)(t_pro - t_start));
            atomicAdd(p.counters + kScCycTotal, (unsigned long long)(t_end - t_start));
            atomicAdd(p.counters + kScCycRounds, st.cyc_rounds);
            atomicAdd(p.counters + kScCycCompact, st.cyc_compact);
            atomicAdd(p.counters + kScCycFinal, (unsigned long long)(t_end - t_final));
        }
    }
}

// Loads the NW code words of record `mr` (8-byte loads when the row stride allows).
template <int NW>
__device__ __forceinline__ void load_codes(const uint8_t* codes, uint32_t stride, uint32_t mr,
                                           uint32_t (&w)[NW]) {
    if ((NW & 1) == 0 && (stride & 7u) == 0) {
        const uint2* cw = reinterpret_cast<const uint2*>(codes + (uint64_t)mr * stride);
#pragma unroll
        for (int i = 0; i < NW / 2; ++i) {
            const uint2 v = __ldg(cw + i);
            w[2 * i] = v.x;
            w[2 * i + 1] = v.y;
        }
    } else {
        const uint32_t* cw = reinterpret_cast<const uint32_t*>(codes + (uint64_t)mr * stride);
#pragma unroll
        for (int i = 0; i < NW; ++i) w[i] = __ldg(cw + i);
    }
}

// NW = code words per record (code_stride / 4); TAB = table variant.
template <int NW, int TAB>
__global__ __launch_bounds__(kThreads, PGPU_SCAN_MIN_BLOCKS) void k_scan_select(ScanParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ ScanState st;
    const uint32_t qi = p.order[blockIdx.x];
    const int tid = threadIdx.x;
    const uint32_t nsq = p.nsq, F = p.F, T = p.T, cap = p.cap;
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem);  // [cap], first (8-byte aligned)
    uint32_t* hist = reinterpret_cast<uint32_t*>(keys + cap);  // [kHistBins]
    float* lut = reinterpret_cast<float*>(hist + kHistBins);
    __half* luth = reinterpret_cast<__half*>(lut);
    constexpr bool HALF = TAB != kTabF32;
    // [F] 2 * cell_dist of the current cluster's cells, after the table
    float* srow = HALF ? reinterpret_cast<float*>(luth + nsq * 256) : lut + nsq * 256;
    float* qv = srow + F;                  // [d]

    if (p.status[qi] != 0) {
        if (tid == 0) p.hcnt[qi] = 0;
        return;
    }
    const long long t_start = clock64();
    for (uint32_t i = tid; i < p.d; i += kThreads) qv[i] = p.q[(uint64_t)qi * p.d + i];
    const float* fdk = p.fd_by_fine + (uint64_t)qi * F;  // fine terms of this query
    if (tid == 0) {
        st.tau = kKeyMax;
        st.count = 0;
        st.evaluated = 0;
        st.looked = 0;
        st.passed = 0;
        st.cyc_rounds = st.cyc_compact = st.n_compact = st.n_records = 0;
    }
    const int lut_e = HALF ? half_lut_exponent(p.qnorm[qi], p.codebook_max) : 0;
    const float inv_scale = HALF ? ldexpf(1.0f, -lut_e) : 1.0f;
    __syncthreads();
    build_table<TAB>(lut, qv, p.codebook, nsq, p.lsq, HALF ? ldexpf(1.0f, lut_e) : 1.0f);
    unsigned long long my_eval = 0, my_look = 0, my_pass = 0;
    const long long t_pro = clock64();
    for (uint32_t l = 0; l < p.P; ++l) {
        // the probed clusters fill a prefix of the slots (the learned probe leaves the
        // rest empty): the first empty slot ends the walk
        if (!scan_cluster_begin(p, st, qi, l)) break;
        const uint32_t r0 = st.r0, i0 = st.i0;
        // the cluster's base records [r0, r1), then its inserted ones (realtime)
        const uint32_t nb = st.r1 - r0, nall = nb + (st.i1 - st.i0);
        if (nall == 0) continue;
        scan_fill_srow(p, srow, fdk, st.c, st.cdl);
        if (tid == 0) st.n_records += nall;
        for (uint32_t base = 0; base < nall; base += kRound) {
            const long long t_round = clock64();
            const uint64_t tau = st.tau;
            // all loads of the thread's records first, so their latencies overlap
            uint32_t fine_id[kRecPerThread];
            float off[kRecPerThread];
            uint32_t words[kRecPerThread][NW];
            uint32_t mem[kRecPerThread];
#pragma unroll
            for (int j = 0; j < kRecPerThread; ++j) {
                const uint32_t v = base + tid + j * kThreads;
                const uint32_t mr = v < nb ? r0 + v : (v < nall ? p.ins_cl_ids[i0 + v - nb] : r0);
                mem[j] = mr;
                fine_id[j] = p.rec_fine[mr];
                off[j] = p.offsets[mr];
                load_codes<NW>(p.codes, p.code_stride, mr, words[j]);
            }
#pragma unroll
            for (int j = 0; j < kRecPerThread; ++j) {
                const uint32_t mi = mem[j];
                bool keep = false;
                uint64_t key = 0;
                if (base + tid + j * kThreads < nall) {
                    // (float)(2.0 * cell_dist + offset): one float add of the exact
                    // 2 * cell_dist (see adc_base)
                    const float t0 = __fadd_rn(srow[fine_id[j]], off[j]);
                    ++my_eval;
                    if (filter_key(t0, mi) < tau) {  // t can only grow past t0
                        ++my_look;
                        float t;
                        if (TAB == kTabF16)
                            t = t0 + lut_sum_words_half<NW>(words[j], luth, nsq) * inv_scale;
                        else
                            t = __fadd_rn(t0, lut_sum_words<NW>(words[j], lut, nsq));
                        key = filter_key(t, mi);
                        keep = key < tau;
                    }
                }
                scan_insert(st, keys, keep, key, my_pass);
            }
            scan_after_round<kThreads>(st, keys, hist, cap, kRound, T, tau, t_round);
        }
    }
    scan_finish<kThreads>(p, st, keys, hist, qi, my_eval, my_look, my_pass, t_start, t_pro);
}

// ------------------------------------------------------------ interleaved kernel
// One block per query. A round is 2 * NT / 32 interleaved record blocks, 2 * NT
// records: thread t takes lane t & 31 of blocks t >> 5 and (t >> 5) + NT / 32, and
// scores the two records together. Rounds arrive in a ring of shared-memory slots
// by one bulk copy each (cp.async.bulk, completion on the slot's mbarrier), issued
// by thread 0 up to a ring's length ahead; the first copies go out before the
// table is built.
//   FP32 table (64 KB): 512 threads, 3 slots, one block per SM.
//   FP16 table (32 KB): 256 threads, 2 slots, two blocks per SM, so one block's
//   table build, cuts and final select overlap the other's rounds.
#ifndef PGPU_SCAN_IL_REC
#define PGPU_SCAN_IL_REC 2
#endif
#ifndef PGPU_SCAN_IL_STAGES32
#define PGPU_SCAN_IL_STAGES32 3
#endif
#ifndef PGPU_SCAN_IL_STAGES16
#define PGPU_SCAN_IL_STAGES16 2
#endif
constexpr int kIlRec = PGPU_SCAN_IL_REC;  // records per thread and round
template <bool HALF>
struct IlShape {
    static constexpr int kThreads = HALF ? 256 : 512;
    static constexpr int kStages = HALF ? PGPU_SCAN_IL_STAGES16 : PGPU_SCAN_IL_STAGES32;
    static constexpr int kMinBlocks = HALF ? 2 : 1;
    static constexpr uint32_t kBlocksPerRound = kThreads / 32 * kIlRec;
    static constexpr int kRound = kThreads * kIlRec;  // records per round
    static_assert(kMaxCap % kThreads == 0 && kHistBins % kThreads == 0, "helper shapes");
};
constexpr uint32_t kIlWaitLimit = 1u << 22;

// Buffer size of the interleaved kernel for filter_topk T (see scan_cap).
template <bool HALF>
__host__ __device__ inline uint32_t il_cap(uint32_t T) {
    constexpr uint32_t NT = IlShape<HALF>::kThreads;
    uint32_t room = T > 1024 ? T : 1024;
    uint32_t c = T + IlShape<HALF>::kRound + room;
    c = (c + NT - 1) / NT * NT;
    return c > kMaxCap ? kMaxCap : c;
}
__host__ __device__ constexpr uint32_t il_table_bytes(bool half) {
    return half ? 256u * 64u * 2u : 256u * 64u * 4u;
}
// Shared memory after the table: the query, the ring, then either the compact table
// being built ([nsq][257] floats) or the cluster's cell terms, the key buffer and the
// cut histogram.
__host__ __device__ inline uint32_t il_query_bytes(uint32_t d) { return (d * 4u + 15u) & ~15u; }
__host__ __device__ inline uint32_t il_srow_bytes(uint32_t F) { return (F * 4u + 7u) & ~7u; }
template <bool HALF>
__host__ __device__ inline uint32_t il_slot_bytes(uint32_t nsq) {
    return IlShape<HALF>::kBlocksPerRound * il_block_bytes(nsq);
}

// Bounded wait on a slot's mbarrier phase. A try_wait may suspend the thread for up
// to PGPU_SCAN_WAIT_HINT ns (0: no hint) while the copy is outstanding.
#ifndef PGPU_SCAN_WAIT_HINT
#define PGPU_SCAN_WAIT_HINT 0
#endif
__device__ __forceinline__ bool il_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < kIlWaitLimit; ++it) {
        uint32_t ok;
        if (PGPU_SCAN_WAIT_HINT > 0)
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
                "selp.b32 %0, 1, 0, p;\n}"
                : "=r"(ok)
                : "r"(bar), "r"(parity), "n"(PGPU_SCAN_WAIT_HINT)
                : "memory");
        else
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                "selp.b32 %0, 1, 0, p;\n}"
                : "=r"(ok)
                : "r"(bar), "r"(parity)
                : "memory");
        if (ok) return true;
    }
    return false;
}

// get_dist_table (quantization.cpp:260-270) of the query qv in the reference's lane
// order, staged as stage[m * 257 + j] (row pitch 257: the expansion reads it without
// bank conflicts), then expanded into the rotated table: column m' < NSQ + 31 of row
// c holds subspace m' mod NSQ (FP32), or the same scaled by 2^lut_e in FP16. Each
// codeword's subspaces go in two halves, a thread per half (NT = 512) or both halves
// by one thread (NT = 256). All NT threads; one barrier inside (after the staging),
// none after the expansion.
// il_load_half issues the codebook loads of a thread's first half (lsq 4), which need
// no query: the caller does so before it reads anything else.
template <int NSQ>
__device__ __forceinline__ void il_load_half(const float* __restrict__ codebook, uint32_t h2,
                                             float4 (&y)[NSQ / 2]) {
    const float4* cb4 =
        reinterpret_cast<const float4*>(codebook) + h2 * (NSQ / 2) * 256u + (threadIdx.x & 255u);
#pragma unroll
    for (int m = 0; m < NSQ / 2; ++m) y[m] = __ldg(cb4 + m * 256);
}
template <int NSQ>
__device__ __forceinline__ void il_stage_half(float* stage, const float* qv, uint32_t h2,
                                              const float4 (&y)[NSQ / 2]) {
    const float4* q4 = reinterpret_cast<const float4*>(qv) + h2 * (NSQ / 2);
    float* out = stage + h2 * (NSQ / 2) * 257u + (threadIdx.x & 255u);
#pragma unroll
    for (int m = 0; m < NSQ / 2; ++m) {
        const float4 x = q4[m];
        const float t0 = __fsub_rn(x.x, y[m].x), t1 = __fsub_rn(x.y, y[m].y);
        const float t2 = __fsub_rn(x.z, y[m].z), t3 = __fsub_rn(x.w, y[m].w);
        out[m * 257] = __fadd_rn(__fadd_rn(__fmul_rn(t0, t0), __fmul_rn(t1, t1)),
                                 __fadd_rn(__fmul_rn(t2, t2), __fmul_rn(t3, t3)));
    }
}

template <int NSQ, bool HALF, int NT, bool WIDE = false>
__device__ __forceinline__ void il_build_table(unsigned char* tab, float* stage, const float* qv,
                                               const float* __restrict__ codebook, uint32_t lsq,
                                               int lut_e, float4 (&y)[NSQ / 2]) {
    static_assert(NT % 256 == 0, "a thread per codeword and half");
    const int tid = threadIdx.x;
    if (lsq == 4) {
        if (NT == 256) {
            float4 z[NSQ / 2];
            il_load_half<NSQ>(codebook, 1, z);
            il_stage_half<NSQ>(stage, qv, 0, y);
            il_stage_half<NSQ>(stage, qv, 1, z);
        } else {
            il_stage_half<NSQ>(stage, qv, tid >> 8, y);
        }
    } else {
        for (uint32_t h2 = tid >> 8; h2 < 2; h2 += NT / 256) {
            const uint32_t j = tid & 255u;
            const int mh = (int)h2 * (NSQ / 2);
            for (int m = mh; m < mh + NSQ / 2; ++m)
                stage[m * 257 + j] =
                    l2sqr_sse(qv + m * lsq, codebook + ((uint64_t)m * 256 + j) * lsq, lsq);
        }
    }
    __syncthreads();
    // a thread keeps its columns and walks down the rows: one load and one store per entry
    // (columns past NSQ + 30 are never read)
    const float scale = HALF ? ldexpf(1.0f, lut_e) : 1.0f;
    if (HALF && !WIDE) {
        const uint32_t m0 = (tid & 31) * 2;
        if (m0 < NSQ + 31) {
            const float* s0 = stage + (m0 % NSQ) * 257;
            const float* s1 = stage + ((m0 + 1) % NSQ) * 257;
            uint32_t* tw = reinterpret_cast<uint32_t*>(tab) + (tid & 31);
#pragma unroll 8
            for (uint32_t c = tid >> 5; c < 256; c += NT / 32) {
                const __half2 h = __halves2half2(__float2half_rn(s0[c] * scale),
                                                 __float2half_rn(s1[c] * scale));
                tw[c * 32] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
    } else {
        const uint32_t m = tid & 63;
        if (m < NSQ + 31) {
            const float* src = stage + (m % NSQ) * 257;
            uint32_t* tw = reinterpret_cast<uint32_t*>(tab) + m;
#pragma unroll 8
            for (uint32_t c = tid >> 6; c < 256; c += NT / 64)
                // WIDE: each FP16 entry in its own 4-byte slot (the FP32 table's addresses)
                tw[c * 64] = HALF ? (uint32_t)__half_as_ushort(__float2half_rn(src[c] * scale))
                                  : __float_as_uint(src[c]);
        }
    }
}

// t of R records (memory ids mr, lanes mr & 31) from their codes (8-byte granules
// of the rotated layout), offsets and fine ids, with srow[f] = 2 * cell_dist of the
// record's cell; the R lookup chains are interleaved. Lookup step s goes to partial
// s mod 4 in FP32; t = (srow[f] + offset) + ((a0 + a1) + (a2 + a3)) (the FP16 table's
// sum scaled back by inv_scale).
template <int NSQ, bool HALF, int R, bool WIDE = false>
__device__ __forceinline__ void il_score(const unsigned char* tab, const float* srow,
                                         const uint2 (&gr)[R][(NSQ + 7) / 8], const float (&off)[R],
                                         const uint32_t (&fine)[R], const uint32_t (&mr)[R],
                                         float inv_scale, float (&t)[R]) {
    float a[R][4];
    uint32_t lb[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
        lb[j] = (mr[j] & 31u) << 2;  // byte 0 of the table address
        a[j][0] = a[j][1] = a[j][2] = a[j][3] = 0.0f;
    }
#pragma unroll
    for (int s2 = 0; s2 < NSQ; ++s2) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t w = (s2 & 4) ? gr[j][s2 >> 3].y : gr[j][s2 >> 3].x;
            // (code << 8) | 4 * lane: the entry of column s2 + lane
            const uint32_t addr = __byte_perm(w, lb[j], 0x5504u | ((uint32_t)(s2 & 3) << 4));
            if (HALF) {
                // compact table: 2-byte entries (one shift); WIDE: one entry per 4-byte slot
                const unsigned short h =
                    WIDE ? *reinterpret_cast<const unsigned short*>(tab + addr + 4 * s2)
                         : *reinterpret_cast<const unsigned short*>(tab + (addr >> 1) + 2 * s2);
                asm("add.f32.f16 %0, %1, %0;" : "+f"(a[j][s2 & 3]) : "h"(h));
            } else {
                // the first four entries start the sums: an entry is never -0, so 0 + x is x
                const float x = *reinterpret_cast<const float*>(tab + addr + 4 * s2);
                a[j][s2 & 3] = s2 < 4 ? x : __fadd_rn(a[j][s2 & 3], x);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const float t0 = __fadd_rn(srow[fine[j]], off[j]);  // (float)(2.0 * cell_dist + offset)
        const float sum = __fadd_rn(__fadd_rn(a[j][0], a[j][1]), __fadd_rn(a[j][2], a[j][3]));
        t[j] = HALF ? t0 + sum * inv_scale : __fadd_rn(t0, sum);
    }
}

template <int NSQ, bool HALF>
__global__ __launch_bounds__(IlShape<HALF>::kThreads, IlShape<HALF>::kMinBlocks) void k_scan_il(
    ScanParams p) {
    constexpr int kIlThreads = IlShape<HALF>::kThreads;
    constexpr int kIlStages = IlShape<HALF>::kStages;
    constexpr uint32_t kIlBlocksPerRound = IlShape<HALF>::kBlocksPerRound;
    constexpr int kIlRound = IlShape<HALF>::kRound;
    static_assert(NSQ % 4 == 0 && NSQ <= 32, "interleaved layout: nsq a multiple of 4, <= 32");
    constexpr int NG = (NSQ + 7) / 8;  // 8-byte code granules per record
    constexpr uint32_t kG = NG * 8;
    constexpr uint32_t kBlk = 32 * kG + 192;  // il_block_bytes
    constexpr uint32_t kSlot = kIlBlocksPerRound * kBlk;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ ScanState st;
    __shared__ __align__(8) uint64_t full[kIlStages];
    __shared__ int il_failed;
    const int tid = threadIdx.x;
    const uint32_t F = p.F, T = p.T, cap = p.cap;
    unsigned char* tab = smem;  // the rotated table, at offset 0
    float* qv = reinterpret_cast<float*>(smem + il_table_bytes(HALF));
    unsigned char* ring = smem + il_table_bytes(HALF) + il_query_bytes(p.d);  // [kIlStages][kSlot]
    unsigned char* rest = ring + kIlStages * kSlot;
    float* stage = reinterpret_cast<float*>(rest);  // [NSQ][257] while the table is built
    float* srow = reinterpret_cast<float*>(rest);   // [F] afterwards
    uint64_t* keys = reinterpret_cast<uint64_t*>(rest + il_srow_bytes(F));  // [cap]
    uint32_t* hist = reinterpret_cast<uint32_t*>(keys + cap);              // [kHistBins]

    // rounds issued and consumed over all the block's queries (slot g % S, parity (g / S) & 1)
    uint32_t g_issued = 0, g_done = 0;
    auto bar_of = [&](uint32_t g) { return (uint32_t)__cvta_generic_to_shared(&full[g % kIlStages]); };
    // thread 0: bulk copy of record blocks [blk0, blk0 + nblk) into round g's slot
    auto issue = [&](uint32_t g, uint64_t blk0, uint32_t nblk) {
        const uint32_t bar = bar_of(g);
        const uint32_t bytes = nblk * kBlk;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + (g % kIlStages) * kSlot);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
                "r"(dst),
            "l"(p.codes_il + blk0 * kBlk), "r"(bytes), "r"(bar)
            : "memory");
    };
    if (tid == 0) {
        for (int i = 0; i < kIlStages; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_of(i)), "r"(1u));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        il_failed = 0;
    }
    const uint32_t nq = p.todo ? *p.ntodo : p.n;
    for (uint32_t qb = blockIdx.x; qb < nq; qb += gridDim.x) {
        const uint32_t qi = p.todo ? p.todo[qb] : p.order[qb];
        if (p.status[qi] != 0) {
            if (tid == 0) p.hcnt[qi] = 0;
            continue;
        }
        const long long t_start = clock64();
        __syncthreads();  // the previous query's buffers are no longer read
        if (tid == 0) {
            st.tau = kKeyMax;
            st.count = 0;
            st.evaluated = st.looked = st.passed = 0;
            st.cyc_rounds = st.cyc_compact = st.n_compact = st.n_records = 0;
        }
        // the first cluster's first rounds go out before the table is built
        uint32_t primed_blk0 = 0, primed_blocks = 0;
        if (tid == 0) {
            const uint32_t c = p.ctag[(uint64_t)qi * p.P];
            if (c < p.C) {
                const uint32_t r0 = p.cell_start[(uint64_t)c * F], r1 = p.cell_start[(uint64_t)c * F + F];
                if (r1 > r0) {
                    const uint32_t b0 = r0 >> 5, nblk = ((r1 - 1) >> 5) - b0 + 1;
                    primed_blk0 = b0;
                    for (uint32_t k = 0; k < (uint32_t)kIlStages && k * kIlBlocksPerRound < nblk; ++k) {
                        const uint32_t m = min(kIlBlocksPerRound, nblk - k * kIlBlocksPerRound);
                        issue(g_issued++, (uint64_t)b0 + k * kIlBlocksPerRound, m);
                        primed_blocks += m;
                    }
                }
            }
        }
        for (uint32_t i = tid; i < p.d; i += kIlThreads) qv[i] = p.q[(uint64_t)qi * p.d + i];
        const float* fdk = p.fd_by_fine + (uint64_t)qi * F;
        // the first cluster's stationary row and this query's fine terms are loaded now,
        // so their latency overlaps the table build (srow is written after it)
        constexpr int kPre = 2;  // float4 per thread and row (F <= kPre * 4 * kIlThreads)
        const uint32_t c_first = p.ctag[(uint64_t)qi * p.P];
        const bool pre = c_first < p.C && (F & 3u) == 0 && F <= kPre * 4 * kIlThreads;
        float4 pre_st[kPre], pre_fd[kPre];
    #pragma unroll
        for (int u = 0; u < kPre; ++u) {
            const uint32_t i = tid + u * kIlThreads;
            if (pre && i < (F >> 2)) {
                pre_st[u] = __ldg(reinterpret_cast<const float4*>(p.stationary + (uint64_t)c_first * F) + i);
                pre_fd[u] = __ldg(reinterpret_cast<const float4*>(fdk) + i);
            }
        }
        const int lut_e = HALF ? half_lut_exponent(p.qnorm[qi], p.codebook_max) : 0;
        const float inv_scale = HALF ? ldexpf(1.0f, -lut_e) : 1.0f;
        float4 y[NSQ / 2];
        if (p.lsq == 4) il_load_half<NSQ>(p.codebook, tid >> 8, y);
        __syncthreads();
        il_build_table<NSQ, HALF, kIlThreads>(tab, stage, qv, p.codebook, p.lsq, lut_e, y);
        unsigned long long my_eval = 0, my_pass = 0;
        const long long t_pro = clock64();

        auto score_records = [&](const uint2 (&gr)[kIlRec][NG], const float (&off)[kIlRec],
                                 const uint32_t (&fine)[kIlRec], const uint32_t (&mr)[kIlRec],
                                 float (&t)[kIlRec]) {
            il_score<NSQ, HALF, kIlRec>(tab, srow, gr, off, fine, mr, inv_scale, t);
        };

        for (uint32_t l = 0; l < p.P && !il_failed; ++l) {
            if (!scan_cluster_begin(p, st, qi, l)) break;  // (its first barrier ends the table)
            const uint32_t r0 = st.r0, r1 = st.r1, i0 = st.i0, ni = st.i1 - st.i0;
            if (r1 - r0 + ni == 0) continue;
            if (tid == 0) st.n_records += r1 - r0 + ni;
            if (l == 0 && pre) {
                // srow from the rows loaded before the table build
                const float cdl = st.cdl;
                float4* s4 = reinterpret_cast<float4*>(srow);
    #pragma unroll
                for (int u = 0; u < kPre; ++u) {
                    const uint32_t i = tid + u * kIlThreads;
                    if (i < (F >> 2)) {
                        const float4 a = pre_st[u], b = pre_fd[u];
                        s4[i] = make_float4(2.0f * __fadd_rn(__fadd_rn(cdl, a.x), b.x),
                                            2.0f * __fadd_rn(__fadd_rn(cdl, a.y), b.y),
                                            2.0f * __fadd_rn(__fadd_rn(cdl, a.z), b.z),
                                            2.0f * __fadd_rn(__fadd_rn(cdl, a.w), b.w));
                    }
                }
                __syncthreads();
            } else {
                scan_fill_srow(p, srow, fdk, st.c, st.cdl);
            }
            uint32_t b0 = 0, nblk = 0, rounds = 0;
            if (r1 > r0) {
                b0 = r0 >> 5;
                nblk = ((r1 - 1) >> 5) - b0 + 1;
                rounds = (nblk + kIlBlocksPerRound - 1) / kIlBlocksPerRound;
            }
            // rounds of this cluster already in flight (the first cluster's, primed)
            uint32_t sent = (l == 0 && primed_blocks > 0 && primed_blk0 == b0)
                                ? (primed_blocks + kIlBlocksPerRound - 1) / kIlBlocksPerRound
                                : 0;
            if (tid == 0) {
                for (; sent < rounds && sent < (uint32_t)kIlStages; ++sent)
                    issue(g_issued++, (uint64_t)b0 + sent * kIlBlocksPerRound,
                          min(kIlBlocksPerRound, nblk - sent * kIlBlocksPerRound));
            }
            sent = rounds < (uint32_t)kIlStages ? rounds : (uint32_t)kIlStages;
            g_issued = g_done + sent;  // every thread tracks the count thread 0 issued
            const uint32_t blk = tid >> 5, lane = tid & 31;
            for (uint32_t k = 0; k < rounds; ++k) {
                const long long t_round = clock64();
                const uint64_t tau = st.tau;
                // tau as (float, id): key(t, id) < tau iff t < tau_f, or t == tau_f and
                // id < tau_id (float compares treat -0 as +0, as the keys do; a bound
                // whose float part is the key of -0 keeps exactly the t < 0)
                float tau_f = tau == kKeyMax ? __int_as_float(0x7f800000) : key_value(tau);
                uint32_t tau_id = tau == kKeyMax ? 0xFFFFFFFFu : (uint32_t)tau;
                if ((uint32_t)(tau >> 32) == 0x7FFFFFFFu) {
                    tau_f = 0.0f;
                    tau_id = 0;
                }
                const uint32_t g = g_done;
                if (!il_wait(bar_of(g), (g / kIlStages) & 1u)) {
                    if (lane == 0) atomicExch(&il_failed, 1);
                }
                uint2 gr[kIlRec][NG];
                float off[kIlRec], t[kIlRec];
                uint32_t fine[kIlRec], rr[kIlRec];
                bool valid[kIlRec];
    #pragma unroll
                for (int j = 0; j < kIlRec; ++j) {
                    const uint32_t bl = blk + j * (kIlThreads / 32);  // block of the round
                    const uint64_t bk = (uint64_t)b0 + k * kIlBlocksPerRound + bl;
                    rr[j] = (uint32_t)(bk * 32 + lane);
                    valid[j] = bk < (uint64_t)b0 + nblk && rr[j] >= r0 && rr[j] < r1 && !il_failed;
                    // out-of-range slots read stale bytes of the slot and are dropped below
                    const unsigned char* rec = ring + (g % kIlStages) * kSlot + bl * kBlk;
    #pragma unroll
                    for (int q2 = 0; q2 < NG; ++q2)
                        gr[j][q2] = *reinterpret_cast<const uint2*>(rec + q2 * 256 + 8 * lane);
                    off[j] = *reinterpret_cast<const float*>(rec + 32 * kG + 4 * lane);
                    fine[j] = valid[j] ? *reinterpret_cast<const uint16_t*>(rec + 32 * kG + 128 + 2 * lane)
                                       : 0u;
                }
                score_records(gr, off, fine, rr, t);
    #pragma unroll
                for (int j = 0; j < kIlRec; ++j) {
                    // key(t, id) < tau by float compares; the key only for kept records
                    const bool keep =
                        valid[j] && (t[j] < tau_f || (t[j] == tau_f && rr[j] < tau_id));
                    my_eval += valid[j] ? 1 : 0;
                    scan_insert(st, keys, keep, keep ? filter_key(t[j], rr[j]) : 0ull, my_pass);
                }
                scan_after_round<kIlThreads>(st, keys, hist, cap, kIlRound, T, tau, t_round);
                if (il_failed) break;  // read after the barrier: the same on every thread
                ++g_done;
                // the slot of round g is free: thread 0 refills it with round k + kIlStages
                const uint32_t kn = k + kIlStages;
                if (kn < rounds) {
                    if (tid == 0)
                        issue(g_issued, (uint64_t)b0 + kn * kIlBlocksPerRound,
                              min(kIlBlocksPerRound, nblk - kn * kIlBlocksPerRound));
                    ++g_issued;
                }
            }
            // realtime: the cluster's inserted records, read from the interleaved copy
            for (uint32_t v0 = 0; v0 < ni; v0 += kIlRound) {
                const long long t_round = clock64();
                const uint64_t tau = st.tau;
                uint2 gr[kIlRec][NG];
                float off[kIlRec], t[kIlRec];
                uint32_t fine[kIlRec], mr[kIlRec];
                bool valid[kIlRec];
    #pragma unroll
                for (int j = 0; j < kIlRec; ++j) {
                    const uint32_t v = v0 + tid + j * kIlThreads;
                    valid[j] = v < ni;
                    mr[j] = valid[j] ? p.ins_cl_ids[i0 + v] : 0u;
    #pragma unroll
                    for (int q2 = 0; q2 < NG; ++q2)
                        gr[j][q2] = __ldg(reinterpret_cast<const uint2*>(
                            p.codes_il + il_granule_offset(mr[j], q2, NSQ)));
                    off[j] = __ldg(reinterpret_cast<const float*>(p.codes_il + il_offset_offset(mr[j], NSQ)));
                    fine[j] = __ldg(reinterpret_cast<const uint16_t*>(p.codes_il + il_fine_offset(mr[j], NSQ)));
                }
                score_records(gr, off, fine, mr, t);
    #pragma unroll
                for (int j = 0; j < kIlRec; ++j) {
                    const uint64_t key = filter_key(t[j], mr[j]);
                    const bool keep = valid[j] && key < tau;
                    my_eval += valid[j] ? 1 : 0;
                    scan_insert(st, keys, keep, key, my_pass);
                }
                scan_after_round<kIlThreads>(st, keys, hist, cap, kIlRound, T, tau, t_round);
            }
        }
        if (il_failed) {
            // a copy did not arrive in time: wait (bounded) for every copy issued, so
            // none lands in shared memory after the block, and report this query and
            // the block's later ones as empty (the rerank reads every count)
            for (uint32_t g = g_done; g < g_issued; ++g) il_wait(bar_of(g), (g / kIlStages) & 1u);
            __syncthreads();
            for (uint64_t i = qb + (uint64_t)tid * gridDim.x; i < nq; i += (uint64_t)kIlThreads * gridDim.x)
                p.hcnt[p.todo ? p.todo[i] : p.order[i]] = 0;
            if (tid == 0) atomicExch(p.err, 1);
            return;
        }
        scan_finish<kIlThreads>(p, st, keys, hist, qi, my_eval, my_eval, my_pass, t_start, t_pro);
    }
}

// Launch order of the scan's blocks. A block's time follows the records of the
// clusters its query probes, and blocks start in index order: queries sorted by
// descending record count start the longest scans first and end the grid with the
// shortest, so fewer SMs sit idle at the tail. The sort is by bucket (4 steps per
// octave of the count), which is all that needs; within a bucket by the first probed
// cluster, in kOrderGroups groups of clusters, so that queries of one cluster run at
// about the same time and find its records, and the rerank its vectors, in L2. The
// results do not depend on it.
constexpr uint32_t kOrderBuckets = 132, kOrderGroups = 62;
constexpr uint32_t kOrderBins = kOrderBuckets * kOrderGroups;
constexpr int kOrderThreads = 1024;
constexpr uint32_t kOrderPer = (kOrderBins + kOrderThreads - 1) / kOrderThreads;
__device__ __forceinline__ uint32_t work_bucket(uint32_t w) {
    if (w == 0) return kOrderBuckets - 1;  // nothing to scan: last
    const int e = 31 - __clz(w);
    const uint32_t frac = e >= 2 ? (w >> (e - 2)) & 3u : (w << (2 - e)) & 3u;
    return (kOrderBuckets - 2) - ((uint32_t)e * 4 + frac);  // more records: earlier
}

// One thread per query: its record count over the probed clusters, as a bin.
__global__ void k_scan_work(const uint32_t* __restrict__ ctag, const int32_t* __restrict__ status,
                            const uint32_t* __restrict__ cell_start,
                            const uint32_t* __restrict__ ins_cl_start, uint32_t n, uint32_t P,
                            uint32_t C, uint32_t F, uint16_t* __restrict__ wbin) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    uint32_t w = 0, first = 0;
    if (status[q] == 0) {
        for (uint32_t l = 0; l < P; ++l) {
            const uint32_t c = ctag[(uint64_t)q * P + l];
            if (c >= C) break;  // the probed clusters fill a prefix of the slots
            if (l == 0) first = (uint32_t)((uint64_t)c * kOrderGroups / C);
            w += cell_start[(uint64_t)c * F + F] - cell_start[(uint64_t)c * F];
            if (ins_cl_start) w += ins_cl_start[c + 1] - ins_cl_start[c];
        }
    }
    wbin[q] = (uint16_t)(work_bucket(w) * kOrderGroups + first);
}

// One block: counting sort of the queries by bin (order within a bin is free). The
// count of queries left to the fused scan starts at 0.
__global__ __launch_bounds__(kOrderThreads) void k_scan_order(const uint16_t* __restrict__ wbin,
                                                              uint32_t n, uint32_t* __restrict__ order,
                                                              uint32_t* __restrict__ ntodo) {
    __shared__ uint32_t hist[kOrderPer * kOrderThreads];
    __shared__ uint32_t wsum[kOrderThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) *ntodo = 0;
    for (uint32_t i = tid; i < kOrderPer * kOrderThreads; i += kOrderThreads) hist[i] = 0;
    __syncthreads();
    for (uint32_t q = tid; q < n; q += kOrderThreads) atomicAdd(&hist[wbin[q]], 1u);
    __syncthreads();
    uint32_t c[kOrderPer], run = 0;
#pragma unroll
    for (uint32_t j = 0; j < kOrderPer; ++j) {
        c[j] = hist[tid * kOrderPer + j];
        run += c[j];
    }
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t at = incl - run;
    for (int w = 0; w < warp; ++w) at += wsum[w];
#pragma unroll
    for (uint32_t j = 0; j < kOrderPer; ++j) {
        hist[tid * kOrderPer + j] = at;
        at += c[j];
    }
    __syncthreads();
    for (uint32_t q = tid; q < n; q += kOrderThreads) order[atomicAdd(&hist[wbin[q]], 1u)] = q;
}

// ------------------------------------------------------------ split scan
// The interleaved layout's scan. One block per query (k_scan_score), two blocks per SM:
//   1. the probed clusters' record ranges and the table (il_build_table);
//   2. a bound on the T-th smallest distance, when the query has more records than the
//      key buffer takes: the r-th smallest t of S records at evenly spaced positions,
//      r far enough above its expectation S T / N that fewer than T records at or below
//      it are improbable (sample_rank);
//   3. records, with no barrier: the clusters go through in groups whose cell terms fit
//      shared memory together; each warp streams its own record blocks of the group
//      straight from the interleaved copy (coalesced 8-byte loads, the next step's loads
//      in flight while the current one is scored, the same il_score arithmetic as
//      k_scan_il) and appends the (t, id) keys at or below the bound to the buffer, one
//      shared atomic per warp and step;
//   4. the exact T smallest keys of the buffer, written unordered: the same set as
//      k_scan_il's, since every record left out lies above T others.
// A query whose buffer overflowed, or got fewer than T keys, goes to k_scan_il's list:
// the bound only decides who answers. The FP16 table (precision form) keeps one entry
// per 4-byte slot, the FP32 table's addresses: a lookup is the same PRMT, load and add
// (the compact 2-byte layout costs a shift per lookup, and its smaller footprint buys
// nothing here).
//
// Bound by the shared-memory pipe and by issue: per record 24 (nsq) lookups of three
// instructions and one 128-byte wavefront each (36 cycles per 32 records measured with
// nothing else, 1.05 ms for the batch below). With two blocks per SM one block's table
// and bound overlap the other's records only in part (a block alone does not fill the
// SM): of a block's 50k SM cycles, in 10k queries over 28.8k records of 24 codes each,
// 33k are the records'. That batch takes 1.63 ms; 2.09 with every distance written out,
// binned and read back, and 25 us more for the record counts and the fused kernel's idle
// blocks.
#ifndef PGPU_SPLIT_REC
#define PGPU_SPLIT_REC 4
#endif
constexpr int kSplitThreads = 256;
constexpr int kSplitWarps = kSplitThreads / 32;
constexpr int kSplitRec = PGPU_SPLIT_REC;    // record blocks per warp and step (il_bytes)
static_assert(kSplitRec <= 4, "il_bytes has room for steps of 4 blocks");
constexpr uint32_t kSplitMaxSlots = 512;     // probed clusters a split query may have

__host__ __device__ inline SplitLayout split_layout(uint32_t nsq, uint32_t d, uint32_t F, uint32_t P,
                                                    uint32_t budget, uint32_t rows) {
    SplitLayout y;
    const uint32_t maxl = P < kSplitMaxSlots ? P : kSplitMaxSlots;
    y.slots = il_table_bytes(false) + il_query_bytes(d);
    y.rows_per = (F + 3u) & ~3u;
    y.group = rows / y.rows_per;
    y.group = y.group < 1 ? 1 : (y.group > maxl ? maxl : y.group);
    y.srow = y.slots + (6u * 4u * (maxl + 1) + 15u) / 16u * 16u;
    y.keys = y.srow + y.group * y.rows_per * 4u;
    const uint32_t stage = (nsq * 257u * 4u + 7u) & ~7u;
    const uint32_t room = budget > y.keys ? budget - y.keys : 0u;
    y.cap = room / 8u;
    y.bytes = room >= stage ? y.keys + y.cap * 8u : 0u;
    return y;
}
// Two blocks per SM when the buffer then takes T keys one and a half times over, else one.
// rows: floats of cell terms that a group of clusters may take (one cluster's at least). A block
// alone on its SM has room for more; with one cluster per group its eight warps wait for each
// cluster's terms in turn: 2000 queries over 300 clusters of 200 records and 4096 fine ids
// took 8.67 ms (8.28 with two blocks and every distance in memory), 6.83 with six clusters to a
// group, 7.22 with four. The buffer keeps room for four times T: at T = 2000 more rows than
// 16384 leave too few keys (500 clusters of 1000 records: 8.50 ms, 9.59 with 24576).
// Either way the buffer has to take the first sampled keys and their select's histogram.
constexpr uint32_t kSplitBudget2 = 111 * 1024, kSplitBudget1 = 220 * 1024;
constexpr uint32_t kSplitLeast = kSplitSampleStep + kSplitHistKeys;
constexpr uint32_t kSplitRows2 = 4096, kSplitRows1[] = {24576, 16384, kSplitRows2};
static uint32_t split_need(uint32_t T) {
    const uint32_t n = T + T / 2 + 512;
    return n > kSplitLeast ? n : kSplitLeast;
}

struct SplitParams {
    const uint32_t* ctag;
    const float* cdist;
    const int32_t* status;
    const uint32_t* cell_start;
    const uint32_t* ins_cl_start;  // realtime: [C+1], or null
    const uint32_t* ins_cl_ids;
    const float* stationary;
    const float* fd_by_fine;
    const float* q;
    const float* qnorm;
    const float* codebook;
    const uint8_t* codes_il;
    const uint32_t* order;
    uint32_t* todo;                // queries left to k_scan_il, and their number
    uint32_t* ntodo;
    float* hdist;
    uint32_t* htag;
    uint32_t* hcnt;
    unsigned long long* counters;
    uint32_t n, d, C, F, lsq, P, T;
    float codebook_max;
    SplitLayout lay;
};

template <int NSQ, bool HALF>
__global__ __launch_bounds__(kSplitThreads, 2) void k_scan_score(const __grid_constant__ SplitParams sp) {
    constexpr int NG = (NSQ + 7) / 8;  // 8-byte code granules per record
    constexpr uint32_t kG = NG * 8;
    constexpr uint32_t kBlk = 32 * kG + 192;  // il_block_bytes
    constexpr int NW = kSplitWarps, RB = kSplitRec, NT = kSplitThreads;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t s_red[NW];
    // select scratch (block_kth_hist) and counters
    __shared__ uint32_t k_red[2 * NW + 2], k_hist256[256], k_cnt, k_count, k_out;
    __shared__ uint64_t k_sel[4];
    const uint32_t qi = sp.order[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t F = sp.F, T = sp.T, cap = sp.lay.cap, Fp = sp.lay.rows_per;
    float4 y[NSQ / 2];
    if (sp.lsq == 4) il_load_half<NSQ>(sp.codebook, 0, y);
    if (sp.status[qi] != 0) {
        if (tid == 0) sp.hcnt[qi] = 0;
        return;
    }
    // more probed clusters than slots: the fused kernel's
    if (sp.P > kSplitMaxSlots && sp.ctag[(uint64_t)qi * sp.P + kSplitMaxSlots] < sp.C) {
        if (tid == 0) sp.todo[atomicAdd(sp.ntodo, 1u)] = qi;
        return;
    }
    unsigned char* tab = smem;
    float* qv = reinterpret_cast<float*>(smem + il_table_bytes(false));
    const uint32_t maxl = sp.P < kSplitMaxSlots ? sp.P : kSplitMaxSlots;
    // per probed cluster: first record position of the query's (one past the last at [L]),
    // base records, first memory id, first inserted slot, id, distance
    uint32_t* sl_start = reinterpret_cast<uint32_t*>(smem + sp.lay.slots);
    uint32_t* sl_nb = sl_start + maxl + 1;
    uint32_t* sl_r0 = sl_nb + maxl + 1;
    uint32_t* sl_i0 = sl_r0 + maxl + 1;
    uint32_t* sl_c = sl_i0 + maxl + 1;
    float* sl_cd = reinterpret_cast<float*>(sl_c + maxl + 1);
    float* srow = reinterpret_cast<float*>(smem + sp.lay.srow);      // [group][Fp] cell terms
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem + sp.lay.keys);  // [cap]
    float* stage = reinterpret_cast<float*>(keys);                   // [NSQ][257] before
    for (uint32_t i = tid; i < sp.d; i += NT) qv[i] = sp.q[(uint64_t)qi * sp.d + i];
    const int lut_e = HALF ? half_lut_exponent(sp.qnorm[qi], sp.codebook_max) : 0;
    const float inv_scale = HALF ? ldexpf(1.0f, -lut_e) : 1.0f;
    if (tid == 0) {
        k_count = 0;
        k_out = 0;
        k_cnt = 0;
    }
    // slot table: PS slots per thread, then an exclusive scan of the records
    constexpr int PS = (int)kSplitMaxSlots / NT;
    static_assert(PS * NT == (int)kSplitMaxSlots, "slots split evenly over the threads");
    uint32_t len[PS], c[PS], run = 0, L = 0;
#pragma unroll
    for (int j = 0; j < PS; ++j) {
        const uint32_t l = tid * PS + j;
        c[j] = l < maxl ? sp.ctag[(uint64_t)qi * sp.P + l] : sp.C;
    }
#pragma unroll
    for (int j = 0; j < PS; ++j) {
        const uint32_t l = tid * PS + j;
        len[j] = 0;
        if (c[j] < sp.C) {
            const uint32_t* cell0 = sp.cell_start + (uint64_t)c[j] * F;
            const uint32_t r0 = cell0[0], r1 = cell0[F];
            uint32_t i0 = 0, i1 = 0;
            if (sp.ins_cl_start) {
                i0 = sp.ins_cl_start[c[j]];
                i1 = sp.ins_cl_start[c[j] + 1];
            }
            sl_c[l] = c[j];
            sl_cd[l] = sp.cdist[(uint64_t)qi * sp.P + l];
            sl_nb[l] = r1 - r0;
            sl_r0[l] = r0;
            sl_i0[l] = i0;
            len[j] = (r1 - r0) + (i1 - i0);
        }
        run += len[j];
    }
    // the probed clusters fill a prefix of the slots
#pragma unroll
    for (int j = 0; j < PS; ++j) L += (uint32_t)__syncthreads_count(c[j] < sp.C);
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_red[warp] = incl;
    const float* fdk = sp.fd_by_fine + (uint64_t)qi * F;
    // cell terms of slots [l0, l1): srow[f] = 2 * cell_dist of cell f, cell_dist =
    // (cd + stationary) + fd (puck_index.cpp:539-540)
    auto fill_rows = [&](uint32_t l0, uint32_t l1) {
        if ((F & 3u) == 0) {
            const uint32_t w4 = ((F >> 2) + 31u) & ~31u;  // a warp stays within a row
#pragma unroll 4
            for (uint32_t e = tid; e < (l1 - l0) * w4; e += NT) {
                const uint32_t l = e / w4, i = e - l * w4;
                if (i < (F >> 2)) {
                    const float cdl = sl_cd[l0 + l];
                    const float4 a =
                        __ldg(reinterpret_cast<const float4*>(sp.stationary + (uint64_t)sl_c[l0 + l] * F) + i);
                    const float4 b = __ldg(reinterpret_cast<const float4*>(fdk) + i);
                    reinterpret_cast<float4*>(srow + l * Fp)[i] =
                        make_float4(2.0f * __fadd_rn(__fadd_rn(cdl, a.x), b.x),
                                    2.0f * __fadd_rn(__fadd_rn(cdl, a.y), b.y),
                                    2.0f * __fadd_rn(__fadd_rn(cdl, a.z), b.z),
                                    2.0f * __fadd_rn(__fadd_rn(cdl, a.w), b.w));
                }
            }
        } else {
            for (uint32_t l = l0; l < l1; ++l)
                for (uint32_t i = tid; i < F; i += NT)
                    srow[(l - l0) * Fp + i] =
                        2.0f * __fadd_rn(__fadd_rn(sl_cd[l], sp.stationary[(uint64_t)sl_c[l] * F + i]), fdk[i]);
        }
    };
    fill_rows(0, min(sp.lay.group, L));
    il_build_table<NSQ, HALF, NT, true>(tab, stage, qv, sp.codebook, sp.lsq, lut_e, y);
    // (its barrier also ends the writes of s_red)
    {
        uint32_t st0 = incl - run;
        for (int w = 0; w < warp; ++w) st0 += s_red[w];
#pragma unroll
        for (int j = 0; j < PS; ++j) {
            const uint32_t l = tid * PS + j;
            if (l < L) {
                sl_start[l] = st0;
                if (l == L - 1) sl_start[L] = st0 + len[j];
            }
            st0 += len[j];
        }
        if (L == 0 && tid == 0) sl_start[0] = 0;
    }
    __syncthreads();
    const uint32_t N = sl_start[L];  // records of all probed clusters
    float tau = __int_as_float(0x7f800000);
    if (N > cap) {
        // the bound, from S sampled records, four or two per thread at a time. Four neighbouring
        // lanes take the records of their own lanes in one record block: whole sectors, and
        // lookups without bank conflicts. The select's histogram follows the S keys.
        static_assert(kSplitSampleStep == 2 * NT && kSplitHistKeys * 2 == kHistBins, "sample_count");
        const uint32_t S = sample_count(cap, T, N);
        const float step = (float)N / (float)S;
        auto sample = [&](uint32_t i0, auto count) {
            constexpr int R = decltype(count)::value;
            uint32_t m[R], f[R];
            uint2 g[R][NG];
            float o[R], t[R], cterm[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint32_t ps = min((uint32_t)((float)((i0 + j * NT) & ~3u) * step), N - 1);
                uint32_t a = 0, b = L;  // the slot holding position ps
                while (b - a > 1) {
                    const uint32_t mid = (a + b) >> 1;
                    if (sl_start[mid] <= ps) a = mid;
                    else b = mid;
                }
                const uint32_t local = ps - sl_start[a], nb = sl_nb[a], r0 = sl_r0[a];
                if (local < nb)
                    m[j] = min(max(((r0 + local) & ~31u) + lane, r0), r0 + nb - 1);
                else
                    m[j] = sp.ins_cl_ids[sl_i0[a] + (local - nb)];
                const uint32_t fi =
                    __ldg(reinterpret_cast<const uint16_t*>(sp.codes_il + il_fine_offset(m[j], NSQ)));
#pragma unroll
                for (int q2 = 0; q2 < NG; ++q2)
                    g[j][q2] = __ldg(
                        reinterpret_cast<const uint2*>(sp.codes_il + il_granule_offset(m[j], q2, NSQ)));
                o[j] = __ldg(reinterpret_cast<const float*>(sp.codes_il + il_offset_offset(m[j], NSQ)));
                cterm[j] = a < sp.lay.group
                               ? srow[a * Fp + fi]
                               : 2.0f * __fadd_rn(__fadd_rn(sl_cd[a], __ldg(sp.stationary +
                                                                            (uint64_t)sl_c[a] * F + fi)),
                                                  __ldg(fdk + fi));
                f[j] = j;
            }
            il_score<NSQ, HALF, R, true>(tab, cterm, g, o, f, m, inv_scale, t);
#pragma unroll
            for (int j = 0; j < R; ++j) keys[i0 + j * NT] = filter_key(t[j], i0 + j * NT);
        };
        uint32_t i0 = tid;
        for (; i0 + 4 * NT <= S + tid; i0 += 4 * NT) sample(i0, std::integral_constant<int, 4>());
        if (i0 < S) sample(i0, std::integral_constant<int, 2>());
        __syncthreads();
        const uint64_t cut = block_cut_bound<NT>(keys, S, min(sample_rank(S, T, N), S),
                                                 reinterpret_cast<uint32_t*>(keys + S), k_red);
        if (cut != kKeyMax) tau = key_value(cut);
    }
    const uint32_t lanes_below = (1u << lane) - 1;
    // keeps the records v with t at or below the bound, as (t bits, id): the warp's take
    // consecutive slots
    auto append = [&](const auto& t, const auto& m, const auto& v) {
        constexpr int R = (int)(sizeof(t) / sizeof(t[0]));
        unsigned b[R];
        uint32_t nk = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            b[r] = __ballot_sync(0xffffffffu, v[r] && t[r] <= tau);
            nk += __popc(b[r]);
        }
        if (nk == 0) return;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&k_count, nk);
        at = __shfl_sync(0xffffffffu, at, 0);
        if (at + nk > cap) return;  // the buffer is full: the query will be left
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (b[r] >> lane & 1u)
                keys[at + __popc(b[r] & lanes_below)] = ((uint64_t)__float_as_uint(t[r]) << 32) | m[r];
            at += __popc(b[r]);
        }
    };
    for (uint32_t g0 = 0; g0 < L; g0 += sp.lay.group) {
        const uint32_t g1 = min(g0 + sp.lay.group, L);
        __syncthreads();  // the previous group's cell terms (the sampled keys) are no longer read
        if (g0 > 0) fill_rows(g0, g1);
        __syncthreads();
        // Cluster by cluster, without barriers: the warp takes record blocks w, w + NW, ...
        // of RB blocks each, w rotating so that the clusters' last blocks spread over the
        // warps. Two register sets, A and B, in turn: step j + 1's loads go into one set
        // while step j is scored from the other (no copies between steps).
        for (uint32_t l = g0; l < g1; ++l) {
            const uint32_t nb = sl_nb[l], r0 = sl_r0[l];
            if (nb == 0) continue;
            const uint32_t nblk = (r0 + nb - 1) / 32 - r0 / 32 + 1;
            const float* const row = srow + (l - g0) * Fp;
            uint32_t bi = ((warp + l) % NW) * RB;
            // a step's loads: whole steps, the blocks past the cluster's last are dropped
            const unsigned char* rec = sp.codes_il + (uint64_t)(r0 / 32 + bi) * kBlk;
            const unsigned char *pg = rec + 8 * lane, *po = rec + 32 * kG + 4 * lane,
                                *pf = rec + 32 * kG + 128 + 2 * lane;
            constexpr uint32_t kStep = NW * RB * kBlk;
            auto load = [&](uint2 (&g)[RB][NG], float (&o)[RB], uint32_t (&f)[RB]) {
#pragma unroll
                for (int r = 0; r < RB; ++r) {
#pragma unroll
                    for (int q2 = 0; q2 < NG; ++q2)
                        g[r][q2] = __ldg(reinterpret_cast<const uint2*>(pg + r * kBlk + q2 * 256));
                    o[r] = __ldg(reinterpret_cast<const float*>(po + r * kBlk));
                    f[r] = __ldg(reinterpret_cast<const uint16_t*>(pf + r * kBlk));
                }
                pg += kStep;
                po += kStep;
                pf += kStep;
            };
            uint32_t u = (r0 & ~31u) + bi * 32 + lane - r0;  // the lane's first record, from r0
            auto emit = [&](const uint2 (&g)[RB][NG], const float (&o)[RB], const uint32_t (&f)[RB]) {
                uint32_t m[RB], fc[RB], ln[RB];
                bool v[RB];
                float t[RB];
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    m[r] = r0 + u + r * 32;
                    v[r] = u + r * 32 < nb;
                    fc[r] = min(f[r], F - 1);  // (a dropped record's may be anything)
                    ln[r] = lane;
                }
                il_score<NSQ, HALF, RB, true>(tab, row, g, o, fc, ln, inv_scale, t);
                append(t, m, v);
                u += NW * RB * 32;
            };
            uint2 ga[RB][NG], gb[RB][NG];
            float oa[RB], ob[RB];
            uint32_t fa[RB], fb[RB];
            if (bi < nblk) load(ga, oa, fa);
            for (; bi < nblk; bi += 2 * NW * RB) {
                if (bi + NW * RB < nblk) load(gb, ob, fb);
                emit(ga, oa, fa);
                if (bi + NW * RB < nblk) {
                    if (bi + 2 * NW * RB < nblk) load(ga, oa, fa);
                    emit(gb, ob, fb);
                }
            }
        }
        // realtime: the clusters' inserted records (gathered from the interleaved copy)
        for (uint32_t l = g0; sp.ins_cl_start != nullptr && l < g1; ++l) {
            const uint32_t i0 = sl_i0[l], ni = sl_start[l + 1] - sl_start[l] - sl_nb[l];
            const float* const row = srow + (l - g0) * Fp;
            for (uint32_t v0 = 0; v0 < ni; v0 += NT) {
                const uint32_t vi = v0 + tid;
                const bool v[1] = {vi < ni};
                const uint32_t m1[1] = {v[0] ? sp.ins_cl_ids[i0 + vi] : 0u};
                uint2 g[1][NG];
#pragma unroll
                for (int q2 = 0; q2 < NG; ++q2)
                    g[0][q2] = __ldg(
                        reinterpret_cast<const uint2*>(sp.codes_il + il_granule_offset(m1[0], q2, NSQ)));
                const float o[1] = {
                    __ldg(reinterpret_cast<const float*>(sp.codes_il + il_offset_offset(m1[0], NSQ)))};
                const uint32_t f[1] = {v[0] ? __ldg(reinterpret_cast<const uint16_t*>(
                                                  sp.codes_il + il_fine_offset(m1[0], NSQ)))
                                            : 0u};
                float t[1];
                il_score<NSQ, HALF, 1, true>(tab, row, g, o, f, m1, inv_scale, t);
                append(t, m1, v);
            }
        }
    }
    __syncthreads();
    const uint32_t m = k_count;
    if (m > cap || m < min(T, N)) {  // the bound was too high or too low
        if (tid == 0) sp.todo[atomicAdd(sp.ntodo, 1u)] = qi;
        return;
    }
    // the exact T smallest, written unordered like k_scan_il's; the table's place is free
    auto put = [&](uint32_t slot, uint64_t k) {
        sp.hdist[(uint64_t)qi * T + slot] = key_value(k);
        sp.htag[(uint64_t)qi * T + slot] = (uint32_t)k;
    };
    // keys[i] below the bound go out, a ballot at a time; one atomic per warp
    constexpr int kPer = 16;  // keys per thread in registers
    uint32_t* hist = reinterpret_cast<uint32_t*>(tab);               // [kHistBins]
    uint64_t* ties = reinterpret_cast<uint64_t*>(hist + kHistBins);  // keys of the T-th's bin
    constexpr uint32_t kTies = 1024;
    uint64_t k[kPer];
    uint32_t lo = 0xFFFFFFFFu, hi = 0, bin = 0xFFFFFFFFu, shift = 0, below = m;
    const bool regs = m <= (uint32_t)(kPer * NT);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint32_t i = j * NT + tid;
        const uint64_t x = regs && i < m ? keys[i] : 0ull;
        k[j] = filter_key(__uint_as_float((uint32_t)(x >> 32)), (uint32_t)x);
        if (regs && i < m) {
            lo = min(lo, (uint32_t)(k[j] >> 32));
            hi = max(hi, (uint32_t)(k[j] >> 32));
        } else {
            k[j] = kKeyMax;
        }
    }
    if (regs && m > T) {
        // the bin of the T-th smallest among kHistBins between the smallest and the largest
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            k_red[warp] = lo;
            k_red[NW + warp] = hi;
        }
        for (uint32_t b = tid; b < kHistBins; b += NT) hist[b] = 0;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            lo = min(lo, k_red[w]);
            hi = max(hi, k_red[NW + w]);
        }
        shift = 32 - min(__clz(hi - lo), 32);
        shift = shift > 10 ? shift - 10 : 0;
        static_assert(kHistBins == 1024, "10 bits of the range");
#pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (j * NT + tid < m) atomicAdd(&hist[((uint32_t)(k[j] >> 32) - lo) >> shift], 1u);
        __syncthreads();
        constexpr uint32_t per = kHistBins / NT;
        uint32_t c[per], sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < per; ++j) {
            c[j] = hist[tid * per + j];
            sum += c[j];
        }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) s_red[warp] = inc;
        __syncthreads();
        uint32_t bl = inc - sum;
        for (int w = 0; w < warp; ++w) bl += s_red[w];
        if (bl < T && T <= bl + sum) {
#pragma unroll
            for (uint32_t j = 0; j < per; ++j) {
                if (bl < T && T <= bl + c[j]) {
                    k_red[0] = tid * per + j;
                    k_red[1] = bl;
                    k_red[2] = c[j];
                }
                bl += c[j];
            }
        }
        __syncthreads();
        bin = k_red[0];
        below = k_red[1];
    }
    if (regs && (m <= T || k_red[2] <= kTies)) {
        // below the bin: out; the bin's own: the first by rank fill up to T
        const uint32_t lim = min(m, T) - (m > T ? below : m);
        uint32_t nout = 0;
        unsigned in[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const bool have = j * NT + tid < m;
            const uint32_t mybin = m > T ? ((uint32_t)(k[j] >> 32) - lo) >> shift : 0u;
            in[j] = __ballot_sync(0xffffffffu, have && mybin < bin);
            nout += __popc(in[j]);
            if (have && mybin == bin) ties[atomicAdd(&k_cnt, 1u)] = k[j];
        }
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&k_out, nout);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (in[j] >> lane & 1u) put(at + __popc(in[j] & ((1u << lane) - 1)), k[j]);
            at += __popc(in[j]);
        }
        if (lim > 0) {
            __syncthreads();
            const uint32_t nt = k_cnt;
            for (uint32_t i = tid; i < nt; i += NT) {
                const uint64_t x = ties[i];
                uint32_t rank = 0;
                for (uint32_t u = 0; u < nt; ++u) rank += ties[u] < x ? 1u : 0u;
                if (rank < lim) put(below + rank, x);
            }
        }
    } else {
        // more keys than the registers take, or in the T-th's bin
        __syncthreads();
        for (uint32_t i = tid; i < m; i += NT) {
            const uint64_t x = keys[i];
            keys[i] = filter_key(__uint_as_float((uint32_t)(x >> 32)), (uint32_t)x);
        }
        __syncthreads();
        const uint64_t bound =
            m > T ? block_kth_hist<NT>(keys, m, T, hist, k_red, &k_cnt, k_hist256, k_sel) + 1 : kKeyMax;
        for (uint32_t i0 = 0; i0 < m; i0 += NT) {
            const uint32_t i = i0 + tid;
            const uint64_t x = i < m ? keys[i] : kKeyMax;
            const unsigned b = __ballot_sync(0xffffffffu, x < bound);
            uint32_t at = 0;
            if (lane == 0 && b) at = atomicAdd(&k_out, (uint32_t)__popc(b));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (x < bound) put(at + __popc(b & ((1u << lane) - 1)), x);
        }
    }
    const uint32_t outn = min(m, T);
    for (uint32_t i = outn + tid; i < T; i += NT) {
        sp.hdist[(uint64_t)qi * T + i] = sentinel_f();
        sp.htag[(uint64_t)qi * T + i] = kNoLabel;
    }
    if (tid == 0) {
        sp.hcnt[qi] = outn;
        if (sp.counters) {
            atomicAdd(sp.counters + kScRecords, (unsigned long long)N);
            atomicAdd(sp.counters + kScKept, (unsigned long long)m);
        }
    }
}

}  // namespace

// Shared memory of the interleaved kernel (il_applies(nsq)) for filter_topk T.
static size_t il_smem_bytes(const DeviceIndex& ix, uint32_t T, bool half) {
    const size_t stage = sizeof(float) * ix.nsq * 257;
    const size_t work = il_srow_bytes(ix.F) +
                        sizeof(uint64_t) * (half ? il_cap<true>(T) : il_cap<false>(T)) +
                        sizeof(uint32_t) * kHistBins;
    const size_t ring = half ? (size_t)IlShape<true>::kStages * il_slot_bytes<true>(ix.nsq)
                             : (size_t)IlShape<false>::kStages * il_slot_bytes<false>(ix.nsq);
    return il_table_bytes(half) + il_query_bytes(ix.d) + ring +
           (stage > work ? stage : work);
}

size_t scan_smem_bytes(const DeviceIndex& ix, uint32_t T) {
    if (il_applies(ix.nsq)) return il_smem_bytes(ix, T, false);
    return sizeof(uint64_t) * scan_cap(T) + sizeof(uint32_t) * kHistBins +
           sizeof(float) * ix.nsq * 256 + sizeof(float) * ix.F + sizeof(float) * ix.d;
}

size_t scan_smem_bytes_half(const DeviceIndex& ix, uint32_t T) {
    if (il_applies(ix.nsq)) return il_smem_bytes(ix, T, true);
    return sizeof(uint64_t) * scan_cap(T) + sizeof(uint32_t) * kHistBins +
           sizeof(__half) * ix.nsq * 256 + sizeof(float) * ix.F + sizeof(float) * ix.d;
}

// The buffer takes T + a round + at least 1024 more keys between cuts.
uint32_t scan_max_filter_topk() { return kMaxCap - kRound - 1024; }

cudaError_t launch_scan_order(const DeviceIndex& ix, uint32_t n, Scratch& s, cudaStream_t stream) {
    if (s.order == nullptr || s.wbin == nullptr) return cudaErrorInvalidValue;
    k_scan_work<<<(n + 255) / 256, 256, 0, stream>>>(s.ctag, s.status, ix.cell_start,
                                                     ix.ins_n ? ix.ins_cl_start : nullptr, n, s.P,
                                                     ix.C, ix.F, s.wbin);
    k_scan_order<<<1, kOrderThreads, 0, stream>>>(s.wbin, n, s.order, s.ntodo);
    return cudaGetLastError();
}

SplitLayout split_choice(const DeviceIndex& ix, uint32_t P, uint32_t T) {
    const SplitLayout two = split_layout(ix.nsq, ix.d, ix.F, P, kSplitBudget2, kSplitRows2);
    if (two.bytes && two.cap >= split_need(T)) return two;
    SplitLayout one{};
    for (uint32_t rows : kSplitRows1) {
        one = split_layout(ix.nsq, ix.d, ix.F, P, kSplitBudget1, rows);
        if (one.bytes && one.cap >= 4 * T + kSplitLeast) return one;
    }
    return one.bytes && one.cap >= T + 512 + kSplitLeast ? one : SplitLayout{};
}

bool scan_split_applies(const DeviceIndex& ix, const Scratch& s) {
    return il_applies(ix.nsq) && ix.codes_il != nullptr && split_choice(ix, s.P, s.T).bytes != 0;
}

static cudaError_t launch_fused(const DeviceIndex& ix, uint32_t n, Scratch& s, bool half_lut,
                                bool left, cudaStream_t stream) {
    ScanParams p;
    p.q = s.q;
    p.qnorm = s.qnorm;
    p.status = s.status;
    p.cdist = s.cdist;
    p.ctag = s.ctag;
    p.fd_by_fine = s.dots;
    p.hdist = s.hdist;
    p.htag = s.htag;
    p.hcnt = s.hcnt;
    p.stationary = ix.stationary;
    p.cell_start = ix.cell_start;
    p.rec_fine = ix.rec_fine;
    p.offsets = ix.offsets;
    p.codes = ix.codes;
    p.codes_il = ix.codes_il;
    p.codebook = ix.codebook;
    p.counters = s.counters;
    p.d = ix.d;
    p.C = ix.C;
    p.F = ix.F;
    p.nsq = ix.nsq;
    p.lsq = ix.lsq;
    p.code_stride = ix.code_stride;
    p.P = s.P;
    p.T = s.T;
    p.cap = scan_cap(s.T);
    p.codebook_max = ix.codebook_max;
    if (s.order == nullptr || s.T > scan_max_filter_topk()) return cudaErrorInvalidValue;
    p.order = s.order;
    p.err = s.tc_err;
    p.ins_cl_start = ix.ins_n ? ix.ins_cl_start : nullptr;
    p.ins_cl_ids = ix.ins_cl_ids;
    p.todo = left ? s.todo : nullptr;
    p.ntodo = s.ntodo;
    p.n = n;
    const size_t smem = half_lut ? scan_smem_bytes_half(ix, s.T) : scan_smem_bytes(ix, s.T);
    const uint32_t nw = ix.code_stride / 4;
    // the queries the split scan left are few, as a rule none: a grid of the blocks that
    // fit the chip loops over them
    const uint32_t fits = 2u * (uint32_t)sm_count();
    auto launch = [&](void (*kernel)(ScanParams), int threads) {
        ensure_max_dynamic_smem(kernel, 220 * 1024);
        kernel<<<left && n > fits ? fits : n, threads, smem, stream>>>(p);
    };
    if (il_applies(ix.nsq)) {
        if (ix.codes_il == nullptr) return cudaErrorInvalidValue;
        p.cap = half_lut ? il_cap<true>(s.T) : il_cap<false>(s.T);
        switch (ix.nsq) {
#define PGPU_IL(N) \
    case N:                                                                                \
        if (half_lut) launch(k_scan_il<N, true>, IlShape<true>::kThreads);                   \
        else launch(k_scan_il<N, false>, IlShape<false>::kThreads);                          \
        break;
            PGPU_IL(4) PGPU_IL(8) PGPU_IL(12) PGPU_IL(16) PGPU_IL(20) PGPU_IL(24) PGPU_IL(28)
            PGPU_IL(32)
#undef PGPU_IL
            default: return cudaErrorInvalidValue;
        }
    } else if (half_lut) {
        if (nw <= 2) launch(k_scan_select<2, kTabF16>, kThreads);
        else if (nw <= 4) launch(k_scan_select<4, kTabF16>, kThreads);
        else if (nw <= 6) launch(k_scan_select<6, kTabF16>, kThreads);
        else if (nw <= 8) launch(k_scan_select<8, kTabF16>, kThreads);
        else launch(k_scan_select<16, kTabF16>, kThreads);
    } else {
        if (nw <= 2) launch(k_scan_select<2, kTabF32>, kThreads);
        else if (nw <= 4) launch(k_scan_select<4, kTabF32>, kThreads);
        else if (nw <= 6) launch(k_scan_select<6, kTabF32>, kThreads);
        else if (nw <= 8) launch(k_scan_select<8, kTabF32>, kThreads);
        else launch(k_scan_select<16, kTabF32>, kThreads);
    }
    return cudaGetLastError();
}

cudaError_t launch_scan_records(const DeviceIndex& ix, uint32_t n, Scratch& s, bool half_lut,
                                cudaStream_t stream) {
    if (!scan_split_applies(ix, s)) return launch_fused(ix, n, s, half_lut, false, stream);
    SplitParams sp;
    sp.ctag = s.ctag;
    sp.cdist = s.cdist;
    sp.status = s.status;
    sp.cell_start = ix.cell_start;
    sp.ins_cl_start = ix.ins_n ? ix.ins_cl_start : nullptr;
    sp.ins_cl_ids = ix.ins_cl_ids;
    sp.stationary = ix.stationary;
    sp.fd_by_fine = s.dots;
    sp.q = s.q;
    sp.qnorm = s.qnorm;
    sp.codebook = ix.codebook;
    sp.codes_il = ix.codes_il;
    sp.order = s.order;
    sp.todo = s.todo;
    sp.ntodo = s.ntodo;
    sp.hdist = s.hdist;
    sp.htag = s.htag;
    sp.hcnt = s.hcnt;
    sp.counters = s.counters;
    sp.n = n;
    sp.d = ix.d;
    sp.C = ix.C;
    sp.F = ix.F;
    sp.lsq = ix.lsq;
    sp.P = s.P;
    sp.T = s.T;
    sp.codebook_max = ix.codebook_max;
    sp.lay = split_choice(ix, s.P, s.T);
    auto score = [&](void (*kernel)(SplitParams)) {
        ensure_max_dynamic_smem(reinterpret_cast<const void*>(kernel), 220 * 1024);
        kernel<<<n, kSplitThreads, sp.lay.bytes, stream>>>(sp);
    };
    switch (ix.nsq) {
#define PGPU_SPLIT(N)                           \
    case N:                                     \
        if (half_lut) score(k_scan_score<N, true>); \
        else score(k_scan_score<N, false>);     \
        break;
        PGPU_SPLIT(4) PGPU_SPLIT(8) PGPU_SPLIT(12) PGPU_SPLIT(16) PGPU_SPLIT(20) PGPU_SPLIT(24)
        PGPU_SPLIT(28) PGPU_SPLIT(32)
#undef PGPU_SPLIT
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_scan_finish(const DeviceIndex& ix, uint32_t n, Scratch& s, bool half_lut,
                               cudaStream_t stream) {
    if (!scan_split_applies(ix, s)) return cudaSuccess;
    return launch_fused(ix, n, s, half_lut, true, stream);
}

}  // namespace pgpu
