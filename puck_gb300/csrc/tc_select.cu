// Exact selections on top of the BF16 tensor-core contraction.
//
// The tensor core gives s^_j ~ s_j for every centroid j, where s_j is the FP32
// value the reference computes (bias_j - q.c_j summed sequentially). With q and
// c_j rounded to BF16 (unit roundoff 2^-8) and any FP32 accumulation order,
//
//   |s^_j - s_j| <= E_j = eps * |q| |c_j| + 2^-20 (|bias_j| + |s^_j|),
//   eps = 2^-7 + 2^-15 + (d + 8) * 2^-21,
//
// (the 2^-7 term bounds the two BF16 roundings of each product, the d term the
// FP32 accumulation of both sides, the last term the final subtractions).
// Let U be the P-th smallest s^_j + E_j. Then every j with s_j <= s_(P) (the
// P-th smallest exact value) has s^_j - E_j <= s_j <= s_(P) <= U, so the window
// W = { j : s^_j - E_j <= U } holds the exact top P and every value tied with
// the P-th. Only W is recomputed in exact FP32 (the reference's operation
// order), sorted by (value, id) and checked for ties among the first P+1
// exactly as k_topsort does; with a tie, or with W beyond its buffer, or when
// the contraction reported a failure, the block recomputes every s_j and
// replays Puck's MaxHeap, so the result is always the reference's.
#include <cfloat>
#include <cstdint>

#include "device_common.cuh"
#include "pgpu_internal.h"

namespace pgpu {
namespace {

constexpr int kWinThreads = 256;
constexpr uint32_t kWinCap = 1024;

__device__ __forceinline__ float window_eps(uint32_t d) {
    return 0.0078125f + 3.0517578125e-05f + (float)(d + 8) * 4.76837158203125e-07f;
}

// Exact top-P of bias_j - q.c_j per row (k_topsort's output and tie rule).
__global__ __launch_bounds__(kWinThreads) void k_window_topk(
    const float* __restrict__ approx, uint32_t ld, const float* __restrict__ Q, uint32_t d,
    const float* __restrict__ qnorm, const float* __restrict__ cents,
    const float* __restrict__ bias, const float* __restrict__ cabs, uint32_t C, uint32_t P,
    uint32_t ld_out, float* __restrict__ out_val, uint32_t* __restrict__ out_idx,
    const int32_t* __restrict__ status,
    const int* __restrict__ tc_err, unsigned long long* __restrict__ fallbacks,
    const int32_t* __restrict__ skip, const uint32_t* __restrict__ qidx,
    const uint32_t* __restrict__ nrows_dev) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* shi = reinterpret_cast<float*>(smem);                 // [C]   s^ + E, later exact s
    float* slo = shi + C;                                        // [C] s^ - E; the heap from here
    float* sq = slo + 2 * (C + 1);                               // [d]
    unsigned long long* ckey = reinterpret_cast<unsigned long long*>(
        (reinterpret_cast<uintptr_t>(sq + d) + 7) & ~uintptr_t(7));  // [kWinCap]
    __shared__ uint32_t hist[256];
    __shared__ uint32_t state[2];
    __shared__ uint32_t ncand;
    // screen row rc; the query it belongs to (a compacted list when a probe answered
    // the others)
    const uint32_t rc = blockIdx.x;
    if (nrows_dev != nullptr && rc >= *nrows_dev) return;
    const uint32_t row = qidx ? qidx[rc] : rc;
    const int tid = threadIdx.x;
    if (skip != nullptr && skip[row]) return;  // the learned probe answered this query
    float* ov = out_val + (uint64_t)row * ld_out;
    uint32_t* oi = out_idx + (uint64_t)row * ld_out;
    // slots past P (a probe's wider cap): unused
    for (uint32_t i = P + tid; i < ld_out; i += kWinThreads) {
        ov[i] = sentinel_f();
        oi[i] = kNoLabel;
    }
    if (status != nullptr && status[row] != 0) {
        for (uint32_t i = tid; i < P; i += kWinThreads) {
            ov[i] = sentinel_f();
            oi[i] = kNoLabel;
        }
        return;
    }
    const float* q = Q + (uint64_t)row * d;
    for (uint32_t k = tid; k < d; k += kWinThreads) sq[k] = q[k];
    if (tid == 0) ncand = 0;
    bool exact_all = (*tc_err != 0);
    if (!exact_all) {
        const float eps = window_eps(d);
        const float qa = sqrtf(qnorm[row]);
        const float* a = approx + (uint64_t)rc * ld;
        for (uint32_t j = tid; j < C; j += kWinThreads) {
            const float s = a[j];
            const float e = eps * qa * cabs[j] + 9.5367431640625e-07f * (fabsf(bias[j]) + fabsf(s)) +
                            1e-30f;
            shi[j] = s + e;
            slo[j] = s - e;
        }
        __syncthreads();
        const float U = key_to_float(block_kth_key<kWinThreads>(shi, C, P, hist, state));
        for (uint32_t j = tid; j < C; j += kWinThreads) {
            if (slo[j] <= U) {
                const uint32_t pos = atomicAdd(&ncand, 1u);
                if (pos < kWinCap) ckey[pos] = j;
            }
        }
        __syncthreads();
        const uint32_t m = ncand;
        if (m > kWinCap) {
            exact_all = true;
        } else {
            uint32_t mp = 1;
            while (mp < m) mp <<= 1;
            for (uint32_t t = tid; t < mp; t += kWinThreads) {
                if (t < m) {
                    const uint32_t j = (uint32_t)ckey[t];
                    const float v =
                        __fsub_rn(bias[j], dot_seq_row(sq, cents + (uint64_t)j * d, d));
                    ckey[t] = ((unsigned long long)ordered_key(v) << 32) | j;
                } else {
                    ckey[t] = ~0ull;
                }
            }
            __syncthreads();
            bitonic_sort_u64<kWinThreads>(ckey, mp);
            int tie = 0;
            const uint32_t last = P < m ? P : m - 1;
            for (uint32_t i = tid; i < last; i += kWinThreads)
                if ((uint32_t)(ckey[i] >> 32) == (uint32_t)(ckey[i + 1] >> 32)) tie = 1;
            tie = __syncthreads_or(tie);
            if (!tie) {
                for (uint32_t i = tid; i < P; i += kWinThreads) {
                    ov[i] = key_to_float((uint32_t)(ckey[i] >> 32));
                    oi[i] = (uint32_t)ckey[i];
                }
                return;
            }
            exact_all = true;
        }
    }
    // Reference path: every exact value, then MaxHeap(P) fed in index order.
    __syncthreads();
    for (uint32_t j = tid; j < C; j += kWinThreads)
        shi[j] = __fsub_rn(bias[j], dot_seq_row(sq, cents + (uint64_t)j * d, d));
    __syncthreads();
    // the heap takes the place of all that follows the values (16-byte aligned)
    uint2* heap = reinterpret_cast<uint2*>((reinterpret_cast<uintptr_t>(slo) + 15) & ~uintptr_t(15));
    if (tid < 32) {
        if (tid == 0) atomicAdd(fallbacks, 1ull);
        warp_heap_replay(heap, shi, nullptr, C, P);
    }
    __syncthreads();
    for (uint32_t i = tid; i < P; i += kWinThreads) {
        ov[i] = __uint_as_float(heap[i + 1].x);
        oi[i] = heap[i + 1].y;
    }
}

// The same selection for small P (P <= kSmallP), one warp per query row: the P-th
// smallest s^ + E by P rounds of warp minima over (value, id), the window's exact
// values recomputed one per lane, a warp bitonic sort of at most 64 candidates,
// and the tie check. With a tie or a wider window the warp feeds every exact
// value, 32 at a time in index order, to lane 0's MaxHeap(P).
constexpr uint32_t kSmallP = 16;
constexpr uint32_t kSmallCap = 64;
// PMAX: compile-time bound on P (1, 4 or 16) for the per-lane sorted lists.
template <uint32_t PMAX>
__global__ __launch_bounds__(256) void k_window_small(
    const float* __restrict__ approx, uint32_t ld, const float* __restrict__ Q, uint32_t d,
    const float* __restrict__ qnorm, const float* __restrict__ cents,
    const float* __restrict__ bias, const float* __restrict__ cabs, uint32_t C, uint32_t P,
    uint32_t ld_out, uint32_t nrows, float* __restrict__ out_val, uint32_t* __restrict__ out_idx,
    const int32_t* __restrict__ status, const int* __restrict__ tc_err,
    unsigned long long* __restrict__ fallbacks, const int32_t* __restrict__ skip,
    const uint32_t* __restrict__ qidx, const uint32_t* __restrict__ nrows_dev) {
    __shared__ unsigned long long wkey[8][kSmallCap];
    __shared__ float hv_s[8][kSmallP + 1];
    __shared__ uint32_t ht_s[8][kSmallP + 1];
    __shared__ float chunk[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rc = blockIdx.x * 8 + warp;  // screen row; its query below
    if (rc >= nrows || (nrows_dev != nullptr && rc >= *nrows_dev)) return;
    const uint32_t row = qidx ? qidx[rc] : rc;
    if (skip != nullptr && skip[row]) return;  // the learned probe answered this query
    float* ov = out_val + (uint64_t)row * ld_out;
    uint32_t* oi = out_idx + (uint64_t)row * ld_out;
    for (uint32_t i = P + lane; i < ld_out; i += 32) {
        ov[i] = sentinel_f();
        oi[i] = kNoLabel;
    }
    if (status != nullptr && status[row] != 0) {
        for (uint32_t i = lane; i < P; i += 32) {
            ov[i] = sentinel_f();
            oi[i] = kNoLabel;
        }
        return;
    }
    const float* q = Q + (uint64_t)row * d;
    const float* a = approx + (uint64_t)rc * ld;
    unsigned long long* keys = wkey[warp];
    bool exact_all = (*tc_err != 0);
    if (!exact_all) {
        const float eps = window_eps(d);
        const float qa = sqrtf(qnorm[row]);
        // P-th smallest (hi, id): each lane keeps its P smallest in ascending order
        // (one pass), then P rounds of warp minima over the lanes' heads
        float tv[PMAX];
        uint32_t ti[PMAX];
#pragma unroll
        for (uint32_t r = 0; r < PMAX; ++r) {
            tv[r] = FLT_MAX;
            ti[r] = 0xFFFFFFFFu;
        }
        float worst = FLT_MAX;  // tv[P - 1]
        for (uint32_t j = lane; j < C; j += 32) {
            const float sv = a[j];
            const float hi = sv + (eps * qa * cabs[j] +
                                   9.5367431640625e-07f * (fabsf(bias[j]) + fabsf(sv)) + 1e-30f);
            if (hi < worst) {  // ids ascend within a lane: equal values keep the earlier
                float v = hi;
                uint32_t id = j;
#pragma unroll
                for (uint32_t r = 0; r < PMAX; ++r) {
                    if (r < P && v < tv[r]) {
                        const float t1 = tv[r];
                        const uint32_t t2 = ti[r];
                        tv[r] = v;
                        ti[r] = id;
                        v = t1;
                        id = t2;
                    }
                    if (r + 1 == P) worst = tv[r];
                }
            }
        }
        uint32_t head = 0;
        float lv = FLT_MAX;
        for (uint32_t r = 0; r < P; ++r) {
            float hv = FLT_MAX;
            uint32_t hid = 0xFFFFFFFFu;
#pragma unroll
            for (uint32_t t = 0; t < PMAX; ++t)
                if (t == head) {
                    hv = tv[t];
                    hid = ti[t];
                }
            float bv = hv;
            uint32_t bi = hid;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov2 = __shfl_xor_sync(0xffffffffu, bv, o);
                const uint32_t oi2 = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov2 < bv || (ov2 == bv && oi2 < bi)) {
                    bv = ov2;
                    bi = oi2;
                }
            }
            if (hid == bi && hv == bv && bi != 0xFFFFFFFFu) ++head;
            lv = bv;
        }
        const float U = lv;
        // window: lo <= U, exact value per candidate
        uint32_t m = 0;
        for (uint32_t j0 = 0; j0 < C; j0 += 32) {
            const uint32_t j = j0 + lane;
            bool in = false;
            if (j < C) {
                const float sv = a[j];
                const float e = eps * qa * cabs[j] + 9.5367431640625e-07f * (fabsf(bias[j]) + fabsf(sv)) +
                                1e-30f;
                in = (sv - e) <= U;
            }
            const unsigned b = __ballot_sync(0xffffffffu, in);
            if (m + __popc(b) > kSmallCap) {
                m = kSmallCap + 1;
                break;
            }
            if (in) keys[m + __popc(b & ((1u << lane) - 1))] = j;
            m += __popc(b);
        }
        __syncwarp();
        if (m <= kSmallCap) {
            // the members' exact values, one member per lane: every dot's loads in flight
            // together instead of one chunk of the screen at a time
            for (uint32_t i = lane; i < m; i += 32) {
                const uint32_t j = (uint32_t)keys[i];
                const float v = __fsub_rn(bias[j], dot_seq_row(q, cents + (uint64_t)j * d, d));
                keys[i] = ((unsigned long long)ordered_key(v) << 32) | j;
            }
            __syncwarp();
        }
        if (m > kSmallCap) {
            exact_all = true;
        } else {
            for (uint32_t i = m + lane; i < kSmallCap; i += 32) keys[i] = ~0ull;
            __syncwarp();
            // bitonic sort of 64 keys, two compare-exchanges per lane and step
            for (uint32_t size = 2; size <= kSmallCap; size <<= 1) {
                for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
                    const uint32_t t = lane;
                    const uint32_t lo = 2 * t - (t & (stride - 1));
                    const uint32_t hi = lo + stride;
                    const unsigned long long x = keys[lo], y = keys[hi];
                    if ((x > y) == ((lo & size) == 0)) {
                        keys[lo] = y;
                        keys[hi] = x;
                    }
                    __syncwarp();
                }
            }
            bool tie = false;
            const uint32_t last = P < m ? P : m - 1;
            for (uint32_t i = lane; i < last; i += 32)
                tie |= (uint32_t)(keys[i] >> 32) == (uint32_t)(keys[i + 1] >> 32);
            if (!__any_sync(0xffffffffu, tie)) {
                for (uint32_t i = lane; i < P; i += 32) {
                    ov[i] = key_to_float((uint32_t)(keys[i] >> 32));
                    oi[i] = (uint32_t)keys[i];
                }
                return;
            }
            exact_all = true;
        }
    }
    // Reference path: every exact value, in index order, into MaxHeap(P).
    float* hv = hv_s[warp];
    uint32_t* ht = ht_s[warp];
    uint32_t dpc = P;
    if (lane == 0) {
        atomicAdd(fallbacks, 1ull);
        for (uint32_t i = 1; i <= P; ++i) hv[i] = sentinel_f();
    }
    for (uint32_t j0 = 0; j0 < C; j0 += 32) {
        const uint32_t j = j0 + lane;
        if (j < C) chunk[warp][lane] = __fsub_rn(bias[j], dot_seq_row(q, cents + (uint64_t)j * d, d));
        __syncwarp();
        if (lane == 0) {
            const uint32_t cnt = C - j0 < 32 ? C - j0 : 32;
            for (uint32_t t = 0; t < cnt; ++t) heap_update(hv, ht, P, dpc, chunk[warp][t], j0 + t);
        }
        __syncwarp();
    }
    if (lane == 0) {
        heap_reorder(hv, ht, P);
        for (uint32_t i = 0; i < P; ++i) {
            ov[i] = hv[i + 1];
            oi[i] = ht[i + 1];
        }
    }
}

// nearest_center, exact part after the MINIMA screen (tc_filter.cu): one warp per point. With
// xa = |x|, dx = |x - bf16(x)| and cmax, dcmax the largest |c| and |c - bf16(c)|, every
// screened score is within
//   E = dx cmax + (xa + dx) dcmax + (d + 8) 2^-21 (xa + dx)(cmax + dcmax)
//       + 2^-21 (xn + cmax^2) + 2^-20 (0.5 cmax^2 + 1.01 xa cmax)
// of the value that orders the centroids like the reference's cur_j = (|x|^2 + |c_j|^2) -
// 2 x.c_j (the roundings of the operands, of both accumulations, of the final subtractions), so
// the centroid with the smallest cur_j, and every one equal to it, lies in a group of 8 whose
// smallest score is at most the row's smallest + 2E. Those groups (1.3 per point where the
// clusters are apart) are measured in the reference's FP32 order, lane = centroid; the smallest
// cur_j with the lowest id wins, as in the reference's strict-< scan. Rows or centroids too
// large for the bound, or a failed screen: every group. Eight lanes per point, four points per
// warp; bound by the centroid rows' loads (their latency, and L1 at two thirds of its rate; 13%
// of the sectors hit there), for which groups of 8 are read by
// the row (groups of 32 read as columns of a transposed copy took 135 us for 77824 points of 96
// dimensions against 2000 centroids, groups of 8 so 160, this 90). The whole call on 262144 such
// points: 3.57 ms with a screen matrix in memory, 0.60 now; 131072 points of 4 dimensions
// against 256 codewords 184 us, now 90.
constexpr int kArgminWarps = 8;
constexpr int kArgminRows = kArgminWarps * 4;  // points per block
struct CentsMax {
    uint32_t norm2_bits;  // largest |c|^2
    uint32_t lost_bits;   // largest |c - bf16(c)|
};
__global__ __launch_bounds__(kArgminWarps * 32) void k_group_argmin(
    const float* __restrict__ gmin, uint32_t G, const float* __restrict__ X, uint64_t row0,
    uint32_t rows, uint32_t d, const float* __restrict__ xnorm, const float* __restrict__ xlost,
    const float* __restrict__ cents, const float* __restrict__ cnorm,
    const CentsMax* __restrict__ cmax, uint32_t K, int vec, const int* __restrict__ tc_err,
    int32_t* __restrict__ assign, float* __restrict__ dis) {
    extern __shared__ __align__(16) float argmin_rows[];  // [kArgminRows][pitch]
    const int lane = threadIdx.x & 31, l8 = lane & 7;
    const uint32_t slot = threadIdx.x >> 3, w = blockIdx.x * kArgminRows + slot;
    const bool valid = w < rows;
    const uint64_t p = row0 + (valid ? w : 0u);
    const uint32_t pitch = ((d + 3u) & ~3u) + 4u;  // the four points of a warp in other banks
    float* x = argmin_rows + (uint64_t)slot * pitch;
    for (uint32_t t = l8; t < d; t += 8) x[t] = X[p * d + t];
    // the row's minima, 256 at a time (32 per lane): one read up to 2048 centroids
    const float4* gm = reinterpret_cast<const float4*>(gmin + (uint64_t)(valid ? w : 0u) * G);
    float4 v[8];
    auto fetch = [&](uint32_t i0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t i = i0 + 8 * u + l8;
            v[u] = i < G / 4 ? gm[i] : make_float4(FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX);
        }
    };
    float U = FLT_MAX;
    for (uint32_t i0 = 0; i0 < G / 4; i0 += 64) {
        fetch(i0);
#pragma unroll
        for (int u = 0; u < 8; ++u) U = fminf(U, fminf(fminf(v[u].x, v[u].y), fminf(v[u].z, v[u].w)));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) U = fminf(U, __shfl_xor_sync(0xffffffffu, U, o));
    const float xn = xnorm[valid ? w : 0u], xa = sqrtf(xn), dx = xlost[valid ? w : 0u];
    const float c2 = __uint_as_float(cmax->norm2_bits), ca = sqrtf(c2) * 1.0000005f;
    const float dc = __uint_as_float(cmax->lost_bits);
    const float E = dx * ca + (xa + dx) * dc +
                    (float)(d + 8) * 4.76837158203125e-07f * (xa + dx) * (ca + dc) +
                    4.76837158203125e-07f * (xn + c2) +
                    9.5367431640625e-07f * (0.5f * c2 + 1.01f * xa * ca) + 1e-30f;
    const bool all = *tc_err != 0 || !(xn < 1e36f) || !(c2 < 1e36f);
    const float thr = U + 2.0f * E * 1.00001f;
    __syncwarp();
    // the reference's scan: min starts at FLT_MAX, strict < in ascending id order (a value of
    // FLT_MAX is none: bidx 0 keeps it out)
    float best = FLT_MAX;
    uint32_t bidx = 0;
    const uint32_t groups = (K + 7) / 8;
    for (uint32_t i0 = 0; i0 < G / 4; i0 += 64) {
        if (G > 256) fetch(i0);
        uint32_t mask = 0;  // bit 4u + e: this lane's group 4 (i0 + 8u + l8) + e
#pragma unroll
        for (int u = 0; u < 8; ++u)
            mask |= ((all || v[u].x <= thr ? 1u : 0u) | (all || v[u].y <= thr ? 2u : 0u) |
                     (all || v[u].z <= thr ? 4u : 0u) | (all || v[u].w <= thr ? 8u : 0u)) << (4 * u);
        if (!valid) mask = 0;
        for (;;) {
            const unsigned left = __ballot_sync(0xffffffffu, mask != 0);
            if (left == 0) break;
            const unsigned team = (left >> (lane & 24)) & 255u;
            const int src = team ? __ffs(team) - 1 : 0;  // a lane of the point with a group
            const uint32_t theirs = __shfl_sync(0xffffffffu, mask, (lane & 24) + src);
            if (team == 0) continue;  // another point of the warp has one
            if (l8 == src) mask &= mask - 1;
            const uint32_t bit = __ffs(theirs) - 1;
            const uint32_t g = (i0 + 8 * (bit >> 2) + src) * 4 + (bit & 3), j = g * 8 + l8;
            if (g >= groups || j >= K) continue;
            const float* cj = cents + (uint64_t)j * d;
            float s = 0.0f;
            if (vec) {
                // 32 bytes per load: each of a warp's loads reads 32 rows, a line each
#pragma unroll 4
                for (uint32_t t = 0; t < d; t += 8) {
                    float y[8];
                    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                        : "=f"(y[0]), "=f"(y[1]), "=f"(y[2]), "=f"(y[3]), "=f"(y[4]), "=f"(y[5]),
                          "=f"(y[6]), "=f"(y[7])
                        : "l"(cj + t));
                    const float4 q0 = *reinterpret_cast<const float4*>(x + t);
                    const float4 q1 = *reinterpret_cast<const float4*>(x + t + 4);
                    s = __fadd_rn(s, __fmul_rn(q0.x, y[0]));
                    s = __fadd_rn(s, __fmul_rn(q0.y, y[1]));
                    s = __fadd_rn(s, __fmul_rn(q0.z, y[2]));
                    s = __fadd_rn(s, __fmul_rn(q0.w, y[3]));
                    s = __fadd_rn(s, __fmul_rn(q1.x, y[4]));
                    s = __fadd_rn(s, __fmul_rn(q1.y, y[5]));
                    s = __fadd_rn(s, __fmul_rn(q1.z, y[6]));
                    s = __fadd_rn(s, __fmul_rn(q1.w, y[7]));
                }
            } else if (d == 4 && (reinterpret_cast<uintptr_t>(cents) & 15) == 0) {
                const float4 y = __ldg(reinterpret_cast<const float4*>(cj));
                s = __fadd_rn(s, __fmul_rn(x[0], y.x));
                s = __fadd_rn(s, __fmul_rn(x[1], y.y));
                s = __fadd_rn(s, __fmul_rn(x[2], y.z));
                s = __fadd_rn(s, __fmul_rn(x[3], y.w));
            } else {
                for (uint32_t t = 0; t < d; ++t) s = __fadd_rn(s, __fmul_rn(x[t], __ldg(cj + t)));
            }
            const float cur = __fsub_rn(__fadd_rn(xn, cnorm[j]), 2.0f * s);
            if (cur < best || (cur == best && j < bidx)) {
                best = cur;
                bidx = j;
            }
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, bidx, o);
        if (ov < best || (ov == best && oi < bidx)) {
            best = ov;
            bidx = oi;
        }
    }
    if (valid && l8 == 0) {
        assign[p] = (int32_t)bidx;
        dis[p] = best;
    }
}

// The screen's bias 0.5|c|^2 (FLT_MAX past the centroids), and the largest norm and rounding
// loss (their bits: the order of non-negative floats; no number is above all).
__global__ void k_cents_bias(const float* __restrict__ cnorm, const float* __restrict__ clost,
                             uint32_t K, uint32_t n, float* __restrict__ bias,
                             CentsMax* __restrict__ cmax) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;  // n: whole blocks
    const float c = j < K ? cnorm[j] : 0.0f, l = j < K ? clost[j] : 0.0f;
    if (j < n) bias[j] = j < K ? 0.5f * c : FLT_MAX;
    const uint32_t mc = __reduce_max_sync(0xffffffffu, __float_as_uint(c));
    const uint32_t ml = __reduce_max_sync(0xffffffffu, __float_as_uint(l));
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&cmax->norm2_bits, mc);
        atomicMax(&cmax->lost_bits, ml);
    }
}

// nearest_center without the selecting screen (dimensions above its limit): one warp per
// point over the whole screen matrix.
// s^_j ~ 0.5|c_j|^2 - x.c_j orders the centroids like the reference's
// cur_j = (|x|^2 + |c_j|^2) - 2 x.c_j; the window around the screened minimum
// is recomputed exactly and the smallest cur_j with the lowest id wins, as in
// the reference's strict-< scan.
__global__ __launch_bounds__(256) void k_window_argmin(
    const float* __restrict__ approx, uint32_t ld, const float* __restrict__ X, uint64_t row0,
    uint32_t rows, uint32_t d, const float* __restrict__ cents, const float* __restrict__ cnorm,
    uint32_t K, const int* __restrict__ tc_err, int32_t* __restrict__ assign,
    float* __restrict__ dis) {
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= rows) return;
    const uint64_t p = row0 + w;
    const float* x = X + p * d;
    float xn = 0.0f;
    if (lane == 0) xn = dot_seq(x, x, d);
    xn = __shfl_sync(0xffffffffu, xn, 0);
    const bool screen = (*tc_err == 0);
    float U = FLT_MAX;
    const float* a = approx + (uint64_t)w * ld;
    const float eps = window_eps(d);
    const float xa = sqrtf(xn);
    if (screen) {
        for (uint32_t j = lane; j < K; j += 32) {
            const float s = a[j];
            const float cn = cnorm[j];
            const float e = eps * xa * sqrtf(cn) + 4.76837158203125e-07f * (xn + cn) +
                            9.5367431640625e-07f * fabsf(s) + 1e-30f;
            U = fminf(U, s + e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) U = fminf(U, __shfl_xor_sync(0xffffffffu, U, o));
    }
    // the reference's scan: min starts at FLT_MAX, strict < in ascending id order
    float best = FLT_MAX;
    uint32_t bidx = 0xFFFFFFFFu;
    for (uint32_t j = lane; j < K; j += 32) {
        if (screen) {
            const float s = a[j];
            const float cn = cnorm[j];
            const float e = eps * xa * sqrtf(cn) + 4.76837158203125e-07f * (xn + cn) +
                            9.5367431640625e-07f * fabsf(s) + 1e-30f;
            if (s - e > U) continue;
        }
        const float cur =
            __fsub_rn(__fadd_rn(xn, cnorm[j]), 2.0f * dot_seq(x, cents + (uint64_t)j * d, d));
        if (cur < best) {  // j ascends within a lane
            best = cur;
            bidx = j;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, bidx, o);
        if (ov < best || (ov == best && oi < bidx)) {
            best = ov;
            bidx = oi;
        }
    }
    if (lane == 0) {
        if (bidx == 0xFFFFFFFFu) {  // nothing below FLT_MAX: the reference keeps id 0
            best = FLT_MAX;
            bidx = 0;
        }
        assign[p] = (int32_t)bidx;
        dis[p] = best;
    }
}

__global__ void k_sqrt_norms(const float* __restrict__ half_norms, uint32_t n, float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = sqrtf(2.0f * half_norms[i]) * 1.0000005f;
}

__global__ void k_halve(const float* __restrict__ x, uint64_t n, float* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = 0.5f * x[i];
}

__global__ void k_norms_seq(const float* __restrict__ X, uint64_t rows, uint32_t d,
                            float* __restrict__ out) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r < rows) out[r] = dot_seq(X + r * d, X + r * d, d);
}

}  // namespace

size_t window_smem_bytes(uint32_t C, uint32_t d) {
    return (size_t)C * 4 + (size_t)(C + 1) * 8 + (size_t)d * 4 + 16 + (size_t)kWinCap * 8;
}

cudaError_t launch_abs_from_half_norms(const float* half_norms, uint32_t n, float* out,
                                       cudaStream_t stream) {
    k_sqrt_norms<<<(n + 255) / 256, 256, 0, stream>>>(half_norms, n, out);
    return cudaGetLastError();
}

cudaError_t launch_coarse_tc(const DeviceIndex& ix, uint32_t n, Scratch& s, cudaStream_t stream) {
    // with a probe, only the queries it left (s.ulist, their count s.ucount on the device)
    TcOperand A{nullptr, ix.d, 1, n, s.qb, s.ulist, s.ucount};
    TcOperand B{nullptr, ix.d, 1, ix.C, ix.coarse_bf16};
    TcEpilogue ep{};
    ep.mode = TC_EPI_SCORE;
    ep.out = s.dots;
    ep.ld = ix.C;
    ep.bias = ix.coarse_norms;
    return launch_tc_gemm(A, B, ix.d, ep, s.tc_err, stream);
}

cudaError_t launch_coarse_window(const DeviceIndex& ix, uint32_t n, Scratch& s,
                                 cudaStream_t stream) {
    if (s.Pfix <= kSmallP) {
        auto kern = s.Pfix == 1 ? k_window_small<1> : s.Pfix <= 4 ? k_window_small<4>
                                                                   : k_window_small<16>;
        kern<<<(n + 7) / 8, 256, 0, stream>>>(
            s.dots, ix.C, s.q, ix.d, s.qnorm, ix.coarse, ix.coarse_norms, ix.coarse_abs, ix.C,
            s.Pfix, s.P, n, s.cdist, s.ctag, s.status, s.tc_err, s.counters + kCounterWindowFallbacks,
            s.pconf, s.ulist, s.ucount);
        return cudaGetLastError();
    }
    const size_t smem = window_smem_bytes(ix.C, ix.d);
    ensure_max_dynamic_smem(k_window_topk, 200 * 1024);
    k_window_topk<<<n, kWinThreads, smem, stream>>>(s.dots, ix.C, s.q, ix.d, s.qnorm, ix.coarse,
                                                    ix.coarse_norms, ix.coarse_abs, ix.C, s.Pfix,
                                                    s.P, s.cdist, s.ctag, s.status, s.tc_err,
                                                    s.counters + kCounterWindowFallbacks, s.pconf,
                                                    s.ulist, s.ucount);
    return cudaGetLastError();
}

// nearest_center through the MINIMA screen (k_tc_filter) and k_group_argmin, in chunks whose
// BF16 rows and group minima stay in L2 between the kernels; a call allocates 50 MB beside the
// centroids' copies, more only above 0.75M centroids (a chunk has 128 rows at least, and a row
// half a byte of minima per centroid: 1 GB at the limit of 2^24).
static cudaError_t nearest_center_screened(uint32_t dim, const float* cents, uint32_t k, const float* x,
                                           uint64_t n, int32_t* assign, float* dis,
                                           cudaStream_t stream) {
    const uint32_t dp = (dim + 7u) & ~7u;
    const uint32_t tiles = (k + kTcFilterTile - 1) / kTcFilterTile, kp = tiles * kTcFilterTile;
    const uint32_t G = tiles * (kTcFilterTile / 8);
    // whole waves of 128-row tiles (one per SM) within 48 MiB of row scratch
    const uint64_t wave = 128ull * (uint64_t)sm_count();
    uint64_t chunk = (48ull << 20) / (2ull * dp + 8 + 4ull * G);
    chunk = chunk >= wave ? chunk / wave * wave : chunk >= 128 ? chunk / 128 * 128 : 128;
    if (chunk > n) chunk = n;
    // one allocation, 256-byte aligned parts
    uint64_t bytes = 0;
    auto part = [&](uint64_t size) {
        const uint64_t at = bytes;
        bytes += (size + 255) & ~255ull;
        return at;
    };
    const uint64_t o_flags = part(sizeof(CentsMax) + 4), o_cb = part(2ull * k * dp), o_cn = part(4ull * k),
                   o_cl = part(4ull * k), o_bias = part(4ull * kp),
                   o_xb = part(2ull * chunk * dp), o_xn = part(4ull * chunk), o_xl = part(4ull * chunk),
                   o_gm = part(4ull * chunk * G);
    uint8_t* base = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&base, bytes, stream);
    if (e != cudaSuccess) return e;
    CentsMax* cmax = reinterpret_cast<CentsMax*>(base + o_flags);
    int* err = reinterpret_cast<int*>(cmax + 1);
    uint16_t* cb = reinterpret_cast<uint16_t*>(base + o_cb);
    uint16_t* xb = reinterpret_cast<uint16_t*>(base + o_xb);
    auto f = [&](uint64_t at) { return reinterpret_cast<float*>(base + at); };
    e = cudaMemsetAsync(cmax, 0, sizeof(CentsMax) + 4, stream);
    if (e == cudaSuccess)
        e = launch_rows_bf16(cents, k, dim, dp, true, 0, cb, f(o_cn), f(o_cl), stream);
    if (e == cudaSuccess) {
        k_cents_bias<<<(kp + 255) / 256, 256, 0, stream>>>(f(o_cn), f(o_cl), k, kp, f(o_bias), cmax);
        e = cudaGetLastError();
    }
    const size_t smem = sizeof(float) * kArgminRows * (((dim + 3u) & ~3u) + 4u);  // <= 33 KB
    const int vec = dim % 8 == 0 && (reinterpret_cast<uintptr_t>(cents) & 31) == 0;
    for (uint64_t r0 = 0; e == cudaSuccess && r0 < n; r0 += chunk) {
        const uint32_t rows = (uint32_t)(n - r0 < chunk ? n - r0 : chunk);
        e = launch_rows_bf16(x + r0 * dim, rows, dim, dp, true, 0, xb, f(o_xn), f(o_xl), stream);
        TcFilter p{};
        p.M = rows;
        p.N = k;
        p.K = dim;
        p.bias = f(o_bias);
        p.pos1 = p.tiles = tiles;
        p.step = 1;
        p.gmin = f(o_gm);
        p.err = err;
        if (e == cudaSuccess) e = launch_tc_filter(kTcMinima, xb, dp, cb, dp, p, stream);
        if (e != cudaSuccess) break;
        k_group_argmin<<<(rows + kArgminRows - 1) / kArgminRows, kArgminWarps * 32, smem, stream>>>(
            f(o_gm), G, x, r0, rows, dim, f(o_xn), f(o_xl), cents, f(o_cn), cmax, k, vec, err, assign, dis);
        e = cudaGetLastError();
    }
    cudaFreeAsync(base, stream);
    return e;
}

cudaError_t launch_nearest_center_tc(uint32_t dim, const float* cents, uint64_t k, const float* x,
                                     uint64_t n, int32_t* assign, float* dis, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    // k below 2^24: the minima of a row stay below 8 MB
    if (tc_filter_applies(dim) && k < (1ull << 24))
        return nearest_center_screened(dim, cents, (uint32_t)k, x, n, assign, dis, stream);
    // screen buffer of at most 256 MiB: rows per chunk, a multiple of 128
    uint64_t chunk = (256ull << 20) / (4 * (k ? k : 1));
    chunk = chunk < 128 ? 128 : (chunk / 128) * 128;
    // the contraction's grid.y (row tiles of 128) is at most 65535
    if (chunk > 65535ull * 128) chunk = 65535ull * 128;
    if (chunk > n) chunk = n;
    float* cnorm = nullptr;
    float* half = nullptr;
    float* screen = nullptr;
    int* err = nullptr;
    cudaError_t e = cudaMallocAsync(&cnorm, sizeof(float) * k, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&half, sizeof(float) * k, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&screen, sizeof(float) * chunk * k, stream);
    if (e == cudaSuccess) e = cudaMallocAsync(&err, sizeof(int), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), stream);
    if (e == cudaSuccess) {
        k_norms_seq<<<(unsigned)((k + 255) / 256), 256, 0, stream>>>(cents, k, dim, cnorm);
        k_halve<<<(unsigned)((k + 255) / 256), 256, 0, stream>>>(cnorm, k, half);
        e = cudaGetLastError();
    }
    for (uint64_t r0 = 0; e == cudaSuccess && r0 < n; r0 += chunk) {
        const uint32_t rows = (uint32_t)(n - r0 < chunk ? n - r0 : chunk);
        TcOperand A{x + r0 * dim, dim, 1, rows};
        TcOperand B{cents, dim, 1, (uint32_t)k};
        TcEpilogue ep{};
        ep.mode = TC_EPI_SCORE;
        ep.out = screen;
        ep.ld = k;
        ep.bias = half;
        e = launch_tc_gemm(A, B, dim, ep, err, stream);
        if (e != cudaSuccess) break;
        k_window_argmin<<<(rows + 7) / 8, 256, 0, stream>>>(screen, (uint32_t)k, x, r0, rows, dim,
                                                           cents, cnorm, (uint32_t)k, err, assign,
                                                           dis);
        e = cudaGetLastError();
    }
    if (cnorm) cudaFreeAsync(cnorm, stream);
    if (half) cudaFreeAsync(half, stream);
    if (screen) cudaFreeAsync(screen, stream);
    if (err) cudaFreeAsync(err, stream);
    return e;
}

}  // namespace pgpu
