// Brute-force k nearest neighbours (squared L2) of a query batch over a base
// set, on the GPU: the training labels of the learned probe.
//
// Every (query, base) pair is screened on the tensor cores: s = 0.5|x|^2 - q.x
// (BF16 operands, FP32 accumulation), which orders the base like |q - x|^2. Per
// query the 64 smallest (s, id) are kept, then rescored in FP32 and the k best
// returned in ascending order. Candidates are exact as long as the true k-th
// neighbour's screened value is among the 64 smallest, i.e. except where more than
// 64 - k points lie within the screen's error of it.
//
// The screen's scores are not written out (k_tc_filter): the first kFirst columns go
// to the queries' lists whole, later ones only where the score is at or below the
// 64th smallest so far, in growing ranges (a range of twice the columns seen adds
// about 128 entries per query to a list of 2048). The ranges are spread over the whole
// base by tiles of 256 rows. A base in the order of its clusters still puts whole tiles
// below a query's threshold; the filter cuts a full part of a list back to its 64
// smallest. Dimensions above the filter's limit: launch_knn_dense, with the screen
// matrix in memory.
// 2048 queries of 96 dimensions over 1M points: 2.08 ms (3.5 in the order of their clusters),
// against 24.5 ms with the screen matrix in memory. The tensor filter's passes are 1.1 ms of it,
// the lists' merges 0.23.
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <numeric>

#include "device_common.cuh"
#include "pgpu_internal.h"

namespace pgpu {
namespace {

constexpr uint32_t kKC = 64;          // candidates per query
static_assert(kKC <= kTcFilterKeep, "a part keeps all of a query's candidates");
constexpr int kWarpsPerBlock = 8;

__global__ void k_half_sq_norms(const float* __restrict__ X, uint64_t rows, uint32_t d,
                                float* __restrict__ out) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const float* x = X + r * d;
    float s = 0.0f;
    for (uint32_t k = 0; k < d; ++k) s += x[k] * x[k];
    out[r] = 0.5f * s;
}

__global__ void k_knn_reset(float* __restrict__ cs, uint32_t* __restrict__ ci,
                            float* __restrict__ thr, uint32_t nq) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (uint64_t)nq * kKC) {
        cs[i] = FLT_MAX;
        ci[i] = kNoLabel;
    }
    if (i < nq) thr[i] = FLT_MAX;
}

// Sorts a warp's 128 (value, id) pairs ascending (4 per lane, bitonic over shared memory).
__device__ void warp_sort128(float* v, uint32_t* id) {
    const int lane = threadIdx.x & 31;
    for (uint32_t size = 2; size <= 128; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t t = lane + 32 * u;  // 64 compare-exchanges
                const uint32_t lo = 2 * t - (t & (stride - 1));
                const uint32_t hi = lo + stride;
                const float a = v[lo], b = v[hi];
                const uint32_t ia = id[lo], ib = id[hi];
                const bool gt = a > b || (a == b && ia > ib);
                if (gt == ((lo & size) == 0)) {
                    v[lo] = b;
                    v[hi] = a;
                    id[lo] = ib;
                    id[hi] = ia;
                }
            }
            __syncwarp();
        }
    }
}

// One warp per query row of the screen chunk S [rows][ld] (base ids base0 + j).
__global__ __launch_bounds__(kWarpsPerBlock * 32) void k_knn_merge(
    const float* __restrict__ S, uint32_t ld, uint32_t rows, uint32_t cols, uint32_t base0,
    float* __restrict__ cs, uint32_t* __restrict__ ci, float* __restrict__ thr) {
    __shared__ float bv[kWarpsPerBlock][2 * kKC];
    __shared__ uint32_t bi[kWarpsPerBlock][2 * kKC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarpsPerBlock + warp;
    if (row >= rows) return;
    float* v = bv[warp];
    uint32_t* id = bi[warp];
    float* rs = cs + (uint64_t)row * kKC;
    uint32_t* ri = ci + (uint64_t)row * kKC;
    for (int u = 0; u < 2; ++u) {
        v[lane + 32 * u] = rs[lane + 32 * u];
        id[lane + 32 * u] = ri[lane + 32 * u];
    }
    float t = thr[row];
    uint32_t nb = 0;  // new candidates in v[64 ..)
    const float* s = S + (uint64_t)row * ld;
    for (uint32_t j0 = 0; j0 < cols; j0 += 32) {
        const uint32_t j = j0 + lane;
        const float x = j < cols ? s[j] : FLT_MAX;
        unsigned b = __ballot_sync(0xffffffffu, x < t);
        if (b == 0) continue;
        if (nb + __popc(b) > kKC) {
            // merge: sort the 64 kept + the nb new ones, keep 64, tighten the threshold
            for (uint32_t e = kKC + nb + lane; e < 2 * kKC; e += 32) {
                v[e] = FLT_MAX;
                id[e] = kNoLabel;
            }
            __syncwarp();
            warp_sort128(v, id);
            t = v[kKC - 1];
            nb = 0;
            b = __ballot_sync(0xffffffffu, x < t);
            if (b == 0) continue;
        }
        if (x < t) {
            const uint32_t pos = kKC + nb + __popc(b & ((1u << lane) - 1));
            v[pos] = x;
            id[pos] = base0 + j;
        }
        nb += __popc(b);
        __syncwarp();
    }
    if (nb > 0) {
        for (uint32_t e = kKC + nb + lane; e < 2 * kKC; e += 32) {
            v[e] = FLT_MAX;
            id[e] = kNoLabel;
        }
        __syncwarp();
        warp_sort128(v, id);
        t = v[kKC - 1];
    }
    for (int u = 0; u < 2; ++u) {
        rs[lane + 32 * u] = v[lane + 32 * u];
        ri[lane + 32 * u] = id[lane + 32 * u];
    }
    if (lane == 0) thr[row] = t;
}

// The queries' lists merged into their 64 smallest (score, id), one warp per query; the
// 64th score becomes the threshold of the next range. A list is `parts` runs of at most
// seg entries, count[row][part] <= seg of them (count null: seg in each).
__global__ __launch_bounds__(kWarpsPerBlock * 32) void k_knn_lists(
    const uint2* __restrict__ cand, uint32_t cap, uint32_t parts, uint32_t seg,
    const uint32_t* __restrict__ count, uint32_t rows, float* __restrict__ cs,
    uint32_t* __restrict__ ci, float* __restrict__ thr) {
    __shared__ float bv[kWarpsPerBlock][2 * kKC];
    __shared__ uint32_t bi[kWarpsPerBlock][2 * kKC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarpsPerBlock + warp;
    if (row >= rows) return;
    float* v = bv[warp];
    uint32_t* id = bi[warp];
    float* rs = cs + (uint64_t)row * kKC;
    uint32_t* ri = ci + (uint64_t)row * kKC;
    for (int u = 0; u < 2; ++u) {
        v[lane + 32 * u] = rs[lane + 32 * u];
        id[lane + 32 * u] = ri[lane + 32 * u];
    }
    __syncwarp();
    float t = v[kKC - 1];
    uint32_t ti = id[kKC - 1];
    uint32_t nb = 0;  // new candidates in v[64 ..)
    auto merge = [&]() {
        for (uint32_t e = kKC + nb + lane; e < 2 * kKC; e += 32) {
            v[e] = FLT_MAX;
            id[e] = kNoLabel;
        }
        __syncwarp();
        warp_sort128(v, id);
        t = v[kKC - 1];
        ti = id[kKC - 1];
        nb = 0;
    };
    const uint2 none = make_uint2(__float_as_uint(FLT_MAX), kNoLabel);
    for (uint32_t p0 = 0; p0 < parts; p0 += 32) {
        // 32 parts' lengths at once
        uint32_t len = 0;
        if (p0 + lane < parts) len = count ? count[(uint64_t)row * parts + p0 + lane] : seg;
        const uint32_t np = parts - p0 < 32 ? parts - p0 : 32;
        // (the loads of two parts are under way while one is merged)
        auto head = [&](uint32_t u) {  // the first entries of part p0 + u
            const uint32_t n = __shfl_sync(0xffffffffu, len, u & 31);
            return u < np && (uint32_t)lane < n
                       ? cand[(uint64_t)row * cap + (uint64_t)(p0 + u) * seg + lane] : none;
        };
        uint2 ahead[2] = {head(0), head(1)};
        for (uint32_t u = 0; u < np; ++u) {
            const uint32_t n = __shfl_sync(0xffffffffu, len, u);
            const uint2* list = cand + (uint64_t)row * cap + (uint64_t)(p0 + u) * seg;
            uint2 c = ahead[0];
            ahead[0] = ahead[1];
            ahead[1] = head(u + 2);
            for (uint32_t e0 = 0; e0 < n; e0 += 32) {
                const uint2 next = e0 + 32 + lane < n ? list[e0 + 32 + lane] : none;
                const float x = __uint_as_float(c.x);
                auto smaller = [&]() { return x < t || (x == t && c.y < ti); };
                unsigned b = __ballot_sync(0xffffffffu, smaller());
                if (b != 0 && nb + __popc(b) > kKC) {
                    merge();
                    b = __ballot_sync(0xffffffffu, smaller());
                }
                if ((b >> lane) & 1u) {
                    const uint32_t pos = kKC + nb + __popc(b & ((1u << lane) - 1));
                    v[pos] = x;
                    id[pos] = c.y;
                }
                nb += __popc(b);
                __syncwarp();
                c = next;
            }
        }
    }
    if (nb > 0) merge();
    for (int u = 0; u < 2; ++u) {
        rs[lane + 32 * u] = v[lane + 32 * u];
        ri[lane + 32 * u] = id[lane + 32 * u];
    }
    if (lane == 0) thr[row] = t;
}

// FP32 rescoring of the 64 candidates, k best ascending (one warp per query).
__global__ __launch_bounds__(kWarpsPerBlock * 32) void k_knn_final(
    const float* __restrict__ base, uint32_t d, const float* __restrict__ Q, uint32_t rows,
    const uint32_t* __restrict__ ci, uint32_t k, int vec, uint32_t* __restrict__ out_ids,
    float* __restrict__ out_dist) {
    __shared__ float bv[kWarpsPerBlock][2 * kKC];
    __shared__ uint32_t bi[kWarpsPerBlock][2 * kKC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * kWarpsPerBlock + warp;
    if (row >= rows) return;
    float* v = bv[warp];
    uint32_t* id = bi[warp];
    const float* q = Q + (uint64_t)row * d;
    for (int u = 0; u < 4; ++u) {
        const uint32_t e = lane + 32 * u;
        uint32_t c = e < kKC ? ci[(uint64_t)row * kKC + e] : kNoLabel;
        float dist = FLT_MAX;
        if (c != kNoLabel) {
            const float* x = base + (uint64_t)c * d;
            float s = 0.0f;
            if (vec) {
#pragma unroll 4
                for (uint32_t t = 0; t < d; t += 4) {
                    const float4 y = __ldg(reinterpret_cast<const float4*>(x + t));
                    const float4 z = __ldg(reinterpret_cast<const float4*>(q + t));
                    const float d0 = z.x - y.x, d1 = z.y - y.y, d2 = z.z - y.z, d3 = z.w - y.w;
                    s += d0 * d0;
                    s += d1 * d1;
                    s += d2 * d2;
                    s += d3 * d3;
                }
            } else {
                for (uint32_t t = 0; t < d; ++t) {
                    const float df = q[t] - x[t];
                    s += df * df;
                }
            }
            dist = s;
        }
        v[e] = dist;
        id[e] = c;
    }
    __syncwarp();
    warp_sort128(v, id);
    for (uint32_t e = lane; e < k; e += 32) {
        out_ids[(uint64_t)row * k + e] = id[e];
        out_dist[(uint64_t)row * k + e] = v[e];
    }
}

// Rows read 16 bytes at a time.
int rows_vec(const float* a, const float* b, uint32_t d) {
    return d % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}

}  // namespace

static cudaError_t launch_knn_dense(const float* base, uint64_t n, uint32_t d, const float* Q,
                                    uint32_t nq, uint32_t k, uint32_t* ids, float* dist, int* err,
                                    cudaStream_t st) {
    if (k == 0 || k > kKC || n == 0 || nq == 0) return cudaErrorInvalidValue;
    constexpr uint32_t kQC = 8192, kBC = 16384;
    float *S = nullptr, *hb = nullptr, *cs = nullptr, *thr = nullptr;
    uint32_t* ci = nullptr;
    cudaError_t e = cudaMallocAsync(&S, sizeof(float) * kQC * kBC, st);
    if (e == cudaSuccess) e = cudaMallocAsync(&hb, sizeof(float) * n, st);
    if (e == cudaSuccess) e = cudaMallocAsync(&cs, sizeof(float) * kQC * kKC, st);
    if (e == cudaSuccess) e = cudaMallocAsync(&ci, sizeof(uint32_t) * kQC * kKC, st);
    if (e == cudaSuccess) e = cudaMallocAsync(&thr, sizeof(float) * kQC, st);
    if (e == cudaSuccess) {
        k_half_sq_norms<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(base, n, d, hb);
        e = cudaGetLastError();
    }
    for (uint32_t q0 = 0; e == cudaSuccess && q0 < nq; q0 += kQC) {
        const uint32_t qr = nq - q0 < kQC ? nq - q0 : kQC;
        k_knn_reset<<<(qr * kKC + 255) / 256, 256, 0, st>>>(cs, ci, thr, qr);
        for (uint64_t b0 = 0; e == cudaSuccess && b0 < n; b0 += kBC) {
            const uint32_t br = (uint32_t)(n - b0 < kBC ? n - b0 : kBC);
            TcEpilogue ep{};
            ep.mode = TC_EPI_SCORE;
            ep.out = S;
            ep.ld = kBC;
            ep.bias = hb + b0;
            e = launch_tc_gemm(TcOperand{Q + (uint64_t)q0 * d, d, 1, qr},
                               TcOperand{base + b0 * d, d, 1, br}, d, ep, err, st);
            if (e != cudaSuccess) break;
            k_knn_merge<<<(qr + kWarpsPerBlock - 1) / kWarpsPerBlock, kWarpsPerBlock * 32, 0, st>>>(
                S, kBC, qr, br, (uint32_t)b0, cs, ci, thr);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) break;
        k_knn_final<<<(qr + kWarpsPerBlock - 1) / kWarpsPerBlock, kWarpsPerBlock * 32, 0, st>>>(
            base, d, Q + (uint64_t)q0 * d, qr, ci, k, rows_vec(base, Q, d), ids + (uint64_t)q0 * k,
            dist + (uint64_t)q0 * k);
        e = cudaGetLastError();
    }
    if (S) cudaFreeAsync(S, st);
    if (hb) cudaFreeAsync(hb, st);
    if (cs) cudaFreeAsync(cs, st);
    if (ci) cudaFreeAsync(ci, st);
    if (thr) cudaFreeAsync(thr, st);
    return e;
}

cudaError_t launch_knn(const float* base, uint64_t n, uint32_t d, const float* Q, uint32_t nq,
                       uint32_t k, uint32_t* ids, float* dist, int* err, cudaStream_t st) {
    if (k == 0 || k > kKC || n == 0 || nq == 0) return cudaErrorInvalidValue;
    if (!tc_filter_applies(d)) return launch_knn_dense(base, n, d, Q, nq, k, ids, dist, err, st);
    constexpr uint32_t kQC = 8192, kFirst = 2048 / kTcFilterTile;
    const uint32_t dp = (d + 7u) & ~7u, qc = nq < kQC ? nq : kQC;
    // base rows held in BF16 at a time: 256 MiB, whole tiles
    uint64_t held = (256ull << 20) / (2ull * dp) / kTcFilterTile * kTcFilterTile;
    if (held > n) held = n;
    const uint64_t padded = (held + kTcFilterTile - 1) / kTcFilterTile * kTcFilterTile;
    // list entries per query: the first columns, or the least that each part takes
    auto cap_of = [](uint32_t rows) { return std::max(2048u, 2 * kTcFilterKeep * tc_filter_splits(rows)); };
    const uint32_t last = nq % kQC ? nq % kQC : qc;  // rows of the last chunk of queries
    uint64_t bytes = 0;
    auto part = [&](uint64_t size) {
        const uint64_t at = bytes;
        bytes += (size + 255) & ~255ull;
        return at;
    };
    const uint64_t o_xb = part(2 * held * dp), o_bias = part(4 * padded), o_qb = part(2ull * qc * dp),
                   o_qn = part(4ull * qc), o_cs = part(4ull * qc * kKC), o_ci = part(4ull * qc * kKC),
                   o_thr = part(4ull * qc),
                   o_cand = part(8 * std::max((uint64_t)qc * cap_of(qc), (uint64_t)last * cap_of(last))),
                   o_cnt = part(8 * std::max((uint64_t)qc * tc_filter_splits(qc),
                                             (uint64_t)last * tc_filter_splits(last)));
    uint8_t* mem = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&mem, bytes, st);
    if (e != cudaSuccess) return e;
    uint16_t* xb = reinterpret_cast<uint16_t*>(mem + o_xb);
    uint16_t* qb = reinterpret_cast<uint16_t*>(mem + o_qb);
    auto f = [&](uint64_t at) { return reinterpret_cast<float*>(mem + at); };
    auto u = [&](uint64_t at) { return reinterpret_cast<uint32_t*>(mem + at); };
    for (uint32_t q0 = 0; e == cudaSuccess && q0 < nq; q0 += kQC) {
        const uint32_t qr = nq - q0 < kQC ? nq - q0 : kQC;
        const unsigned blocks = (qr + kWarpsPerBlock - 1) / kWarpsPerBlock;
        e = launch_rows_bf16(Q + (uint64_t)q0 * d, qr, d, dp, false, 0, qb, f(o_qn), nullptr, st);
        if (e != cudaSuccess) break;
        k_knn_reset<<<(qr * kKC + 255) / 256, 256, 0, st>>>(f(o_cs), u(o_ci), f(o_thr), qr);
        uint64_t seen = 0;  // base rows screened
        for (uint64_t b0 = 0; e == cudaSuccess && b0 < n; b0 += held) {
            const uint64_t br = n - b0 < held ? n - b0 : held;
            const uint32_t tiles = (uint32_t)((br + kTcFilterTile - 1) / kTcFilterTile);
            if (q0 == 0 || n > held)
                e = launch_rows_bf16(base + b0 * d, br, d, dp, false, tiles * kTcFilterTile - (uint32_t)br,
                                     xb, f(o_bias), nullptr, st);
            TcFilter p{};
            p.M = qr;
            p.N = (uint32_t)br;
            p.K = d;
            p.bias = f(o_bias);
            p.tiles = tiles;
            // a stride near the golden section of the tiles, coprime to them
            p.step = (uint32_t)(tiles * 0.6180339887);
            if (p.step == 0) p.step = 1;
            while (std::gcd(p.step, tiles) != 1) ++p.step;
            p.thr = f(o_thr);
            p.count = u(o_cnt);
            p.cand = reinterpret_cast<uint2*>(mem + o_cand);
            p.cap = cap_of(qr);
            p.id0 = (uint32_t)b0;
            p.err = err;
            for (uint32_t pos = 0; e == cudaSuccess && pos < tiles;) {
                const bool first = seen == 0;
                const uint64_t room = first ? kFirst : 2 * (seen / kTcFilterTile);
                p.pos0 = pos;
                p.pos1 = tiles - pos < room ? tiles : pos + (uint32_t)room;
                e = launch_tc_filter(first ? kTcDense : kTcBelow, qb, dp, xb, dp, p, st);
                if (e != cudaSuccess) break;
                k_knn_lists<<<blocks, kWarpsPerBlock * 32, 0, st>>>(
                    p.cand, p.cap, first ? 1u : 2 * p.splits,
                    first ? (p.pos1 - pos) * kTcFilterTile : p.seg, first ? nullptr : p.count, qr,
                    f(o_cs), u(o_ci), f(o_thr));
                e = cudaGetLastError();
                seen += (uint64_t)(p.pos1 - pos) * kTcFilterTile;
                pos = p.pos1;
            }
        }
        if (e != cudaSuccess) break;
        k_knn_final<<<blocks, kWarpsPerBlock * 32, 0, st>>>(base, d, Q + (uint64_t)q0 * d, qr, u(o_ci), k, rows_vec(base, Q, d),
                                                            ids + (uint64_t)q0 * k, dist + (uint64_t)q0 * k);
        e = cudaGetLastError();
    }
    cudaFreeAsync(mem, st);
    return e;
}

}  // namespace pgpu
