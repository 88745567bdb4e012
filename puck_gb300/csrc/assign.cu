// pgpu_puck_assign: the build's encoder, PuckIndex::puck_assign
// (puck/puck/puck_index.cpp:602-709), for points whose cells are already known.
//
// Per point, in the reference's float order:
//   r = (x - coarse[c]) - fine[f]                     saxpy(-1) twice (:638-643)
//   per filter subspace k: code_k = nearest_center of r's slice over the 256
//     codewords (kmeans.cpp:221-258: (|r_k|^2 + |w|^2) - 2 r_k.w, first minimum
//     wins), then r_k -= w[code_k]                    (:649-679)
//   the second-level PQ (whether_pq) encodes what is left of r the same way
//   offset = 2 * sdot(decode(codes), vocab), vocab = coarse[c] + fine[f], and for
//     the second-level PQ vocab += the filter decode   (set_static_value_of_formula,
//     quantization.cpp:244-258)
// Every dot product sums sequentially from 0, one rounding per product and sum.
// The reference subtracts 2*dot in double after a float sum; that is one
// correctly rounded operation on two floats, so one float subtraction gives the
// same bits.
//
// Subspaces of up to 8 dimensions run in three kernels, parallel over what the float order
// leaves free:
//   k_encode      (point, subspace) pairs: a thread measures four points against the 256
//                 codewords of one subspace, which sit in shared memory and are read by
//                 broadcast; the second quantizer's residual is formed again from x, the
//                 cell and the filter code, so nothing but codes goes through memory;
//   k_encode_1d   a second quantizer of one-dimensional subspaces (the default): per value a
//                 search in the sorted codewords and the exact test of the few whose
//                 rounded distance can be the smallest, instead of all 256;
//   k_offsets     one thread per point: the two sequential offset sums.
// Wider subspaces: k_puck_assign, one warp per point, the 32 lanes splitting the codewords.
#include <cuda_runtime.h>

#include <cfloat>
#include <string>

#include "device_common.cuh"
#include "pgpu_internal.h"

namespace {

constexpr int kAssignWarps = 8;

__global__ void k_codeword_norms(const float* __restrict__ cb, uint64_t rows, uint32_t lsq,
                                 float* __restrict__ out) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r < rows) out[r] = pgpu::dot_seq(cb + r * lsq, cb + r * lsq, lsq);
}

struct AssignParams {
    const float* base;          // [n][d]
    const uint32_t* cell_assign;
    const float* coarse;        // [C][d]
    const float* fine;          // [F][d]
    const float* fcb;           // [fnsq][256][flsq]
    const float* fcb_norm;      // [fnsq][256]
    const float* pcb;           // [pnsq][256][plsq] (pnsq = 0: none)
    const float* pcb_norm;
    float* f_off;
    uint8_t* f_codes;           // [n][fnsq]
    float* p_off;
    uint8_t* p_codes;           // [n][pnsq]
    int* err;                   // set to 1 for a cell id out of range
    uint64_t n;
    uint32_t d, C, F, fnsq, flsq, pnsq, plsq, stride;  // stride: shared floats per warp
};

// One quantizer's pass over the residual r (shared memory); codes to cs (shared) and out.
__device__ void warp_encode(float* r, const float* __restrict__ cb, const float* __restrict__ cbn,
                            uint32_t nsq, uint32_t lsq, uint8_t* cs, uint8_t* out, int lane) {
    for (uint32_t k = 0; k < nsq; ++k) {
        float* s = r + (uint64_t)k * lsq;
        const float pn = pgpu::dot_seq(s, s, lsq);
        float best = FLT_MAX;
        uint32_t bi = 0;
        for (uint32_t c = lane; c < 256; c += 32) {  // ascending within a lane: first wins
            const float* w = cb + ((uint64_t)k * 256 + c) * lsq;
            float dt = 0.0f;
            for (uint32_t t = 0; t < lsq; ++t) dt = __fadd_rn(dt, __fmul_rn(s[t], __ldg(w + t)));
            const float cur = __fsub_rn(__fadd_rn(pn, __ldg(cbn + (uint64_t)k * 256 + c)), 2.0f * dt);
            if (cur < best) {
                best = cur;
                bi = c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov < best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            cs[k] = (uint8_t)bi;
            out[k] = (uint8_t)bi;
        }
        const float* w = cb + ((uint64_t)k * 256 + bi) * lsq;
        for (uint32_t t = lane; t < lsq; t += 32) s[t] = __fsub_rn(s[t], __ldg(w + t));
        __syncwarp();
    }
}

// 2 * sum_t decode(codes)[t] * v[t], sequential (lane 0 only).
__device__ float decode_dot(const float* __restrict__ cb, const uint8_t* cs, uint32_t lsq,
                            const float* v, uint32_t d) {
    float s = 0.0f;
    for (uint32_t t = 0; t < d; ++t) {
        const uint32_t k = t / lsq;
        const float dec = __ldg(cb + ((uint64_t)k * 256 + cs[k]) * lsq + (t - k * lsq));
        s = __fadd_rn(s, __fmul_rn(dec, v[t]));
    }
    return 2.0f * s;
}

__global__ __launch_bounds__(kAssignWarps * 32) void k_puck_assign(AssignParams p) {
    extern __shared__ float assign_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t i = (uint64_t)blockIdx.x * kAssignWarps + warp;
    if (i >= p.n) return;  // whole warps only; no block barrier follows
    const uint32_t d = p.d;
    float* r = assign_smem + (uint64_t)warp * p.stride;
    float* v = r + d;
    uint8_t* fcs = reinterpret_cast<uint8_t*>(v + d);
    uint8_t* pcs = fcs + p.fnsq;
    const uint32_t cell = p.cell_assign[i];
    if ((uint64_t)cell >= (uint64_t)p.C * p.F) {
        if (lane == 0) atomicExch(p.err, 1);
        return;
    }
    const uint32_t c = cell / p.F, f = cell % p.F;
    const float* x = p.base + i * d;
    const float* cv = p.coarse + (uint64_t)c * d;
    const float* fv = p.fine + (uint64_t)f * d;
    for (uint32_t t = lane; t < d; t += 32) r[t] = __fsub_rn(__fsub_rn(x[t], cv[t]), fv[t]);
    __syncwarp();
    warp_encode(r, p.fcb, p.fcb_norm, p.fnsq, p.flsq, fcs, p.f_codes + i * p.fnsq, lane);
    if (p.pnsq) warp_encode(r, p.pcb, p.pcb_norm, p.pnsq, p.plsq, pcs, p.p_codes + i * p.pnsq, lane);
    for (uint32_t t = lane; t < d; t += 32) v[t] = __fadd_rn(cv[t], fv[t]);
    __syncwarp();
    if (lane == 0) {
        p.f_off[i] = decode_dot(p.fcb, fcs, p.flsq, v, d);
        if (p.pnsq) {
            for (uint32_t t = 0; t < d; ++t) {
                const uint32_t k = t / p.flsq;
                v[t] = __fadd_rn(v[t], __ldg(p.fcb + ((uint64_t)k * 256 + fcs[k]) * p.flsq +
                                             (t - k * p.flsq)));
            }
            p.p_off[i] = decode_dot(p.pcb, pcs, p.plsq, v, d);
        }
    }
}

// Residual value of dimension t of point i in cell (c, f): x - coarse - fine, and for the
// second quantizer less the filter codeword's value.
template <bool SECOND>
__device__ __forceinline__ float residual(const AssignParams& p, uint64_t i, uint32_t c, uint32_t f,
                                          uint32_t t) {
    float r = __fsub_rn(__fsub_rn(__ldg(p.base + i * p.d + t), __ldg(p.coarse + (uint64_t)c * p.d + t)),
                        __ldg(p.fine + (uint64_t)f * p.d + t));
    if (SECOND) {
        const uint32_t fk = t / p.flsq;
        const uint32_t code = p.f_codes[i * p.fnsq + fk];
        r = __fsub_rn(r, __ldg(p.fcb + ((uint64_t)fk * 256 + code) * p.flsq + (t - fk * p.flsq)));
    }
    return r;
}

// Codes of subspace blockIdx.y. Bound by instruction issue: per (point, codeword) LSQ
// products, LSQ - 1 sums, (|r|^2 + |w|^2), the subtraction of 2 dot (one fused step: the
// doubling is exact, so it rounds once like the reference's) and one minimum. A thread
// measures four points against each broadcast codeword. The index is not carried along:
// codewords go in groups of 8, the first group that lowers the minimum is kept, and its 8
// values are formed once more to find the first that equals it. The residual slices are read
// 16 bytes at a time where the rows allow it (vec): read by the float, the loads took as long
// as the arithmetic. Packed f32x2 arithmetic has no higher rate here.
// 500k points, 24 subspaces of 4 and 96 one-dimensional second codes, the whole call: 42.0 ms
// with a warp per point, 2.67 with float loads of the slices, 2.29 now; the multiplies and
// adds alone are 0.7 ms of it at full rate.
constexpr int kEncThreads = 256;
constexpr int kEncPoints = 4;  // per thread
template <int LSQ, bool SECOND>
__global__ __launch_bounds__(kEncThreads) void k_encode(AssignParams p, int vec) {
    constexpr int STR = (LSQ + 4) / 4 * 4;  // floats per codeword: values, norm
    __shared__ __align__(16) float sw[256 * STR];
    const uint32_t k = blockIdx.y;
    const int tid = threadIdx.x;
    {
        const float* cb = (SECOND ? p.pcb : p.fcb) + ((uint64_t)k * 256 + tid) * LSQ;
#pragma unroll
        for (int t = 0; t < LSQ; ++t) sw[tid * STR + t] = __ldg(cb + t);
        sw[tid * STR + LSQ] = (SECOND ? p.pcb_norm : p.fcb_norm)[(uint64_t)k * 256 + tid];
    }
    __syncthreads();
    const uint64_t i0 = (uint64_t)blockIdx.x * (kEncThreads * kEncPoints) + tid;
    float s[kEncPoints][LSQ], pn[kEncPoints], best[kEncPoints];
    int grp[kEncPoints];
    bool ok[kEncPoints];
#pragma unroll
    for (int j = 0; j < kEncPoints; ++j) {
        const uint64_t i = i0 + (uint64_t)j * kEncThreads;
        bool in = i < p.n;
        const uint32_t cell = in ? p.cell_assign[i] : 0u;
        if ((uint64_t)cell >= (uint64_t)p.C * p.F) {
            atomicExch(p.err, 1);
            in = false;
        }
        ok[j] = in;
        const uint32_t c = cell / p.F, f = cell % p.F;
        if (!SECOND && LSQ % 4 == 0 && vec) {
#pragma unroll
            for (int t = 0; t < LSQ; t += 4) {
                const uint32_t at = k * LSQ + t;
                const float4 x = in ? __ldg(reinterpret_cast<const float4*>(p.base + i * p.d + at))
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 u = in ? __ldg(reinterpret_cast<const float4*>(p.coarse + (uint64_t)c * p.d + at))
                                    : x;
                const float4 v = in ? __ldg(reinterpret_cast<const float4*>(p.fine + (uint64_t)f * p.d + at))
                                    : x;
                s[j][t] = __fsub_rn(__fsub_rn(x.x, u.x), v.x);
                s[j][t + 1] = __fsub_rn(__fsub_rn(x.y, u.y), v.y);
                s[j][t + 2] = __fsub_rn(__fsub_rn(x.z, u.z), v.z);
                s[j][t + 3] = __fsub_rn(__fsub_rn(x.w, u.w), v.w);
            }
        } else {
#pragma unroll
            for (int t = 0; t < LSQ; ++t) s[j][t] = in ? residual<SECOND>(p, i, c, f, k * LSQ + t) : 0.0f;
        }
        pn[j] = pgpu::dot_seq(s[j], s[j], LSQ);
        best[j] = FLT_MAX;
        grp[j] = -1;
    }
    // (|r|^2 + |w|^2) - 2 r.w of point j and the codeword at w
    auto measure = [&](int j, const float (&w)[STR]) {
        float dt = __fmul_rn(s[j][0], w[0]);
#pragma unroll
        for (int t = 1; t < LSQ; ++t) dt = __fadd_rn(dt, __fmul_rn(s[j][t], w[t]));
        return __fmaf_rn(dt, -2.0f, __fadd_rn(pn[j], w[LSQ]));
    };
    auto codeword = [&](int c, float (&w)[STR]) {
#pragma unroll
        for (int t = 0; t < STR; t += 4) {
            const float4 v = *reinterpret_cast<const float4*>(&sw[c * STR + t]);
            w[t] = v.x;
            w[t + 1] = v.y;
            w[t + 2] = v.z;
            w[t + 3] = v.w;
        }
    };
#pragma unroll 1
    for (int g = 0; g < 32; ++g) {
        float gm[kEncPoints];
#pragma unroll
        for (int j = 0; j < kEncPoints; ++j) gm[j] = FLT_MAX;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            float w[STR];
            codeword(g * 8 + u, w);
#pragma unroll
            for (int j = 0; j < kEncPoints; ++j) gm[j] = fminf(gm[j], measure(j, w));
        }
#pragma unroll
        for (int j = 0; j < kEncPoints; ++j)
            if (gm[j] < best[j]) {
                best[j] = gm[j];
                grp[j] = g;
            }
    }
#pragma unroll
    for (int j = 0; j < kEncPoints; ++j) {
        if (!ok[j]) continue;
        uint32_t bi = 0;
        for (int u = 7; u >= 0 && grp[j] >= 0; --u) {  // the last match found is the first in order
            float w[STR];
            codeword(grp[j] * 8 + u, w);
            if (measure(j, w) == best[j]) bi = grp[j] * 8 + u;
        }
        const uint64_t i = i0 + (uint64_t)j * kEncThreads;
        if (SECOND) p.p_codes[i * p.pnsq + k] = (uint8_t)bi;
        else p.f_codes[i * p.fnsq + k] = (uint8_t)bi;
    }
}

// One-dimensional codewords of each subspace in ascending order (value, then index), their
// indexes, and whether any is too large (or not a number) for the search below.
__global__ __launch_bounds__(256) void k_sort_levels(const float* __restrict__ cb,
                                                     float* __restrict__ val, uint8_t* __restrict__ idx,
                                                     int* __restrict__ bad) {
    __shared__ float w[256];
    const int tid = threadIdx.x;
    const float x = cb[(uint64_t)blockIdx.x * 256 + tid];
    w[tid] = x;
    const int any = __syncthreads_or(!(fabsf(x) <= 1e18f));
    int rank = 0;
    for (int j = 0; j < 256; ++j) rank += (w[j] < x || (w[j] == x && j < tid)) ? 1 : 0;
    if (tid == 0) bad[blockIdx.x] = any;
    if (!any) {
        val[(uint64_t)blockIdx.x * 256 + rank] = x;
        idx[(uint64_t)blockIdx.x * 256 + rank] = (uint8_t)tid;
    }
}

// The second quantizer over one-dimensional subspaces. The reference takes the smallest
// cur_c = fl(fl(s^2 + w^2) - 2 fl(s w)), lowest index first; with u = 2^-24 each rounding is
// within u of its operands' size, |cur_c - (s - w)^2| <= 8 u (s^2 + w^2). So no codeword is
// the smallest whose (s - w)^2 less 16 u (s^2 + w^2) lies above a cur already found (twice
// the bound: the test is in floats too), and once |s - w| > 2^-18 |w| that difference only
// grows away from s: the scan from s's place in the sorted codewords stops there on each
// side, after two or three codewords in practice. A warp takes a point's 32 dimensions,
// block tiles of 32 dimensions keep the sorted codewords in shared memory (pitch 257: the
// first steps of the 32 searches read 32 banks). 500k x 96 values
// in 0.44 ms; all 256 distances of each would be 1.9 ms at full rate.
constexpr int k1dThreads = 512;
constexpr int k1dPitch = 257;
__global__ __launch_bounds__(k1dThreads) void k_encode_1d(AssignParams p, const float* __restrict__ val,
                                                          const uint8_t* __restrict__ idx,
                                                          const int* __restrict__ bad) {
    __shared__ float sv[32 * k1dPitch];
    __shared__ uint8_t si[32 * k1dPitch];
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t t0 = blockIdx.y * 32, nt = p.d - t0 < 32 ? p.d - t0 : 32;
    for (uint32_t e = tid; e < nt * 256; e += k1dThreads) {
        sv[(e >> 8) * k1dPitch + (e & 255)] = val[(uint64_t)t0 * 256 + e];
        si[(e >> 8) * k1dPitch + (e & 255)] = idx[(uint64_t)t0 * 256 + e];
    }
    __syncthreads();
    const uint32_t t = t0 + lane;
    const bool mine = (uint32_t)lane < nt;
    const bool slow = mine && bad[t] != 0;
    const float* w = sv + lane * k1dPitch;
    const uint8_t* wi = si + lane * k1dPitch;
    constexpr float kRel = 9.5367431640625e-07f;   // 2^-20 = 16 u
    constexpr float kFar = 3.814697265625e-06f;    // 2^-18
    constexpr float kTiny = 1e-36f;                // roundings of products below the normal range
    const uint64_t step = (uint64_t)gridDim.x * (k1dThreads / 32);
    for (uint64_t i = (uint64_t)blockIdx.x * (k1dThreads / 32) + (tid >> 5); i < p.n; i += step) {
        const uint32_t cell = p.cell_assign[i];
        if ((uint64_t)cell >= (uint64_t)p.C * p.F || !mine) continue;  // flagged by k_encode
        const float s = residual<true>(p, i, cell / p.F, cell % p.F, t);
        const float pn = __fmul_rn(s, s);
        float best = FLT_MAX;
        uint32_t bi = 0;
        if (slow || !(fabsf(s) <= 1e18f)) {
            for (uint32_t c = 0; c < 256; ++c) {
                const float y = __ldg(p.pcb + (uint64_t)t * 256 + c);
                const float cur = __fsub_rn(__fadd_rn(pn, __fmul_rn(y, y)), 2.0f * __fmul_rn(s, y));
                if (cur < best) {
                    best = cur;
                    bi = c;
                }
            }
        } else {
            uint32_t pos = 0;  // codewords below s, at most 255
#pragma unroll
            for (int b = 128; b > 0; b >>= 1)
                if (w[pos + b - 1] < s) pos += b;
            bi = 256;
            auto take = [&](int j) {  // false: no codeword further out can be the smallest
                const float y = w[j];
                const float yn = __fmul_rn(y, y), dd = fabsf(s - y);
                if (dd > kFar * fabsf(y) && dd * dd - kRel * (dd * dd + pn + yn) - kTiny > best)
                    return false;
                const float cur = __fsub_rn(__fadd_rn(pn, yn), 2.0f * __fmul_rn(s, y));
                const uint32_t c = wi[j];
                if (cur < best || (cur == best && c < bi)) {
                    best = cur;
                    bi = c;
                }
                return true;
            };
            for (int j = (int)pos; j < 256; ++j)
                if (!take(j)) break;
            for (int j = (int)pos - 1; j >= 0; --j)
                if (!take(j)) break;
        }
        p.p_codes[i * p.pnsq + t] = (uint8_t)bi;
    }
}

// The offsets of a point, one thread each: 2 * sum_t decode(codes)[t] * vocab[t] with vocab =
// coarse + fine, and for the second quantizer its decode against vocab + filter decode, the
// sums sequential in t.
__global__ __launch_bounds__(128) void k_offsets(AssignParams p, int vec) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const uint32_t cell = p.cell_assign[i];
    if ((uint64_t)cell >= (uint64_t)p.C * p.F) return;
    const float* cv = p.coarse + (uint64_t)(cell / p.F) * p.d;
    const float* fv = p.fine + (uint64_t)(cell % p.F) * p.d;
    const uint8_t* fc = p.f_codes + i * p.fnsq;
    const uint8_t* pc = p.p_codes + i * p.pnsq;
    float a = 0.0f, b = 0.0f;
    if (vec) {
        // four dimensions per step: d % 4 == 0, four-dimensional filter subspaces,
        // 16-byte aligned centroids and codewords, one-dimensional second subspaces
        for (uint32_t t = 0; t < p.d; t += 4) {
            const float4 c4 = __ldg(reinterpret_cast<const float4*>(cv + t));
            const float4 f4 = __ldg(reinterpret_cast<const float4*>(fv + t));
            const float4 w4 = __ldg(reinterpret_cast<const float4*>(p.fcb) +
                                    (uint64_t)(t >> 2) * 256 + fc[t >> 2]);
            const float v[4] = {__fadd_rn(c4.x, f4.x), __fadd_rn(c4.y, f4.y), __fadd_rn(c4.z, f4.z),
                                __fadd_rn(c4.w, f4.w)};
            const float w[4] = {w4.x, w4.y, w4.z, w4.w};
            float y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                y[u] = p.pnsq ? __ldg(p.pcb + (uint64_t)(t + u) * 256 + pc[t + u]) : 0.0f;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a = __fadd_rn(a, __fmul_rn(w[u], v[u]));
                b = __fadd_rn(b, __fmul_rn(y[u], __fadd_rn(v[u], w[u])));
            }
        }
    } else {
        for (uint32_t t = 0; t < p.d; ++t) {
            const float v = __fadd_rn(__ldg(cv + t), __ldg(fv + t));
            const uint32_t k = t / p.flsq;
            const float w = __ldg(p.fcb + ((uint64_t)k * 256 + fc[k]) * p.flsq + (t - k * p.flsq));
            a = __fadd_rn(a, __fmul_rn(w, v));
            if (p.pnsq) {
                const uint32_t m = t / p.plsq;
                const float y = __ldg(p.pcb + ((uint64_t)m * 256 + pc[m]) * p.plsq + (t - m * p.plsq));
                b = __fadd_rn(b, __fmul_rn(y, __fadd_rn(v, w)));
            }
        }
    }
    p.f_off[i] = 2.0f * a;
    if (p.pnsq) p.p_off[i] = 2.0f * b;
}

template <bool SECOND>
void launch_encode(const AssignParams& p, uint32_t nsq, uint32_t lsq, int vec, cudaStream_t st) {
    constexpr uint32_t per = kEncThreads * kEncPoints;
    const dim3 grid((unsigned)((p.n + per - 1) / per), nsq);
    switch (lsq) {
#define PGPU_ENC(L) \
    case L:         \
        k_encode<L, SECOND><<<grid, kEncThreads, 0, st>>>(p, vec); \
        break;
        PGPU_ENC(1) PGPU_ENC(2) PGPU_ENC(3) PGPU_ENC(4) PGPU_ENC(5) PGPU_ENC(6) PGPU_ENC(7) PGPU_ENC(8)
#undef PGPU_ENC
    }
}

}  // namespace

extern "C" int pgpu_puck_assign(uint32_t d, uint64_t n, const float* base,
                                const uint32_t* cell_assign, const float* coarse, uint32_t C,
                                const float* fine, uint32_t F, const float* filter_codebook,
                                uint32_t filter_nsq, const float* pq_codebook, uint32_t pq_nsq,
                                float* filter_offsets, uint8_t* filter_codes, float* pq_offsets,
                                uint8_t* pq_codes, void* stream) {
    if (d == 0 || C == 0 || F == 0 || filter_nsq == 0 || base == nullptr || cell_assign == nullptr ||
        coarse == nullptr || fine == nullptr || filter_codebook == nullptr ||
        filter_offsets == nullptr || filter_codes == nullptr ||
        (pq_nsq > 0 && (pq_codebook == nullptr || pq_offsets == nullptr || pq_codes == nullptr)))
        return pgpu::set_last_error(PGPU_E_INVALID, "invalid argument");
    if (d % filter_nsq != 0 || (pq_nsq > 0 && d % pq_nsq != 0))
        return pgpu::set_last_error(PGPU_E_UNSUPPORTED, "feature_dim must be a multiple of nsq");
    if (d > pgpu::kMaxDim)
        return pgpu::set_last_error(PGPU_E_LIMIT, "feature_dim above the supported limit");
    if ((uint64_t)C * F > 0xFFFFFFFFull)
        return pgpu::set_last_error(PGPU_E_LIMIT, "more than 2^32-1 cells");
    if (n == 0) return PGPU_OK;
    cudaStream_t st = (cudaStream_t)stream;
    AssignParams p;
    p.base = base;
    p.cell_assign = cell_assign;
    p.coarse = coarse;
    p.fine = fine;
    p.fcb = filter_codebook;
    p.pcb = pq_codebook;
    p.f_off = filter_offsets;
    p.f_codes = filter_codes;
    p.p_off = pq_offsets;
    p.p_codes = pq_codes;
    p.n = n;
    p.d = d;
    p.C = C;
    p.F = F;
    p.fnsq = filter_nsq;
    p.flsq = d / filter_nsq;
    p.pnsq = pq_nsq;
    p.plsq = pq_nsq ? d / pq_nsq : 0;
    // residual and vocab floats, then the two code rows, rounded up to whole floats
    p.stride = 2 * d + (filter_nsq + pq_nsq + 3) / 4;
    const size_t smem = sizeof(float) * kAssignWarps * p.stride;  // <= 72 KB (d <= kMaxDim)
    const uint64_t nnorm = (uint64_t)(filter_nsq + pq_nsq) * 256;
    // subspaces of at most 8 dimensions (every shape of the configurations): the kernels
    // that are parallel over subspaces, 2.29 ms against 42.0 on 500k points of 96 dimensions
    const bool split = p.flsq <= 8 && p.plsq <= 8;
    const bool sorted = split && pq_nsq && p.plsq == 1;
    float* norms = nullptr;
    int* err = nullptr;
    cudaError_t e = cudaMallocAsync(
        (void**)&norms,
        sizeof(float) * nnorm + sizeof(int) + (sorted ? d * (256ull * 5 + sizeof(int)) : 0), st);
    if (e != cudaSuccess)
        return pgpu::set_last_error(e == cudaErrorMemoryAllocation ? PGPU_E_NOMEM : PGPU_E_CUDA,
                                    std::string("puck_assign scratch: ") + cudaGetErrorString(e));
    err = reinterpret_cast<int*>(norms + nnorm);
    p.fcb_norm = norms;
    p.pcb_norm = norms + (uint64_t)filter_nsq * 256;
    p.err = err;
    pgpu::ensure_max_dynamic_smem(k_puck_assign, 100 * 1024);
    e = cudaMemsetAsync(err, 0, sizeof(int), st);
    if (e == cudaSuccess) {
        k_codeword_norms<<<(unsigned)((filter_nsq * 256ull + 255) / 256), 256, 0, st>>>(
            filter_codebook, filter_nsq * 256ull, p.flsq, norms);
        if (pq_nsq)
            k_codeword_norms<<<(unsigned)((pq_nsq * 256ull + 255) / 256), 256, 0, st>>>(
                pq_codebook, pq_nsq * 256ull, p.plsq, norms + (uint64_t)filter_nsq * 256);
        if (split) {
            const auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
            const bool rows = d % 4 == 0 && aligned(coarse) && aligned(fine);
            launch_encode<false>(p, filter_nsq, p.flsq, rows && aligned(base), st);
            if (sorted) {
                int* bad = err + 1;
                float* val = reinterpret_cast<float*>(bad + d);
                uint8_t* idx = reinterpret_cast<uint8_t*>(val + (uint64_t)d * 256);
                k_sort_levels<<<d, 256, 0, st>>>(pq_codebook, val, idx, bad);
                const uint64_t want = (n + k1dThreads / 32 - 1) / (k1dThreads / 32);
                const dim3 grid((unsigned)(want < 2048 ? want : 2048), (d + 31) / 32);
                k_encode_1d<<<grid, k1dThreads, 0, st>>>(p, val, idx, bad);
            } else if (pq_nsq) {
                launch_encode<true>(p, pq_nsq, p.plsq, 0, st);
            }
            const int vec = rows && p.flsq == 4 && p.plsq <= 1 && aligned(filter_codebook);
            k_offsets<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(p, vec);
        } else {
            k_puck_assign<<<(unsigned)((n + kAssignWarps - 1) / kAssignWarps), kAssignWarps * 32, smem,
                            st>>>(p);
        }
        e = cudaGetLastError();
    }
    int flag = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&flag, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(norms, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return pgpu::set_last_error(PGPU_E_CUDA, std::string("puck_assign: ") + cudaGetErrorString(e));
    if (flag) return pgpu::set_last_error(PGPU_E_INVALID, "cell_assign entry out of range");
    return PGPU_OK;
}
