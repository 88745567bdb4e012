// Learned probe predictor: a small MLP (query -> coarse-cluster scores) trained
// and evaluated on the GPU with the BF16 tensor-core contraction (tc_gemm.cu).
//
//   H1 = GELU(X W1^T + b1)      X [n][d],  W1 [h][d]
//   H2 = GELU(H1 W2^T + b2)     W2 [h][h]
//   Z  = H2 W3^T + b3           W3 [C][h]  (scores of the C coarse clusters)
//
// Training target of a query: the distribution of the coarse clusters that hold
// its exact top-L neighbours (L ids per query, kNoLabel for none); the loss is
// the softmax cross-entropy against it, mean over the batch; Adam on FP32
// master weights. Every GEMM of the forward and backward passes runs on the
// tensor cores in BF16 with FP32 accumulation; softmax, bias gradients and the
// optimizer are FP32 CUDA kernels.
//
// The GEMMs of a training step read BF16 copies, row-major along the contraction, so
// that the operands arrive by TMA and are rounded once instead of once per tile. Each
// product's epilogue is a plain store; k_prep reads it once and writes what follows from
// it: the activation or the gradient through it, in BF16 as it stands and transposed (for
// the weight gradients, which contract over the batch). No product splits its K range: the
// sums keep one order, and Adam makes much of a gradient's last bits (its own sums are
// fused one way for the same reason). A step of 2048 queries,
// 96 -> 512 -> 512 -> 4000, takes 0.31 ms; with operands rounded in every tile, strided
// transposed reads and column sums by one thread per column it took 1.42. What is left: the
// contractions 0.12 (64 bytes per cycle and SM of operands), the copies 0.05, softmax and
// column sums 0.02 each, the rest launches.
//
// Search with a probe attached (scan mode): per query the clusters are taken in
// descending predicted probability until their mass reaches `mass` (adaptive
// search_coarse_count); when max_probe clusters do not reach it, the query keeps
// the plain fixed-count coarse selection (confidence fallback). The coarse
// distance of a chosen cluster is the reference's exact FP32 value.
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <initializer_list>

#include "device_common.cuh"
#include "pgpu_internal.h"
#include "tc_common.cuh"

namespace pgpu {
namespace {

constexpr int kProbeThreads = 256;

uint32_t round8(uint32_t v) { return (v + 7u) & ~7u; }

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// uniform(-a, a) from a counter-based hash: deterministic for a seed
__global__ void k_init_uniform(float* __restrict__ w, uint64_t n, float a, uint64_t seed) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t r = splitmix64(seed * 0x100000001B3ull + i);
    const float u = (float)(r >> 40) * (1.0f / 16777216.0f);  // [0, 1)
    w[i] = (2.0f * u - 1.0f) * a;
}

// Per row: softmax of the scores, the soft target from the row's label ids, the
// row loss, and dZ = (softmax - target) / n in place of the scores.
__global__ __launch_bounds__(kProbeThreads) void k_softmax_xent(
    float* __restrict__ Z, uint32_t C, const uint32_t* __restrict__ labels, uint32_t L,
    uint32_t n, float* __restrict__ row_loss) {
    __shared__ float red[2][kProbeThreads / 32];
    __shared__ uint32_t nvalid;
    const uint32_t row = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* z = Z + (uint64_t)row * C;
    const uint32_t* lab = labels + (uint64_t)row * L;
    float m = -FLT_MAX;
#pragma unroll 8
    for (uint32_t c = tid; c < C; c += kProbeThreads) m = fmaxf(m, z[c]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[0][warp] = m;
    if (warp == 0) {
        uint32_t valid = 0;
        for (uint32_t t = lane; t < L; t += 32) valid += lab[t] < C;
        valid = __reduce_add_sync(0xffffffffu, valid);
        if (lane == 0) nvalid = valid;
    }
    __syncthreads();
    m = red[0][0];
    for (int w = 1; w < kProbeThreads / 32; ++w) m = fmaxf(m, red[0][w]);
    float s = 0.0f;
#pragma unroll 8
    for (uint32_t c = tid; c < C; c += kProbeThreads) s += expf(z[c] - m);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[1][warp] = s;
    __syncthreads();
    s = 0.0f;
    for (int w = 0; w < kProbeThreads / 32; ++w) s += red[1][w];
    const float lse = m + logf(s);
    const float w = nvalid ? 1.0f / (float)nvalid : 0.0f;
    const float inv_n = 1.0f / (float)n;
    if (warp == 0) {
        float l = 0.0f;  // the same in every lane: the labels' terms in their order
        for (uint32_t t0 = 0; t0 < L; t0 += 32) {
            const uint32_t c = t0 + lane < L ? lab[t0 + lane] : C;
            const float zc = c < C ? z[c] : 0.0f;
            for (uint32_t t = 0; t < 32 && t0 + t < L; ++t) {
                const float zt = __shfl_sync(0xffffffffu, zc, t);
                if (__shfl_sync(0xffffffffu, c, t) < C) l += w * (lse - zt);
            }
        }
        if (lane == 0) row_loss[row] = l * inv_n;
    }
    __syncthreads();  // the labels' scores are read
#pragma unroll 8
    for (uint32_t c = tid; c < C; c += kProbeThreads) z[c] = expf(z[c] - lse) * inv_n;
    __syncthreads();
    // a repeated label's decrements are taken in turn, by the thread of its first place
    for (uint32_t t = tid; t < L; t += kProbeThreads) {
        const uint32_t c = lab[t];
        bool first = c < C;
        for (uint32_t u = 0; first && u < t; ++u) first = lab[u] != c;
        if (!first) continue;
        float g = z[c];
        for (uint32_t u = t; u < L; ++u)
            if (lab[u] == c) g -= w * inv_n;
        z[c] = g;
    }
}

// One matrix of k_prep: v[i][j] = f(src[i][j]), rows x cols.
enum { kPrepCopy = 0, kPrepGelu = 1, kPrepGeluBwd = 2 };
struct PrepJob {
    const float* src;
    uint32_t rows, cols;
    int f;              // GELU: gelu(src + bias[j]); GELU_BWD: src * gelu'(pre[i][j] + bias[j])
    const float* bias;
    const float* pre;
    uint16_t* out;      // BF16 [rows][ld], columns cols..ld zero, or null
    uint32_t ld;
    uint16_t* outT;     // BF16 [cols][ldT], columns rows..ldT zero, or null
    uint32_t ldT;
    float* v32;         // v in FP32, or null
};
struct PrepJobs {
    PrepJob j[4];
    uint32_t end[4];    // first block past each job
};

// Bound by memory: 64 x 64 tiles, each value read once; both BF16 forms are written as
// pairs, 128 bytes per warp, the transposed one through shared memory.
constexpr uint32_t kPrepTile = 64;
__global__ __launch_bounds__(kProbeThreads) void k_prep(const __grid_constant__ PrepJobs jobs) {
    constexpr uint32_t T = kPrepTile, kW = kProbeThreads / 32;
    __shared__ __align__(4) uint16_t tile[T][T + 2];  // [column][row]
    uint32_t k = 0;
    while (blockIdx.x >= jobs.end[k]) ++k;
    const PrepJob& J = jobs.j[k];
    const uint32_t blk = blockIdx.x - (k ? jobs.end[k - 1] : 0u), tc = (J.cols + T - 1) / T;
    const uint32_t r0 = blk / tc * T, c0 = blk % tc * T;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ja = c0 + lane * 2;
    const bool in[2] = {ja < J.cols, ja + 1 < J.cols};
    float bias[2] = {0.0f, 0.0f};
    if (J.f != kPrepCopy)
        for (int u = 0; u < 2; ++u)
            if (in[u]) bias[u] = J.bias[ja + u];
    float v[T / kW][2], pre[T / kW][2];
#pragma unroll
    for (uint32_t a = 0; a < T / kW; ++a) {
        const uint32_t i = r0 + warp + a * kW;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool ok = in[u] && i < J.rows;
            const uint64_t at = (uint64_t)i * J.cols + ja + u;
            v[a][u] = ok ? J.src[at] : 0.0f;
            pre[a][u] = ok && J.f == kPrepGeluBwd ? J.pre[at] : 0.0f;
        }
    }
#pragma unroll
    for (uint32_t a = 0; a < T / kW; ++a) {
        const uint32_t il = warp + a * kW, i = r0 + il;
        uint16_t h[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float x = v[a][u];
            if (in[u] && i < J.rows) {
                if (J.f == kPrepGelu) x = gelu_f(x + bias[u]);
                if (J.f == kPrepGeluBwd) x *= gelu_grad_f(pre[a][u] + bias[u]);
                if (J.v32 != nullptr) J.v32[(uint64_t)i * J.cols + ja + u] = x;
            }
            h[u] = __bfloat16_as_ushort(__float2bfloat16_rn(x));
            tile[lane * 2 + u][il] = h[u];
        }
        if (J.out != nullptr && i < J.rows && ja < J.ld)  // ld and ja are even
            *reinterpret_cast<uint32_t*>(J.out + (uint64_t)i * J.ld + ja) = h[0] | ((uint32_t)h[1] << 16);
    }
    __syncthreads();
    if (J.outT != nullptr) {
        const uint32_t i = r0 + lane * 2;
#pragma unroll
        for (uint32_t a = 0; a < T / kW; ++a) {
            const uint32_t jl = warp + a * kW, j = c0 + jl;
            if (j < J.cols && i < J.ldT)
                *reinterpret_cast<uint32_t*>(J.outT + (uint64_t)j * J.ldT + i) =
                    *reinterpret_cast<const uint32_t*>(&tile[jl][lane * 2]);
        }
    }
}

cudaError_t launch_prep(const PrepJob* job, int count, cudaStream_t st) {
    PrepJobs p{};
    uint32_t blocks = 0;
    for (int k = 0; k < 4; ++k) {
        if (k < count) {
            p.j[k] = job[k];
            blocks += ((job[k].rows + kPrepTile - 1) / kPrepTile) *
                      ((job[k].cols + kPrepTile - 1) / kPrepTile);
        }
        p.end[k] = blocks;
    }
    k_prep<<<blocks, kProbeThreads, 0, st>>>(p);
    return cudaGetLastError();
}

// out[j] = sum_i G[i][j] (bias gradients) for up to three matrices of the same rows. Bound by
// latency: a column's sum is a chain of FP32 additions in row order. A block takes 32 columns;
// all its warps load the next rows while one adds the rows at hand out of shared memory.
// One more block adds up the rows' losses, in a fixed order.
struct ColsumJobs {
    const float* G[3];
    float* out[3];
    uint32_t cols[3], end[3];
};
constexpr uint32_t kColsumRows = 128;
__global__ __launch_bounds__(kProbeThreads) void k_colsum(const __grid_constant__ ColsumJobs p,
                                                          uint32_t rows,
                                                          const float* __restrict__ row_loss,
                                                          float* __restrict__ loss_sum) {
    constexpr uint32_t kW = kProbeThreads / 32, kPer = kColsumRows / kW;
    __shared__ float buf[2][kColsumRows][32];
    uint32_t k = 0;
    if (blockIdx.x == p.end[2]) {  // the batch's loss: threads' sums, then theirs in pairs
        float* part = &buf[0][0][0];
        float s = 0.0f;
        for (uint32_t i = threadIdx.x; i < rows; i += kProbeThreads) s += row_loss[i];
        part[threadIdx.x] = s;
        for (uint32_t o = kProbeThreads / 2; o > 0; o >>= 1) {
            __syncthreads();
            if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        }
        if (threadIdx.x == 0) *loss_sum = part[0];
        return;
    }
    while (blockIdx.x >= p.end[k]) ++k;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cols = p.cols[k];
    const uint32_t j = (blockIdx.x - (k ? p.end[k - 1] : 0u)) * 32 + lane;
    const float* G = p.G[k] + j;
    float v[kPer];
    auto fetch = [&](uint32_t r0) {
#pragma unroll
        for (uint32_t a = 0; a < kPer; ++a) {
            const uint32_t r = r0 + warp + a * kW;
            v[a] = j < cols && r < rows ? G[(uint64_t)r * cols] : 0.0f;
        }
    };
    fetch(0);
    float s = 0.0f;
    for (uint32_t r0 = 0, b = 0; r0 < rows; r0 += kColsumRows, b ^= 1u) {
#pragma unroll
        for (uint32_t a = 0; a < kPer; ++a) buf[b][warp + a * kW][lane] = v[a];
        __syncthreads();  // the other buffer's rows were added before this barrier's arrival
        if (r0 + kColsumRows < rows) fetch(r0 + kColsumRows);
        if (warp == 0) {
            const uint32_t m = min(kColsumRows, rows - r0);
            if (m == kColsumRows) {
#pragma unroll 16
                for (uint32_t r = 0; r < kColsumRows; ++r) s += buf[b][r][lane];
            } else {
                for (uint32_t r = 0; r < m; ++r) s += buf[b][r][lane];
            }
        }
    }
    if (warp == 0 && j < cols) p.out[k][j] = s;
}

__global__ void k_to_bf16(const float* __restrict__ x, uint64_t n, uint16_t* __restrict__ y) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __bfloat16_as_ushort(__float2bfloat16_rn(x[i]));
}

// Adam; the weights' BF16 copies lie in the parameters' order without the biases: weights
// end at e1, e2 and e3, each matrix followed by its bias (h values after the first two).
__global__ __launch_bounds__(kProbeThreads) void k_adam(
    float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
    float* __restrict__ v, uint64_t n, float lr, float b1, float b2, float eps, float c1, float c2,
    uint16_t* __restrict__ wb, uint64_t e1, uint64_t e2, uint64_t e3, uint32_t h) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = fmaf(1.0f - b1, gi, __fmul_rn(b1, m[i]));
    const float vi = fmaf((1.0f - b2) * gi, gi, __fmul_rn(b2, v[i]));
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    const uint16_t hw = __bfloat16_as_ushort(__float2bfloat16_rn(wi));
    if (i < e1)
        wb[i] = hw;
    else if (i >= e1 + h && i < e2)
        wb[i - h] = hw;
    else if (i >= e2 + h && i < e3)
        wb[i - 2ull * h] = hw;
}

// Adaptive cluster choice from the probe's scores (see the file comment). Rows
// that the probe answers get their clusters in ctag/cdist [n][Pcap] (unused slots
// kNoLabel) and pconf = 1; the others get pconf = 0 and are left to the
// fixed-count selection.
__global__ __launch_bounds__(kProbeThreads) void k_probe_select(
    const float* __restrict__ Z, uint32_t C, const float* __restrict__ Q, uint32_t d,
    const float* __restrict__ cents, const float* __restrict__ bias, const int32_t* __restrict__ status,
    float mass, uint32_t max_probe, uint32_t Pcap, float* __restrict__ cdist,
    uint32_t* __restrict__ ctag, int32_t* __restrict__ pconf,
    unsigned long long* __restrict__ counters, uint32_t* __restrict__ ulist,
    uint32_t* __restrict__ ucount) {
    extern __shared__ float sp[];  // [C] probabilities
    __shared__ float red_v[kProbeThreads / 32];
    __shared__ uint32_t red_i[kProbeThreads / 32];
    __shared__ float sp_top[kProbeThreads / 32];
    __shared__ float bcast;
    __shared__ uint32_t pick[64];
    __shared__ uint32_t npick;
    __shared__ int confident;
    const uint32_t row = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) pconf[row] = 0;
    // a row the probe does not answer goes to the fixed-count selection's list
    auto leave = [&]() {
        if (tid == 0 && ulist != nullptr) ulist[atomicAdd(ucount, 1u)] = row;
    };
    if (status[row] != 0) {
        leave();
        return;
    }
    const float* z = Z + (uint64_t)row * C;
    float m = -FLT_MAX;
    for (uint32_t c = tid; c < C; c += kProbeThreads) m = fmaxf(m, z[c]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red_v[warp] = m;
    __syncthreads();
    if (tid == 0) {
        float v = red_v[0];
        for (int w = 1; w < kProbeThreads / 32; ++w) v = fmaxf(v, red_v[w]);
        bcast = v;
    }
    __syncthreads();
    m = bcast;
    float s = 0.0f;
    float ev = -1.0f;  // the largest exp value, lowest id: the first cluster of the order below
    uint32_t ei = 0xFFFFFFFFu;
    for (uint32_t c = tid; c < C; c += kProbeThreads) {
        const float e = expf(z[c] - m);
        sp[c] = e;
        s += e;
        if (e > ev) {  // c ascends within a thread
            ev = e;
            ei = c;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        const float ov = __shfl_xor_sync(0xffffffffu, ev, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, ei, o);
        if (ov > ev || (ov == ev && oi < ei)) {
            ev = ov;
            ei = oi;
        }
    }
    __syncthreads();
    if (lane == 0) {
        red_v[warp] = s;
        red_i[warp] = ei;
        sp_top[warp] = ev;
    }
    __syncthreads();
    if (tid == 0) {
        float v = 0.0f, bv = -1.0f;
        uint32_t bi = 0xFFFFFFFFu;
        for (int w = 0; w < kProbeThreads / 32; ++w) {
            v += red_v[w];
            if (sp_top[w] > bv || (sp_top[w] == bv && red_i[w] < bi)) {
                bv = sp_top[w];
                bi = red_i[w];
            }
        }
        bcast = v;
        npick = 0;
        confident = 0;
        // one cluster already holds the mass: no ranking rounds
        if (bv * (1.0f / v) >= mass && max_probe >= 1) {
            pick[0] = bi;
            npick = 1;
            confident = 1;
        }
    }
    __syncthreads();
    const float inv = 1.0f / bcast;
    float acc = 0.0f;
    // descending probability, ties to the lower id, until the mass is reached
    for (uint32_t r = 0; !confident && r < max_probe; ++r) {
        float bv = -1.0f;
        uint32_t bi = 0xFFFFFFFFu;
        for (uint32_t c = tid; c < C; c += kProbeThreads) {
            const float v = sp[c];
            if (v > bv || (v == bv && c < bi)) {
                bv = v;
                bi = c;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) {
                bv = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            red_v[warp] = bv;
            red_i[warp] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            float fv = red_v[0];
            uint32_t fi = red_i[0];
            for (int w = 1; w < kProbeThreads / 32; ++w)
                if (red_v[w] > fv || (red_v[w] == fv && red_i[w] < fi)) {
                    fv = red_v[w];
                    fi = red_i[w];
                }
            pick[r] = fi;
            npick = r + 1;
            sp[fi] = -1.0f;
            bcast = fv * inv;
        }
        __syncthreads();
        acc += bcast;
        if (acc >= mass) {
            if (tid == 0) confident = 1;
            break;
        }
    }
    __syncthreads();
    if (!confident) {
        if (tid == 0) atomicAdd(counters + kCounterProbeFallbacks, 1ull);
        leave();
        return;  // the fixed-count selection fills this row
    }
    if (tid == 0) pconf[row] = 1;
    const uint32_t np = npick;
    const float* q = Q + (uint64_t)row * d;
    for (uint32_t i = tid; i < Pcap; i += kProbeThreads) {
        if (i < np) {
            const uint32_t c = pick[i];
            cdist[(uint64_t)row * Pcap + i] = __fsub_rn(bias[c], dot_seq_row(q, cents + (uint64_t)c * d, d));
            ctag[(uint64_t)row * Pcap + i] = c;
        } else {
            cdist[(uint64_t)row * Pcap + i] = sentinel_f();
            ctag[(uint64_t)row * Pcap + i] = kNoLabel;
        }
    }
    if (tid == 0) atomicAdd(counters + kCounterProbeClusters, (unsigned long long)np);
}

}  // namespace

uint64_t ProbeNet::param_count() const {
    return (uint64_t)h * d + h + (uint64_t)h * h + h + (uint64_t)C * h + C;
}

size_t probe_work_layout(const ProbeNet& net, uint32_t n, ProbeWork* w) {
    const uint64_t d = net.d, h = net.h, C = net.C;
    const uint64_t dp = round8(net.d), hp = round8(net.h), Cp = round8(net.C), np = round8(n);
    const struct {
        uint16_t** p;
        uint64_t n;
    } halves[] = {{&w->Xb, n * dp},   {&w->XT, d * np},   {&w->W1b, h * dp},  {&w->W2b, h * hp},
                  {&w->W3b, C * hp},  {&w->W2T, h * hp},  {&w->W3T, h * Cp},  {&w->H1b, n * hp},
                  {&w->H1T, h * np},  {&w->H2b, n * hp},  {&w->H2T, h * np},  {&w->dZb, n * Cp},
                  {&w->dZT, C * np},  {&w->dH2b, n * hp}, {&w->dH2T, h * np}, {&w->dH1T, h * np}};
    const struct {
        float** p;
        uint64_t n;
    } floats[] = {{&w->A1, n * h},
                  {&w->A2, n * h},
                  {&w->Z, n * C},
                  {&w->dH1, n * h},
                  {&w->dH2, n * h},
                  {&w->loss, n}};
    size_t at = 0;
    auto take = [&](uint64_t bytes) {
        const size_t a = at;
        at += (bytes + 255) / 256 * 256;
        return a;
    };
    for (const auto& b : halves) {
        const size_t a = take(b.n * 2);
        if (w->block) *b.p = reinterpret_cast<uint16_t*>(w->block + a);
    }
    for (const auto& b : floats) {
        const size_t a = take(b.n * 4);
        if (w->block) *b.p = reinterpret_cast<float*>(w->block + a);
    }
    return at;
}

cudaError_t probe_sync_bf16(const ProbeNet& net, cudaStream_t st) {
    const struct {
        const float* w;
        uint16_t* b;
        uint64_t n;
    } mats[] = {{net.W1, net.W1b, (uint64_t)net.h * net.d},
                {net.W2, net.W2b, (uint64_t)net.h * net.h},
                {net.W3, net.W3b, (uint64_t)net.C * net.h}};
    for (const auto& m : mats)
        k_to_bf16<<<(unsigned)((m.n + 255) / 256), 256, 0, st>>>(m.w, m.n, m.b);
    return cudaGetLastError();
}

cudaError_t probe_infer(const ProbeNet& net, const float* X, const uint16_t* Xb, uint32_t n,
                        uint16_t* H1b, uint16_t* H2b, float* Z, int* err, cudaStream_t st) {
    TcEpilogue e1{};
    e1.mode = TC_EPI_BIAS_GELU;
    e1.out_bf16 = H1b;
    e1.ld = net.h;
    e1.bias = net.b1;
    TcOperand w1{nullptr, net.d, 1, net.h, net.W1b};
    cudaError_t e = launch_tc_gemm(TcOperand{X, net.d, 1, n, Xb}, w1, net.d, e1, err, st);
    if (e != cudaSuccess) return e;
    TcEpilogue e2{};
    e2.mode = TC_EPI_BIAS_GELU;
    e2.out_bf16 = H2b;
    e2.ld = net.h;
    e2.bias = net.b2;
    e = launch_tc_gemm(TcOperand{nullptr, net.h, 1, n, H1b},
                       TcOperand{nullptr, net.h, 1, net.h, net.W2b}, net.h, e2, err, st);
    if (e != cudaSuccess) return e;
    TcEpilogue e3{};
    e3.mode = TC_EPI_BIAS;
    e3.out = Z;
    e3.ld = net.C;
    e3.bias = net.b3;
    return launch_tc_gemm(TcOperand{nullptr, net.h, 1, n, H2b},
                          TcOperand{nullptr, net.h, 1, net.C, net.W3b}, net.h, e3, err, st);
}

cudaError_t probe_backward(const ProbeNet& net, const float* X, uint32_t n,
                           const uint32_t* labels, uint32_t L, ProbeWork& w, ProbeNet& grad,
                           float* loss_sum, int* err, cudaStream_t st) {
    const uint32_t d = net.d, h = net.h, C = net.C;
    const uint32_t dp = round8(d), hp = round8(h), Cp = round8(C), np = round8(n);
    cudaError_t e = cudaSuccess;
    // out [M][N] = A B^T over K, A [M][lda], B [N][ldb]
    auto gemm = [&](const uint16_t* A, uint32_t lda, uint32_t M, const uint16_t* B, uint32_t ldb,
                    uint32_t N, uint32_t K, float* out, const float* bias = nullptr) {
        if (e != cudaSuccess) return;
        TcEpilogue ep{};
        ep.mode = bias ? TC_EPI_BIAS : TC_EPI_STORE;
        ep.alpha = 1.0f;
        ep.out = out;
        ep.ld = N;
        ep.bias = bias;
        e = launch_tc_gemm(TcOperand{nullptr, lda, 1, M, A}, TcOperand{nullptr, ldb, 1, N, B}, K, ep,
                           err, st);
    };
    auto prep = [&](std::initializer_list<PrepJob> jobs) {
        if (e == cudaSuccess) e = launch_prep(jobs.begin(), (int)jobs.size(), st);
    };
    // the network's own BF16 copies where their rows keep the 16-byte alignment
    const bool own = d % 8 == 0 && h % 8 == 0;
    const uint16_t *W1b = own ? net.W1b : w.W1b, *W2b = own ? net.W2b : w.W2b,
                   *W3b = own ? net.W3b : w.W3b;
    const PrepJob x{X, n, d, kPrepCopy, nullptr, nullptr, w.Xb, dp, w.XT, np, nullptr};
    const PrepJob w1{net.W1, h, d, kPrepCopy, nullptr, nullptr, w.W1b, dp, nullptr, 0, nullptr};
    const PrepJob w2{net.W2, h, h, kPrepCopy, nullptr, nullptr, own ? nullptr : w.W2b,
                     hp,     w.W2T, hp, nullptr};
    const PrepJob w3{net.W3, C, h, kPrepCopy, nullptr, nullptr, own ? nullptr : w.W3b,
                     hp,     w.W3T, Cp, nullptr};
    if (own)
        prep({x, w2, w3});
    else
        prep({x, w1, w2, w3});
    gemm(w.Xb, dp, n, W1b, dp, h, dp, w.A1);
    prep({{w.A1, n, h, kPrepGelu, net.b1, nullptr, w.H1b, hp, w.H1T, np, nullptr}});
    gemm(w.H1b, hp, n, W2b, hp, h, hp, w.A2);
    prep({{w.A2, n, h, kPrepGelu, net.b2, nullptr, w.H2b, hp, w.H2T, np, nullptr}});
    gemm(w.H2b, hp, n, W3b, hp, C, hp, w.Z, net.b3);
    if (e != cudaSuccess) return e;
    k_softmax_xent<<<n, kProbeThreads, 0, st>>>(w.Z, C, labels, L, n, w.loss);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prep({{w.Z, n, C, kPrepCopy, nullptr, nullptr, w.dZb, Cp, w.dZT, np, nullptr}});
    // dW3 = dZ^T H2                                     [C][h], contraction over the batch
    gemm(w.dZT, np, C, w.H2T, np, h, np, grad.W3);
    // dZ2 = (dZ W3) * GELU'(Z2)                          [n][h], contraction over C
    gemm(w.dZb, Cp, n, w.W3T, Cp, h, Cp, w.dH2);
    prep({{w.dH2, n, h, kPrepGeluBwd, net.b2, w.A2, w.dH2b, hp, w.dH2T, np, w.dH2}});
    // dW2 = dZ2^T H1
    gemm(w.dH2T, np, h, w.H1T, np, h, np, grad.W2);
    // dZ1 = (dZ2 W2) * GELU'(Z1)
    gemm(w.dH2b, hp, n, w.W2T, hp, h, hp, w.dH1);
    prep({{w.dH1, n, h, kPrepGeluBwd, net.b1, w.A1, nullptr, 0, w.dH1T, np, w.dH1}});
    // dW1 = dZ1^T X
    gemm(w.dH1T, np, h, w.XT, np, d, np, grad.W1);
    if (e != cudaSuccess) return e;
    const uint32_t ch = (h + 31) / 32, cc = (C + 31) / 32;
    const ColsumJobs sums{{w.Z, w.dH2, w.dH1}, {grad.b3, grad.b2, grad.b1}, {C, h, h},
                          {cc, cc + ch, cc + 2 * ch}};
    k_colsum<<<cc + 2 * ch + 1, kProbeThreads, 0, st>>>(sums, n, w.loss, loss_sum);
    return cudaGetLastError();
}

cudaError_t probe_init(ProbeNet& net, uint64_t seed, cudaStream_t st) {
    struct L {
        float* w;
        uint64_t n;
        float a;
    } layers[] = {{net.W1, (uint64_t)net.h * net.d, sqrtf(3.0f / net.d)},
                  {net.W2, (uint64_t)net.h * net.h, sqrtf(3.0f / net.h)},
                  {net.W3, (uint64_t)net.C * net.h, sqrtf(3.0f / net.h)}};
    uint64_t k = 0;
    for (const L& l : layers) {
        k_init_uniform<<<(unsigned)((l.n + 255) / 256), 256, 0, st>>>(l.w, l.n, l.a, seed * 3 + k++);
    }
    cudaMemsetAsync(net.b1, 0, sizeof(float) * net.h, st);
    cudaMemsetAsync(net.b2, 0, sizeof(float) * net.h, st);
    cudaMemsetAsync(net.b3, 0, sizeof(float) * net.C, st);
    return cudaGetLastError();
}

cudaError_t probe_adam(ProbeNet& net, const ProbeNet& grad, ProbeNet& m, ProbeNet& v, float lr,
                       uint64_t step, cudaStream_t st) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    // the parameters are one contiguous block in every ProbeNet
    const uint64_t n = net.param_count();
    const uint64_t e1 = (uint64_t)net.h * net.d, e2 = e1 + net.h + (uint64_t)net.h * net.h;
    const uint64_t e3 = e2 + net.h + (uint64_t)net.C * net.h;
    k_adam<<<(unsigned)((n + kProbeThreads - 1) / kProbeThreads), kProbeThreads, 0, st>>>(
        net.W1, grad.W1, m.W1, v.W1, n, lr, b1, b2, eps, c1, c2, net.W1b, e1, e2, e3, net.h);
    return cudaGetLastError();
}

cudaError_t launch_probe_select(const ProbeNet& net, const DeviceIndex& ix, uint32_t n,
                                const float* Z, float mass, uint32_t max_probe, Scratch& s,
                                cudaStream_t st) {
    ensure_max_dynamic_smem(k_probe_select, 200 * 1024);
    k_probe_select<<<n, kProbeThreads, sizeof(float) * net.C, st>>>(
        Z, net.C, s.q, ix.d, ix.coarse, ix.coarse_norms, s.status, mass, max_probe, s.P, s.cdist,
        s.ctag, s.pconf, s.counters, s.ulist, s.ucount);
    return cudaGetLastError();
}

}  // namespace pgpu
