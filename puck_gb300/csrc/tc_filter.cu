// Tensor-core contraction with a selecting epilogue: scores s_ij = bias_j - a_i.b_j of BF16
// rows (FP32 accumulation) that are reduced where they are formed, in tensor memory, and
// never written out whole. Two selections:
//   MINIMA  the smallest score of every 8 consecutive columns of a row: the screen of
//           nearest_center. The centroid nearest to a point lies in a group whose minimum is
//           within twice the screen's error of the row's smallest; only those groups are
//           measured exactly.
//   BELOW   the (score, column) pairs at or below a row's threshold, in its list: the screen of
//           the brute-force neighbours. A row's list has a part for each warp that works on the
//           row, so an entry costs no atomic (one with its result on the way took 3 of the 6 ms
//           of a million columns). A part that cannot take the entries of 32 more columns is
//           cut back, with them, to its kTcFilterKeep smallest, which are all that the row's smallest
//           can need of it, and the last of them is the row's threshold there: no order of the
//           columns overflows a list. DENSE fills the lists for the first columns.
//
// One CTA per SM loops over items, an item being a 128-row tile of A and every splits-th of a
// range of 256-column tiles of B (position p stands for tile (p * step) mod tiles: a range of
// positions is spread over all of B). 320 threads, roles as in tc_gemm.cu's persistent kernel:
//   warp 0, one lane: TMA producer. The A tile of an item is loaded once, all of K (at most
//     kMaxResident chunks of 64; up to 2 chunks, the next item's tile while one is in use); the
//     B chunks go through a ring of kRing stages.
//   warp 1, one lane: MMA issuer (M = 128, N = 256, K = 16 per instruction, no instruction for
//     K past the end), one of two 256-column TMEM accumulators per tile in turn.
//   warps 2-9: the selection, lane = row, half a tile's columns each (two warps per scheduler:
//     one alone waits for its own loads most of the time). The next 32 columns are on their way
//     from TMEM while 32 are reduced.
// Bound by the selection: a subtraction and a minimum per score, 16 million warp-wide scores
// for 262144 x 2000 of 96 dimensions (0.2 ms in all; its product alone is 0.07). Eight warps do
// it in a chain of TMEM and bias loads: 28% of the issue slots and 21% of the tensor pipe are
// used. Keeping A resident takes a third off the L2 traffic of reloading it with every B chunk. Every wait is bounded; on expiry *err is set, the roles stop,
// the copies in flight are waited for (bounded) and the TMEM is released.
#include <cuda_bf16.h>

#include <cfloat>
#include <cstdint>

#include "device_common.cuh"
#include "pgpu_internal.h"
#include "tc_common.cuh"

namespace pgpu {
namespace {

constexpr int kThreads = 320;
constexpr uint32_t kSelectWarps = 8;
constexpr uint32_t kNT = kTcFilterTile;  // 256 columns of B per tile
constexpr uint32_t kRing = 4;
constexpr uint32_t kMaxResident = 4;
constexpr uint32_t kABytes = 128u * 64u * 2u, kBBytes = kNT * 64u * 2u;

// A tiles held: two where they fit beside the ring.
__host__ __device__ constexpr uint32_t a_buffers(uint32_t nch) { return nch <= 2 ? 2u : 1u; }

// A part of a list, n entries, and up to 32 new ones (a key per lane, ~0: none) cut back to the
// kTcFilterKeep smallest (score, column) by one warp: the smallest so far sorted in registers (0
// and 1; two per lane), the rest brought in 64 at a time (2 and 3) and the 128 sorted. Returns the
// largest score kept. More than kTcFilterKeep entries in all. The new ones come from registers, so
// that a part needs room for the kept ones alone and a call no more memory than without (it is
// allocated by the call, and each further 32 MB of it cost 130 us): one million rows in the order
// of 1024 clusters, 2048 queries, take 3.5 ms (28 where an overflowing part had the call repeated
// with the screen in memory). One thread replacing the largest of its full part took 9.3 ms.
__device__ __forceinline__ float cut_back(uint2* list, uint32_t n, unsigned long long extra) {
    static_assert(kTcFilterKeep == 64, "two keys per lane");
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();  // the lane that wrote the entries is another
    unsigned long long a[4];
    auto fetch = [&](uint32_t i) {
        if (i >= n) return ~0ull;
        const uint2 e = list[i];
        return ((unsigned long long)ordered_key(__uint_as_float(e.x) + 0.0f) << 32) | e.y;  // -0 is 0
    };
    a[0] = fetch(lane);
    a[1] = fetch(lane + 32);
    for (uint32_t i0 = 64;; i0 += 64) {
        const bool last = i0 >= n;
        a[2] = last ? extra : fetch(i0 + lane);
        a[3] = last ? ~0ull : fetch(i0 + lane + 32);
        // bitonic over elements 32 t + lane
#pragma unroll 1
        for (uint32_t size = 2; size <= 128; size <<= 1) {
#pragma unroll 1
            for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
                if (stride >= 32) {
                    const bool far = stride == 64;
                    const unsigned long long b0 = a[far ? 2 : 1], b1 = a[far ? 3 : 0];
                    const unsigned long long b2 = a[far ? 0 : 3], b3 = a[far ? 1 : 2];
                    const unsigned long long b[4] = {b0, b1, b2, b3};
#pragma unroll
                    for (uint32_t t = 0; t < 4; ++t) {
                        const uint32_t e = 32 * t + lane;
                        const bool low = ((e & size) == 0) == ((e & stride) == 0);
                        a[t] = (b[t] < a[t]) == low ? b[t] : a[t];
                    }
                } else {
#pragma unroll
                    for (uint32_t t = 0; t < 4; ++t) {
                        const unsigned long long b = __shfl_xor_sync(0xffffffffu, a[t], stride);
                        const uint32_t e = 32 * t + lane;
                        const bool low = ((e & size) == 0) == ((e & stride) == 0);
                        a[t] = (b < a[t]) == low ? b : a[t];
                    }
                }
            }
        }
        if (last) break;
    }
    __syncwarp();  // every entry is read
#pragma unroll
    for (int t = 0; t < 2; ++t)
        list[32 * t + lane] = make_uint2(__float_as_uint(key_to_float((uint32_t)(a[t] >> 32))), (uint32_t)a[t]);
    __syncwarp();
    return key_to_float((uint32_t)(__shfl_sync(0xffffffffu, a[1], 31) >> 32));
}

template <int MODE>
__global__ __launch_bounds__(kThreads, 1) void k_tc_filter(const __grid_constant__ CUtensorMap tma_a,
                                                           const __grid_constant__ CUtensorMap tma_b,
                                                           TcFilter p) {
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kNT >> 3) << 17) |
                                ((128u >> 4) << 24);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t afull[2], aempty[2], bfull[kRing], bempty[kRing], tfull[2], tempty[2];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms: 1024 bytes
    const uint32_t nch = (p.K + 63) / 64;
    const uint32_t abufs = a_buffers(nch), ring = sbase + abufs * nch * kABytes;
    const uint32_t items = ((p.M + 127) / 128) * p.splits;
    if (threadIdx.x == 0) {
        failed = 0;
        auto init = [](uint64_t* b, uint32_t n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n));
        };
        for (uint32_t i = 0; i < kRing; ++i) {
            init(&bfull[i], 1);
            init(&bempty[i], 1);
        }
        for (uint32_t i = 0; i < 2; ++i) {
            init(&afull[i], 1);
            init(&aempty[i], 1);
            init(&tfull[i], 1);
            init(&tempty[i], kSelectWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_base)),
                     "r"(2u * kNT)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;
    auto fail = [&]() {
        failed = 1;
        atomicExch(p.err, 1);
    };
    auto tile_of = [&](uint32_t pos) { return (uint32_t)((uint64_t)pos * p.step % p.tiles); };
    auto commit = [](uint64_t* b) {
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b))
            : "memory");
    };

    if (warp == 0) {
        if (lane == 0) {
            auto load = [](uint32_t dst, const CUtensorMap* map, uint32_t k0, uint32_t row, uint32_t bar) {
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                    " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                    "l"(reinterpret_cast<uint64_t>(map)), "r"((int32_t)k0), "r"((int32_t)row), "r"(bar)
                    : "memory");
            };
            auto expect = [](uint32_t bar, uint32_t bytes) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                             : "memory");
            };
            uint32_t it = 0, ai = 0;
            for (uint32_t item = blockIdx.x; item < items && !failed; item += gridDim.x) {
                const uint32_t m0 = item / p.splits * 128u, first = p.pos0 + item % p.splits;
                if (first >= p.pos1) continue;
                const uint32_t ab = ai % abufs, use = ai / abufs;
                if (use > 0 && !tma_wait(smem_u32(&aempty[ab]), (use - 1) & 1u, &failed)) {
                    fail();
                    break;
                }
                ++ai;
                expect(smem_u32(&afull[ab]), nch * kABytes);
                for (uint32_t c = 0; c < nch; ++c)
                    load(sbase + (ab * nch + c) * kABytes, &tma_a, c * 64, m0, smem_u32(&afull[ab]));
                for (uint32_t pos = first; pos < p.pos1 && !failed; pos += p.splits) {
                    const uint32_t n0 = tile_of(pos) * kNT;
                    for (uint32_t c = 0; c < nch; ++c, ++it) {
                        const uint32_t st = it % kRing;
                        if (it >= kRing &&
                            !tma_wait(smem_u32(&bempty[st]), ((it / kRing) & 1u) ^ 1u, &failed)) {
                            fail();
                            break;
                        }
                        expect(smem_u32(&bfull[st]), kBBytes);
                        load(ring + st * kBBytes, &tma_b, c * 64, n0, smem_u32(&bfull[st]));
                    }
                }
            }
            // no copy may land after the CTA: wait (bounded) for the last one of each buffer
            for (uint32_t i = ai > abufs ? ai - abufs : 0u; i < ai; ++i)
                tma_wait(smem_u32(&afull[i % abufs]), (i / abufs) & 1u, &failed);
            for (uint32_t st = 0; st < kRing && st < it; ++st) {
                const uint32_t last = it - 1 - ((it - 1 - st) % kRing);
                tma_wait(smem_u32(&bfull[st]), (last / kRing) & 1u, &failed);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t it = 0, lt = 0, ai = 0;
            bool ok = true;
            for (uint32_t item = blockIdx.x; item < items && ok && !failed; item += gridDim.x) {
                const uint32_t first = p.pos0 + item % p.splits;
                if (first >= p.pos1) continue;
                const uint32_t ab = ai % abufs;
                if (!tma_wait(smem_u32(&afull[ab]), (ai / abufs) & 1u, &failed)) {
                    fail();
                    break;
                }
                for (uint32_t pos = first; pos < p.pos1 && ok; pos += p.splits, ++lt) {
                    const uint32_t acc = lt & 1u;
                    if (lt >= 2 && !tma_wait(smem_u32(&tempty[acc]), ((lt >> 1) - 1) & 1u, &failed)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    for (uint32_t c = 0; c < nch; ++c, ++it) {
                        const uint32_t st = it % kRing;
                        if (!tma_wait(smem_u32(&bfull[st]), (it / kRing) & 1u, &failed)) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;");
                        const uint32_t left = p.K - c * 64, n16 = left >= 64 ? 4u : (left + 15) / 16;
                        for (uint32_t k = 0; k < n16; ++k) {
                            const uint64_t ad = sw128_desc(sbase + (ab * nch + c) * kABytes + k * 32u);
                            const uint64_t bd = sw128_desc(ring + st * kBBytes + k * 32u);
                            const uint32_t accum = (c > 0 || k > 0) ? 1u : 0u;
                            asm volatile(
                                "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(
                                    tmem + acc * kNT),
                                "l"(ad), "l"(bd), "r"(kIdesc), "r"(accum)
                                : "memory");
                        }
                        commit(&bempty[st]);
                    }
                    if (ok) commit(&tfull[acc]);
                }
                if (!ok) {
                    fail();
                    break;
                }
                commit(&aempty[ab]);
                ++ai;
            }
            // the last commit covers every MMA issued before it
            for (uint32_t i = ai > abufs ? ai - abufs : 0u; i < ai; ++i)
                tma_wait(smem_u32(&aempty[i % abufs]), (i / abufs) & 1u, &failed);
        }
    } else {
        const uint32_t quarter = (uint32_t)(warp & 3);          // TMEM lanes 32 * (warp % 4)
        const uint32_t half = (uint32_t)(warp - 2) >> 2;        // columns [128 half, +128)
        constexpr uint32_t kCols = kNT / 2;
        uint32_t lt = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x) {
            const uint32_t first = p.pos0 + item % p.splits;
            if (first >= p.pos1) continue;
            const uint32_t row = item / p.splits * 128u + quarter * 32u + lane;
            const bool in = row < p.M;
            float thr = MODE == kTcBelow && in ? p.thr[row] : -FLT_MAX;
            // this warp's part of the row's list: no other warp of the grid writes it
            const uint32_t part = item % p.splits * 2 + half;
            uint2* list = p.cand + (uint64_t)row * p.cap + part * p.seg;
            uint32_t found = 0;
            for (uint32_t pos = first; pos < p.pos1; pos += p.splits, ++lt) {
                const uint32_t acc = lt & 1u;
                const uint32_t n0 = tile_of(pos) * kNT + half * kCols;
                // the bias of 32 columns is loaded while the 32 before it are reduced (a tile's
                // first ones while its product is waited for)
                const float4* bias = reinterpret_cast<const float4*>(p.bias + n0);
                float4 bq[2][8];
                auto fetch_bias = [&](uint32_t cg, float4 (&b)[8]) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) b[j] = __ldg(bias + cg * 8 + j);
                };
                fetch_bias(0, bq[0]);
                if (!tma_wait(smem_u32(&tfull[acc]), (lt >> 1) & 1u, &failed)) {
                    if (lane == 0) fail();
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t taddr = tmem + acc * kNT + half * kCols + ((quarter * 32u) << 16);
                uint32_t r[2][32];
                auto fetch = [&](uint32_t cg, uint32_t (&v)[32]) {
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
                        "%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,"
                        "%31}, [%32];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                          "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]),
                          "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
                          "=r"(v[30]), "=r"(v[31])
                        : "r"(taddr + cg * 32));
                };
                // the loaded registers are operands of the wait: nothing reads them before it
                auto arrived = [](uint32_t (&v)[32]) {
                    asm volatile("tcgen05.wait::ld.sync.aligned;"
                                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), 
                                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), 
                                   "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), 
                                   "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                                 :
                                 : "memory");
                };
                fetch(0, r[0]);
                arrived(r[0]);
                float4* out_min = MODE == kTcMinima && in
                                      ? reinterpret_cast<float4*>(p.gmin + (uint64_t)row * p.tiles * (kNT / 8) +
                                                                  n0 / 8)
                                      : nullptr;
                float prev[4];
#pragma unroll
                for (uint32_t cg = 0; cg < kCols / 32; ++cg) {
                    uint32_t(&v)[32] = r[cg & 1];
                    if (cg + 1 < kCols / 32) {
                        fetch(cg + 1, r[(cg + 1) & 1]);
                        fetch_bias(cg + 1, bq[(cg + 1) & 1]);
                    }
                    float gm[4];
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 b = bq[cg & 1][j / 4];
                        const float s0 = __fsub_rn(b.x, __uint_as_float(v[j]));
                        const float s1 = __fsub_rn(b.y, __uint_as_float(v[j + 1]));
                        const float s2 = __fsub_rn(b.z, __uint_as_float(v[j + 2]));
                        const float s3 = __fsub_rn(b.w, __uint_as_float(v[j + 3]));
                        const float m = fminf(fminf(s0, s1), fminf(s2, s3));
                        gm[j / 8] = j % 8 == 0 ? m : fminf(gm[j / 8], m);
                        if (MODE != kTcMinima) {
                            v[j] = __float_as_uint(s0);
                            v[j + 1] = __float_as_uint(s1);
                            v[j + 2] = __float_as_uint(s2);
                            v[j + 3] = __float_as_uint(s3);
                        }
                    }
                    // two groups of 32 columns per store: whole 32-byte sectors
                    if (MODE == kTcMinima && (cg & 1) == 0) {
#pragma unroll
                        for (int t = 0; t < 4; ++t) prev[t] = gm[t];
                    } else if (MODE == kTcMinima && in) {
                        asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(out_min + cg - 1),
                                     "f"(prev[0]), "f"(prev[1]), "f"(prev[2]), "f"(prev[3]), "f"(gm[0]),
                                     "f"(gm[1]), "f"(gm[2]), "f"(gm[3])
                                     : "memory");
                    }
                    const uint32_t col = n0 + cg * 32;
                    if (MODE == kTcBelow) {
                        float lim = thr;
                        if (__any_sync(0xffffffffu, found + 32 > p.seg)) {
                            // a part may not take these columns' entries: look who has how many
                            // (first the load under way: this path may move registers)
                            if (cg + 1 < kCols / 32) arrived(r[(cg + 1) & 1]);
                            uint32_t hits = 0;
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                hits |= (__uint_as_float(v[j]) <= thr && col + j < p.N ? 1u : 0u) << j;
                            unsigned over = __ballot_sync(0xffffffffu, found + __popc(hits) > p.seg);
                            while (over) {
                                const int r0 = __ffs(over) - 1;
                                over &= over - 1;
                                uint32_t x = 0;  // that row's score of column `lane`
#pragma unroll
                                for (int j = 0; j < 32; ++j) {
                                    const uint32_t u = __shfl_sync(0xffffffffu, v[j], r0);
                                    x = lane == j ? u : x;
                                }
                                const bool hit = __shfl_sync(0xffffffffu, hits, r0) >> lane & 1u;
                                const float t = cut_back(
                                    reinterpret_cast<uint2*>(__shfl_sync(
                                        0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(list), r0)),
                                    __shfl_sync(0xffffffffu, found, r0),
                                    hit ? ((unsigned long long)ordered_key(__uint_as_float(x) + 0.0f) << 32) |
                                              (p.id0 + col + lane)
                                        : ~0ull);
                                if (lane == r0) {
                                    found = kTcFilterKeep;
                                    thr = t;
                                    lim = __int_as_float(0x7fffffff);  // these columns are done
                                }
                            }
                        }
                        // entries are rare: eight columns with one are looked through
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            if (gm[t] <= lim) {
#pragma unroll
                                for (int j = 8 * t; j < 8 * t + 8; ++j)
                                    if (__uint_as_float(v[j]) <= lim && col + j < p.N)
                                        list[found++] = make_uint2(v[j], p.id0 + col + j);
                            }
                    }
                    if (MODE == kTcDense && in) {
                        uint2* out = p.cand + (uint64_t)row * p.cap + (pos - p.pos0) * kNT + half * kCols +
                                     cg * 32;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            out[j] = make_uint2(v[j], col + j < p.N ? p.id0 + col + j : kNoLabel);
                    }
                    if (cg + 1 < kCols / 32) arrived(r[(cg + 1) & 1]);
                }
                // this accumulator may take the next tile's MMAs
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[acc]))
                                 : "memory");
            }
            if (MODE == kTcBelow && in) p.count[(uint64_t)row * 2 * p.splits + part] = found;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kNT)
                     : "memory");
    }
}

// BF16 copies of rows (out: [rows][dp], dp - d zeros) and their squared norms, one warp per 32
// rows: read and written coalesced through shared memory, then each lane sums its row in
// order. Products and sums rounded separately (seq), or fused and halved into `norm` with
// `pad` entries of FLT_MAX after the rows (the bias of a contraction). lost, if not null: a
// bound on the length of what the BF16 rounding took from each row.
constexpr int kRowWarps = 2;  // small blocks: a few thousand centroids still fill the chip
__global__ __launch_bounds__(kRowWarps * 32) void k_rows_bf16(const float* __restrict__ X, uint64_t rows,
                                                              uint32_t d, uint32_t dp, int seq,
                                                              uint32_t pad, uint16_t* __restrict__ out,
                                                              float* __restrict__ norm,
                                                              float* __restrict__ lost) {
    __shared__ float tile[kRowWarps][32][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t r0 = ((uint64_t)blockIdx.x * kRowWarps + warp) * 32;
    if (r0 >= rows + pad) return;
    const uint32_t nr = r0 >= rows ? 0u : rows - r0 < 32 ? (uint32_t)(rows - r0) : 32u;
    float s = 0.0f, l2 = 0.0f;
    for (uint32_t c0 = 0; c0 < dp && nr > 0; c0 += 32) {
        const uint32_t w = d > c0 ? (d - c0 < 32 ? d - c0 : 32u) : 0u, wp = dp - c0 < 32 ? dp - c0 : 32u;
        if (w == 32 && nr == 32) {
            // whole tile: every load in flight, then the sums without loop overhead
            float v[32];
#pragma unroll
            for (int r = 0; r < 32; ++r) v[r] = X[(r0 + r) * d + c0 + lane];
#pragma unroll
            for (int r = 0; r < 32; ++r) {
                tile[warp][r][lane] = v[r];
                out[(r0 + r) * dp + c0 + lane] = __bfloat16_as_ushort(__float2bfloat16_rn(v[r]));
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 32; ++c) v[c] = tile[warp][lane][c];
            if (seq) {
#pragma unroll
                for (int c = 0; c < 32; ++c) s = __fadd_rn(s, __fmul_rn(v[c], v[c]));
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) s = __fmaf_rn(v[c], v[c], s);
            }
            if (lost) {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const float e = v[c] - __bfloat162float(__float2bfloat16_rn(v[c]));  // exact
                    l2 += e * e;
                }
            }
            __syncwarp();
            continue;
        }
        if (wp == 32) {
            for (uint32_t r = 0; r < nr; ++r) {
                const float v = (uint32_t)lane < w ? X[(r0 + r) * d + c0 + lane] : 0.0f;
                tile[warp][r][lane] = v;
                out[(r0 + r) * dp + c0 + lane] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
            }
        } else {  // narrow rows: several per step
            for (uint32_t e = lane; e < nr * wp; e += 32) {
                const uint32_t r = e / wp, c = e - r * wp;
                const float v = c < w ? X[(r0 + r) * d + c0 + c] : 0.0f;
                tile[warp][r][c] = v;
                out[(r0 + r) * dp + c0 + c] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
            }
        }
        __syncwarp();
        if (seq)
            for (uint32_t c = 0; c < w; ++c) s = __fadd_rn(s, __fmul_rn(tile[warp][lane][c], tile[warp][lane][c]));
        else
            for (uint32_t c = 0; c < w; ++c) s = __fmaf_rn(tile[warp][lane][c], tile[warp][lane][c], s);
        if (lost)
            for (uint32_t c = 0; c < w; ++c) {
                const float v = tile[warp][lane][c];
                const float e = v - __bfloat162float(__float2bfloat16_rn(v));  // exact
                l2 += e * e;
            }
        __syncwarp();
    }
    if (lost && r0 + lane < rows) lost[r0 + lane] = sqrtf(l2) * 1.0001f + 1e-30f;
    if (r0 + lane < rows) norm[r0 + lane] = seq ? s : 0.5f * s;
    else if (r0 + lane < rows + pad) norm[r0 + lane] = FLT_MAX;
}

}  // namespace

// A row tile's columns are split until the items fill the SMs.
uint32_t tc_filter_splits(uint32_t M) {
    const uint32_t sms = (uint32_t)sm_count(), mt = (M + 127) / 128;
    return mt >= sms ? 1u : sms / mt;
}

// (without tensor maps nearest_center and knn take the forms with a screen matrix)
bool tc_filter_applies(uint32_t K) { return K > 0 && K <= kMaxResident * 64 && tensor_maps_available(); }

cudaError_t launch_rows_bf16(const float* X, uint64_t rows, uint32_t d, uint32_t dp, bool seq,
                             uint32_t pad, uint16_t* out, float* norm, float* lost,
                             cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    const uint64_t per = kRowWarps * 32;
    k_rows_bf16<<<(unsigned)((rows + pad + per - 1) / per), kRowWarps * 32, 0, stream>>>(
        X, rows, d, dp, seq ? 1 : 0, pad, out, norm, lost);
    return cudaGetLastError();
}

cudaError_t launch_tc_filter(int mode, const uint16_t* A, uint64_t a_rs, const uint16_t* B,
                             uint64_t b_rs, TcFilter& p, cudaStream_t stream) {
    if (p.M == 0 || p.N == 0 || p.pos1 <= p.pos0) return cudaSuccess;
    CUtensorMap ma, mb;
    if (!encode_bf16_rows(&ma, A, p.M, a_rs, p.K, 128) || !encode_bf16_rows(&mb, B, p.N, b_rs, p.K, kNT))
        return cudaErrorInvalidValue;
    const uint32_t sms = (uint32_t)sm_count(), mt = (p.M + 127) / 128;
    p.splits = tc_filter_splits(p.M);
    if (p.splits > p.pos1 - p.pos0) p.splits = p.pos1 - p.pos0;
    p.seg = p.cap / (2 * p.splits);
    if (mode == kTcBelow && p.seg < kTcFilterKeep) return cudaErrorInvalidValue;
    const uint32_t items = mt * p.splits, nch = (p.K + 63) / 64;
    const size_t smem = (size_t)a_buffers(nch) * nch * kABytes + kRing * kBBytes + 1024;
    const unsigned grid = items < sms ? items : sms;
    auto run = [&](auto* kernel) {
        ensure_max_dynamic_smem(kernel, (int)(kMaxResident * kABytes + kRing * kBBytes + 1024));
        kernel<<<grid, kThreads, smem, stream>>>(ma, mb, p);
    };
    if (mode == kTcMinima) run(k_tc_filter<kTcMinima>);
    else if (mode == kTcBelow) run(k_tc_filter<kTcBelow>);
    else run(k_tc_filter<kTcDense>);
    return cudaGetLastError();
}

}  // namespace pgpu
