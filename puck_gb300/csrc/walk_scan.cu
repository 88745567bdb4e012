// k_walk_scan: the cell walk and filter-PQ ADC scan of
// PuckIndex::search_nearest_filter_points (puck/puck/puck_index.cpp:485-557) and
// compute_quantized_distance (puck_index.cpp:346-390), bit-exact.
//
// The reference walks, for each probed coarse cluster c (ascending coarse term),
// the fine cells k in ascending fine-term order fd, breaks when
// fd + min_dist >= pivot, skips cells with stationary[c][k] >= max_stationary_dist,
// and scans the others into a bounded max-heap; pivot and max_stationary_dist only
// decrease as the heap fills. One block per query reproduces it:
//
//   candidate generation (all threads, against the current pivot/max_stat, which
//   bound every later value):
//     enumeration: cells of c in ascending stationary order (sorted at load) below
//                  max_stat and before the break, re-ordered by fine rank. Used
//                  when they fit one block-wide chunk of the sorted row.
//     fd-order   : 128 consecutive fine ranks per chunk, break/skip tests per cell
//                  (the heap-fill phase, where nothing is pruned yet).
//   speculative ADC: every point of every candidate cell (one thread per point). Points
//     whose distance is below the heap's top at that time, the only ones that can still
//     enter the heap, go to a list in order.
//   replay (warp 0): the candidates in fine-rank order with the exact pivot,
//     max_stationary_dist and heap; it only prunes further, never adds.
// Every test is monotone in pivot/max_stat, so the replay inserts exactly the points the
// sequential walk inserts, in the same order. The walk also stops inside a cell at the first
// point whose part without the table sum is not below the top: such a point and those after
// it cannot enter the heap (the sum is not negative), so the stop only matters for the count
// of scanned records, which all threads form after the replay from the heap's tops.
//
// What bounds it: the sequential replay, a chain of shared-memory reads and warp votes (25 to
// 45 cycles each). So
//   * a cell without list entries costs two tests and a minimum, its record prefetched;
//   * an insert reads five heap levels at once (lane i decides node i of the subtree, two
//     votes give every lane its place on or off the way down), two rounds for a heap of
//     1100 instead of ten dependent levels; slots of the heap's lower half, filled first,
//     have no children and take a cell's entries together;
//   * the double-precision division of the pivot is left out at radius_rate 1 (halving a
//     float is exact): it alone cost 800 cycles per cell;
//   * clusters that can hold no candidate (their smallest stationary term is not below
//     max_stat, or rank 0 breaks) are passed over a block's width at a time.
// Measured on a GB300, whole calls: one query over 200k points with filter_topk 1100 (57k
// records and 3.4k inserts) 9.9 ms with a one-thread replay, 2.7 ms now; 10k queries over 1M
// points with filter_topk 200 15.1 ms, now 6.7 ms (the walk itself 10.9 and 4.4 ms, where three
// of a block's four warps wait at its barrier for the replay: 19% of the issue slots are used).
#include "device_common.cuh"
#include "pgpu_internal.h"

namespace pgpu {
namespace {

constexpr int kSlots = 128;     // candidate slots per round
constexpr int kMaxWarps = 16;   // of the widest block
constexpr int kPointBuf = 512;  // points whose distances are formed per batch

struct WalkParams {
    const float* q;
    const float* qnorm;
    const int32_t* status;
    const float* cdist;
    const uint32_t* ctag;
    const float* fdist;       // [B][F] fine terms in ascending (rank) order
    const uint32_t* ftag;     // [B][F] fine id at each rank
    const float* fd_by_fine;  // [B][F] fine term indexed by fine id
    float* hdist;
    uint32_t* htag;
    uint32_t* hcnt;
    const float* stationary;  // [C][F]
    const float* stat_sorted; // [C][F] stationary ascending per coarse row
    const uint32_t* stat_fine;// [C][F] fine id of each sorted entry
    const uint32_t* cell_start;
    const float* mdo;
    const float* offsets;
    const uint8_t* codes;
    const float* codebook;
    unsigned long long* counters;
    const int32_t* ins_head;  // realtime: [C*F] newest insert of each cell, or null
    const int32_t* ins_next;
    uint32_t n_base;          // memory id of insert 0
    uint32_t d, C, F, nsq, lsq, code_stride, P, T;
    double rr;
    int rr_one;  // rr == 1
};

// Diagnostic counters accumulated per launch (pgpu_walk_counters): records and
// cells scanned, fd-order chunks, enumerations, fd-order coarse clusters, heap
// inserts, and thread-0 clock cycles spent in replay / whole walk / prologue /
// candidate generation / speculative ADC.
enum { kCntRecords, kCntCells, kCntChunks, kCntEnum, kCntFdOrder, kCntInserts, kCycReplay,
       kCycTotal, kCycPrologue, kCycCand, kCycAdc, kNumCounters };

// Heap slots held in shared memory: 0 (unused) to T, an even number.
__host__ __device__ inline uint32_t heap_slots(uint32_t T) { return (T + 2) & ~1u; }

// A block's state in static shared memory; the table, the heap, the query and the fine ranks
// follow in dynamic shared memory.
struct WalkState {
    uint4 rec[kSlots];           // for the replay: fine term, stationary term, list entries [z, w)
    uint2 list[kPointBuf + 2];   // points below the heap's top: distance, memory id
    float evtop[kPointBuf];      // the heap's top after each list entry
    float pt0[kPointBuf];        // points' distances without the table sum
    // candidates
    uint32_t fine[kSlots];
    float fd[kSlots], stat[kSlots], dist[kSlots];
    uint32_t start[kSlots], cnt_pts[kSlots], pref[kSlots];
    float top[kSlots];           // the heap's top when the cell's turn came, -inf: not scanned
    float pivot, max_stat, min_dist, cdl;
    uint32_t c, dpc, broke, part_upd, part_cells;
    unsigned votes[kPointBuf / 32];  // points of the batch below the heap's top
    uint32_t live[kMaxWarps];        // clusters of the window that may hold candidates
    uint32_t warp_tot[kMaxWarps];
    unsigned long long cnt[kNumCounters];
};

// The rare steps of the replay, kept out of its loop.
__device__ __noinline__ float pivot_general(float top, float qn, double rr) {
    return pivot_of(top, qn, rr);
}
__device__ __noinline__ float point_distance(const WalkParams& p, const float* lut, float dist,
                                             uint32_t mi) {
    return __fadd_rn(adc_base(dist, p.offsets[mi]),
                     lut_sum(p.codes + (uint64_t)mi * p.code_stride, lut, p.nsq));
}

// The replay of candidates [b0, last] by warp 0; see the file comment. A cell of more points
// than the buffer comes in parts: resumed, cell b0 has passed its tests; partial, it is the
// only one and its updates wait for its last part.
__device__ __forceinline__ void replay(const WalkParams& p, WalkState& st, uint32_t b0,
                                       uint32_t last, const float* lut, uint2* heap,
                                       float qn, bool resumed, bool partial, const HeapLane& hl) {
    const int lane = threadIdx.x & 31;
    const long long t_rep = clock64();
    const uint32_t T = p.T;
    const float md = st.min_dist, cdl = st.cdl;
    float pivot = st.pivot, max_stat = st.max_stat, top = __uint_as_float(heap[1].x);
    float room = __fsub_rn(pivot, cdl);  // max_stat after a cell: room - its fine term
    uint32_t dpc = st.dpc, cells = 0, ins = 0;
    bool broke = false;
    // one value below the top: the slot it takes, as MaxHeap::insert
    auto insert = [&](float v, uint32_t tag) {
        uint32_t f = 1;
        if (dpc > 0) f = dpc--;
        const float landed = warp_heap_insert(heap, T, f, v, tag, hl);
        if (f == 1) top = landed;
    };
    uint4 rec = st.rec[b0];
    for (uint32_t i = b0; i <= last; ++i) {
        const uint4 next = st.rec[i < last ? i + 1 : i];
        const float fdi = __uint_as_float(rec.x), stat = __uint_as_float(rec.y);
        uint32_t upd = 0;
        if (resumed && i == b0) {
            upd = st.part_upd;
            ins -= upd;  // counted with their part
        } else {
            if (__fadd_rn(fdi, md) >= pivot) {
                broke = true;
                break;
            }
            if (stat >= max_stat) {
                rec = next;
                continue;
            }
            ++cells;
        }
        if (lane == 0) st.top[i] = top;
        uint2 ev = st.list[rec.z];
        for (uint32_t e = rec.z; e < rec.w;) {
            if (dpc > T / 2 && dpc > 1) {
                // leaf slots of a heap not yet full: the top does not change
                const uint32_t free = dpc - T / 2, m = free < rec.w - e ? free : rec.w - e;
                for (uint32_t r = lane; r < m; r += 32) {
                    heap[dpc - r] = st.list[e + r];
                    st.evtop[e + r] = top;
                }
                __syncwarp();
                dpc -= m;
                e += m;
                upd += m;
                ev = st.list[e];
                continue;
            }
            const uint2 after = st.list[e + 1];
            const float tf = __uint_as_float(ev.x);
            if (!(tf >= top)) {
                insert(tf, ev.y);
                ++upd;
            }
            if (lane == 0) st.evtop[e] = top;
            ev = after;
            ++e;
        }
        if (!partial) {
            if (p.ins_head) {
                // realtime: the cell's inserted points, newest first, none skipped,
                // each counted as an update (realtime_insert_puck_index.cpp:398-453)
                uint32_t sp = 0;
                const uint64_t cell = (uint64_t)st.c * p.F + st.fine[i];
                for (int32_t id = p.ins_head[cell]; id >= 0; id = p.ins_next[id]) {
                    const uint32_t mi = p.n_base + (uint32_t)id;
                    const float tf = point_distance(p, lut, st.dist[i], mi);
                    ++sp;
                    ++upd;
                    if (!(tf >= top)) insert(tf, mi);
                }
                if (lane == 0) st.cnt[kCntRecords] += sp;
            }
            if (upd > 0) {
                // (top - |q|^2) / 1.0 / 2.0 in double and rounded is half the float
                if (p.rr_one) pivot = 0.5f * __fsub_rn(top, qn);
                else pivot = pivot_general(top, qn, p.rr);
                room = __fsub_rn(pivot, cdl);
            }
            const float cand_ms = __fsub_rn(room, fdi);
            if (cand_ms < max_stat) max_stat = cand_ms;
        }
        ins += upd;
        rec = next;
    }
    __syncwarp();  // part_upd is read above
    if (lane == 0) {
        st.pivot = pivot;
        st.max_stat = max_stat;
        st.dpc = dpc;
        st.broke = broke ? 1u : 0u;
        st.part_upd = ins + (resumed ? st.part_upd : 0u);  // read after a partial replay only
        st.part_cells = cells;
        st.cnt[kCntCells] += cells;
        st.cnt[kCntInserts] += ins;
        st.cnt[kCycReplay] += (unsigned long long)(clock64() - t_rep);
    }
}

// Scans candidates [0, n) (sorted by fine rank) in batches whose points fit the
// point buffer. Returns true when the walk broke inside this coarse cluster.
template <int NT>
__device__ __forceinline__ bool process_candidates(const WalkParams& p, WalkState& st, uint32_t n,
                                                   const float* lut, uint2* heap, const uint32_t* cs,
                                                   float qn, const HeapLane& hl) {
    constexpr int kIter = kPointBuf / NT;  // points per thread and batch
    static_assert(kPointBuf % NT == 0 && kPointBuf / 32 <= 31, "a lane per vote word");
    const int tid = threadIdx.x, lane = tid & 31;
    const float cdl = st.cdl;
    if ((uint32_t)tid < n) {
        const uint32_t k = st.fine[tid];
        const uint32_t s0 = cs[k];
        st.start[tid] = s0;
        st.cnt_pts[tid] = cs[k + 1] - s0;
        st.dist[tid] = __fadd_rn(__fadd_rn(cdl, st.stat[tid]), st.fd[tid]);
    }
    __syncthreads();
    uint32_t b0 = 0, part = 0;  // part: points of cell b0 already done (a cell in parts)
    while (b0 < n) {
        const bool mine = (uint32_t)tid >= b0 && (uint32_t)tid < n;
        const uint32_t cnt = mine ? st.cnt_pts[tid] - ((uint32_t)tid == b0 ? part : 0u) : 0u;
        uint32_t total;
        const uint32_t incl = block_scan_incl<NT / 32>(cnt, st.warp_tot, &total);
        if (mine) st.pref[tid] = incl - cnt;
        const int fits = __syncthreads_count(mine && incl <= (uint32_t)kPointBuf);
        long long t_adc = clock64();
        const uint32_t n_used = fits > 0 ? (uint32_t)fits : 1u;
        const uint32_t last = b0 + n_used - 1;
        const uint32_t full = st.pref[last] + st.cnt_pts[last] - (last == b0 ? part : 0u);
        const uint32_t npts = fits > 0 ? full : (uint32_t)kPointBuf;
        const float top = __uint_as_float(heap[1].x);
        float tf[kIter];
        uint32_t mem[kIter];
        unsigned vote[kIter];
#pragma unroll
        for (int u = 0; u < kIter; ++u) {
            const uint32_t j = tid + u * NT;
            vote[u] = 0;
            if ((j & ~31u) >= npts) continue;  // the whole warp
            bool below = false;
            if (j < npts) {
                uint32_t lo = b0, hi = b0 + n_used;  // last candidate with pref <= j
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (st.pref[mid] <= j) lo = mid;
                    else hi = mid;
                }
                const uint32_t mi = st.start[lo] + (j - st.pref[lo]) + (lo == b0 ? part : 0u);
                const float t0 = adc_base(st.dist[lo], p.offsets[mi]);
                st.pt0[j] = t0;
                mem[u] = mi;
                tf[u] = __fadd_rn(t0, lut_sum(p.codes + (uint64_t)mi * p.code_stride, lut, p.nsq));
                below = !(tf[u] >= top);
            }
            vote[u] = __ballot_sync(0xffffffffu, below);
            if (lane == 0) st.votes[j >> 5] = vote[u];
        }
        __syncthreads();
        // the list: entries before each vote word (lane w holds word w; past the last: all)
        const unsigned word = (uint32_t)lane * 32 < npts ? st.votes[lane] : 0u;
        uint32_t before = __popc(word);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        before -= __popc(word);
#pragma unroll
        for (int u = 0; u < kIter; ++u) {
            const uint32_t base = __shfl_sync(0xffffffffu, before, (tid + u * NT) >> 5);
            if ((vote[u] >> lane) & 1u)
                st.list[base + __popc(vote[u] & ((1u << lane) - 1))] =
                    make_uint2(__float_as_uint(tf[u]), mem[u]);
        }
        // entries before point j (j <= npts)
        auto rank = [&](uint32_t j) {
            const uint32_t b = __shfl_sync(0xffffffffu, before, j >> 5);
            const unsigned w = __shfl_sync(0xffffffffu, word, j >> 5);
            return b + __popc(w & ((1u << (j & 31)) - 1));
        };
        const bool used = (uint32_t)tid >= b0 && (uint32_t)tid <= last;
        const uint32_t p0 = used ? st.pref[tid] : 0u;
        const uint32_t pe = used ? ((uint32_t)tid == last ? npts : p0 + cnt) : 0u;
        const uint32_t e0 = rank(p0), e1 = rank(pe);
        if (used) {
            st.rec[tid] = make_uint4(__float_as_uint(st.fd[tid]), __float_as_uint(st.stat[tid]), e0, e1);
            st.top[tid] = -__int_as_float(0x7f800000);  // not scanned
        }
        if (tid == 0) st.cnt[kCycAdc] += (unsigned long long)(clock64() - t_adc);
        __syncthreads();
        if (tid < 32) replay(p, st, b0, last, lut, heap, qn, part > 0, fits == 0, hl);
        __syncthreads();
        // records scanned: per cell the points before the first whose part without the table
        // is not below the top at its turn (tops fall and the parts ascend: binary search)
        const float none = -__int_as_float(0x7f800000);
        uint32_t lo = p0, hi = used && st.top[tid] > none ? pe : p0;
        while (__any_sync(0xffffffffu, lo < hi)) {
            const uint32_t mid = (lo + hi) >> 1;
            const uint32_t e = rank(mid);
            if (lo < hi) {
                if (st.pt0[mid] >= (e > e0 ? st.evtop[e - 1] : st.top[tid])) hi = mid;
                else lo = mid + 1;
            }
        }
        const uint32_t scanned = __reduce_add_sync(0xffffffffu, lo - p0);
        if (lane == 0 && scanned) atomicAdd(&st.cnt[kCntRecords], (unsigned long long)scanned);
        if (st.broke) return true;
        if (fits == 0 && part + st.part_cells > 0) {
            part += kPointBuf;  // points past the cell's stop add nothing
        } else {
            b0 += n_used;
            part = 0;
        }
    }
    return false;
}

template <int NT>
__global__ __launch_bounds__(NT, NT == 128 ? 4 : 1) void k_walk_scan(WalkParams p) {
    constexpr int kWarps = NT / 32;
    static_assert(NT >= kSlots && kWarps <= kMaxWarps, "a thread per candidate slot");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ WalkState st;
    const uint32_t qi = blockIdx.x;
    const int tid = threadIdx.x;
    const uint32_t nsq = p.nsq, T = p.T, F = p.F;
    float* lut = reinterpret_cast<float*>(smem);
    uint2* heap = reinterpret_cast<uint2*>(lut + nsq * 256);  // 1-based [1..T], 16-byte aligned
    float* qv = reinterpret_cast<float*>(heap + heap_slots(T));
    uint16_t* rank_s = reinterpret_cast<uint16_t*>(qv + p.d);  // [F] fine id -> rank
    // enumeration staging, in the list's place (the list is filled after it)
    uint32_t* e_fine = reinterpret_cast<uint32_t*>(&st.list[0]);
    uint32_t* e_rank = e_fine + kSlots;
    float* e_fd = reinterpret_cast<float*>(e_rank + kSlots);
    float* e_stat = e_fd + kSlots;
    static_assert(4 * kSlots <= 2 * kPointBuf, "the staging fits the list");

    if (p.status[qi] != 0) {
        if (tid == 0) p.hcnt[qi] = 0;
        return;
    }
    const long long t_start = clock64();
    const float* fd = p.fdist + (uint64_t)qi * F;
    const uint32_t* ftag = p.ftag + (uint64_t)qi * F;
    const float* fdk = p.fd_by_fine + (uint64_t)qi * F;
    for (uint32_t i = tid; i < p.d; i += NT) qv[i] = p.q[(uint64_t)qi * p.d + i];
    for (uint32_t i = tid; i < heap_slots(T); i += NT) heap[i] = make_uint2(kHeapSentinelBits, 0u);
    for (uint32_t i = tid; i < F; i += NT) {
        const uint32_t k = ftag[i];
        if (k < F) rank_s[k] = (uint16_t)i;
    }
    __syncthreads();
    // get_dist_table (quantization.cpp:260-270)
    build_lut(lut, qv, p.codebook, nsq, p.lsq, NT);
    const float qn = p.qnorm[qi];
    if (tid == 0) {
        st.dpc = T;
        st.pivot = pivot_of(sentinel_f(), qn, p.rr);
        for (int i = 0; i < kNumCounters; ++i) st.cnt[i] = 0;
        st.cnt[kCycPrologue] = (unsigned long long)(clock64() - t_start);
    }
    __syncthreads();

    const float fd0 = fd[0];
    const HeapLane hl = heap_lane();
    // windows of NT probed clusters, one per thread
    for (uint32_t lb = 0; lb < p.P; lb += NT) {
      const uint32_t wl = lb + tid;
      const uint32_t wc = wl < p.P ? p.ctag[(uint64_t)qi * p.P + wl] : p.C;
      const bool wvalid = wc < p.C;
      const float wcdl = wvalid ? p.cdist[(uint64_t)qi * p.P + wl] : 0.0f;
      const float wmd = wvalid ? __fadd_rn(p.mdo[wc], wcdl) : 0.0f;
      const float wst = wvalid ? p.stat_sorted[(uint64_t)wc * F] : 0.0f;
      const int wcount = __syncthreads_count(wvalid);
      if (tid == 0) st.cnt[kCntEnum] += (unsigned long long)wcount;  // less the fine-order ones
      for (uint32_t from = 0; from < (uint32_t)NT;) {
        // the window's next cluster that may hold a candidate: its first cell in
        // stationary order is below max_stat and rank 0 does not break (both tests can
        // only turn against it as the pivot falls)
        const float pw = st.pivot;
        const float wms = __fsub_rn(__fsub_rn(pw, wcdl), fd0);
        const unsigned lv = __ballot_sync(0xffffffffu, wvalid && (uint32_t)tid >= from && wst < wms &&
                                                           !(__fadd_rn(fd0, wmd) >= pw));
        if ((tid & 31) == 0) st.live[tid >> 5] = lv;
        __syncthreads();
        uint32_t next = NT;
#pragma unroll
        for (int w = kWarps - 1; w >= 0; --w)
            if (st.live[w]) next = 32 * w + __ffs(st.live[w]) - 1;
        if ((uint32_t)tid == next) {
            st.c = wc;
            st.cdl = wcdl;
            st.min_dist = wmd;
            st.max_stat = wms;
        }
        __syncthreads();
        from = next + 1;
        if (next == (uint32_t)NT) break;
        const uint32_t c = st.c;
        const uint32_t* cs = p.cell_start + (uint64_t)c * F;
        float pv = st.pivot, ms = st.max_stat;
        const float md = st.min_dist;
        long long t_cand = clock64();

        // ---- enumeration through the stationary-sorted row of c
        bool below = false;
        uint32_t k = 0;
        float sv = 0.0f;
        if (tid < kSlots && (uint32_t)tid < F) {
            sv = p.stat_sorted[(uint64_t)c * F + tid];
            k = p.stat_fine[(uint64_t)c * F + tid];
            below = sv < ms;
        }
        const bool fallback = __syncthreads_and(below || tid >= kSlots) && F > (uint32_t)kSlots;
        if (tid == 0 && fallback) {
            st.cnt[kCntFdOrder] += 1;
            st.cnt[kCntEnum] -= 1;
        }
        // one pass over the enumeration, or the fd-order chunks (nothing pruned yet)
        const float* statrow = p.stationary + (uint64_t)c * F;
        for (uint32_t base = 0;;) {
            uint32_t n, bpos = 0;
            bool cand = false;
            if (!fallback) {
                float fv = 0.0f;
                uint32_t r = 0;
                if (below && k < F) {
                    fv = fdk[k];
                    r = rank_s[k];
                    cand = !(__fadd_rn(fv, md) >= pv);
                }
                const uint32_t pos = block_scan_incl<NT / 32>(cand ? 1u : 0u, st.warp_tot, &n) - 1;
                if (cand) {
                    e_fine[pos] = k;
                    e_rank[pos] = r;
                    e_fd[pos] = fv;
                    e_stat[pos] = sv;
                }
                __syncthreads();
                if ((uint32_t)tid < n) {  // order by fine rank (ranks are distinct)
                    const uint32_t myr = e_rank[tid];
                    uint32_t o = 0;
                    for (uint32_t j = 0; j < n; ++j) o += e_rank[j] < myr;
                    st.fine[o] = e_fine[tid];
                    st.fd[o] = e_fd[tid];
                    st.stat[o] = e_stat[tid];
                }
            } else {
                t_cand = clock64();
                pv = st.pivot;
                ms = st.max_stat;
                const uint32_t idx = base + tid;
                const bool valid = tid < kSlots && idx < F;
                const float fdv = valid ? fd[idx] : 0.0f;
                const bool brk = !valid || (__fadd_rn(fdv, md) >= pv);
                // first break position in the chunk: everything before it is a candidate
                // unless skipped; breaks are monotone in idx, so the non-breaking threads
                // are a prefix
                bpos = __syncthreads_count(!brk);
                float stv = 0.0f;
                uint32_t kk = 0;
                if ((uint32_t)tid < bpos) {
                    kk = ftag[idx];
                    if (kk >= F) kk = 0;  // never taken for finite queries
                    stv = statrow[kk];
                    cand = !(stv >= ms);
                }
                const uint32_t pos = block_scan_incl<NT / 32>(cand ? 1u : 0u, st.warp_tot, &n) - 1;
                if (cand) {
                    st.fine[pos] = kk;
                    st.fd[pos] = fdv;
                    st.stat[pos] = stv;
                }
                if (tid == 0) st.cnt[kCntChunks] += 1;
            }
            __syncthreads();
            if (tid == 0) st.cnt[kCycCand] += (unsigned long long)(clock64() - t_cand);
            const bool broke = n > 0 && process_candidates<NT>(p, st, n, lut, heap, cs, qn, hl);
            base += kSlots;
            if (!fallback || broke || bpos < (uint32_t)kSlots || base >= F) break;
        }
        __syncthreads();
      }
    }
    if (tid < 32 && st.dpc > 0) warp_heap_reorder(heap, T, hl);  // a heap not full
    if (tid == 0) {
        p.hcnt[qi] = T - st.dpc;
        st.cnt[kCycTotal] = (unsigned long long)(clock64() - t_start);
        if (p.counters)
            for (int i = 0; i < kNumCounters; ++i) atomicAdd(p.counters + i, st.cnt[i]);
    }
    __syncthreads();
    for (uint32_t i = tid; i < T; i += NT) {
        p.hdist[(uint64_t)qi * T + i] = __uint_as_float(heap[i + 1].x);
        p.htag[(uint64_t)qi * T + i] = heap[i + 1].y;
    }
}

}  // namespace

size_t walk_smem_bytes(const DeviceIndex& ix, uint32_t T) {
    return sizeof(float) * ix.nsq * 256 + sizeof(uint2) * heap_slots(T) + sizeof(float) * ix.d +
           sizeof(uint16_t) * ((ix.F + 1) & ~1u) + sizeof(WalkState);
}

cudaError_t launch_walk_scan(const DeviceIndex& ix, const SearchConfig& cfg, uint32_t n,
                             Scratch& s, cudaStream_t stream) {
    WalkParams p;
    p.q = s.q;
    p.qnorm = s.qnorm;
    p.status = s.status;
    p.cdist = s.cdist;
    p.ctag = s.ctag;
    p.fdist = s.fdist;
    p.ftag = s.ftag;
    p.fd_by_fine = s.dots;
    p.hdist = s.hdist;
    p.htag = s.htag;
    p.hcnt = s.hcnt;
    p.stationary = ix.stationary;
    p.ins_head = ix.ins_n ? ix.ins_head : nullptr;
    p.ins_next = ix.ins_next;
    p.n_base = ix.n;
    p.stat_sorted = ix.stat_sorted;
    p.stat_fine = ix.stat_fine;
    p.cell_start = ix.cell_start;
    p.mdo = ix.min_dist_offset;
    p.offsets = ix.offsets;
    p.codes = ix.codes;
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
    p.rr = cfg.radius_rate;
    p.rr_one = cfg.radius_rate == 1.0;
    const size_t smem = walk_smem_bytes(ix, s.T) - sizeof(WalkState);  // the dynamic part
    // Wide blocks where there is at most one per SM: only the distances of candidate cells
    // are parallel over a query's threads. One query over 200k points: the
    // walk's distances take 0.37 ms of it with 512 threads, 0.52 with 128; with more queries than
    // SMs four narrow blocks per SM hide each other's latency.
    if (n <= (uint32_t)sm_count()) {
        ensure_max_dynamic_smem(k_walk_scan<512>, 208 * 1024);
        k_walk_scan<512><<<n, 512, smem, stream>>>(p);
    } else {
        ensure_max_dynamic_smem(k_walk_scan<128>, 208 * 1024);
        k_walk_scan<128><<<n, 128, smem, stream>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace pgpu
