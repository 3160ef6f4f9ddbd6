// K4 (batched form): candidate gather / dedup / distance / top-K as one
// persistent work-stealing kernel.
//
// Same results as k_candidates (query.cu), organised for heavy-tailed
// candidate counts and for CUDA-graph capture (no host round trip):
//  * k_plan_items turns every query with C > 0 non-unique candidates into
//    P = min(64, ceil(C / chunk)) work items; item p of a query owns the
//    candidate ids whose hash h (32 bits) has floor(h * P / 2^32) = p, so the items of a query
//    deduplicate disjoint id sets (each fits the shared-memory set) and can be
//    processed by different CTAs. Queries without candidates get their padded
//    output ((-1, FLT_MAX) x K) right there.
//    Queries of at most kSmallMax go to k_candidates_small (one warp each), dense
//    ones to the membership rows below.
//  * k_candidates_ws is a persistent grid that claims items with an atomic
//    counter (work stealing). Each item yields an exact top-K over its id
//    partition; the last item of a query to finish merges the P partial lists
//    (threadfence + arrival counter) into the final ascending (distance, id)
//    top-K. Distances follow the reference's lane order (cuLSH_Kernels.cu:301-348)
//    exactly as in k_candidates.
//  * A partition that does not fit the shared-memory set raises an overflow
//    count instead of spilling; the host then re-runs the search through the
//    arena-based kernel (rare: more than ~65k non-unique candidates for one
//    query).
#include <atomic>
#include <cfloat>

#include <cuda_bf16.h>

#include <algorithm>

#include "culsh_internal.cuh"
#include "topk_common.cuh"

namespace culsh {
namespace {

constexpr uint32_t kPartSalt = 0x5bd1e995u;
constexpr int GCH = 256;               // bucket slots scanned per gather chunk

constexpr int PT_PLAN = 256;           // queries per planning block

// One thread per query: partition count, a block scan, one atomic range
// reservation per block, so every query's items are contiguous.
__global__ void __launch_bounds__(PT_PLAN) k_plan_items(WsArgs a) {
    __shared__ uint32_t ws[PT_PLAN / 32];
    __shared__ uint32_t s_base;
    __shared__ uint8_t s_empty[PT_PLAN];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int q0 = blockIdx.x * PT_PLAN;
    const int q = q0 + tid < a.Q ? (a.order ? (int)a.order[q0 + tid] : q0 + tid) : a.Q;
    uint32_t P = 0;
    bool dense = false, small = false;
    if (q < a.Q) {
        const unsigned long long C = a.cnu[q];
        // near-exhaustive candidate sets go to the bitmap kernel instead
        dense = C >= a.dense_min;
        // (FP32 form, enough queries to fill the device: one item while its set
        // holds every candidate, since each item scans the query's whole list)
        P = (C == 0 || dense) ? 0u
            : C <= a.whole        ? 1u
                                  : (uint32_t)min((unsigned long long)a.pmax, (C + a.chunk - 1) / a.chunk);
        if (dense) a.dense_q[atomicAdd(a.n_dense, 1u)] = q;
        // a handful of candidates: one warp each (k_candidates_small)
        small = !dense && C > 0 && C <= a.small_max;
        if (small) P = 0;
    }
    const uint32_t sm = __ballot_sync(0xffffffffu, small);
    if (sm) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(a.n_small, (uint32_t)__popc(sm));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(sm & ((1u << lane) - 1u));
        if (small) a.small_q[at] = q;
    }
    s_empty[tid] = q < a.Q && P == 0 && !dense && !small;
    uint32_t x = P;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (tid == 0) {
        uint32_t t = 0;
        for (int i = 0; i < PT_PLAN / 32; ++i) {
            const uint32_t v = ws[i];
            ws[i] = t;
            t += v;
        }
        // More items than the partial-list buffers hold: the work-stealing
        // kernel then runs nothing and the host uses the per-query kernel.
        const uint32_t base = t ? atomicAdd(a.n_items, t) : 0u;
        if (t && (unsigned long long)base + t > a.item_cap) atomicOr(a.overflow, 1u);
        s_base = base;
    }
    __syncthreads();
    if (q < a.Q) {
        const uint32_t off = s_base + ws[w] + x - P;
        a.q_items[q] = (int)P;
        a.q_off[q] = (int)off;
        a.q_done[q] = 0;
        a.cu[q] = 0;
        for (uint32_t k = 0; k < P && off + k < a.item_cap; ++k) {
            a.item_q[off + k] = q;
            a.item_p[off + k] = (uint8_t)k;
        }
    }
    // Queries without candidates: padded output ((-1, FLT_MAX) x K), written
    // cooperatively so that the stores coalesce.
    const int nq = min(PT_PLAN, a.Q - q0);
    const int K = a.K;
    for (int i = tid; i < nq * K; i += PT_PLAN) {
        const int ql = i / K;
        if (s_empty[ql]) {
            const int64_t qq = a.order ? (int64_t)a.order[q0 + ql] : (int64_t)(q0 + ql);
            const int64_t o = qq * K + (i - ql * K);
            a.out_ids[o] = -1;
            a.out_d[o] = FLT_MAX;
        }
    }
}

// Locality order of the queries: a counting sort into kOrderBins bins of the
// home bucket of table 0 (bucket indices follow the lexicographic order of
// the codes, so nearby bins hold nearby points); queries without a home
// bucket go to the last bin. Order within a bin is arbitrary.
__device__ __forceinline__ uint32_t order_bin(const WsArgs& a, int q) {
    const int32_t b = a.qbuckets[(int64_t)q * a.T];   // table 0, probe 0
    const uint64_t b0 = a.boff[1] - a.boff[0];
    return b < 0 || b0 == 0 ? (uint32_t)kOrderBins : (uint32_t)((uint64_t)b * kOrderBins / b0);
}

__global__ void k_order_hist(WsArgs a) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < a.Q) atomicAdd(a.order_bins + order_bin(a, q), 1u);
}

// Exclusive scan of kOrderBins + 1 counters in one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_order_scan(WsArgs a) {
    constexpr int PER = (kOrderBins + 1 + 1023) / 1024;
    __shared__ uint32_t warp_sum[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t v[PER], tot = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid * PER + k;
        v[k] = i <= kOrderBins ? a.order_bins[i] : 0u;
        tot += v[k];
    }
    uint32_t x = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t s = warp_sum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sum[lane] = s - warp_sum[lane];
    }
    __syncthreads();
    uint32_t run = warp_sum[w] + x - tot;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = tid * PER + k;
        if (i <= kOrderBins) a.order_bins[i] = run;
        run += v[k];
    }
}

__global__ void k_order_scatter(WsArgs a) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < a.Q) a.order[atomicAdd(a.order_bins + order_bin(a, q), 1u)] = (uint32_t)q;
}

// ---- FP32 form ----
// Top-K of an item by selection instead of insertion: the item's distances
// take the place of its hash set as (distance bits, id) words, one histogram
// pass over the distances' range (two or three where many share a bin) finds a
// threshold that K of them and few more do not exceed, and those few are
// sorted. Kept sorted lists (one per warp, merged by one warp) cost a warp-wide
// insertion of some 150 cycles per entry, and with K = 100 nearly every
// candidate of an item was inserted (a serving burst over 10M points, K 10 and
// 100: 8.5 ms of this kernel, now 4.6).

struct SelectSmem {
    uint32_t hist[256];
    uint32_t lo, hi, valid;   // range and count of the finite distances
    uint32_t m, bin, rest;
};
constexpr uint32_t kNoDist = 0xFFFFFFFFu;   // distance bits of an entry that is never listed

// Chooses from ent[0 .. n) at least the min(K, valid) smallest (distance, id)
// entries, sorts them and leaves their positions in idx; returns
// min(K, valid). All WT threads; sm.lo, hi and valid are set and visible.
template <int WT>
__device__ __forceinline__ uint32_t block_top(const unsigned long long* ent, uint32_t n, uint32_t K, uint32_t* idx,
                                              SelectSmem& sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lo = sm.lo, valid = sm.valid;
    uint32_t edge = 0, sh = 32;   // chosen: (bits - lo) >> sh <= edge
    if (valid > K && valid > 32) {
        uint32_t prefix = 0, want = K;
        for (int top = 32 - __clz((int)(sm.hi - lo)); top > 0;) {
            const int s = max(top - 8, 0);
            for (int b = tid; b < 256; b += WT) sm.hist[b] = 0;
            __syncthreads();
            for (uint32_t e = tid; e < n; e += WT) {
                const uint32_t v = (uint32_t)(ent[e] >> 32) - lo;
                if ((uint32_t)(ent[e] >> 32) != kNoDist && (top >= 32 ? 0u : v >> top) == prefix)
                    atomicAdd(&sm.hist[(v >> s) & ((1u << (top - s)) - 1u)], 1u);
            }
            __syncthreads();
            if (warp == 0) {
                uint32_t mine = 0;
#pragma unroll
                for (int b = 0; b < 8; ++b) mine += sm.hist[lane * 8 + b];
                uint32_t x = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == __ffs((int)__ballot_sync(0xffffffffu, x >= want)) - 1) {
                    uint32_t r = want - (x - mine), b = (uint32_t)lane * 8;
                    while (sm.hist[b] < r) r -= sm.hist[b++];
                    sm.bin = b;
                    sm.rest = r;
                }
            }
            __syncthreads();
            prefix = (prefix << (top - s)) | sm.bin;
            want = sm.rest;
            top = s;
            edge = prefix;
            sh = (uint32_t)s;
            // entries up to this bin: K - want below it and the bin itself
            const bool few = K - want + sm.hist[sm.bin] <= max(K + K / 2, 32u);
            __syncthreads();
            if (few) break;   // uniform
        }
    }
    if (tid == 0) sm.m = 0;
    __syncthreads();
    for (uint32_t b = warp * 32; b < n; b += WT) {
        const uint32_t e = b + lane;
        const uint32_t bits = e < n ? (uint32_t)(ent[e] >> 32) : kNoDist;
        const bool take = bits != kNoDist && (sh >= 32 || ((bits - lo) >> sh) <= edge);
        const uint32_t bal = __ballot_sync(0xffffffffu, take);
        uint32_t at = 0;
        if (lane == 0 && bal) at = atomicAdd(&sm.m, (uint32_t)__popc(bal));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & ((1u << lane) - 1u));
        if (take) idx[at] = e;
    }
    __syncthreads();
    const uint32_t m = sm.m;
    auto key = [&](uint32_t i) { return i == 0xFFFFFFFFu ? ~0ull : ent[i]; };
    if (m <= 32) {
        if (warp == 0) {
            uint32_t i = lane < (int)m ? idx[lane] : 0xFFFFFFFFu;
            unsigned long long v = key(i);
#pragma unroll
            for (int a = 2; a <= 32; a <<= 1) {
#pragma unroll
                for (int b = a >> 1; b > 0; b >>= 1) {
                    const unsigned long long ov = __shfl_xor_sync(0xffffffffu, v, b);
                    const uint32_t oi = __shfl_xor_sync(0xffffffffu, i, b);
                    const bool keep_min = ((lane & b) == 0) == ((lane & a) == 0);
                    if (ov != v && (ov < v) == keep_min) {
                        v = ov;
                        i = oi;
                    }
                }
            }
            if (lane < (int)m) idx[lane] = i;
        }
        __syncthreads();
        return min(K, valid);
    }
    uint32_t P = 64;
    while (P < m) P <<= 1;
    for (uint32_t e = m + tid; e < P; e += WT) idx[e] = 0xFFFFFFFFu;
    __syncthreads();
    for (uint32_t a = 2; a <= P; a <<= 1)
        for (uint32_t b = a >> 1; b > 0; b >>= 1) {
            for (uint32_t t = tid; t < P / 2; t += WT) {
                const uint32_t x = 2 * t - (t & (b - 1)), y = x + b;
                const uint32_t ix = idx[x], iy = idx[y];
                if ((key(ix) > key(iy)) == ((x & a) == 0)) {
                    idx[x] = iy;
                    idx[y] = ix;
                }
            }
            __syncthreads();
        }
    return min(K, valid);
}

// Hash of an id for the set and the partitions.
__device__ __forceinline__ uint32_t id_hash(uint32_t x) {
    x *= 0x9E3779B1u;
    x ^= x >> 15;
    x *= 0x85EBCA77u;
    return x ^ (x >> 13);
}

// Queries of at most kSmallMax non-unique candidates, one warp each: bucket list,
// ids, duplicates (lanes that hold the same id), distances and order all within
// the warp. As items of k_candidates_ws they took a block, a cleared hash set
// and a dozen block barriers each: 103 us for 9,700 look-ups of one point, now
// 48 us.
constexpr int SMW = 8;   // warps per block
__global__ void __launch_bounds__(32 * SMW) k_candidates_small(WsArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t s_base[SMW][32];
    __shared__ uint32_t s_pre[SMW][32], s_id[SMW][32];
    __shared__ float s_d[SMW][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int D = a.D, K = a.K, T = a.T, LT = a.L * T;
    float* qs = reinterpret_cast<float*>(smem) + (size_t)w * ((D + 3) & ~3);
    const bool vec = (D & 3) == 0;
    const unsigned int n = *a.n_small;
    unsigned long long tu = 0, tn = 0;
    for (unsigned int i = blockIdx.x * SMW + w; i < n; i += gridDim.x * SMW) {
        const int q = a.small_q[i];
        for (int d = lane; d < D; d += 32) qs[d] = __ldg(a.queries + (int64_t)q * D + d);
        uint32_t nl = 0, C = 0;   // lists, ids
        for (int e0 = 0; e0 < LT; e0 += 128) {
            int32_t j[4];
            uint32_t st[4], sz[4];
            uint64_t gi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * 32 + lane;
                j[u] = -1;
                if (e < LT) {
                    const int l = e / T;
                    j[u] = __ldg(a.qbuckets + (int64_t)l * a.Q * T + (int64_t)q * T + (e - l * T));
                    gi[u] = __ldg(a.boff + l) + (uint32_t)max(j[u], 0);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                sz[u] = 0;
                if (j[u] >= 0) {
                    st[u] = __ldg(a.starts + gi[u]);
                    sz[u] = __ldg(a.sizes + gi[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t has = __ballot_sync(0xffffffffu, sz[u] > 0);
                if (has == 0) continue;
                uint32_t x = sz[u];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (sz[u] > 0) {
                    const uint32_t k = nl + __popc(has & ((1u << lane) - 1u));
                    s_base[w][k] = (uint64_t)((e0 + u * 32 + lane) / T) * (uint64_t)a.N + st[u];
                    s_pre[w][k] = C + x;   // ids up to and including this list
                }
                nl += __popc(has);
                C += __shfl_sync(0xffffffffu, x, 31);
            }
        }
        __syncwarp();
        const bool on = lane < (int)C;
        uint32_t id = 0;
        if (on) {
            uint32_t k = 0;
            while (s_pre[w][k] <= (uint32_t)lane) ++k;
            id = __ldg(a.ids + s_base[w][k] + (lane - (k ? s_pre[w][k - 1] : 0u)));
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, on);
        bool first = false;
        if (on) first = __ffs((int)__match_any_sync(mask, id)) - 1 == lane;
        const uint32_t uniq = __ballot_sync(0xffffffffu, first);
        const uint32_t U = __popc(uniq);
        if (first) s_id[w][__popc(uniq & ((1u << lane) - 1u))] = id;
        __syncwarp();
        const uint32_t per = vec ? 16 : 4, sub = vec ? lane >> 1 : lane >> 3;
        for (uint32_t b = 0; b < U; b += per) {
            const uint32_t e = b + sub;
            const float d = row_distance<2>(a.X + (int64_t)(e < U ? s_id[w][e] : 0u) * D, D, qs, vec, e < U);
            if (e < U && (lane & (vec ? 1 : 7)) == 0) s_d[w][e] = d;
        }
        __syncwarp();
        unsigned long long v = ~0ull;
        if (lane < (int)U && s_d[w][lane] < FLT_MAX)
            v = ((unsigned long long)__float_as_uint(s_d[w][lane]) << 32) | s_id[w][lane];
#pragma unroll
        for (int x = 2; x <= 32; x <<= 1) {
#pragma unroll
            for (int y = x >> 1; y > 0; y >>= 1) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, y);
                if ((o < v) == (((lane & y) == 0) == ((lane & x) == 0))) v = o;
            }
        }
        int32_t* oid = a.out_ids + (int64_t)q * K;
        float* od = a.out_d + (int64_t)q * K;
        for (int k = lane; k < K; k += 32) {
            const bool have = k < 32 && v != ~0ull;
            oid[k] = have ? (int32_t)(uint32_t)v : -1;
            od[k] = have ? __uint_as_float((uint32_t)(v >> 32)) : FLT_MAX;
        }
        if (lane == 0) a.cu[q] = U;
        tu += U;
        tn += C;
        __syncwarp();
    }
    if (lane == 0 && tn) {
        atomicAdd(a.totals + 0, tu);
        atomicAdd(a.totals + 1, tn);
    }
}

// Registers for the row loads in flight: as many blocks per SM are asked for as
// a set of 4,096 slots leaves room for (30 KB each: 7 of 128 threads) or 32
// warps' registers do, which gives 64 to 72 registers; left alone, the compiler
// took 40 to 128 as the code around the loads changed. 10,000 queries of 12,900
// candidates, K = 10, after the gather's change (gather_bucket_ids): 16.0 ms at
// 128 threads and sets of 4,096, 9.6 at 256 and 8,192, now 15.2 and 8.8; 2,000
// queries of 13,800 at 10M x 96 5.6, now 4.8.
constexpr int ws_min_blocks(int WT) { return WT == 512 ? 2 : WT == 256 ? 4 : WT == 128 ? 7 : 8; }
template <int WT, int W_SLOTS, bool STAGED>
__global__ void __launch_bounds__(WT, ws_min_blocks(WT)) k_candidates_ws(WsArgs a) {
    constexpr int WW = WT / 32;
    constexpr uint32_t W_CAP = W_SLOTS / 2;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_ucount, s_skip;
    __shared__ int s_item, s_last;
    __shared__ GatherSmem<WT, GCH> s_gather;
    __shared__ SelectSmem s_sel;
    __shared__ uint64_t s_bar[WW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = a.D, K = a.K, L = a.L, T = a.T;
    const int Dp = (D + 3) & ~3;
    // rows staged by bulk copies where they start on 16-byte boundaries
    const size_t stage_bytes = STAGED ? row_stage_bytes(D) : 0;
    const bool staged = STAGED && row_staged(D) && (reinterpret_cast<uintptr_t>(a.X) & 15) == 0;
    float* stage = reinterpret_cast<float*>(smem + warp * stage_bytes);
    uint32_t phase = 0;
    float* qs = reinterpret_cast<float*>(smem + WW * stage_bytes);
    uint32_t* hset = reinterpret_cast<uint32_t*>(qs + Dp);                        // [W_SLOTS], then the entries
    unsigned long long* ent = reinterpret_cast<unsigned long long*>(hset);       // [W_CAP]
    uint32_t* ulist = hset + W_SLOTS;                                            // [W_CAP], then positions
    float* wd = reinterpret_cast<float*>(ulist + W_CAP);                         // [K] merge of very large partial lists
    uint32_t* wi = reinterpret_cast<uint32_t*>(wd + K);
    // Bit 0 of the overflow word: the plan did not fit (set by k_plan_items,
    // which has finished). Read once and broadcast, so that the whole block
    // returns or none of it does; bit 1 (a set overflow) may be raised by
    // other blocks meanwhile and is left to the host.
    // Thread 0 claims the next item while the block works on the current one.
    if (tid == 0) {
        s_skip = *(volatile unsigned int*)a.overflow & 1u;
        s_item = s_skip ? 0 : (int)atomicAdd(a.next_item, 1u);
        for (int w = 0; w < WW; ++w) stage_bar_init(s_bar + w);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (s_skip) return;
    const int n_items = (int)*a.n_items;
    const bool vec = (D & 3) == 0;
    for (;;) {
        const int item = s_item;
        if (item >= n_items) break;
        int next = 0;
        if (tid == 0) next = (int)atomicAdd(a.next_item, 1u);
        const int q = a.item_q[item];
        const uint32_t p = a.item_p[item];
        const uint32_t P = (uint32_t)a.q_items[q];
        const unsigned long long C = a.cnu[q];
        // as many set slots as the item can need: twice its candidates
        uint32_t slots = W_SLOTS;
        if (P == 1 && C < W_CAP) slots = max(32u, 2u << (31 - __clz((int)C)) << (((uint32_t)C & ((uint32_t)C - 1)) != 0));
        for (int i = tid; i < Dp; i += WT) qs[i] = i < D ? a.queries[(int64_t)q * D + i] : 0.0f;
        for (uint32_t i = tid; i < slots; i += WT) hset[i] = kEmpty32;
        if (tid == 0) s_ucount = 0;
        __syncthreads();

        // Gather this item's id partition from every matched bucket.
        const BucketView bv{a.qbuckets, a.boff, a.starts, a.sizes, a.ids, a.N, L, T, a.Q};
        gather_bucket_ids<WT, GCH, (WT < 256 ? 2 : 1)>(bv, q, s_gather, [&](uint32_t id) {
            const uint32_t h = id_hash(id);
            if (P > 1 && __umulhi(h, P) != p) return;
            set_insert_at(hset, slots - 1, ulist, W_CAP, &s_ucount, id, h);
        });
        __syncthreads();
        uint32_t U = s_ucount;
        if (U > W_CAP) {   // the set overflowed: flag it, finish the protocol with no candidates
            if (tid == 0) atomicOr(a.overflow, 2u);
            U = 0;
        }
        if (tid == 0) {
            s_sel.lo = kNoDist;
            s_sel.hi = s_sel.valid = 0;
        }
        __syncthreads();   // the set is no longer read: its place takes the entries

        // Exact FP32 distances in the reference lane order.
        {
            const uint32_t per = vec ? 16 : 4, sub = vec ? lane >> 1 : lane >> 3;
            const bool lead = (lane & (vec ? 1 : 7)) == 0;
            uint32_t lo = kNoDist, hi = 0, valid = 0;
            for (uint32_t b = warp * per; b < U; b += WW * per) {
                const uint32_t e = b + sub;
                const bool on = e < U;
                const uint32_t id = on ? ulist[e] : 0u;
                const float d = staged ? staged_distance(a.X, D, qs, ulist, b, U, stage, s_bar + warp, phase, a.overflow)
                                       : row_distance(a.X + (int64_t)id * D, D, qs, vec, on);
                if (on && lead) {
                    const uint32_t bits = d < FLT_MAX ? __float_as_uint(d) : kNoDist;
                    ent[e] = ((unsigned long long)bits << 32) | id;
                    if (bits != kNoDist) {
                        lo = min(lo, bits);
                        hi = max(hi, bits);
                        ++valid;
                    }
                }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            valid = __reduce_add_sync(0xffffffffu, valid);
            if (lane == 0 && valid) {
                atomicMin(&s_sel.lo, lo);
                atomicMax(&s_sel.hi, hi);
                atomicAdd(&s_sel.valid, valid);
            }
        }
        __syncthreads();
        uint32_t n = block_top<WT>(ent, U, (uint32_t)K, ulist, s_sel);
        if (tid == 0) {
            atomicAdd(a.cu + q, (unsigned long long)U);
            atomicAdd(a.totals + 0, (unsigned long long)U);
        }
        bool write = P == 1;
        if (P > 1) {
            // Publish this partition's list; the last partition to finish merges.
            float* pd = a.part_d + (int64_t)item * K;
            uint32_t* pi = a.part_i + (int64_t)item * K;
            for (uint32_t k = tid; k < n; k += WT) {
                const unsigned long long v = ent[ulist[k]];
                pd[k] = __uint_as_float((uint32_t)(v >> 32));
                pi[k] = (uint32_t)v;
            }
            if (tid == 0) a.part_n[item] = (int)n;
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.q_done + q, 1u) == P - 1;
            __syncthreads();
            if (s_last) {   // uniform
                __threadfence();
                const int first = a.q_off[q];
                if (P * (uint32_t)K <= W_CAP) {
                    if (tid == 0) {
                        s_sel.lo = kNoDist;
                        s_sel.hi = s_sel.valid = 0;
                    }
                    __syncthreads();
                    for (uint32_t e = tid; e < P * (uint32_t)K; e += WT) {
                        const uint32_t it = e / K, k = e - it * K;
                        unsigned long long v = ~0ull;
                        if ((int)k < *(volatile const int*)(a.part_n + first + it)) {
                            const int64_t o = (int64_t)(first + it) * K + k;
                            const uint32_t bits = __float_as_uint(*(volatile const float*)(a.part_d + o));
                            v = ((unsigned long long)bits << 32) | *(volatile const uint32_t*)(a.part_i + o);
                            atomicMin(&s_sel.lo, bits);
                            atomicMax(&s_sel.hi, bits);
                            atomicAdd(&s_sel.valid, 1u);
                        }
                        ent[e] = v;
                    }
                    __syncthreads();
                    n = block_top<WT>(ent, P * (uint32_t)K, (uint32_t)K, ulist, s_sel);
                    write = true;
                } else if (warp == 0) {
                    int m = 0;
                    float thr_d = FLT_MAX;
                    uint32_t thr_i = 0;
                    for (uint32_t k = 0; k < P; ++k) {
                        const int it = first + (int)k;
                        const int cnt = *(volatile const int*)(a.part_n + it);
                        const float* pd2 = a.part_d + (int64_t)it * K;
                        const uint32_t* pi2 = a.part_i + (int64_t)it * K;
                        for (int e = 0; e < cnt; ++e) {
                            const float d = *(volatile const float*)(pd2 + e);
                            const uint32_t id = *(volatile const uint32_t*)(pi2 + e);
                            if (!lessp(d, id, thr_d, thr_i)) break;
                            warp_insert(wd, wi, m, K, d, id, thr_d, thr_i);
                        }
                    }
                    int32_t* oid = a.out_ids + (int64_t)q * K;
                    float* od = a.out_d + (int64_t)q * K;
                    for (int k = lane; k < K; k += 32) {
                        oid[k] = k < m ? (int32_t)wi[k] : -1;
                        od[k] = k < m ? wd[k] : FLT_MAX;
                    }
                    if (lane == 0) atomicAdd(a.totals + 1, C);
                }
            }
        }
        if (write) {   // uniform
            int32_t* oid = a.out_ids + (int64_t)q * K;
            float* od = a.out_d + (int64_t)q * K;
            for (uint32_t k = tid; k < (uint32_t)K; k += WT) {
                const unsigned long long v = k < n ? ent[ulist[k]] : 0ull;
                oid[k] = k < n ? (int32_t)(uint32_t)v : -1;
                od[k] = k < n ? __uint_as_float((uint32_t)(v >> 32)) : FLT_MAX;
            }
            if (tid == 0) atomicAdd(a.totals + 1, C);
        }
        if (tid == 0) s_item = next;
        __syncthreads();
    }
}

// ---- BF16 form ----
// WT threads per item: WT / 32 warps each keep a sorted top-K list over a
// strided share of the item's candidates (tuned: 64, 128, 256 or 512; wide
// items keep more row gathers in flight per block of shared memory).
// W_SLOTS: shared hash-set slots per item (4096, 8192 or 16384, tuned); an
// item holds at most W_CAP = W_SLOTS / 2 distinct ids. Every item of a query
// scans the query's whole id list and keeps its partition, so larger sets
// (fewer, larger partitions) scan less at the cost of occupancy.
template <int WT, int W_SLOTS>
__global__ void __launch_bounds__(WT) k_candidates_ws_bf16(WsArgs a) {
    constexpr int WW = WT / 32;
    constexpr int W_CAP = W_SLOTS / 2;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_ucount;
    __shared__ int s_item, s_last, s_wn[WW];
    __shared__ GatherSmem<WT, GCH> s_gather;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = a.D, K = a.K, L = a.L, T = a.T;
    const int Dp = (D + 3) & ~3;
    float* qs = reinterpret_cast<float*>(smem);
    uint32_t* hset = reinterpret_cast<uint32_t*>(qs + Dp);
    uint32_t* ulist = hset + W_SLOTS;
    float* wd_all = reinterpret_cast<float*>(ulist + W_CAP);
    uint32_t* wi_all = reinterpret_cast<uint32_t*>(wd_all + WW * K);
    float* wd = wd_all + warp * K;
    uint32_t* wi = wi_all + warp * K;
    // BF16 form: approximate distance and error bound of each candidate.
    float* dA = reinterpret_cast<float*>(wi_all + WW * K);
    float* eA = dA + W_CAP;
    __shared__ float s_tau;
    __shared__ uint32_t s_scount, s_recheck, s_skip;
    // Bit 0 of the overflow word: the plan did not fit (set by k_plan_items,
    // which has finished). Read once and broadcast, so that the whole block
    // returns or none of it does; bit 1 (a set overflow) may be raised by
    // other blocks meanwhile and is left to the host.
    if (tid == 0) s_skip = *(volatile unsigned int*)a.overflow & 1u;
    __syncthreads();
    if (s_skip) return;
    const unsigned int n_items = *a.n_items;
    const bool vec = (D & 3) == 0;

    for (;;) {
        if (tid == 0) s_item = (int)atomicAdd(a.next_item, 1u);
        __syncthreads();
        const int item = s_item;
        if (item >= (int)n_items) break;
        const int q = a.item_q[item];
        const uint32_t p = a.item_p[item];
        const uint32_t P = (uint32_t)a.q_items[q];
        const unsigned long long C = a.cnu[q];
        for (int i = tid; i < Dp; i += WT) qs[i] = i < D ? a.queries[(int64_t)q * D + i] : 0.0f;
        for (int i = tid; i < W_SLOTS; i += WT) hset[i] = kEmpty32;
        if (tid == 0) s_ucount = 0;
        __syncthreads();

        // Gather this item's id partition from every matched bucket.
        const BucketView bv{a.qbuckets, a.boff, a.starts, a.sizes, a.ids, a.N, L, T, a.Q};
        gather_bucket_ids<WT, GCH, 4>(bv, q, s_gather, [&](uint32_t id) {
            if (P > 1 && (uint32_t)(((uint64_t)mix32(id ^ kPartSalt) * P) >> 32) != p) return;
            set_insert(hset, W_SLOTS - 1, ulist, W_CAP, &s_ucount, id);
        });
        __syncthreads();
        uint32_t U = s_ucount;
        if (U > W_CAP) {   // the set overflowed: flag it, finish the protocol with no candidates
            if (tid == 0) atomicOr(a.overflow, 2u);
            U = 0;
        }

        // Exact FP32 distances in the reference lane order over list entries
        // [0, cnt) (entry j is ulist[idx_of(j)]), into per-warp sorted top-K
        // lists; an entry whose distance is already exact (pre) is not loaded.
        int n = 0;
        float thr_d = FLT_MAX;
        uint32_t thr_i = 0;
        auto fp32_pass = [&](uint32_t cnt, auto idx_of, auto pre) {
            fp32_dist_pass<WW>(a.X, D, qs, vec, cnt, idx_of, [&](uint32_t ci) { return ulist[ci]; }, pre, wd, wi, K,
                               n, thr_d, thr_i);
        };
        {
            // Pass 1: BF16 rows. d~ is computed in the reference lane order
            // from the bf16 copy; E bounds |d~ - d| where d is the FP32
            // distance (exact rows: E = 0, since d~ is then d itself; rows
            // with extreme magnitudes: E = inf). Each warp keeps the K
            // smallest upper ends d~ + E; tau, the K-th smallest over the
            // item, caps the distance of its K nearest, so only candidates
            // with d~ - E <= tau can be among them.
            const int per = vec ? 16 : 4;
            for (uint32_t base = warp * per; base < U; base += WW * per) {
                float dt = 0.f, b1 = 0.f, b2 = 0.f;
                uint32_t ci, id;
                bool own;
                if (vec) {
                    ci = base + (lane >> 1);
                    const int h = lane & 1;
                    const bool valid = ci < U;
                    id = valid ? ulist[ci] : 0u;
                    const uint16_t* rowp = a.xb + (int64_t)id * D;
                    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
                    if (valid) {
#pragma unroll 8
                        for (int c = 4 * h; c < D; c += 8) {
                            const uint2 raw = __ldg(reinterpret_cast<const uint2*>(rowp + c));
                            const float x0 = __uint_as_float(raw.x << 16), x1 = __uint_as_float(raw.x & 0xFFFF0000u);
                            const float x2 = __uint_as_float(raw.y << 16), x3 = __uint_as_float(raw.y & 0xFFFF0000u);
                            const float4 qv = *reinterpret_cast<const float4*>(qs + c);
                            const float d0 = __fsub_rn(qv.x, x0), d1 = __fsub_rn(qv.y, x1);
                            const float d2 = __fsub_rn(qv.z, x2), d3 = __fsub_rn(qv.w, x3);
                            s0 = __fmaf_rn(d0, d0, s0);
                            s1 = __fmaf_rn(d1, d1, s1);
                            s2 = __fmaf_rn(d2, d2, s2);
                            s3 = __fmaf_rn(d3, d3, s3);
                            b1 = __fmaf_rn(fabsf(x0), fabsf(d0), b1);
                            b1 = __fmaf_rn(fabsf(x1), fabsf(d1), b1);
                            b1 = __fmaf_rn(fabsf(x2), fabsf(d2), b1);
                            b1 = __fmaf_rn(fabsf(x3), fabsf(d3), b1);
                            b2 = __fmaf_rn(x0, x0, b2);
                            b2 = __fmaf_rn(x1, x1, b2);
                            b2 = __fmaf_rn(x2, x2, b2);
                            b2 = __fmaf_rn(x3, x3, b2);
                        }
                    }
                    const float o0 = __shfl_xor_sync(0xffffffffu, s0, 1), o1 = __shfl_xor_sync(0xffffffffu, s1, 1);
                    const float o2 = __shfl_xor_sync(0xffffffffu, s2, 1), o3 = __shfl_xor_sync(0xffffffffu, s3, 1);
                    const float t0 = __fadd_rn(s0, o0), t1 = __fadd_rn(s1, o1), t2 = __fadd_rn(s2, o2),
                                t3 = __fadd_rn(s3, o3);
                    dt = __fadd_rn(__fadd_rn(t0, t2), __fadd_rn(t1, t3));
                    b1 = __fadd_rn(b1, __shfl_xor_sync(0xffffffffu, b1, 1));
                    b2 = __fadd_rn(b2, __shfl_xor_sync(0xffffffffu, b2, 1));
                    own = valid && h == 0;
                } else {
                    ci = base + (lane >> 3);
                    const int r = lane & 7;
                    const bool valid = ci < U;
                    id = valid ? ulist[ci] : 0u;
                    const uint16_t* rowp = a.xb + (int64_t)id * D;
                    float sacc = 0.f;
                    if (valid)
#pragma unroll 4
                        for (int c = r; c < D; c += 8) {
                            const float x = __uint_as_float((uint32_t)__ldg(rowp + c) << 16);
                            const float df = __fsub_rn(qs[c], x);
                            sacc = __fmaf_rn(df, df, sacc);
                            b1 = __fmaf_rn(fabsf(x), fabsf(df), b1);
                            b2 = __fmaf_rn(x, x, b2);
                        }
                    const float t = __fadd_rn(sacc, __shfl_xor_sync(0xffffffffu, sacc, 4));
                    const float u = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 2));
                    dt = __fadd_rn(u, __shfl_xor_sync(0xffffffffu, u, 1));
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) {
                        b1 = __fadd_rn(b1, __shfl_xor_sync(0xffffffffu, b1, o));
                        b2 = __fadd_rn(b2, __shfl_xor_sync(0xffffffffu, b2, o));
                    }
                    own = valid && r == 0;
                }
                float e = 0.f, up = 0.f;
                if (own) {
                    const uint8_t fl = __ldg(a.xflag + id);
                    if (fl == 1) {
                        e = 0.f;
                    } else if (fl == 2 || !(dt <= FLT_MAX)) {
                        e = __int_as_float(0x7f800000);
                    } else {
                        // E = c1 * d~ + c2 * (2 rho b1 + rho^2 b2), upward roundings
                        const float rho = 0.00393676758f;   // 2^-8 (1 + 2^-7), bf16 rounding relative to |x~|
                        const float delta = __fmaf_ru(rho * rho, b2, __fmul_ru(2.0f * rho, b1));
                        e = __fmaf_ru(a.e_c1, dt, __fmul_ru(a.e_c2, delta));
                    }
                    dA[ci] = dt;
                    eA[ci] = e;
                    up = __fadd_ru(dt, e);
                }
                uint32_t want = __ballot_sync(0xffffffffu, own && lessp(up, ci, thr_d, thr_i));
                while (want) {
                    const int src = __ffs(want) - 1;
                    want &= want - 1;
                    const float cdv = __shfl_sync(0xffffffffu, up, src);
                    const uint32_t cid = __shfl_sync(0xffffffffu, ci, src);
                    if (lessp(cdv, cid, thr_d, thr_i)) warp_insert(wd, wi, n, K, cdv, cid, thr_d, thr_i);
                }
            }
            if (lane == 0) s_wn[warp] = n;
            if (tid == 0) s_scount = s_recheck = 0;
            __syncthreads();
            if (warp == 0) {
                for (int w = 1; w < WW; ++w) {
                    const int nw = s_wn[w];
                    for (int e = 0; e < nw; ++e) {
                        const float d = wd_all[w * K + e];
                        const uint32_t id = wi_all[w * K + e];
                        if (!lessp(d, id, thr_d, thr_i)) break;
                        warp_insert(wd, wi, n, K, d, id, thr_d, thr_i);
                    }
                }
                if (lane == 0) s_tau = n == K ? wd[K - 1] : __int_as_float(0x7f800000);
            }
            __syncthreads();
            // Shortlist (into the free hash-set memory): d~ - E <= tau.
            const float tau = s_tau;
            uint32_t* slist = hset;
            uint32_t rc = 0;
            for (uint32_t ci = tid; ci < U; ci += WT)
                if (__fsub_rd(dA[ci], eA[ci]) <= tau) {
                    slist[atomicAdd(&s_scount, 1u)] = ci;
                    rc += eA[ci] != 0.f;
                }
            if (rc) atomicAdd(&s_recheck, rc);
            __syncthreads();
            if (tid == 0 && s_recheck) atomicAdd(a.rechecked, (unsigned long long)s_recheck);
            // Pass 2: exact distances of the shortlist (re-read in FP32 only
            // for rows whose bf16 copy is inexact).
            n = 0;
            thr_d = FLT_MAX;
            thr_i = 0;
            fp32_pass(s_scount, [&](uint32_t j) { return slist[j]; }, [&](uint32_t ci, float& d) {
                if (eA[ci] != 0.f) return false;
                d = dA[ci];
                return true;
            });
        }
        if (lane == 0) s_wn[warp] = n;
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < WW; ++w) {
                const int nw = s_wn[w];
                for (int e = 0; e < nw; ++e) {
                    const float d = wd_all[w * K + e];
                    const uint32_t id = wi_all[w * K + e];
                    if (!lessp(d, id, thr_d, thr_i)) break;
                    warp_insert(wd, wi, n, K, d, id, thr_d, thr_i);
                }
            }
            if (lane == 0) {
                atomicAdd(a.cu + q, (unsigned long long)U);
                atomicAdd(a.totals + 0, (unsigned long long)U);
            }
        }
        if (P == 1) {
            if (warp == 0) {
                int32_t* oid = a.out_ids + (int64_t)q * K;
                float* od = a.out_d + (int64_t)q * K;
                for (int k = lane; k < K; k += 32) {
                    oid[k] = k < n ? (int32_t)wi[k] : -1;
                    od[k] = k < n ? wd[k] : FLT_MAX;
                }
                if (lane == 0) atomicAdd(a.totals + 1, C);
            }
        } else {
            // Publish this partition's list; the last partition to finish merges.
            if (warp == 0) {
                float* pd = a.part_d + (int64_t)item * K;
                uint32_t* pi = a.part_i + (int64_t)item * K;
                for (int k = lane; k < n; k += 32) {
                    pd[k] = wd[k];
                    pi[k] = wi[k];
                }
                if (lane == 0) a.part_n[item] = n;
                __threadfence();
                __syncwarp();
                if (lane == 0) s_last = atomicAdd(a.q_done + q, 1u) == P - 1;
                __syncwarp();
                if (s_last) {
                    __threadfence();
                    n = 0;
                    thr_d = FLT_MAX;
                    thr_i = 0;
                    const int first = a.q_off[q];
                    for (uint32_t k = 0; k < P; ++k) {
                        const int it = first + (int)k;
                        const int m = *(volatile const int*)(a.part_n + it);
                        const float* pd2 = a.part_d + (int64_t)it * K;
                        const uint32_t* pi2 = a.part_i + (int64_t)it * K;
                        for (int e = 0; e < m; ++e) {
                            const float d = *(volatile const float*)(pd2 + e);
                            const uint32_t id = *(volatile const uint32_t*)(pi2 + e);
                            if (!lessp(d, id, thr_d, thr_i)) break;
                            warp_insert(wd, wi, n, K, d, id, thr_d, thr_i);
                        }
                    }
                    int32_t* oid = a.out_ids + (int64_t)q * K;
                    float* od = a.out_d + (int64_t)q * K;
                    for (int k = lane; k < K; k += 32) {
                        oid[k] = k < n ? (int32_t)wi[k] : -1;
                        od[k] = k < n ? wd[k] : FLT_MAX;
                    }
                    if (lane == 0) atomicAdd(a.totals + 1, C);
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace

// Dense form: a query whose non-unique candidates reach dense_min (a large
// share of the dataset) is deduplicated in an N-bit bitmap in shared memory
// rather than in id partitions; the bitmap is then compacted 8,192 bits at a
// time into a candidate list for the exact distance pass. Persistent grid,
// one query per CTA at a time.
constexpr int DT = 256;
constexpr int DW = DT / 32;

// Shared memory of scan_words: candidate ids of DT words, per-warp lists.
struct ScanSmem {
    uint32_t* clist;   // [DT * 32]
    float* wd;         // [DW][K]
    uint32_t* wi;      // [DW][K]
};
__device__ __forceinline__ ScanSmem scan_smem(void* p, int K) {
    ScanSmem s;
    s.clist = static_cast<uint32_t*>(p);
    s.wd = reinterpret_cast<float*>(s.clist + DT * 32);
    s.wi = reinterpret_cast<uint32_t*>(s.wd + DW * K);
    return s;
}
constexpr size_t scan_bytes(int K) { return 4 * (size_t)DT * 32 + (size_t)DW * K * (sizeof(float) + sizeof(uint32_t)); }

// Exact top-K of the points whose bits are set in words word(0 .. nwords),
// DT words at a time, written padded to oid / od by one block; returns the
// number of set bits (every thread).
template <class Word>
__device__ __forceinline__ unsigned long long scan_words(const float* __restrict__ X, int D, int K, uint32_t nwords,
                                                         Word word, const float* qs, bool vec, const ScanSmem& sc,
                                                         int32_t* oid, float* od) {
    __shared__ uint32_t s_ws[DW], s_wn[DW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* wd = sc.wd + warp * K;
    uint32_t* wi = sc.wi + warp * K;
    int n = 0;
    float thr_d = FLT_MAX;
    uint32_t thr_i = 0;
    unsigned long long U = 0;
    for (uint32_t w0 = 0; w0 < nwords; w0 += DT) {
        const uint32_t w = w0 + tid;
        const uint32_t bits = w < nwords ? word(w) : 0u;
        // block exclusive scan of the set-bit counts
        const uint32_t c = __popc(bits);
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_ws[warp] = x;
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (int i = 0; i < DW; ++i) {
            const uint32_t v = s_ws[i];
            before += i < warp ? v : 0u;
            total += v;
        }
        uint32_t k = before + x - c;
        for (uint32_t m = bits; m; m &= m - 1) sc.clist[k++] = w * 32 + (uint32_t)(__ffs((int)m) - 1);
        __syncthreads();
        fp32_dist_pass<DW>(X, D, qs, vec, total, [](uint32_t j) { return j; },
                           [&](uint32_t ci) { return sc.clist[ci]; }, [](uint32_t, float&) { return false; }, wd, wi,
                           K, n, thr_d, thr_i);
        U += total;
        __syncthreads();
    }
    if (lane == 0) s_wn[warp] = n;
    __syncthreads();
    if (warp == 0) {
        for (int ww = 1; ww < DW; ++ww) {
            const int nw = s_wn[ww];
            for (int e = 0; e < nw; ++e) {
                const float d = sc.wd[ww * K + e];
                const uint32_t id = sc.wi[ww * K + e];
                if (!lessp(d, id, thr_d, thr_i)) break;
                warp_insert(wd, wi, n, K, d, id, thr_d, thr_i);
            }
        }
        for (int k = lane; k < K; k += 32) {
            oid[k] = k < n ? (int32_t)wi[k] : -1;
            od[k] = k < n ? wd[k] : FLT_MAX;
        }
    }
    return U;
}

__global__ void __launch_bounds__(DT, 1) k_candidates_dense(WsArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ GatherSmem<DT, GCH> s_gather;
    __shared__ int s_q;
    const int tid = threadIdx.x;
    const int D = a.D, K = a.K, L = a.L, T = a.T;
    const int Dp = (D + 3) & ~3;
    const uint32_t nwords = (uint32_t)((a.N + 31) >> 5);
    const uint32_t nwp = (nwords + 3) & ~3u;
    float* qs = reinterpret_cast<float*>(smem);
    uint32_t* bits = reinterpret_cast<uint32_t*>(qs + Dp);
    const ScanSmem sc = scan_smem(bits + nwp, K);
    const bool vec = (D & 3) == 0;
    const unsigned int ndense = *a.n_dense;

    for (;;) {
        if (tid == 0) {
            const unsigned int k = atomicAdd(a.dense_next, 1u);
            s_q = k < ndense ? a.dense_q[k] : -1;
        }
        __syncthreads();
        const int q = s_q;
        if (q < 0) break;
        for (int i = tid; i < Dp; i += DT) qs[i] = i < D ? a.queries[(int64_t)q * D + i] : 0.0f;
        for (uint32_t i = tid; i < nwords; i += DT) bits[i] = 0u;
        __syncthreads();
        const BucketView bv{a.qbuckets, a.boff, a.starts, a.sizes, a.ids, a.N, L, T, a.Q};
        gather_bucket_ids<DT, GCH, 4>(bv, q, s_gather,
                                      [&](uint32_t id) { atomicOr(&bits[id >> 5], 1u << (id & 31)); });
        __syncthreads();

        const unsigned long long U = scan_words(a.X, D, K, nwords, [&](uint32_t w) { return bits[w]; }, qs, vec, sc,
                                                a.out_ids + (int64_t)q * K, a.out_d + (int64_t)q * K);
        if (tid == 0) {
            a.cu[q] = U;
            atomicAdd(a.totals + 0, U);
            atomicAdd(a.totals + 1, a.cnu[q]);
        }
        __syncthreads();
    }
}

// Exact scan of the queries the tensor-core merge could not finish (their
// survivors outgrew its lists): the candidates come from the query's
// membership row, distances and top-K as in k_candidates_dense.
__global__ void __launch_bounds__(DT, 1) k_knn_scan_rows(KnnSearch k) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, D = k.D, K = k.K;
    float* qs = reinterpret_cast<float*>(smem);
    const ScanSmem sc = scan_smem(qs + ((D + 3) & ~3), K);
    const unsigned int nf = *k.n_fallback;
    for (unsigned int f = blockIdx.x; f < nf; f += gridDim.x) {
        const int i = k.fallback[f], q = k.dense_q[i];
        for (int d = tid; d < D; d += DT) qs[d] = k.queries[(int64_t)q * D + d];
        __syncthreads();
        const uint32_t* row = k.bm + (int64_t)i * k.nwp;
        scan_words(k.X, D, K, (uint32_t)((k.N + 31) >> 5), [&](uint32_t w) { return __ldg(row + w); }, qs,
                   (D & 3) == 0, sc, k.out_ids + (int64_t)q * K, k.out_d + (int64_t)q * K);
        __syncthreads();
    }
}

// Membership rows of the dense queries for the tensor-core path
// (knn_tc.cu): query k of the dense list gets row bm[k][0 .. nwp) with bit i
// set when point i is one of its candidates (nwp - ceil(N/32) padding words
// stay zero). The bits are set in an N-bit bitmap in shared memory from the
// query's bucket ids (every matched bucket over the L tables and T probes,
// as the reference's candidate lists, cuLSH_SearchTables.cu:321-364) and
// copied out once; their count is the query's unique candidate count.
// Persistent grid, one query per CTA at a time, 1024 threads. A dataset whose
// bits do not fit shared memory (more than about 1.6M points) takes one sweep
// over the query's ids per segment of it. The matched buckets of a chunk of
// slots form one flattened list of ids; warps take 32 x BU of them in turn
// (BU loads in flight per lane) and OR their bits in. Two kinds of buckets do
// better, both laid out once per index; the set is the same either way:
//  - a bucket row (a.big_rows, of the largest buckets; up to BROWS of them per
//    query) is ORed into the words as they are copied out: one 16-byte load
//    per four words instead of one shared-memory atomic per id;
//  - a bank list (k_bank_fill, other buckets of 512 ids or more, where one
//    segment holds the dataset): 16-bit entries, 32 of which a warp ORs into
//    32 different banks.
// Bound by the shared-memory atomics. 10,000 queries of 743k ids each over 1M
// points: 4.65 ms id by id, 3.8 with bucket rows, 3.45 with bank lists too.
// Prefetching the next entries into registers spills (4.23 ms when the rest
// took 3.6); padding entries that are compared instead of ORed into a spare
// row 4.97.
constexpr int BT = 1024;
constexpr int BU = 8;
constexpr int BCH = 512;   // (table, probe) slots per compaction chunk
constexpr uint32_t BROWS = 64;

struct BitmapSmem {
    // id lists of a chunk's matched buckets (whole buckets, or the tails of
    // bank lists), as one flattened range
    uint64_t lbase[BCH];    // offset of each list (top bit: in the tails)
    uint32_t lpre[BCH];     // ids up to and including each list
    // bank lists: first entry and units up to and including each list
    uint64_t bbase[BCH];
    uint32_t bsize[BCH];    // groups of 128 entries
    uint32_t bpre[BCH];
    uint32_t wsum[2][BT / 32];
    uint32_t nl, nb;
    uint32_t nrow;          // matched buckets with a bucket row (may exceed BROWS)
    uint32_t row[BROWS];    // their rows
};

// First of the n ascending inclusive prefixes that exceeds i.
__device__ __forceinline__ uint32_t list_of(const uint32_t* pre, uint32_t n, uint32_t i) {
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (pre[mid] > i) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Row of global bucket gi among the n ascending bucket numbers of big_gi, -1
// if it has none.
__device__ __forceinline__ int big_row(const uint64_t* __restrict__ big_gi, int n, uint64_t gi) {
    int lo = 0, hi = n - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const uint64_t v = __ldg(big_gi + mid);
        if (v == gi) return mid;
        if (v < gi) lo = mid + 1;
        else hi = mid - 1;
    }
    return -1;
}

// Ids of the ascending list b[0 .. n) below p.
__device__ __forceinline__ uint32_t ids_below(const uint32_t* __restrict__ b, uint32_t n, uint32_t p) {
    uint32_t lo = 0;
    while (n > 0) {
        const uint32_t half = n >> 1;
        const bool below = __ldg(b + lo + half) < p;
        lo = below ? lo + half + 1 : lo;
        n = below ? n - half - 1 : half;
    }
    return lo;
}

// Sets the bit of a bank-list entry (the low 16 bits of e: word row << 5 | bit)
// in the column of words at `col`.
__device__ __forceinline__ void or_entry(uint32_t* col, uint32_t e) {
    atomicOr(col + (e & 0xFFE0u), __funnelshift_l(0u, 1u, e));   // 1 << (e & 31)
}

// Sample words of a segment for f = 32 / G: chunk c's i-th point is bit
// (c % G) f of word c / G + i s32 / G, so G chunks share their reads.
template <int G>
__device__ __forceinline__ void sample_words(const uint32_t* bits, uint32_t* srow, int s32) {
    const int step = s32 / G;   // s32 is a multiple of 4
    for (int c = threadIdx.x; c < step; c += BT) {
        uint32_t word[G];
#pragma unroll
        for (int j = 0; j < G; ++j) word[j] = 0;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
            const uint32_t w = bits[c + i * step];
#pragma unroll
            for (int j = 0; j < G; ++j) word[j] |= ((w >> (j * (32 / G))) & 1u) << i;
        }
#pragma unroll
        for (int j = 0; j < G; ++j) srow[c * G + j] = word[j];
    }
}

// ORs unit u of the bank lists of g (BU groups of one list) into the bitmap;
// one warp, every load in flight before the first is ORed in.
__device__ __forceinline__ void or_bank_unit(const WsArgs& a, const BitmapSmem& g, uint32_t u, uint32_t* bits) {
    const int lane = threadIdx.x & 31;
    const uint32_t h = list_of(g.bpre, g.nb, u);
    const uint32_t first = (u - (h ? g.bpre[h - 1] : 0u)) * BU;
    const uint32_t cnt = min((uint32_t)BU, g.bsize[h] - first);
    // lane b's four entries of a group are bits of words with bank b, so a
    // warp's atomics never share a bank
    const uint2* src = reinterpret_cast<const uint2*>(a.bank + g.bbase[h]) + (size_t)first * 32 + lane;
    uint32_t* col = bits + lane;
    uint2 v[BU];
#pragma unroll
    for (int b = 0; b < BU; ++b)
        if (b < (int)cnt) v[b] = __ldg(src + b * 32);
#pragma unroll
    for (int b = 0; b < BU; ++b) {
        if (b >= (int)cnt) break;   // warp-uniform
        or_entry(col, v[b].x);
        or_entry(col, v[b].x >> 16);
        or_entry(col, v[b].y);
        or_entry(col, v[b].y >> 16);
    }
}

// ORs ids [32 BU u, 32 BU (u + 1)) of the flattened id lists into the bitmap
// (one warp): short lists share a unit, so that its loads are in flight
// together whatever the list lengths.
__device__ __forceinline__ void or_id_unit(const WsArgs& a, const BitmapSmem& g, uint32_t u, uint32_t total,
                                           uint32_t* bits, uint32_t p0) {
    const int lane = threadIdx.x & 31;
    uint32_t h = list_of(g.lpre, g.nl, u * (32 * BU));
    uint32_t v[BU];
#pragma unroll
    for (int b = 0; b < BU; ++b) {
        const uint32_t i = u * (32 * BU) + b * 32 + lane;
        if (i < total) {
            while (g.lpre[h] <= i) ++h;
            const uint64_t base = g.lbase[h];
            const uint32_t* src = (base >> 63 ? a.bank_tail : a.ids) + (base & ~(1ull << 63));
            v[b] = __ldg(src + (i - (h ? g.lpre[h - 1] : 0u)));
        }
    }
#pragma unroll
    for (int b = 0; b < BU; ++b)
        if (u * (32 * BU) + b * 32 + lane < total) {
            const uint32_t w = v[b] - p0;   // p0 is a multiple of 32
            atomicOr(&bits[w >> 5], __funnelshift_l(0u, 1u, w));
        }
}

__global__ void __launch_bounds__(BT, 1) k_cand_bitmap(WsArgs a, KnnSearch k, uint32_t* __restrict__ bm) {
    extern __shared__ __align__(16) uint32_t bits[];
    __shared__ BitmapSmem g;
    __shared__ int s_q;
    __shared__ unsigned int s_item;
    __shared__ unsigned long long s_cnt[BT / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = BT / 32;
    const unsigned int nseg = (unsigned int)k.nseg;
    const unsigned int nitems = (unsigned int)k.nd * nseg;
    const int T = a.T, LT = a.L * a.T;
    // Thread 0 claims the next item while the block works on the current
    // one (the claim's round trip overlaps the work) and publishes it at the
    // end of the item, before the block's last barrier.
    if (tid == 0) {
        const unsigned int it = atomicAdd(a.dense_next, 1u);
        s_item = it;
        s_q = it < nitems ? k.dense_q[it / nseg] : -1;
    }
    __syncthreads();
    for (;;) {
        const int q = s_q;
        if (q < 0) break;
        const unsigned int kq = s_item / nseg, g0 = s_item % nseg;
        // the item's points: [p0, p1), word offset w0 of its row
        const uint32_t p0 = g0 * (uint32_t)k.seg;
        const uint32_t p1 = g0 + 1 == nseg ? (uint32_t)a.N : p0 + (uint32_t)k.seg;
        const int w0 = (int)(p0 >> 5);
        const int nwp = (g0 + 1 == nseg ? k.nwp : (int)(p1 >> 5)) - w0;
        unsigned int knext = 0;
        if (tid == 0) knext = atomicAdd(a.dense_next, 1u);
        for (int i = tid * 4; i < nwp; i += BT * 4) *reinterpret_cast<uint4*>(bits + i) = make_uint4(0u, 0u, 0u, 0u);
        for (int c0 = 0; c0 < LT; c0 += BCH) {
            // matched buckets of this chunk of (table, probe) slots, with sizes
            if (tid == 0) {
                g.nl = g.nb = 0;
                if (c0 == 0) g.nrow = 0;
            }
            __syncthreads();
            const int c1 = min(LT, c0 + BCH);
            for (int e = c0 + tid; e < c1; e += BT) {
                const int l = e / T, t = e - l * T;
                const int32_t j = __ldg(a.qbuckets + (int64_t)l * a.Q * T + (int64_t)q * T + t);
                if (j >= 0) {
                    const uint64_t gi = __ldg(a.boff + l) + (uint32_t)j;
                    uint32_t st = __ldg(a.starts + gi), sz = __ldg(a.sizes + gi);
                    if (a.nbig > 0 && sz >= a.big_min) {
                        const int r = big_row(a.big_gi, a.nbig, gi);
                        if (r >= 0) {
                            const uint32_t kr = atomicAdd(&g.nrow, 1u);
                            if (kr < BROWS) {
                                g.row[kr] = (uint32_t)r;
                                continue;
                            }
                        }
                    }
                    if (nseg > 1 && sz) {
                        // the bucket's ids ascend: its part inside the segment
                        const uint32_t* b = a.ids + (uint64_t)l * (uint64_t)a.N + st;
                        const uint32_t lo = ids_below(b, sz, p0), hi = ids_below(b, sz, p1);
                        st += lo;
                        sz = hi - lo;
                    }
                    const uint64_t off = (uint64_t)l * (uint64_t)a.N + st;
                    uint64_t lb = off;
                    uint32_t ls = sz;
                    if (a.bank_meta && sz >= a.bank_min) {
                        const uint2 mt = __ldg(a.bank_meta + gi);
                        if (mt.x) {
                            const uint32_t kk = atomicAdd(&g.nb, 1u);
                            g.bbase[kk] = (off + 3) & ~3ull;
                            g.bsize[kk] = mt.x;
                        }
                        lb = off | (1ull << 63);
                        ls = mt.y;
                    }
                    if (ls) {
                        const uint32_t kk = atomicAdd(&g.nl, 1u);
                        g.lbase[kk] = lb;
                        g.lpre[kk] = ls;
                    }
                }
            }
            __syncthreads();
            const uint32_t nl = g.nl, nb = g.nb;
            if (nl + nb == 0) continue;   // uniform
            {
                // inclusive scans: ids per list (threads of the lower half),
                // units per bank list (upper half)
                static_assert(2 * BCH <= BT && BCH % 32 == 0, "one list per thread");
                const int half = tid / BCH, t = tid % BCH;
                uint32_t c = 0;
                if (half == 0 && t < (int)nl) c = g.lpre[t];
                if (half == 1 && t < (int)nb) c = (g.bsize[t] + BU - 1) / BU;
                uint32_t x = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                constexpr int HW = BCH / 32;   // warps per half
                if (half < 2 && lane == 31) g.wsum[half][warp % HW] = x;
                __syncthreads();
                if (half < 2) {
                    uint32_t before = lane < warp % HW ? g.wsum[half][lane] : 0u;
                    before = __reduce_add_sync(0xffffffffu, before);
                    if (half == 0 && t < (int)nl) g.lpre[t] = before + x;
                    if (half == 1 && t < (int)nb) g.bpre[t] = before + x;
                }
            }
            __syncthreads();
            const uint32_t bunits = nb ? g.bpre[nb - 1] : 0u;
            const uint32_t ids = nl ? g.lpre[nl - 1] : 0u;
            const uint32_t units = bunits + (ids + 32 * BU - 1) / (32 * BU);
            for (uint32_t u = warp; u < units; u += NW) {
                if (u < bunits) or_bank_unit(a, g, u, bits);
                else or_id_unit(a, g, u - bunits, ids, bits, p0);
            }
            __syncthreads();
        }
        uint32_t* row = bm + (int64_t)kq * k.nwp + w0;
        const uint32_t nrow = min(g.nrow, BROWS);
        unsigned long long cnt = 0;
        for (int i = tid * 4; i < nwp; i += BT * 4) {
            uint4 v = *reinterpret_cast<const uint4*>(bits + i);
#pragma unroll 4
            for (uint32_t r = 0; r < nrow; ++r) {
                const uint4 w = __ldg(reinterpret_cast<const uint4*>(a.big_rows + (size_t)g.row[r] * k.nwp + w0 + i));
                v.x |= w.x;
                v.y |= w.y;
                v.z |= w.z;
                v.w |= w.w;
            }
            *reinterpret_cast<uint4*>(row + i) = v;
            if (nrow > 0 && k.f > 0) *reinterpret_cast<uint4*>(bits + i) = v;   // for the sample words
            cnt += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) s_cnt[warp] = cnt;
        __syncthreads();
        // the segment's sample chunks: chunk c holds points (i s32 + c) f of it
        uint32_t* srow = k.bm_sample + (int64_t)kq * k.nws + g0 * k.s32;
        if (k.f == 16) sample_words<2>(bits, srow, k.s32);
        else if (k.f == 8) sample_words<4>(bits, srow, k.s32);
        else
            for (int c = tid; c < k.s32; c += BT) {
                uint32_t word = 0, p = (uint32_t)c * k.f;
#pragma unroll 8
                for (int i = 0; i < 32; ++i, p += (uint32_t)k.s32 * k.f) word |= ((bits[p >> 5] >> (p & 31)) & 1u) << i;
                srow[c] = word;
            }
        if (tid == 0) {
            unsigned long long U = 0;
            for (int w = 0; w < NW; ++w) U += s_cnt[w];
            if (nseg == 1) a.cu[q] = U;
            else atomicAdd(a.cu + q, U);   // zeroed by the planner
            atomicAdd(a.totals + 0, U);
            if (g0 == 0) atomicAdd(a.totals + 1, a.cnu[q]);
            s_item = knext;
            s_q = knext < nitems ? k.dense_q[knext / nseg] : -1;
        }
        __syncthreads();
    }
}

__global__ void k_big_find(const uint32_t* __restrict__ sizes, uint64_t totB, uint32_t big_min, uint64_t* gi,
                           uint32_t* sz, unsigned int* cnt, unsigned int cap) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < totB; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = sizes[i];
        if (s >= big_min) {
            const unsigned int k = atomicAdd(cnt, 1u);
            if (k < cap) {
                gi[k] = i;
                sz[k] = s;
            }
        }
    }
}

// Bank lists (one block per bucket of the list gi): a bucket's ids as 16-bit
// entries (word row << 5 | bit of the id in an N-bit bitmap whose words are 32
// banks wide), arranged so that a warp of the membership kernel ORs 32
// entries into 32 different banks: entry slot [group][bank][4] holds four
// ids of one bank. Every bank gets as many slots as an even split of the
// bucket would fill; a bank with fewer ids fills the rest with an entry of the
// word row past the bitmap (never copied out), one with more sends the remaining
// ids to the bucket's tail (32-bit ids). The order within a bank is arbitrary: the
// entries are ORed. 32 random banks cost 3.5 cycles a warp instruction, distinct
// ones 1.6, and an entry is half an id (figures at k_cand_bitmap).
constexpr int BF = 256;
__global__ void __launch_bounds__(BF) k_bank_fill(const uint64_t* __restrict__ gi, const unsigned int* __restrict__ n,
                                                 unsigned int cap, const uint64_t* __restrict__ boff, int L,
                                                 const uint32_t* __restrict__ starts, const uint32_t* __restrict__ sizes,
                                                 const uint32_t* __restrict__ ids, int64_t N, uint16_t* bank,
                                                 uint32_t* tail, uint2* meta) {
    __shared__ uint32_t cnt[32], ntail;
    const unsigned int nb = min(*n, cap);
    const uint16_t dummy = (uint16_t)(((uint32_t)(N + 1023) >> 10) << 5);
    for (unsigned int r = blockIdx.x; r < nb; r += gridDim.x) {
        const uint64_t b = gi[r];
        int l = 0;
        while (l + 1 < L && boff[l + 1] <= b) ++l;
        const uint64_t off = (uint64_t)l * N + starts[b], base = (off + 3) & ~3ull;
        const uint32_t sz = sizes[b];
        const uint32_t R = ((sz - 3) / 32) & ~3u;   // slots per bank; 32 R entries fit from base on
        __syncthreads();
        if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
        if (threadIdx.x == 32) ntail = 0;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < sz; j += BF) {
            const uint32_t v = ids[off + j], bk = (v >> 5) & 31u;
            const uint32_t k = atomicAdd(&cnt[bk], 1u);
            if (k < R) bank[base + (uint64_t)(k >> 2) * 128 + bk * 4 + (k & 3)] = (uint16_t)(((v >> 10) << 5) | (v & 31u));
            else tail[off + atomicAdd(&ntail, 1u)] = v;
        }
        __syncthreads();
        for (uint32_t s = threadIdx.x; s < 32 * R; s += BF) {
            const uint32_t bk = (s >> 2) & 31u, k = ((s >> 7) << 2) | (s & 3u);
            if (k >= cnt[bk]) bank[base + s] = dummy;
        }
        if (threadIdx.x == 0) meta[b] = make_uint2(R / 4, ntail);
    }
}

cudaError_t launch_bank_fill(const uint64_t* gi, const unsigned int* n, unsigned int cap, const uint64_t* boff, int L,
                             const uint32_t* starts, const uint32_t* sizes, const uint32_t* ids, int64_t N,
                             uint16_t* bank, uint32_t* tail, uint2* meta, cudaStream_t st) {
    k_bank_fill<<<152 * 8, BF, 0, st>>>(gi, n, cap, boff, L, starts, sizes, ids, N, bank, tail, meta);
    return cudaGetLastError();
}

// Row r (blockIdx.y) gets the bits of bucket gi[r]'s ids (table tl[r]).
__global__ void k_big_fill(const uint64_t* __restrict__ gi, const int32_t* __restrict__ tl,
                           const uint32_t* __restrict__ starts, const uint32_t* __restrict__ sizes,
                           const uint32_t* __restrict__ ids, int64_t N, uint32_t* rows, int nwp) {
    const int r = blockIdx.y;
    const uint64_t b = gi[r];
    const uint32_t st = starts[b], sz = sizes[b];
    const uint32_t* src = ids + (uint64_t)tl[r] * N + st;
    uint32_t* row = rows + (size_t)r * nwp;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < sz; j += gridDim.x * blockDim.x) {
        const uint32_t v = src[j];
        atomicOr(row + (v >> 5), 1u << (v & 31));
    }
}

cudaError_t launch_big_find(const uint32_t* sizes, uint64_t totB, uint32_t big_min, uint64_t* gi, uint32_t* sz,
                            unsigned int* cnt, unsigned int cap, cudaStream_t st) {
    if (totB == 0) return cudaSuccess;
    const unsigned g = (unsigned)std::min<uint64_t>((totB + 255) / 256, 4096);
    k_big_find<<<g, 256, 0, st>>>(sizes, totB, big_min, gi, sz, cnt, cap);
    return cudaGetLastError();
}

cudaError_t launch_big_fill(const uint64_t* gi, const int32_t* tl, int nbig, const uint32_t* starts,
                            const uint32_t* sizes, const uint32_t* ids, int64_t N, uint32_t* rows, int nwp,
                            cudaStream_t st) {
    if (nbig <= 0) return cudaSuccess;
    k_big_fill<<<dim3(16, (unsigned)nbig), 256, 0, st>>>(gi, tl, starts, sizes, ids, N, rows, nwp);
    return cudaGetLastError();
}

// (less the block's lists and the bank lists' word row)
size_t bitmap_smem(int max_smem) { return (size_t)max_smem - sizeof(BitmapSmem) - 2048; }

cudaError_t launch_cand_bitmap(const WsArgs& a, const KnnSearch& k, uint32_t* bm, int grid, cudaStream_t st) {
    static std::atomic<size_t> cap{0};
    // the longest segment is the last one
    size_t smem = 4 * (size_t)(k.nwp - (k.nseg - 1) * (k.seg >> 5));
    if (a.bank_meta) smem = 4 * ((size_t)((a.N + 1023) >> 10) + 1) * 32;   // and the word row of unused entries
    const cudaError_t e = opt_in_smem(k_cand_bitmap, smem, cap);
    if (e != cudaSuccess) return e;
    k_cand_bitmap<<<grid, BT, smem, st>>>(a, k, bm);
    return cudaGetLastError();
}

size_t knn_scan_smem(int D, int K) { return sizeof(float) * (size_t)((D + 3) & ~3) + scan_bytes(K); }

cudaError_t launch_knn_scan_rows(const KnnSearch& k, int grid, cudaStream_t st) {
    static std::atomic<size_t> cap{0};
    const size_t smem = knn_scan_smem(k.D, k.K);
    const cudaError_t e = opt_in_smem(k_knn_scan_rows, smem, cap);
    if (e != cudaSuccess) return e;
    k_knn_scan_rows<<<grid, DT, smem, st>>>(k);
    return cudaGetLastError();
}

size_t dense_smem_bytes(int64_t N, int D, int K) {
    const size_t nwp = (size_t)((((N + 31) >> 5) + 3) & ~3ll);
    return sizeof(float) * (size_t)((D + 3) & ~3) + 4 * nwp + scan_bytes(K);
}

size_t ws_smem_bytes(int D, int K, int wt, WsForm form, int slots) {
    const size_t cap = (size_t)slots / 2;
    const bool bf16 = form == WsForm::bf16;
    return (form == WsForm::staged ? (size_t)(wt / 32) * row_stage_bytes(D) : 0) + sizeof(float) * (size_t)((D + 3) & ~3) +
           sizeof(uint32_t) * ((size_t)slots + cap) + (size_t)(bf16 ? wt / 32 : 1) * K * (sizeof(float) + sizeof(uint32_t)) +
           (bf16 ? 2 * sizeof(float) * cap : 0);
}

cudaError_t launch_order_queries(const WsArgs& a, cudaStream_t st) {
    if (a.Q <= 0 || !a.order) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.order_bins, 0, sizeof(uint32_t) * (kOrderBins + 1), st);
    if (e != cudaSuccess) return e;
    const unsigned g = (unsigned)((a.Q + 255) / 256);
    k_order_hist<<<g, 256, 0, st>>>(a);
    k_order_scan<<<1, 1024, 0, st>>>(a);
    k_order_scatter<<<g, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_plan_items(const WsArgs& a, cudaStream_t st) {
    if (a.Q <= 0) return cudaSuccess;
    k_plan_items<<<(a.Q + PT_PLAN - 1) / PT_PLAN, PT_PLAN, 0, st>>>(a);
    return cudaGetLastError();
}

namespace {
template <int WT, WsForm kForm, int SL>
std::atomic<size_t>& ws_smem_cap() {
    static std::atomic<size_t> cap{0};   // dynamic shared memory this kernel is opted into
    return cap;
}

template <int WT, WsForm kForm, int SL>
constexpr auto ws_kernel() {
    if constexpr (kForm == WsForm::bf16) return &k_candidates_ws_bf16<WT, SL>;
    else return &k_candidates_ws<WT, SL, kForm == WsForm::staged>;
}

template <int WT, WsForm kForm, int SL>
cudaError_t launch_ws_v(const WsArgs& a, int grid, cudaStream_t st) {
    const size_t smem = ws_smem_bytes(a.D, a.K, WT, kForm, SL);
    const cudaError_t e = opt_in_smem(ws_kernel<WT, kForm, SL>(), smem, ws_smem_cap<WT, kForm, SL>());
    if (e != cudaSuccess) return e;
    ws_kernel<WT, kForm, SL>()<<<grid, WT, smem, st>>>(a);
    return cudaGetLastError();
}

template <int WT, WsForm kForm, int SL>
int ws_bps_v(int D, int K) {
    int n = 0;
    const size_t smem = ws_smem_bytes(D, K, WT, kForm, SL);
    if (opt_in_smem(ws_kernel<WT, kForm, SL>(), smem, ws_smem_cap<WT, kForm, SL>()) != cudaSuccess) return 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ws_kernel<WT, kForm, SL>(), WT, smem) != cudaSuccess)
        n = 1;
    return n > 0 ? n : 1;
}

template <WsForm kForm, int SL>
cudaError_t launch_ws_w(const WsArgs& a, int grid, cudaStream_t st) {
    switch (a.wt) {
        case 64: return launch_ws_v<64, kForm, SL>(a, grid, st);
        case 256: return launch_ws_v<256, kForm, SL>(a, grid, st);
        case 512: return launch_ws_v<512, kForm, SL>(a, grid, st);
        default: return launch_ws_v<128, kForm, SL>(a, grid, st);
    }
}

template <WsForm kForm, int SL>
int ws_bps_w(int D, int K, int wt) {
    switch (wt) {
        case 64: return ws_bps_v<64, kForm, SL>(D, K);
        case 256: return ws_bps_v<256, kForm, SL>(D, K);
        case 512: return ws_bps_v<512, kForm, SL>(D, K);
        default: return ws_bps_v<128, kForm, SL>(D, K);
    }
}

// BF16 copy of the dataset (round to nearest even) and a per-row flag:
// 1 when every element is exact in bf16, 2 when a nonzero element has a
// magnitude outside [2^-100, 2^100] (the search then always re-checks the
// row in FP32), 0 otherwise. One warp per row.
__global__ void k_bf16_rows(const float* __restrict__ X, int64_t N, int D, uint16_t* __restrict__ xb,
                            uint8_t* __restrict__ flag) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = w0; r < N; r += nw) {
        bool exact = true, special = false;
        for (int d = lane; d < D; d += 32) {
            const float x = __ldg(X + r * D + d);
            const uint16_t h = __bfloat16_as_ushort(__float2bfloat16_rn(x));
            xb[r * D + d] = h;
            exact &= __uint_as_float((uint32_t)h << 16) == x;
            const float ax = fabsf(x);
            special |= x != 0.0f && !(ax >= 7.88860905e-31f && ax <= 1.26765060e30f);
        }
        exact = __all_sync(0xffffffffu, exact);
        special = __any_sync(0xffffffffu, special);
        if (lane == 0) flag[r] = special ? 2 : (exact ? 1 : 0);
    }
}
}  // namespace

cudaError_t launch_candidates_small(const WsArgs& a, int sms, cudaStream_t st) {
    const size_t smem = sizeof(float) * SMW * (size_t)((a.D + 3) & ~3);
    static std::atomic<size_t> cap{0};
    const cudaError_t e = opt_in_smem(k_candidates_small, smem, cap);
    if (e != cudaSuccess) return e;
    const int grid = std::min((a.Q + SMW - 1) / SMW, sms * 8);
    k_candidates_small<<<grid, 32 * SMW, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_candidates_ws(const WsArgs& a, int grid, cudaStream_t st) {
    const bool bf16 = a.form == WsForm::bf16;
    if (a.slots == 16384)
        return bf16 ? launch_ws_w<WsForm::bf16, 16384>(a, grid, st) : launch_ws_w<WsForm::direct, 16384>(a, grid, st);
    if (a.slots == 8192)
        return bf16 ? launch_ws_w<WsForm::bf16, 8192>(a, grid, st) : launch_ws_w<WsForm::direct, 8192>(a, grid, st);
    if (a.form == WsForm::staged) return launch_ws_w<WsForm::staged, 4096>(a, grid, st);
    return bf16 ? launch_ws_w<WsForm::bf16, 4096>(a, grid, st) : launch_ws_w<WsForm::direct, 4096>(a, grid, st);
}

int ws_blocks_per_sm(int D, int K, int wt, WsForm form, int slots) {
    const bool bf16 = form == WsForm::bf16;
    if (slots == 16384)
        return bf16 ? ws_bps_w<WsForm::bf16, 16384>(D, K, wt) : ws_bps_w<WsForm::direct, 16384>(D, K, wt);
    if (slots == 8192) return bf16 ? ws_bps_w<WsForm::bf16, 8192>(D, K, wt) : ws_bps_w<WsForm::direct, 8192>(D, K, wt);
    if (form == WsForm::staged) return ws_bps_w<WsForm::staged, 4096>(D, K, wt);
    return bf16 ? ws_bps_w<WsForm::bf16, 4096>(D, K, wt) : ws_bps_w<WsForm::direct, 4096>(D, K, wt);
}

cudaError_t launch_candidates_dense(const WsArgs& a, int grid, cudaStream_t st) {
    static std::atomic<size_t> cap{0};   // dynamic shared memory this kernel is opted into
    const size_t smem = dense_smem_bytes(a.N, a.D, a.K);
    const cudaError_t e = opt_in_smem(k_candidates_dense, smem, cap);
    if (e != cudaSuccess) return e;
    k_candidates_dense<<<grid, DT, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_bf16_rows(const float* X, int64_t N, int D, uint16_t* xb, uint8_t* flag, cudaStream_t st) {
    if (N <= 0) return cudaSuccess;
    const int64_t warps = std::min<int64_t>(N, 152 * 64);
    k_bf16_rows<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(X, N, D, xb, flag);
    return cudaGetLastError();
}

}  // namespace culsh
